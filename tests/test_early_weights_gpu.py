"""Weights that are read before the kernel in front has finished: calls back to back on a stream, without a synchronisation between
them, so that a read that comes too early finds the weight of nobody.  s32 sums are exact; each call's result is its own buffer."""
import pytest

from test_matmul_gpu import capi  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu

ROWS = (1, 2, 9, 16, 17, 33, 48, 200)


def ints(torch, *shape):
    return torch.randint(-128, 128, shape, dtype=torch.int8, device="cuda")


def exact(a, w):
    return (a.double() @ w.double()).int()


def s32_call(capi, torch, a, w, **kw):
    (M, K), N = a.shape, kw.pop("N")
    out = torch.full((M, N), 77, dtype=torch.int32, device="cuda")
    return capi.make_matmul(M, N, K, a, w, out, src_dt=capi.DT["s8"], dst_dt=capi.DT["s32"], flags=capi.FLAG_STABLE_WEIGHTS, **kw), out


def test_prepacked_weights_in_turn(capi):
    """Six weights that were in place before, several row counts: every call may read its weight while the one in front still runs."""
    import torch
    K, N = 6016, 4224                               # large enough for the few-row kernel below 17 rows
    st = torch.cuda.current_stream().cuda_stream
    ws, packs = [ints(torch, K, N) for _ in range(6)], []
    for w in ws:
        p = torch.empty(capi.lib.b200dnn_prepack_size(K, N, 0), dtype=torch.uint8, device="cuda")
        capi.check(capi.lib.b200dnn_prepack(w.data_ptr(), K, N, N, 0, 0, p.data_ptr(), st))
        packs.append(p)
    a = {M: ints(torch, M, K) for M in ROWS}
    todo = [(M, i) for rep in range(3) for i in range(6) for M in ROWS]
    descs = [s32_call(capi, torch, a[M], packs[i], N=N, wei_format="r") for M, i in todo]
    torch.cuda.synchronize()
    for d, _ in descs:
        capi.check(capi.matmul(d, st))
    torch.cuda.synchronize()
    ref = {(M, i): exact(a[M], ws[i]) for M in ROWS for i in range(6)}
    for (M, i), (_, out) in zip(todo, descs):
        assert torch.equal(out, ref[M, i]), (M, i)


@pytest.mark.parametrize("first", [200, 20, 2])
@pytest.mark.parametrize("other_stream", [False, True])
def test_cached_weight_behind_its_packing(capi, first, other_stream):
    """The first call packs the raw weight into the library's cache; the calls right behind it, on the same stream or another, find it
    there while the packing may still be under way."""
    import torch
    K, N = 6016, 4224
    s0 = torch.cuda.current_stream()
    s1 = torch.cuda.Stream() if other_stream else s0
    a = {M: ints(torch, M, K) for M in ROWS + (first,)}
    ws = [ints(torch, K, N) for _ in range(6)]
    torch.cuda.synchronize()
    res = []
    for w in ws:
        d, out = s32_call(capi, torch, a[first], w, N=N, weights_const=True)
        later = [(M,) + s32_call(capi, torch, a[M], w, N=N, weights_const=True) for M in ROWS]
        torch.cuda.synchronize()                    # (the outputs' fill)
        capi.check(capi.matmul(d, s0.cuda_stream))
        for _, e, _ in later:
            capi.check(capi.matmul(e, s1.cuda_stream))
        res.append((w, out, later))
    torch.cuda.synchronize()
    capi.lib.b200dnn_clear_caches()
    for w, out, later in res:
        assert torch.equal(out, exact(a[first], w))
        for M, _, o in later:
            assert torch.equal(o, exact(a[M], w)), M


def test_dynamic_quantisation_behind_the_prepack(capi):
    """Prepack and the call that quantises its rows, back to back: the GEMM reads the weight while its rows are being quantised."""
    import torch
    K, N = 6016, 4224
    st = torch.cuda.current_stream().cuda_stream
    packs = [torch.empty(capi.lib.b200dnn_prepack_size(K, N, 0), dtype=torch.uint8, device="cuda") for _ in range(4)]
    ws = [ints(torch, K, N) for _ in packs]
    x = {M: torch.randn(M, K, device="cuda").bfloat16() for M in ROWS}
    one = torch.full((N,), 0.01, device="cuda")

    def call(M, p):
        out = torch.zeros(M, N, device="cuda")
        return capi.make_matmul(M, N, K, x[M], p, out, src_dt=capi.DT["bf16"], dst_dt=capi.DT["f32"], dynamic_quant=True,
                                src_scale=capi.quant(None, M, capi.DT["f32"]), wei_format="r", wei_scale=one), out
    ref = []
    for i, w in enumerate(ws):                      # each call alone
        capi.check(capi.lib.b200dnn_prepack(w.data_ptr(), K, N, N, 0, 0, packs[i].data_ptr(), st))
        torch.cuda.synchronize()
        for M in ROWS:
            d, out = call(M, packs[i])
            capi.check(capi.matmul(d, st))
            torch.cuda.synchronize()
            ref.append(out)
    for p in packs:
        p[4096:] = 0                                # (behind the header)
    got = [[call(M, p) for M in ROWS] for p in packs]
    torch.cuda.synchronize()
    for i, w in enumerate(ws):
        capi.check(capi.lib.b200dnn_prepack(w.data_ptr(), K, N, N, 0, 0, packs[i].data_ptr(), st))
        for d, _ in got[i]:
            capi.check(capi.matmul(d, st))
    torch.cuda.synchronize()
    for r, (_, out) in zip(ref, [g for row in got for g in row]):
        assert torch.equal(r, out)


def test_bf16_weights_in_turn(capi):
    """The same weight as a call alone gives: a cached bf16 weight behind its packing and, later, read early among other weights."""
    import torch
    K, N = 2048, 4224
    st = torch.cuda.current_stream().cuda_stream
    ws = [(torch.randn(K, N, device="cuda") * 0.02).bfloat16() for _ in range(4)]
    x = {M: torch.randn(M, K, device="cuda").bfloat16() for M in (1, 8, 33, 64, 200)}

    def call(M, w):
        out = torch.zeros(M, N, device="cuda")
        return capi.make_matmul(M, N, K, x[M], w, out, src_dt=capi.DT["bf16"], wei_dt=capi.DT["bf16"], dst_dt=capi.DT["f32"],
                                flags=capi.FLAG_STABLE_WEIGHTS), out
    todo = [(M, i) for i in range(4) for M in x] + [(M, i) for M in x for i in range(4)]
    descs = [call(M, ws[i]) for M, i in todo]
    torch.cuda.synchronize()
    for d, _ in descs:
        capi.check(capi.matmul(d, st))
    torch.cuda.synchronize()
    for (M, i), (d, out) in zip(todo, descs):
        got = out.clone()
        out.zero_()
        torch.cuda.synchronize()
        capi.check(capi.matmul(d, st))
        torch.cuda.synchronize()
        assert torch.equal(got, out), (M, i)
        # f32 sums of K exact products: each addition rounds by at most 2^-23 of a partial sum, which is at most sum |x||w|
        a, w = x[M].double(), ws[i].double()
        assert ((out - a @ w).abs() <= K * 2.0 ** -23 * (a.abs() @ w.abs())).all()
    capi.lib.b200dnn_clear_caches()

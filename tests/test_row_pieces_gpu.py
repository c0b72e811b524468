"""Results in rows without 16-byte alignment, written as aligned 32-byte pieces that span the sixteen columns an epilogue step has and those before them: every distance of
a row from a piece's boundary (odd N and ldc, destinations that begin in the middle of one), every length of the last 32 columns, tiles of every form and grouped ones, in bf16,
f32 and s32, against exact products; what lies between the rows and behind them stays as it was."""
import pytest

from test_matmul_gpu import capi  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu

TORCH = {"bf16": "bfloat16", "f32": "float32", "s32": "int32"}


@pytest.mark.parametrize("dt", ["bf16", "f32", "s32"])
@pytest.mark.parametrize("M,N", [(200, n) for n in [*range(1, 34), 48, 63, 65, 80, 95, 112, 127, 129, 130, 144, 255, 257, 272, 500, 501]] + [(600, 3001), (2300, 1029)])
@pytest.mark.parametrize("pad,start", [(0, 0), (3, 1), (8, 5), (1, 7)])
def test_every_distance_from_a_boundary(capi, monkeypatch, dt, M, N, pad, start):
    import torch
    torch.manual_seed(N + pad)
    K, ldc = 160, N + pad
    a, w = (torch.randint(-9, 10, s, dtype=torch.int8, device="cuda") for s in ((M, K), (K, N)))
    want = (a.float() @ w.float()).to(getattr(torch, TORCH[dt]))
    pool = torch.full((start + M * ldc + 40,), 77, dtype=want.dtype, device="cuda")
    out = pool[start:start + M * ldc].view(M, ldc)
    for pair, split in (("0", "1"), ("0", "2"), ("1", "0")):       # one CTA a tile, a tile's K shared by two, pairs of CTAs
        monkeypatch.setenv("B200DNN_TC_PAIR", pair)
        monkeypatch.setenv("B200DNN_TC_KSPLIT", split)
        pool.fill_(77)
        d = capi.make_matmul(M, N, K, a, w, out, src_dt=capi.DT["s8"], dst_dt=capi.DT[dt], force_kernel=2, ldc=ldc)
        capi.check(capi.matmul(d, torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert torch.equal(out[:, :N], want), (dt, N, pad, start, pair, split)
        assert (pool[:start] == 77).all() and (pool[start + M * ldc:] == 77).all() and (out[:, N:] == 77).all()
    capi.lib.b200dnn_clear_caches()


@pytest.mark.parametrize("dt", ["bf16", "f32"])
@pytest.mark.parametrize("wdt", ["s8", "bf16"])
@pytest.mark.parametrize("N,pad", [(16, 1), (48, 3), (112, 1), (144, 5), (33, 0), (272, 1)])
def test_grouped(capi, dt, wdt, N, pad):
    """One grouped launch over experts whose results have odd pitches."""
    import torch
    torch.manual_seed(N)
    K, ldc, Ms = 160, N + pad, (33, 0, 200, 1)
    descs, outs, wants, keep = (capi.MatmulDesc * len(Ms))(), [], [], []
    for g, M in enumerate(Ms):
        a, w = (torch.randint(-9, 10, s, dtype=torch.int8, device="cuda") for s in ((max(M, 1), K), (K, N)))
        wants.append((a.float() @ w.float()).to(getattr(torch, TORCH[dt])))
        outs.append(torch.full((max(M, 1), ldc), 77, dtype=wants[-1].dtype, device="cuda"))
        if wdt == "bf16":
            a, w, kw = a.bfloat16(), w.bfloat16(), {}
        else:
            one = torch.ones(max(M, 1, N), device="cuda")
            kw = dict(src_scale=capi.quant(one, count=M), wei_scale=one[:N])
            keep.append(one)
        keep += [a, w]
        descs[g] = capi.make_matmul(M, N, K, a, w, outs[-1], src_dt=capi.DT[wdt], wei_dt=capi.DT[wdt], dst_dt=capi.DT[dt], ldc=ldc, **kw)
    st = torch.cuda.current_stream().cuda_stream
    capi.check(capi.lib.b200dnn_group_matmul(len(Ms), descs, st))              # (packs the weights)
    before = capi.lib.b200dnn_launch_count()
    capi.check(capi.lib.b200dnn_group_matmul(len(Ms), descs, st))
    torch.cuda.synchronize()
    assert capi.lib.b200dnn_launch_count() - before == 1
    for M, out, want in zip(Ms, outs, wants):
        assert torch.equal(out[:M, :N], want[:M]) and (out[:, N:] == 77).all() and (M or (out == 77).all()), (dt, wdt, N, M)
    capi.lib.b200dnn_clear_caches()

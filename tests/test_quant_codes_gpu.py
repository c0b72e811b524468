"""Codes of the per-token quantisation where a quotient lies on, or one float beside, the middle of two codes: they must be those of the IEEE
division (the oracle's), in every kernel that a row length and a number of rows can reach."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(oracle, x, dt, K):
    from zendnn_b200 import capi
    M = x.shape[0]
    q_ref, s_ref = oracle.quant_per_token(x)
    q, s = np.zeros((M, K), dtype=np.int8), np.zeros(M, dtype=np.float32)
    capi.check(capi.lib.b200dnn_quant_per_token(capi.ptr(x), capi.DT[dt], M, K, K, capi.ptr(q), K, capi.ptr(s), capi.DT["f32"], None))
    assert (s == s_ref).all()
    assert (q == q_ref).all(), np.argwhere(q != q_ref)[:5]


# 2562: rows of codes that do not all start on a vector (test_each_kernel forces a warp and a CTA per row)
@pytest.mark.parametrize("K,rows", [(2560, 128), (2562, 128), (5120, 128), (2560, 40)])
def test_bf16_every_pair_of_significands(oracle, K, rows):
    """Rows with abs-max b/128 (b = 128 ... 255) holding every bf16 of both signs down to 2^-9 of it; the last row has elements that are not finite."""
    step = 128 // rows if rows < 128 else 1
    b = (128 + step * np.arange(rows)).astype(np.float32) / 128
    a = np.arange(128, 256, dtype=np.float32) / 128
    one = np.concatenate([a * np.float32(2.0) ** -e for e in range(10)])
    one = np.concatenate([one, -one])
    x = np.zeros((rows, K), dtype=np.float32)
    x[:, :one.size] = np.where(np.abs(one)[None, :] <= b[:, None], one[None, :], 0)
    x[np.arange(rows), 7] = b
    x[-1, 11], x[-1, 300], x[-1, K - 1] = np.inf, np.nan, -np.inf
    _check(oracle, oracle.f32_to_bf16(x), "bf16", K)


@pytest.mark.parametrize("K,rows", [(1024, 64), (1022, 64), (4096, 8)])
def test_f32_beside_the_middle_of_two_codes(oracle, K, rows):
    rng = np.random.default_rng(K)
    x = np.zeros((rows, K), dtype=np.float32)
    for r in range(rows):
        absmax = np.float32(rng.uniform(0.5, 300.0))
        s = np.float32(absmax / np.float32(127))
        v = ((rng.integers(-127, 127, K) + np.float32(0.5)) * s).astype(np.float32)
        v = (v.view(np.int32) + rng.integers(-2, 3, K).astype(np.int32)).view(np.float32)
        x[r] = np.clip(v, -absmax, absmax)
        x[r, 5] = absmax
    x[0, 9], x[0, 10] = np.nan, np.inf
    _check(oracle, x, "f32", K)


@pytest.mark.parametrize("warp", ["0", "1"])
@pytest.mark.parametrize("dt,K,rows", [("bf16", 2560, 128), ("bf16", 4096, 128), ("f32", 1024, 64), ("f32", 2048, 64)])
def test_middle_of_two_codes_in_either_kernel(oracle, monkeypatch, warp, dt, K, rows):
    monkeypatch.setenv("B200DNN_QUANT_WARP", warp)
    (test_bf16_every_pair_of_significands if dt == "bf16" else test_f32_beside_the_middle_of_two_codes)(oracle, K, rows)


# a warp and a CTA per row, one and two vectors past a multiple, the longest rows of a warp, rows beyond a CTA's registers
@pytest.mark.parametrize("dt", ["bf16", "f32"])
@pytest.mark.parametrize("rows,K", [(70, 1), (70, 17), (64, 1999), (64, 2047), (5, 1001), (5, 4097), (64, 16385 + 8)])
def test_rows_of_any_alignment(oracle, dt, rows, K):
    """Source rows that start and end anywhere, into rows of codes that start on a vector: the bytes behind a row of codes stay as they were."""
    import torch
    from zendnn_b200 import capi
    rng = np.random.default_rng(K)
    ld, dld = K + 3, (K + 15) // 16 * 16 + 16
    full = rng.normal(size=(rows, ld)).astype(np.float32)
    full[rows // 2, K - 1], full[0, 0] = 50.0, np.inf if K > 1 else 3.0
    if dt == "bf16":
        full = oracle.f32_to_bf16(full)
    x = np.concatenate([full[:1].ravel()[:1], full.ravel()])           # one element in front: no row is aligned to more than an element
    dev = torch.from_numpy(x.view(np.int16 if dt == "bf16" else np.int32)).cuda()
    q = torch.full((rows, dld), 99, dtype=torch.int8, device="cuda")
    s = torch.zeros(rows, device="cuda")
    es = 2 if dt == "bf16" else 4
    capi.check(capi.lib.b200dnn_quant_per_token(dev.data_ptr() + es, capi.DT[dt], rows, K, ld, q.data_ptr(), dld, s.data_ptr(), capi.DT["f32"],
                                                torch.cuda.current_stream().cuda_stream))
    q_ref, s_ref = oracle.quant_per_token(np.ascontiguousarray(full[:, :K]))
    assert (s.cpu().numpy() == s_ref).all()
    got = q.cpu().numpy()
    assert (got[:, :K] == q_ref).all() and (got[:, K:] == 99).all()


def _device_rows(oracle, dt, rows, K, ld, seed):
    """Rows `ld` elements apart behind one element (ld = K: aligned, behind sixteen bytes), with an infinity, a NaN and one large element."""
    import torch
    rng = np.random.default_rng(seed)
    full = rng.normal(size=(rows, ld)).astype(np.float32)
    full[rows // 2, K - 1], full[0, 0], full[rows - 1, K // 2] = 50.0, np.inf, np.nan
    if dt == "bf16":
        full = oracle.f32_to_bf16(full)
    pad = 1 if ld != K else 16 // full.itemsize
    dev = torch.from_numpy(np.concatenate([full.ravel()[:pad], full.ravel()]).view(np.int16 if dt == "bf16" else np.int32)).cuda()
    return dev, dev.data_ptr() + pad * full.itemsize, np.ascontiguousarray(full[:, :K])


# two, four, eight and sixteen vectors a lane of a warp (one short of that where the rows are odd); two and eight vectors a thread of a CTA, and rows beyond that
@pytest.mark.parametrize("warp", ["0", "1"])
@pytest.mark.parametrize("dt", ["bf16", "f32"])
@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("vecs", [64, 128, 256, 512, 513, 2048 + 40])
@pytest.mark.parametrize("rows", [9, 150])
def test_each_kernel(oracle, monkeypatch, warp, dt, odd, vecs, rows):
    import torch
    from zendnn_b200 import capi
    monkeypatch.setenv("B200DNN_QUANT_WARP", warp)
    K = vecs * (8 if dt == "bf16" else 4) - (3 if odd else 0)
    dld = (K + 15) // 16 * 16 + 16
    dev, src, x = _device_rows(oracle, dt, rows, K, K + 3 if odd else K, vecs)
    q, s = torch.full((rows, dld), 99, dtype=torch.int8, device="cuda"), torch.zeros(rows, device="cuda")
    capi.check(capi.lib.b200dnn_quant_per_token(src, capi.DT[dt], rows, K, K + 3 if odd else K, q.data_ptr(), dld, s.data_ptr(), capi.DT["f32"],
                                                torch.cuda.current_stream().cuda_stream))
    q_ref, s_ref = oracle.quant_per_token(x)
    assert (s.cpu().numpy() == s_ref).all()
    got = q.cpu().numpy()
    assert (got[:, :K] == q_ref).all() and (got[:, K:] == 99).all()


@pytest.mark.parametrize("dt", ["bf16", "f32"])
@pytest.mark.parametrize("odd", [(False, False), (False, True), (True, True)])
@pytest.mark.parametrize("vecs,rows", [(65, (3, 0, 70)), (513, (1, 2, 4)), (520, (90, 0, 80))])
def test_groups(oracle, dt, odd, vecs, rows):
    """Several matrices in one launch, aligned, odd and of both kinds."""
    import ctypes as C
    import torch
    from zendnn_b200 import capi
    G, K = len(rows), vecs * (8 if dt == "bf16" else 4) - (3 if all(odd) else 0)
    lds = [K + 3 if odd[g % 2] else K for g in range(G)]
    made = [_device_rows(oracle, dt, max(r, 1), K, lds[g], vecs + g) for g, r in enumerate(rows)]
    dld = (K + 15) // 16 * 16
    qs = [torch.full((max(r, 1), dld), 99, dtype=torch.int8, device="cuda") for r in rows]
    ss = [torch.zeros(max(r, 1), device="cuda") for r in rows]
    ptrs = lambda v: (C.c_void_p * G)(*v)
    capi.check(capi.lib.b200dnn_group_quant_per_token(G, ptrs([m[1] for m in made]), capi.DT[dt], (C.c_int32 * G)(*rows), (C.c_int32 * G)(*[K] * G),
                                                      (C.c_int64 * G)(*lds), ptrs([q.data_ptr() for q in qs]), (C.c_int64 * G)(*[dld] * G),
                                                      ptrs([s.data_ptr() for s in ss]), capi.DT["f32"], torch.cuda.current_stream().cuda_stream))
    for g, r in enumerate(rows):
        if r:
            q_ref, s_ref = oracle.quant_per_token(made[g][2])
            got = qs[g].cpu().numpy()
            assert (ss[g].cpu().numpy() == s_ref).all() and (got[:, :K] == q_ref).all() and (got[:, K:] == 99).all(), g


@pytest.mark.parametrize("warp", ["0", "1"])
@pytest.mark.parametrize("dt", ["bf16", "f32"])
@pytest.mark.parametrize("vecs,short,rows", [(64, 0, 9), (128, 0, 20), (256, 0, 70), (512, 0, 9), (513, 0, 9), (513, 0, 150), (130, 3, 9)])
def test_scattered(oracle, monkeypatch, warp, dt, vecs, short, rows):
    """A row goes to up to three places, some to none; a row length that is no multiple of a vector goes element by element."""
    import torch
    from zendnn_b200 import capi
    monkeypatch.setenv("B200DNN_QUANT_WARP", warp)
    n, K = 3, vecs * (8 if dt == "bf16" else 4) - short
    dev, src, x = _device_rows(oracle, dt, rows, K, K, vecs)
    rng = np.random.default_rng(rows)
    to = rng.permutation(rows * n).astype(np.int32)
    to[rng.random(rows * n) < 0.3] = -1
    dld = (K + 15) // 16 * 16
    q, s = torch.full((rows * n, dld), 99, dtype=torch.int8, device="cuda"), torch.full((rows * n,), -1.0, device="cuda")
    to_dev = torch.from_numpy(to).cuda()
    capi.check(capi.lib.b200dnn_quant_per_token_scatter(src, capi.DT[dt], K, K, to_dev.data_ptr(), n, rows, q.data_ptr(), dld, s.data_ptr(),
                                                        torch.cuda.current_stream().cuda_stream))
    q_ref, s_ref = oracle.quant_per_token(x)
    q_all, s_all = np.full((rows * n, dld), 99, dtype=np.int8), np.full(rows * n, -1.0, dtype=np.float32)
    for i, d in enumerate(to):
        if d >= 0:
            q_all[d, :K], s_all[d] = q_ref[i // n], s_ref[i // n]
    assert (s.cpu().numpy() == s_all).all() and (q.cpu().numpy() == q_all).all()

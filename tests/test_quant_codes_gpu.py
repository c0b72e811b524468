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


# 2560: a warp per row; 2562: element by element; 5120 and (with few rows) 2560: a CTA per row
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

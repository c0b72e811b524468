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

"""The one-launch routing of a small MoE batch against the launches it stands for: a layer over T tokens (one launch up to 64) gives, row by
row, what the same tokens give at the head of a larger batch (the general launches)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    from zendnn_b200 import capi as c
    assert c.lib.b200dnn_device_count() > 0, "no CUDA device"
    return c


@pytest.mark.parametrize("T,E,topk,S", [(1, 4, 2, 0), (32, 64, 6, 2), (64, 16, 16, 1), (33, 8, 1, 0), (64, 255, 3, 1), (7, 130, 5, 0)])
def test_small_route_matches_general(capi, oracle, T, E, topk, S):
    rng = np.random.default_rng(T + E)
    H, I, big = 128, 64, 96
    x = oracle.f32_to_bf16(rng.standard_normal((big, H)).astype(np.float32))
    logits = rng.standard_normal((big, E)).astype(np.float32)
    logits[:, : E // 2] = np.round(logits[:, : E // 2])     # ties
    ex = (capi.MoeExpert * (E + S))()
    keep = []
    for e in range(E + S):
        w13, w2 = rng.integers(-127, 128, (H, 2 * I), dtype=np.int8), rng.integers(-127, 128, (I, H), dtype=np.int8)
        s13, s2 = np.full(2 * I, 1e-3, np.float32), np.full(H, 1e-3, np.float32)
        keep.append((w13, w2, s13, s2))
        ex[e].w13, ex[e].ldb13, ex[e].w13_scale = w13.ctypes.data, 2 * I, s13.ctypes.data
        ex[e].w2, ex[e].ldb2, ex[e].w2_scale = w2.ctypes.data, H, s2.ctypes.data

    def run(t):
        out = np.zeros((t, H), dtype=np.uint16)
        capi.check(capi.lib.b200dnn_moe_layer(capi.ptr(x), H, capi.ptr(logits), t, E, S, topk, ex, H, I, H, 0, capi.ACT["silu_and_mul"],
                                              capi.ptr(out), H, None))
        return out
    whole = run(big)
    small = run(T)
    capi.lib.b200dnn_clear_caches()
    # a row depends on its own token alone: INT8 sums are exact and the rest is computed row by row
    assert (small == whole[:T]).all()

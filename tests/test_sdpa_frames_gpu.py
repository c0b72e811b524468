"""The prompt kernel's exponentials: sums kept in a frame that follows the row maximum only when a score lies far above it.  Scores that jump by less and by far more than that
reach, block by block, within one half of a block and in one half only; scores so large that the frame is shifted; head dimensions at the edges of the
kernel's instantiations; rows whose keys fill one block, and one key more.  Against the CPU oracle with the tolerance of the operator's tests."""
import numpy as np
import pytest

from test_sdpa_gpu import capi, close, make, run  # noqa: F401  (capi: fixture)

pytestmark = pytest.mark.gpu


def stepped(oracle, rng, S, KV, D, steps):
    """Scores of a few units, plus steps[i] on the keys from i * KV / len(steps) on.  All of them are exact in f32 whatever the order of the products (multiples of 1/16;
    steps beyond 2^19 alone), so that kernel and oracle exponentiate the same numbers."""
    q, k = np.zeros((1, 2, S, D), np.float32), np.zeros((1, 2, KV, D), np.float32)
    if max(abs(x) for x in steps) < 2.0 ** 19:
        q[..., 1:5] = rng.integers(-4, 5, (1, 2, S, 4)) / 4.0
        k[..., 1:5] = rng.integers(-4, 5, (1, 2, KV, 4)) / 4.0
    q[..., 0] = 1.0
    k[..., 0] = np.repeat(np.asarray(steps, np.float32), -(-KV // len(steps)))[:KV]
    v = rng.standard_normal((1, 2, KV, D)).astype(np.float32)
    return tuple(oracle.f32_to_bf16(a) for a in (q, k, v))


STEPS = {"within the reach": (0, 4, 8, 12), "up, block by block": (0, 16, 48, 112, 240), "far up": (0, 1024, 65536), "down": (240, 112, 48, 0),
         "up and down": (0, 64, 0, 128, 0, 96), "shifted frames": (-2.0 ** 33, 2.0 ** 33), "one frame in the shifted range": (0, 2.0 ** 30),
         "below the range": (-2.0 ** 31, -2.0 ** 20, -64)}


@pytest.mark.parametrize("steps", STEPS)
@pytest.mark.parametrize("KV", [127, 129, 700])
def test_scores_in_steps(capi, oracle, steps, KV):
    rng = np.random.default_rng(KV)
    q, k, v = stepped(oracle, rng, 150, KV, 64, STEPS[steps])
    st, out = run(capi, q, k, v, scale=1.0)
    assert st == capi.SUCCESS, capi.last_error()
    close(oracle, out, oracle.sdpa(q, k, v, scale=1.0), v, (steps, KV))


@pytest.mark.parametrize("D", [64, 72, 80, 88, 96, 104])
@pytest.mark.parametrize("S,KV", [(128, 128), (150, 129), (300, 300)])
def test_head_dimensions(capi, oracle, D, S, KV):
    rng = np.random.default_rng(D + S)
    q, k, v = make(oracle, rng, 2, 2, S, KV, D)
    m = rng.standard_normal((2, 1, 1, KV)).astype(np.float32)
    m[1, ..., KV // 2:] = -np.inf
    for mask, causal in ((None, False), (None, True), (m, False)):
        st, out = run(capi, q, k, v, mask=mask, causal=causal)
        assert st == capi.SUCCESS, capi.last_error()
        close(oracle, out, oracle.sdpa(q, k, v, mask, causal=causal), v, (D, S, KV, causal))

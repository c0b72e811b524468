"""Attention with the values that break a softmax: scores far above the others.  The few-query kernel (up to 16 rows), the prompt kernel
and the three-step form (scores, softmax and product one after the other) have to agree with the oracle."""
import numpy as np
import pytest

from test_sdpa_gpu import capi, close, make, run  # noqa: F401  (capi: fixture)

pytestmark = pytest.mark.gpu

GAPS = (60.0, 89.0, 100.0, 150.0, 200.0, 400.0)


def one_large_key(oracle, rng, B, S, KV, D, keys):
    """Scores of about unit size but for one key per batch entry (keys[b]), which lies GAPS[h] above them (natural units, scale 1)."""
    H = len(GAPS)
    q, k, v = (rng.standard_normal((B, H, n, D)).astype(np.float32) for n in (S, KV, KV))
    q *= 0.3
    k *= 0.3
    q[..., 0] = 8.0
    k[..., 0] = 0.0
    for b in range(B):
        for h in range(H):
            k[b, h, keys[b], 0] = GAPS[h] / 8.0
    return tuple(oracle.f32_to_bf16(a) for a in (q, k, v))


@pytest.mark.parametrize("half", [0, 1])
@pytest.mark.parametrize("S", [7, 20])
def test_one_dominating_key_at_every_position(capi, oracle, S, half):
    """A middle block of 128 keys; every position of both 32-score chunks that a thread reads of its half."""
    rng = np.random.default_rng(S + half)
    keys = [128 + 64 * half + i for i in range(64)]
    q, k, v = one_large_key(oracle, rng, len(keys), S, 384, 64, keys)
    st, out = run(capi, q, k, v, scale=1.0)
    assert st == capi.SUCCESS, capi.last_error()
    close(oracle, out, oracle.sdpa(q, k, v, scale=1.0), v, (S, half))


def test_one_dominating_key_causal(capi, oracle):
    rng = np.random.default_rng(9)
    keys = [128 + 11 * i for i in range(12)]
    q, k, v = one_large_key(oracle, rng, len(keys), 400, 400, 64, keys)
    st, out = run(capi, q, k, v, scale=1.0, causal=True)
    assert st == capi.SUCCESS, capi.last_error()
    close(oracle, out, oracle.sdpa(q, k, v, scale=1.0, causal=True), v, "causal")

"""Attention with the values that break a softmax: one key whose score towers over the others, masks of the type's lowest finite
value, masks of any size on every key of a row, infinities and NaN.  The few-query kernel (up to 16 rows), the prompt kernel and the
three-step form (scores, softmax and product one after the other) have to agree with the oracle, and with each other where the
oracle is not defined."""
import numpy as np
import pytest

from test_sdpa_gpu import capi, close, make, run  # noqa: F401  (capi: fixture)

pytestmark = pytest.mark.gpu

GAPS = (60.0, 89.0, 100.0, 150.0, 200.0, 400.0)
FORMS = {"few queries": (7, "1"), "prompt": (150, "1"), "three steps": (150, "0")}


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


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("value", ["lowest", -1e9, -1e4, 1e4])
@pytest.mark.parametrize("causal", [False, True])
def test_rows_that_carry_one_finite_mask_value(capi, oracle, monkeypatch, form, bf16, value, causal):
    """Padding is usually written as the lowest finite value.  A row whose keys all carry it is a softmax over what is left of the
    scores after the addition (equal ones for the lowest value), not a row without keys."""
    S, fused = FORMS[form]
    monkeypatch.setenv("B200DNN_SDPA_FUSED", fused)
    lowest = np.float32(-3.3895313892515355e38) if bf16 else np.finfo(np.float32).min
    low = lowest if value == "lowest" else np.float32(value)
    rng = np.random.default_rng(S)
    B, H, KV, D = 2, 2, 300, 64
    q, k, v = make(oracle, rng, B, H, S, KV, D)
    m = np.zeros((B, 1, S, KV), dtype=np.float32)
    m[0, :, :, :140] = low                              # left padding: under the causal mask the first rows see nothing else
    m[1, :, S // 2] = low                               # a padding query
    m[1, :, :, 200:] = low
    mask = oracle.f32_to_bf16(m) if bf16 else m
    st, out = run(capi, q, k, v, mask=mask, causal=causal)
    assert st == capi.SUCCESS, capi.last_error()
    close(oracle, out, oracle.sdpa(q, k, v, oracle.bf16_to_f32(mask) if bf16 else m, causal=causal), v, (form, bf16, value, causal))


@pytest.mark.parametrize("S", [7, 150])
@pytest.mark.parametrize("what", ["nan key", "inf key", "nan query", "inf query", "nan mask", "inf mask"])
def test_non_finite_scores(capi, oracle, monkeypatch, S, what):
    """A NaN or an infinite score reaches its row as it does in the three-step form, wherever the key lies."""
    rng = np.random.default_rng(S)
    B, H, KV, D = 40, 1, 384, 64
    q, k, v = make(oracle, rng, B, H, S, KV, D)
    mask = None
    bad = {"nan": 0x7FC0, "inf": 0x7F80}[what[:3]]
    keys = [(b if b < 32 else 16 * (b - 32)) + (0, 128, 256)[b % 3] for b in range(B)]
    if what.endswith("key"):
        for b in range(B):
            k[b, 0, keys[b], 5] = bad
    elif what.endswith("query"):
        q[:, 0, S // 2, 5] = bad
        q[1:4, 0, S // 2, :] = bad
    else:
        mask = np.zeros((B, 1, S, KV), dtype=np.float32)
        for b in range(B):
            mask[b, 0, :, keys[b]] = np.nan if what[:3] == "nan" else np.inf
        mask[5, 0, 2] = np.nan
    got = {}
    for fused in ("0", "1"):
        monkeypatch.setenv("B200DNN_SDPA_FUSED", fused)
        st, out = run(capi, q, k, v, mask=mask)
        assert st == capi.SUCCESS, capi.last_error()
        got[fused] = oracle.bf16_to_f32(out)
    a, b = got["0"], got["1"]
    assert (np.isnan(a) == np.isnan(b)).all(), (what, int(np.isnan(a).sum()), int(np.isnan(b).sum()))
    ok = ~np.isnan(a)
    assert (np.abs(a - b)[ok] <= 2.0 ** -7 * np.abs(a[ok]) + 1e-3 * np.abs(oracle.bf16_to_f32(v)).max()).all()


@pytest.mark.parametrize("S", [7, 150])
@pytest.mark.parametrize("base", [2.0 ** 10, 2.0 ** 16, -2.0 ** 16])
def test_scores_with_a_large_common_part(capi, oracle, S, base):
    """Scores of one size far from 0: what counts is their distance from the row maximum, which f32 holds exactly here (the products of
    the common part are powers of two, the rest small integers over 16), so probabilities keep their precision at any size."""
    rng = np.random.default_rng(S)
    B, H, KV, D = 1, 2, 300, 64
    q, k = np.zeros((B, H, S, D), np.float32), np.zeros((B, H, KV, D), np.float32)
    q[..., 0], k[..., 0] = 2.0 ** 5, base / 2.0 ** 5
    q[..., 1:5] = rng.integers(-8, 9, (B, H, S, 4)) / 4.0
    k[..., 1:5] = rng.integers(-8, 9, (B, H, KV, 4)) / 4.0
    v = rng.standard_normal((B, H, KV, D)).astype(np.float32)
    q, k, v = (oracle.f32_to_bf16(a) for a in (q, k, v))
    st, out = run(capi, q, k, v, scale=1.0)
    assert st == capi.SUCCESS, capi.last_error()
    close(oracle, out, oracle.sdpa(q, k, v, scale=1.0), v, (S, base))

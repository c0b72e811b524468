"""The vector form of the row normalisations at rows of any length: rows that are no whole 16-byte vectors, one behind the other in memory (each row meets its
neighbours' elements in its first and last vector), around the widths at which the number of threads and of vectors per thread changes, against the CPU oracle
with the tolerance of the operator's tests."""
import numpy as np
import pytest

from test_norm_gpu import capi, close, run  # noqa: F401  (capi: fixture)

pytestmark = pytest.mark.gpu

WIDTHS = (1, 7, 9, 255, 257, 505, 844, 4081, 4083, 4089, 8178, 8191, 8200, 11072, 12274, 12275, 12289, 16370, 16371, 16376, 16384)


@pytest.mark.parametrize("n", WIDTHS)
@pytest.mark.parametrize("kind", ["rms_norm", "fused_add_rms_norm", "layer_norm"])
def test_rows_of_any_length(capi, oracle, kind, n):
    rng = np.random.default_rng(n)
    rows = 11                                           # every distance from a 16-byte boundary
    x = rng.normal(size=(rows, n)).astype(np.float32) * 2 + 0.3
    x[4] *= 1e4                                         # a row that a neighbour must not see
    x = oracle.f32_to_bf16(x)
    res = oracle.f32_to_bf16(rng.normal(size=(rows, n)).astype(np.float32)) if kind == "fused_add_rms_norm" else None
    params = rng.normal(size=(2, n)).astype(np.float32)
    for bf16 in (False, True):
        gamma, beta = (oracle.f32_to_bf16(p) if bf16 else p for p in params)
        if kind != "layer_norm":
            beta = None
        st, out, res_out, q, s = run(capi, kind, x, gamma, beta, residual=res, quant=True)
        assert st == capi.SUCCESS, capi.last_error()
        ref = oracle.normalization(kind, x, gamma, beta, **({} if res is None else dict(residual=res)))
        if res is not None:
            ref, ref_res = ref
            assert (res_out == ref_res).all()
        close(oracle, out, ref, (kind, n, bf16))
        qr, sr = oracle.quant_per_token(out)
        assert (q == qr).all() and (s == sr).all(), (kind, n, bf16)


@pytest.mark.parametrize("n", [41, 844])
def test_infinities_and_nan_stay_in_their_row(capi, oracle, n):
    rng = np.random.default_rng(n)
    x = rng.normal(size=(9, n)).astype(np.float32)
    clean = oracle.f32_to_bf16(x)
    x[2, 0], x[4, n - 1], x[6, n // 2] = np.inf, np.nan, -np.inf
    gamma = rng.normal(size=n).astype(np.float32)
    for kind, beta in (("rms_norm", None), ("layer_norm", gamma)):
        want = run(capi, kind, clean, gamma, beta, quant=True)
        got = run(capi, kind, oracle.f32_to_bf16(x), gamma, beta, quant=True)
        assert want[0] == capi.SUCCESS and got[0] == capi.SUCCESS
        for row in (0, 1, 3, 5, 7, 8):
            for i in (1, 3, 4):
                assert (got[i][row] == want[i][row]).all(), (kind, row, i)


@pytest.mark.parametrize("rows", [253, 506, 1100, 1265, 2101])
@pytest.mark.parametrize("n", [505, 844, 1024, 1536, 2056, 2999, 4104, 6152, 6400, 8192, 8200])
@pytest.mark.parametrize("kind", ["fused_add_rms_norm", "layer_norm"])
def test_many_rows(capi, oracle, kind, n, rows):
    """As many rows as make a thread hold two or four vectors: the same eleven rows again and again."""
    rng = np.random.default_rng(n)
    x = oracle.f32_to_bf16(rng.normal(size=(11, n)).astype(np.float32) * 2 + 0.3)
    res = oracle.f32_to_bf16(rng.normal(size=(11, n)).astype(np.float32)) if kind == "fused_add_rms_norm" else None
    gamma, beta = (rng.normal(size=n).astype(np.float32) for _ in range(2))
    if kind != "layer_norm":
        beta = None
    times = (rows // 11, 1)
    st, out, res_out, q, s = run(capi, kind, np.tile(x, times), gamma, beta, residual=None if res is None else np.tile(res, times), quant=True)
    assert st == capi.SUCCESS, capi.last_error()
    ref = oracle.normalization(kind, x, gamma, beta, **({} if res is None else dict(residual=res)))
    if res is not None:
        ref, ref_res = ref
        assert (res_out == np.tile(ref_res, times)).all()
    close(oracle, out, np.tile(ref, times), (kind, n, rows))
    for part in (slice(0, 11), slice(rows - 11, rows)):
        qr, sr = oracle.quant_per_token(np.ascontiguousarray(out[part]))
        assert (q[part] == qr).all() and (s[part] == sr).all(), (kind, n, rows)

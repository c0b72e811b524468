"""Every form and width of the tcgen05 tile kernel that the cost model may choose for a plain call: one CTA a tile, a pair, shares of K over a cluster, at each
width.  That the form ran is read from a captured graph.  INT8 sums are exact and the float epilogue gives the bytes of the default form; bf16 within
the bound of its f32 sums."""
import numpy as np
import pytest

from helpers import kernel_grids
from test_matmul_gpu import capi  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu

FORMS = [(0, bn, 1) for bn in (32, 64, 96, 128, 160, 192, 224, 256)] + [(1, bn, 1) for bn in (64, 96, 128, 160, 192, 224, 256)] + \
        [(0, 64, 2), (0, 128, 2), (0, 128, 3), (0, 128, 4), (0, 256, 2), (0, 256, 3), (0, 256, 4)]


def _force(monkeypatch, pair, bn, splits):
    for name, v in (("PAIR", pair), ("BN", bn), ("KSPLIT", splits)):
        monkeypatch.setenv("B200DNN_TC_" + name, str(v))


def _ctas(M, N, pair, bn, splits):
    import torch
    sms, tiles = torch.cuda.get_device_properties(0).multi_processor_count, -(-M // (256 if pair else 128)) * -(-N // bn)
    return 2 * min(tiles, sms // 2) if pair else tiles * splits if splits > 1 else min(tiles, sms)


# ragged rows and columns, K with a short last block; more tiles than SMs where the tiles are narrow
@pytest.mark.parametrize("pair,bn,splits", FORMS)
@pytest.mark.parametrize("M,K,N", [(100, 1296, 1000), (300, 2064, 264), (770, 912, 2100)])
def test_int8(capi, oracle, monkeypatch, pair, bn, splits, M, K, N):
    import torch
    rng = np.random.default_rng(M + bn)
    A, W = rng.integers(-128, 128, (M, K), dtype=np.int8), rng.integers(-128, 128, (K, N), dtype=np.int8)
    sa, sw, bias = rng.uniform(0.01, 0.05, M).astype(np.float32), rng.uniform(1e-4, 5e-4, N).astype(np.float32), rng.normal(size=N).astype(np.float32)
    dA, dW, dsa, dsw, db = (torch.from_numpy(x).cuda() for x in (A, W, sa, sw, bias))
    s32, out = torch.zeros(M, N, dtype=torch.int32, device="cuda"), torch.zeros(M, N, dtype=torch.bfloat16, device="cuda")
    d32 = capi.make_matmul(M, N, K, dA, dW, s32, src_dt=capi.DT["s8"], dst_dt=capi.DT["s32"], force_kernel=2)
    f32 = torch.zeros(M, N, device="cuda")
    df = capi.make_matmul(M, N, K, dA, dW, f32, src_dt=capi.DT["s8"], dst_dt=capi.DT["f32"], src_scale=dsa, wei_scale=dsw, bias=db, postops=["relu"], force_kernel=2)
    d16 = capi.make_matmul(M, N, K, dA, dW, out, src_dt=capi.DT["s8"], dst_dt=capi.DT["bf16"], src_scale=dsa, wei_scale=dsw, bias=db, postops=["gelu_tanh"], force_kernel=2)
    st = torch.cuda.current_stream().cuda_stream
    capi.check(capi.matmul(d16, st))
    default = out.clone()
    _force(monkeypatch, pair, bn, splits)
    assert _ctas(M, N, pair, bn, splits) in [n for n, _ in kernel_grids(lambda st: capi.check(capi.matmul(d32, st)))]
    s32.zero_()
    out.zero_()
    capi.check(capi.matmul(d32, st))
    capi.check(capi.matmul(d16, st))
    capi.check(capi.matmul(df, st))
    acc = oracle.gemm_s32(A, W)
    assert (s32.cpu().numpy() == acc).all()
    assert torch.equal(out, default)
    # one rounding per operation, none of them contracted
    assert (f32.cpu().numpy() == np.maximum(acc.astype(np.float32) * sa[:, None] * sw[None, :] + bias[None, :], np.float32(0))).all()
    capi.lib.b200dnn_clear_caches()


@pytest.mark.parametrize("pair,bn,splits", FORMS)
@pytest.mark.parametrize("M,K,N", [(100, 1048, 1000), (770, 456, 1300)])
def test_bf16(capi, monkeypatch, pair, bn, splits, M, K, N):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M + bn)
    A, W = (torch.randn(s, device="cuda", generator=g).bfloat16() for s in ((M, K), (K, N)))
    bias = torch.randn(N, device="cuda", generator=g)
    out = torch.zeros(M, N, device="cuda")
    d = capi.make_matmul(M, N, K, A, W, out, src_dt=capi.DT["bf16"], wei_dt=capi.DT["bf16"], dst_dt=capi.DT["f32"], bias=bias, force_kernel=2)
    _force(monkeypatch, pair, bn, splits)
    assert _ctas(M, N, pair, bn, splits) in [n for n, _ in kernel_grids(lambda st: capi.check(capi.matmul(d, st)))]
    out.zero_()
    capi.check(capi.matmul(d, torch.cuda.current_stream().cuda_stream))
    a, w = A.double(), W.double()
    # f32 sums of K exact products, see test_skinny_gpu.py
    assert ((out - (a @ w + bias)).abs() <= K * 2.0 ** -23 * (a.abs() @ w.abs() + bias.abs())).all()
    capi.lib.b200dnn_clear_caches()


@pytest.mark.parametrize("M", [20, 400])
def test_gelu_tanh_rounds_where_it_did(capi, M):
    """x / (1 + 2^(-2 u log2 e)) with u = (c x) (1 + (f x) x), the last sum in one rounding (few rows and tiles).  From the argument on, what is left
    are 2^x (2^-22), the reciprocal (2^-23) and three roundings (2^-24); a rounding more in u moves the result by 14 to 25 times 2^-24 or 2^-23."""
    import torch
    rng = np.random.default_rng(M)
    K, N, f4 = 16, 256, np.float32
    A, W = np.zeros((M, K), dtype=np.int8), np.zeros((K, N), dtype=np.int8)
    A[:, 0], W[0] = 1, -(np.arange(N) % 16 + 112).astype(np.int8)
    s = rng.uniform(4.6 / 112, 5.7 / 127, M).astype(f4)
    out = torch.zeros(M, N, device="cuda")
    dA, dW, ds, dw = torch.from_numpy(A).cuda(), torch.from_numpy(W).cuda(), torch.from_numpy(s).cuda(), torch.ones(N, device="cuda")
    d = capi.make_matmul(M, N, K, dA, dW, out, src_dt=capi.DT["s8"], dst_dt=capi.DT["f32"], src_scale=ds, wei_scale=dw, weights_const=False, postops=["gelu_tanh"])
    capi.check(capi.matmul(d, torch.cuda.current_stream().cuda_stream))
    x = W[0].astype(f4)[None, :] * s[:, None]
    c, f = f4(0.79788458347320556640625), f4(0.044715)
    t = ((f * x).astype(np.float64) * x + 1).astype(f4)                         # (the product is exact in double)
    arg = ((c * x) * t) * f4(-2.0 * 1.44269504088896340736)
    ref = x / (1 + np.exp2(arg.astype(np.float64)))
    err = np.abs(out.cpu().numpy() - ref) / np.abs(ref)
    assert err.max() <= 2.0 ** -22 + 2.0 ** -23 + 3 * 2.0 ** -24, err.max()

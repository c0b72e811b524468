"""INT8 GEMMs whose rows start anywhere: activations whose base or row stride is not a multiple of 16 bytes (re-pitched in front of
the tcgen05 kernel, funnel-shifted into shared memory by the decode kernels) and destinations without 16-byte alignment (stored
along the rows through the epilogue's staging blocks).  s32 sums and the bf16 / f32 results without a transcendental are exact,
and nothing outside the destination's columns is written."""
import numpy as np
import pytest

from test_matmul_gpu import capi  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 2, 7, 16, 17, 129, 300])
@pytest.mark.parametrize("K,lda_pad,a_off", [(31, 0, 0), (128, 1, 0), (333, 3, 5), (1027, 13, 2), (256, 0, 1)])
@pytest.mark.parametrize("N,ldc_pad,d_off", [(1, 0, 0), (33, 2, 1), (130, 1, 3), (259, 0, 0)])
def test_any_alignment(capi, oracle, M, K, lda_pad, a_off, N, ldc_pad, d_off):
    import torch
    rng = np.random.default_rng(M * 7 + K + N)
    lda, ldc = K + lda_pad, N + ldc_pad
    A = rng.integers(0, 256, (M, K), dtype=np.uint8)
    W = rng.integers(-128, 128, (K, N), dtype=np.int8)
    bias = rng.normal(size=N).astype(np.float32)
    ws = rng.uniform(0.001, 0.01, N).astype(np.float32)
    abuf = torch.full((a_off + M * lda,), 7, dtype=torch.uint8, device="cuda")
    abuf[a_off:].view(M, lda)[:, :K] = torch.from_numpy(A).cuda()
    w_dev, b_dev, ws_dev = torch.from_numpy(W).cuda(), torch.from_numpy(bias).cuda(), torch.from_numpy(ws).cuda()
    ss, zp = torch.full((1,), 0.02, device="cuda"), torch.full((1,), 37, dtype=torch.int32, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    for name, tdt, kw in (("s32", torch.int32, {}),
                          ("f32", torch.float32, dict(src_scale=ss, wei_scale=ws_dev, src_zp=zp, bias=b_dev, postops=["relu"])),
                          ("bf16", torch.int16, dict(src_scale=ss, wei_scale=ws_dev, src_zp=zp, bias=b_dev, postops=["relu"]))):
        dbuf = torch.full((d_off + M * ldc,), 99, dtype=tdt, device="cuda")
        dst = dbuf[d_off:]
        d = capi.make_matmul(M, N, K, abuf.data_ptr() + a_off, w_dev, dst, src_dt=capi.DT["u8"], dst_dt=capi.DT[name], lda=lda, ldc=ldc,
                             weights_const=False, **kw)
        assert capi.matmul(d, st) == capi.SUCCESS, capi.last_error()
        torch.cuda.synchronize()
        got = dst.view(M, ldc).cpu().numpy()
        ref = oracle.matmul_w8a8(A, W, name, src_scale=None if name == "s32" else np.array([0.02], dtype=np.float32),
                                 wei_scale=None if name == "s32" else ws, src_zp=0 if name == "s32" else 37,
                                 bias=None if name == "s32" else bias, postops=[] if name == "s32" else ["relu"])
        res = np.ascontiguousarray(got[:, :N])
        assert (res.view(np.uint16 if name == "bf16" else res.dtype) == ref).all(), name
        assert (got[:, N:] == 99).all() and (dbuf[:d_off] == 99).all(), name

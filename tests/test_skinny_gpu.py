"""The few-row tcgen05 kernel (weight as the MMA's 128 rows, shares of K added over a cluster) at the edges of its range: row
counts beside multiples of 16, column tiles with a remainder, K with a remainder and with too few blocks to share, every result type."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def capi():
    from zendnn_b200 import capi as c
    assert c.lib.b200dnn_device_count() > 0, "no CUDA device"
    return c


@pytest.mark.parametrize("M,K,N", [(17, 128, 128), (17, 1100, 130), (33, 4096, 1000), (48, 2064, 513), (16, 8192, 3080), (31, 544, 4097)])
@pytest.mark.parametrize("out", ["s32", "f32", "bf16"])
def test_skinny_int8(capi, oracle, M, K, N, out):
    rng = np.random.default_rng(M * 7 + N)
    K16 = K + (-K) % 16                                     # rows at a pitch the copy engine takes
    A = np.zeros((M, K16), dtype=np.uint8)
    A[:, :K] = rng.integers(0, 256, (M, K))
    W = rng.integers(-128, 128, (K, N), dtype=np.int8)
    zp = np.array([131], dtype=np.int32)
    acc = (A[:, :K].astype(np.int64) - 131) @ W.astype(np.int64)
    kw = dict(lda=K16, src_dt=capi.DT["u8"], dst_dt=capi.DT[out], src_zp=zp, weights_const=False)
    if out == "s32":
        dst = np.zeros((M, N), dtype=np.int32)
        capi.check(capi.matmul(capi.make_matmul(M, N, K, A, W, dst, **kw)))
        assert (dst == acc).all()
        return
    ss, sw, bias = np.array([0.013], dtype=np.float32), rng.uniform(0.001, 0.01, N).astype(np.float32), rng.standard_normal(N).astype(np.float32)
    dst = np.zeros((M, N), dtype=np.float32 if out == "f32" else np.uint16)
    capi.check(capi.matmul(capi.make_matmul(M, N, K, A, W, dst, src_scale=ss, wei_scale=sw, bias=bias, postops=["relu"], **kw)))
    ref = np.maximum((acc.astype(np.float32) * ss) * sw + bias, np.float32(0))      # one rounding per operation, as in the kernel
    if out == "f32":
        assert (dst == ref).all()
    else:
        assert (dst == oracle.f32_to_bf16(ref)).all()


@pytest.mark.parametrize("M,K,N", [(1, 64, 16), (1, 4096, 1000), (15, 1096, 257), (16, 8192, 384), (49, 2048, 1030), (64, 520, 4100)])
@pytest.mark.parametrize("out", ["f32", "bf16"])
def test_skinny_bf16(capi, oracle, M, K, N, out):
    rng = np.random.default_rng(M * 5 + K)
    A, W = (oracle.f32_to_bf16(rng.standard_normal(s).astype(np.float32)) for s in ((M, K), (K, N)))
    bias = rng.standard_normal(N).astype(np.float32)
    dst = np.zeros((M, N), dtype=np.float32 if out == "f32" else np.uint16)
    d = capi.make_matmul(M, N, K, A, W, dst, src_dt=capi.DT["bf16"], wei_dt=capi.DT["bf16"], dst_dt=capi.DT[out], bias=bias, weights_const=True,
                         flags=capi.FLAG_STABLE_WEIGHTS)
    a, w = ((x.astype(np.uint32) << 16).view(np.float32).astype(np.float64) for x in (A, W))
    ref = a @ w + bias
    # f32 sums of K exact products: each of the K additions rounds by at most 2^-24 of a partial sum (2^-23 where the tensor core cuts
    # instead), and a partial sum is at most sum |a||w|; bf16 rounds the result by 2^-9 of itself on top
    tol = K * 2.0 ** -23 * (np.abs(a) @ np.abs(w) + np.abs(bias))
    for _ in range(2):                                      # the second call finds the packed weight, complete, and reads it early
        dst[:] = 0
        capi.check(capi.matmul(d))
        got = dst.astype(np.float64) if out == "f32" else (dst.astype(np.uint32) << 16).view(np.float32).astype(np.float64)
        assert (np.abs(got - ref) <= tol + (0 if out == "f32" else 2.0 ** -8 * np.abs(ref))).all()
    capi.lib.b200dnn_clear_caches()


@pytest.mark.parametrize("kernel", [4, 5, -1])
def test_other_kernel_numbers_stay_with_the_tile_kernel(capi, oracle, kernel):
    """force_kernel names the kernels 1 to 3; any other number runs the tcgen05 tile kernel, which refuses rows that the copy engine
    cannot read."""
    rng = np.random.default_rng(kernel + 1)
    for M, K in ((5, 64), (20, 160)):
        A, W = rng.integers(-128, 128, (M, K), dtype=np.int8), rng.integers(-128, 128, (K, 72), dtype=np.int8)
        dst = np.zeros((M, 72), dtype=np.int32)
        capi.check(capi.matmul(capi.make_matmul(M, 72, K, A, W, dst, src_dt=capi.DT["s8"], dst_dt=capi.DT["s32"], weights_const=False, force_kernel=kernel)))
        assert (dst == A.astype(np.int32) @ W.astype(np.int32)).all()
    A, dst = rng.integers(-128, 128, (20, 33), dtype=np.int8), np.zeros((20, 72), dtype=np.int32)
    d = capi.make_matmul(20, 72, 33, A, W, dst, src_dt=capi.DT["s8"], dst_dt=capi.DT["s32"], weights_const=False, force_kernel=kernel)
    assert capi.matmul(d) == capi.FAILURE and "16-byte aligned" in capi.last_error()


# both sides of the lines that the choice of kernel draws: rows against bytes of a column, one wave of column tiles (148 x 128 columns) and
# how full the last one is, rows of 16 x K that the decode kernel has no room for
@pytest.mark.parametrize("M,K,N", [(24, 512, 300), (25, 1008, 300), (25, 1024, 300), (33, 1536, 300), (33, 1520, 300), (48, 1024, 18944), (9, 2048, 18945),
                                   (17, 3072, 18945), (24, 3072, 37889), (25, 512, 25600), (24, 512, 18945), (16, 14336, 18960), (9, 8192, 18944),
                                   (49, 2048, 300), (64, 2048, 5120), (64, 2048, 5121), (49, 4096, 5121), (64, 4080, 9472), (33, 3056, 9473), (48, 3072, 9473),
                                   (48, 8192, 9473), (64, 8192, 9473), (65, 8192, 9473)])
def test_lines_of_the_choice_int8(capi, M, K, N):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    A, W = (torch.randint(-128, 128, s, dtype=torch.int8, device="cuda", generator=g) for s in ((M, K), (K, N)))
    dst = torch.full((M, N), 7, dtype=torch.int32, device="cuda")
    capi.check(capi.matmul(capi.make_matmul(M, N, K, A, W, dst, src_dt=capi.DT["s8"], dst_dt=capi.DT["s32"], weights_const=False),
                           torch.cuda.current_stream().cuda_stream))
    assert torch.equal(dst, (A.double() @ W.double()).int())


@pytest.mark.parametrize("M,K,N", [(64, 1024, 300), (64, 1016, 300), (48, 768, 300), (48, 760, 300), (8, 512, 18944), (8, 512, 18945), (8, 512, 25300),
                                   (9, 1536, 25300), (24, 1536, 25300), (24, 1528, 25300), (25, 1536, 25300), (64, 1024, 5121), (64, 2048, 5121), (48, 1528, 9473),
                                   (48, 1536, 9473), (64, 4088, 9473), (64, 4096, 9473)])
def test_lines_of_the_choice_bf16(capi, M, K, N):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M + K + N)
    A, W = (torch.randn(s, device="cuda", generator=g).bfloat16() for s in ((M, K), (K, N)))
    dst = torch.zeros(M, N, device="cuda")
    capi.check(capi.matmul(capi.make_matmul(M, N, K, A, W, dst, src_dt=capi.DT["bf16"], wei_dt=capi.DT["bf16"], dst_dt=capi.DT["f32"], weights_const=False),
                           torch.cuda.current_stream().cuda_stream))
    a, w = A.double(), W.double()
    assert ((dst - a @ w).abs() <= K * 2.0 ** -23 * (a.abs() @ w.abs())).all()      # see test_skinny_bf16

"""W4A8 in its tensor-core form against the oracle: edges of its tiles (rows, columns, a last block of K that is short), every class of group size, shares
of K over a cluster, more tiles than SMs, and its bounded waits.  Within 1 bf16 ulp, as the other W4A8 forms."""
import ctypes as C

import numpy as np
import pytest

from helpers import assert_bf16_close, kernel_grids

pytestmark = pytest.mark.gpu


def _case(oracle, M, K, N, gs, transB=False, bias=True, po=("swish",)):
    from zendnn_b200 import capi
    G = K // gs
    rng = np.random.default_rng(M * 3 + K + N + gs)
    X = oracle.f32_to_bf16(rng.normal(size=(M, K)).astype(np.float32))
    X[M // 2, K // 3] = 0x7FC0          # a NaN entry quantises to 0
    W = rng.integers(-8, 8, (K, N), dtype=np.int8)
    sw = rng.uniform(1e-3, 5e-3, (G, N)).astype(np.float32)
    b = rng.normal(size=N).astype(np.float32) if bias else None
    A, sa = oracle.quant_per_token(X)
    ref = oracle.matmul_group_scaled(A, W, sa.reshape(M, 1), sw, "bf16", bias=b, postops=list(po))
    packed, out, sc = oracle.pack_s4(W, transB), np.zeros((M, N), dtype=np.uint16), np.zeros(M, dtype=np.float32)
    d = capi.make_matmul(M, N, K, X, packed, out, src_dt=capi.DT["bf16"], dst_dt=capi.DT["bf16"], transB=transB, bias=b, src_scale=capi.quant(sc, count=M),
                         wei_scale=capi.quant(sw, count=G * N), weights_const=False, dynamic_quant=True, wei_dt=capi.DT["s4"], postops=po)
    return capi, d, out, ref, sc, sa, (X, W, sw, b, packed)


@pytest.mark.parametrize("split", [1, 2, 4])
@pytest.mark.parametrize("gs", [32, 64, 128, 256, 384])
@pytest.mark.parametrize("M,N", [(1, 8), (16, 136), (17, 130), (33, 1000), (64, 256), (65, 127), (129, 264)])
def test_edges(oracle, monkeypatch, M, N, gs, split):
    monkeypatch.setenv("B200DNN_GS_TC", "1")
    monkeypatch.setenv("B200DNN_GS_TC_SPLIT", str(split if split > 1 else 99))
    K = 3072 if gs == 384 else 1024 + (gs if gs <= 64 else 0)     # groups of 32 and 64: the last block of 128 k is a quarter or half full
    if gs == 256:
        K = 2048
    capi, d, out, ref, sc, sa, keep = _case(oracle, M, K, N, gs, transB=bool(split & 2))
    capi.check(capi.matmul(d))
    assert (sc == sa).all()
    assert_bf16_close(out, ref, 1, "M=%d K=%d N=%d gs=%d split=%d" % (M, K, N, gs, split), atol=1e-5)


def _device_case(oracle, M, K, N, gs):
    """The same on device memory, with a stream to call on: the call, what it launches per grid and block, its result and the oracle's."""
    import torch
    capi, d, out, ref, _, _, keep = _case(oracle, M, K, N, gs)
    X, W, sw, b, packed = (torch.from_numpy(np.ascontiguousarray(x).view(np.int16) if x.dtype == np.uint16 else np.ascontiguousarray(x)).cuda() for x in keep)
    o = torch.zeros((M, N), dtype=torch.int16, device="cuda")
    d = capi.make_matmul(M, N, K, X, packed, o, src_dt=capi.DT["bf16"], dst_dt=capi.DT["bf16"], bias=b, src_scale=capi.quant(None, count=M),
                         wei_scale=capi.quant(sw, K // gs * N, capi.DT["f32"]), dynamic_quant=True, wei_dt=capi.DT["s4"], postops=("swish",))
    launched = kernel_grids(lambda st: capi.check(capi.matmul(d, st)))
    o.zero_()
    capi.check(capi.matmul(d, torch.cuda.current_stream().cuda_stream))
    got = o.cpu().numpy().view(np.uint16)
    capi.lib.b200dnn_clear_caches()
    return launched, got, ref


GS_TC_THREADS = {16: 608, 32: 608, 64: 864, 128: 864}      # of a CTA, by its rows


@pytest.mark.parametrize("split", [3, 5, 6, 7, 8])
@pytest.mark.parametrize("gs", [32, 64, 128, 256])
@pytest.mark.parametrize("bm,M", [(16, 11), (32, 27), (64, 70), (128, 100)])
def test_shares(oracle, monkeypatch, bm, M, gs, split):
    """Shares of the groups that do not come out even (17 over a cluster; with groups of 32 and 64 the last block of 128 k is a quarter or half full)."""
    monkeypatch.setenv("B200DNN_GS_TC", "1")
    monkeypatch.setenv("B200DNN_GS_TC_BM", str(bm))
    monkeypatch.setenv("B200DNN_GS_TC_SPLIT", str(split))
    K = 16 * 128 + gs if gs <= 128 else 17 * gs
    N = 200
    launched, got, ref = _device_case(oracle, M, K, N, gs)
    assert (2 * -(-M // bm) * split, GS_TC_THREADS[bm]) in launched, launched
    assert_bf16_close(got, ref, 1, "bm=%d gs=%d split=%d" % (bm, gs, split), atol=1e-5)


# both sides of each line of the choice, up to 16 rows: K, rows, columns against the decode form; the group and the columns against the general
# form (fewer than eight groups); odd columns and rows that the decode form has no room for
@pytest.mark.parametrize("M,K,N,gs,tensor_cores", [(1, 2048, 512, 32, False), (1, 4096, 512, 32, True), (16, 4096, 512, 128, False), (16, 8192, 512, 128, True),
                                                   (2, 1024, 256, 64, False), (16, 1024, 28672, 64, True), (1, 256, 512, 128, False), (1, 256, 4864, 128, True),
                                                   (1, 1024, 512, 1024, True), (12, 14336, 128, 128, True), (3, 1024, 333, 128, True), (3, 1024, 334, 128, False)])
def test_lines_of_the_choice(oracle, monkeypatch, M, K, N, gs, tensor_cores):
    launched, got, ref = _device_case(oracle, M, K, N, gs)
    assert any(threads == 608 for _, threads in launched) == tensor_cores, launched
    assert_bf16_close(got, ref, 1, "M=%d K=%d N=%d gs=%d" % (M, K, N, gs), atol=1e-5)


@pytest.mark.parametrize("gs", [32, 128])
@pytest.mark.parametrize("bm", [16, 32, 64, 128])
def test_more_tiles_than_sms(oracle, monkeypatch, gs, bm):
    """The persistent walk: rings and barriers go on from one tile to the next."""
    monkeypatch.setenv("B200DNN_GS_TC_BM", str(bm))
    M, K, N = 150, 640, 128 * (160 if bm == 128 else 60) + 24
    capi, d, out, ref, _, _, keep = _case(oracle, M, K, N, gs, bias=False, po=())
    capi.check(capi.matmul(d))
    assert_bf16_close(out, ref, 1, "bm=%d gs=%d" % (bm, gs), atol=1e-5)


@pytest.mark.parametrize("bm", [1, 48, 256, -16])
@pytest.mark.parametrize("M", [4, 150])
def test_tile_rows_that_do_not_exist(oracle, monkeypatch, M, bm):
    """Refused on the host (the kernel divides by the number of shares, which nothing would have set)."""
    monkeypatch.setenv("B200DNN_GS_TC", "1")
    monkeypatch.setenv("B200DNN_GS_TC_BM", str(bm))
    capi, d, out, _, _, _, keep = _case(oracle, M, 256, 136, 32)
    assert capi.matmul(d) == capi.FAILURE and "bad tile rows %d" % bm in capi.last_error()
    assert (out == 0).all()


@pytest.mark.parametrize("M", [4, 200])
def test_waits_run_out(monkeypatch, M):
    import torch
    from zendnn_b200 import capi
    st = torch.cuda.current_stream().cuda_stream
    K, N, gs = 4096, 640, 128
    x = torch.randn(M, K, device="cuda").bfloat16()
    w = torch.randint(0, 256, (K * N // 2,), dtype=torch.uint8, device="cuda")
    ws = torch.rand(K // gs, N, device="cuda") * 4e-3 + 1e-3
    o = torch.zeros(M, N, dtype=torch.bfloat16, device="cuda")
    d = capi.make_matmul(M, N, K, x, w, o, src_dt=capi.DT["bf16"], wei_dt=capi.DT["s4"], dst_dt=capi.DT["bf16"], dynamic_quant=True,
                         src_scale=capi.quant(None, M, capi.DT["f32"]), wei_scale=capi.quant(ws, ws.numel(), capi.DT["f32"]))
    monkeypatch.setenv("B200DNN_GS_TC", "1")
    capi.check(capi.matmul(d, st))
    assert capi.lib.b200dnn_stream_status(C.c_void_p(st)) == capi.SUCCESS
    ref = o.clone()
    monkeypatch.setenv("B200DNN_TEST_NO_LOADS", "1")
    capi.check(capi.matmul(d, st))
    assert capi.lib.b200dnn_stream_status(C.c_void_p(st)) == capi.FAILURE
    assert "gave up waiting" in capi.last_error()
    monkeypatch.delenv("B200DNN_TEST_NO_LOADS")
    o.zero_()
    capi.check(capi.matmul(d, st))
    assert capi.lib.b200dnn_stream_status(C.c_void_p(st)) == capi.SUCCESS
    assert torch.equal(o, ref)
    capi.lib.b200dnn_clear_caches()

"""Dynamic quantisation inside the decode kernels: results and row scales equal, bit for bit, those of the call whose rows a kernel of its own quantises, at the edges
of the split of rows over warps (1 to 16 rows, few and many vectors a lane) and for rows with infinities, NaN and zeros; sources that the fused form does not take."""
import numpy as np
import pytest

from test_matmul_gpu import capi  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


def call(capi, monkeypatch, fused, x, w, ws, sdt="f32", K=None, out=None, ring=None):
    import torch
    M, N = x.shape[0], w.shape[1]
    K = K or x.shape[1]
    monkeypatch.setenv("B200DNN_FUSED_QUANT", fused)
    monkeypatch.setenv("B200DNN_DECODE_KERNEL", "2" if ring else "1")
    scale = torch.zeros(M, dtype=torch.float32 if sdt == "f32" else torch.bfloat16, device="cuda")
    y = torch.zeros(M, N, device="cuda") if out is None else out
    before = capi.lib.b200dnn_launch_count()
    d = capi.make_matmul(M, N, K, x, w, y, src_dt=capi.DT["bf16"], dst_dt=capi.DT["f32"], dynamic_quant=True, src_scale=capi.quant(scale, M, capi.DT[sdt]), wei_scale=ws, lda=x.stride(0))
    capi.check(capi.matmul(d, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return y, scale, capi.lib.b200dnn_launch_count() - before


def weights(torch, K, N):
    return torch.randint(-127, 128, (K, N), dtype=torch.int8, device="cuda"), torch.rand(N, device="cuda") * 0.01


@pytest.mark.parametrize("ring", [False, True])
@pytest.mark.parametrize("M", [1, 2, 3, 5, 7, 8, 11, 16])
@pytest.mark.parametrize("K", [8, 264, 2048, 6152])
def test_bits_of_the_separate_kernel(capi, monkeypatch, M, K, ring):
    import torch
    torch.manual_seed(M + K)
    w, ws = weights(torch, K, 136)
    x = (torch.randn(M, K, device="cuda") * torch.logspace(-3, 3, M, device="cuda")[:, None]).bfloat16()
    capi.lib.b200dnn_clear_caches()
    call(capi, monkeypatch, "0", x, w, ws)                       # (packs the weight)
    for sdt in ("f32", "bf16"):
        want, want_s, n0 = call(capi, monkeypatch, "0", x, w, ws, sdt, ring=ring)
        got, got_s, n1 = call(capi, monkeypatch, "1", x, w, ws, sdt, ring=ring)
        # (the ring form has eight warps, and a row needs one at least)
        assert n1 == (n0 if ring and M > 8 else n0 - 1) and torch.equal(got, want) and torch.equal(got_s, want_s), (M, K, sdt)
    capi.lib.b200dnn_clear_caches()


@pytest.mark.parametrize("M", [1, 4, 16])
def test_rows_that_are_not_finite(capi, monkeypatch, M):
    import torch
    torch.manual_seed(M)
    K = 1032
    w, ws = weights(torch, K, 72)
    for bad in (float("inf"), -float("inf"), float("nan")):
        x = torch.randn(M, K, device="cuda").bfloat16()
        x[M // 2, 5], x[M - 1, K - 1], x[0, 700:] = bad, bad, 0.0
        if M > 1:
            x[1] = 0.0
        want, want_s, _ = call(capi, monkeypatch, "0", x, w, ws)
        got, got_s, _ = call(capi, monkeypatch, "1", x, w, ws)
        assert torch.equal(got, want) and torch.equal(got_s, want_s), (M, bad)
    capi.lib.b200dnn_clear_caches()


def test_sources_that_stay_with_the_separate_kernel(capi, monkeypatch):
    """Rows that do not start on 16 bytes, and results that lie over the source."""
    import torch
    torch.manual_seed(0)
    w, ws = weights(torch, 256, 64)
    pool = torch.randn(4 * 264 + 8, device="cuda").bfloat16()
    call(capi, monkeypatch, "0", pool[:4 * 256].view(4, 256), w, ws)          # (packs the weight)
    for x in (pool[1:1 + 4 * 256].view(4, 256), pool[:4 * 257].view(4, 257)):
        a, _, n0 = call(capi, monkeypatch, "0", x, w, ws, K=256)
        b, _, n1 = call(capi, monkeypatch, "1", x, w, ws, K=256)
        assert n0 == n1 and torch.equal(a, b)
    x = pool[:4 * 256].view(4, 256)
    want, _, _ = call(capi, monkeypatch, "0", x.clone(), w, ws)
    over = x.view(-1).view(torch.float32)[:4 * 64].view(4, 64)              # the first 1 KiB of the source
    got, _, _ = call(capi, monkeypatch, "1", x, w, ws, out=over)
    assert torch.equal(got, want)
    capi.lib.b200dnn_clear_caches()

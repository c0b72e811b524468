"""The bounded waits of the few-row GEMM and of both attention kernels: with the producers' copies switched off every wait runs out after
about a second, the kernel leaves with a status that b200dnn_stream_status reports, and the next call on the same context is correct."""
import ctypes as C

import pytest

from test_matmul_gpu import capi  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["int8 few rows", "bf16 few rows, split", "sdpa prompt", "sdpa prompt, mask", "sdpa few queries", "sdpa few queries, split"])
def test_waits_run_out(capi, monkeypatch, kind):
    import torch
    st = torch.cuda.current_stream().cuda_stream
    BF16 = capi.DT["bf16"]
    mask = None
    if "sdpa" in kind:
        S, KV = (3 if "few" in kind else 200), (2000 if "split" in kind else 100)
        q, k, v, o = (torch.randn(1, 2, n, 64, device="cuda").bfloat16() for n in (S, KV, KV, S))
        d = capi.SdpaDesc()
        d.batch, d.num_heads, d.seq_len, d.kv_seq_len, d.head_dim = 1, 2, S, KV, 64
        for name, x in (("q_stride", q), ("k_stride", k), ("v_stride", v), ("o_stride", o)):
            setattr(d, name, (C.c_int64 * 4)(*x.stride()))
        d.qkv_dt = d.out_dt = BF16
        if "mask" in kind:
            mask = torch.randn(S, KV, device="cuda")
            d.mask_ndims, d.mask_dt, d.attn_mask = 2, capi.DT["f32"], mask.data_ptr()
            d.mask_sizes, d.mask_strides = (C.c_int64 * 4)(S, KV, 0, 0), (C.c_int64 * 4)(KV, 1, 0, 0)
        d.query, d.key, d.value, d.output = (x.data_ptr() for x in (q, k, v, o))
        call = lambda: capi.lib.b200dnn_sdpa(C.byref(d), st)  # noqa: E731
    else:
        M, K, N = (20, 512, 300) if "int8" in kind else (8, 4096, 300)
        if "int8" in kind:
            x, w = (torch.randint(-128, 128, s, dtype=torch.int8, device="cuda") for s in ((M, K), (K, N)))
            o = torch.zeros(M, N, dtype=torch.int32, device="cuda")
            d = capi.make_matmul(M, N, K, x, w, o, src_dt=capi.DT["s8"], dst_dt=capi.DT["s32"])
        else:
            x, w, o = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(K, N, device="cuda").bfloat16(), torch.zeros(M, N, device="cuda")
            d = capi.make_matmul(M, N, K, x, w, o, src_dt=BF16, wei_dt=BF16, dst_dt=capi.DT["f32"])
        call = lambda: capi.matmul(d, st)  # noqa: E731
    capi.check(call())
    assert capi.lib.b200dnn_stream_status(st) == capi.SUCCESS, capi.last_error()
    ref = o.clone()
    monkeypatch.setenv("B200DNN_TEST_NO_LOADS", "1")
    assert call() == capi.SUCCESS                       # device pointers: the call only enqueues
    assert capi.lib.b200dnn_stream_status(st) == capi.FAILURE
    assert "gave up waiting" in capi.last_error()
    monkeypatch.delenv("B200DNN_TEST_NO_LOADS")
    o.zero_()
    torch.cuda.synchronize()
    capi.check(call())
    assert capi.lib.b200dnn_stream_status(st) == capi.SUCCESS, capi.last_error()
    assert torch.equal(o, ref)
    capi.lib.b200dnn_clear_caches()

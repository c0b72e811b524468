"""A host thread whose first CUDA call is one of the library's, with device buffers throughout: nothing has made a context current there."""
import ctypes as C
import threading

import pytest

from test_matmul_gpu import capi  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["bf16 few rows", "bf16 tile", "int8 few rows", "int8 tile", "sdpa few queries", "sdpa prompt", "norm"])
def test_first_call_of_a_thread(capi, kind):
    import torch
    st = torch.cuda.current_stream().cuda_stream
    BF16 = capi.DT["bf16"]
    M = 200 if "tile" in kind else 20
    if "sdpa" in kind:
        S = 3 if "few" in kind else 40
        q, k, v, o = (torch.randn(1, 2, n, 64, device="cuda").bfloat16() for n in (S, 200, 200, S))
        d = capi.SdpaDesc()
        d.batch, d.num_heads, d.seq_len, d.kv_seq_len, d.head_dim = 1, 2, S, 200, 64
        for name, x in (("q_stride", q), ("k_stride", k), ("v_stride", v), ("o_stride", o)):
            setattr(d, name, (C.c_int64 * 4)(*x.stride()))
        d.qkv_dt = d.out_dt = BF16
        d.query, d.key, d.value, d.output = (x.data_ptr() for x in (q, k, v, o))
        call = lambda: capi.lib.b200dnn_sdpa(C.byref(d), st)  # noqa: E731
    elif kind == "norm":
        x, o, g = torch.randn(8, 512, device="cuda").bfloat16(), torch.empty(8, 512, device="cuda", dtype=torch.bfloat16), torch.ones(512, device="cuda")
        d = capi.NormDesc()
        d.norm_type, d.batch, d.norm_size, d.epsilon, d.use_scale = capi.NORM["rms_norm"], 8, 512, 1e-6, 1
        d.src_dt = d.dst_dt = BF16
        d.gamma_dt = capi.DT["f32"]
        d.input, d.output, d.gamma = x.data_ptr(), o.data_ptr(), g.data_ptr()
        call = lambda: capi.lib.b200dnn_normalization(C.byref(d), st)  # noqa: E731
    else:
        K, N = 256, 128
        o = torch.empty(M, N, device="cuda", dtype=torch.bfloat16 if "bf16" in kind else torch.int32)
        if "bf16" in kind:
            x, w = torch.randn(M, K, device="cuda").bfloat16(), torch.randn(K, N, device="cuda").bfloat16()
            d = capi.make_matmul(M, N, K, x, w, o, src_dt=BF16, wei_dt=BF16, dst_dt=BF16)
        else:
            x, w = (torch.randint(-128, 128, s, dtype=torch.int8, device="cuda") for s in ((M, K), (K, N)))
            d = capi.make_matmul(M, N, K, x, w, o, src_dt=capi.DT["s8"], dst_dt=capi.DT["s32"])
        call = lambda: capi.matmul(d, st)  # noqa: E731
    capi.check(call())                              # here: weights are packed, the stream's context exists
    torch.cuda.synchronize()
    ref = o.clone()
    o.zero_()
    torch.cuda.synchronize()
    rc = []
    t = threading.Thread(target=lambda: rc.append((call(), capi.last_error())))
    t.start()
    t.join()
    torch.cuda.synchronize()
    assert rc[0][0] == capi.SUCCESS, rc[0][1]
    assert torch.equal(ref, o)
    capi.lib.b200dnn_clear_caches()

"""Overlapped launches (programmatic dependent launch): the switch that turns them off, seen in the edges of a captured graph."""
import ctypes as C

import pytest

from test_matmul_gpu import capi  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


def calls(capi, torch):
    """One descriptor per kind of overlapped launch, with what it points to."""
    keep = []

    def t(*shape, dtype=torch.bfloat16):
        x = (torch.randn(*shape, device="cuda") if dtype.is_floating_point else torch.randint(-8, 9, shape, device="cuda")).to(dtype)
        keep.append(x)
        return x

    def sdpa(S):
        q, k, v, o = t(1, 2, S, 64), t(1, 2, 200, 64), t(1, 2, 200, 64), t(1, 2, S, 64)
        d = capi.SdpaDesc()
        d.batch, d.num_heads, d.seq_len, d.kv_seq_len, d.head_dim = 1, 2, S, 200, 64
        for name, x in (("q_stride", q), ("k_stride", k), ("v_stride", v), ("o_stride", o)):
            setattr(d, name, (C.c_int64 * 4)(*x.stride()))
        d.qkv_dt = d.out_dt = capi.DT["bf16"]
        d.query, d.key, d.value, d.output = (x.data_ptr() for x in (q, k, v, o))
        return lambda st: capi.lib.b200dnn_sdpa(C.byref(d), st)

    def norm():
        x, y, g = t(8, 512), t(8, 512), t(512, dtype=torch.float32)
        d = capi.NormDesc()
        d.norm_type, d.batch, d.norm_size, d.epsilon, d.use_scale = capi.NORM["rms_norm"], 8, 512, 1e-6, 1
        d.src_dt = d.dst_dt = capi.DT["bf16"]
        d.gamma_dt = capi.DT["f32"]
        d.input, d.output, d.gamma = x.data_ptr(), y.data_ptr(), g.data_ptr()
        return lambda st: capi.lib.b200dnn_normalization(C.byref(d), st)

    def matmul(M, dyn):
        x, w, y = t(M, 256), t(256, 128, dtype=torch.int8 if dyn else torch.bfloat16), t(M, 128)
        ws = torch.rand(128, device="cuda")
        keep.append(ws)
        kw = dict(dynamic_quant=True, src_scale=capi.quant(None, M, capi.DT["f32"]), wei_scale=ws) if dyn else dict(wei_dt=capi.DT["bf16"])
        d = capi.make_matmul(M, 128, 256, x, w, y, src_dt=capi.DT["bf16"], dst_dt=capi.DT["bf16"], **kw)
        return lambda st: capi.matmul(d, st)

    return {"sdpa few queries": sdpa(3), "sdpa prompt": sdpa(40), "norm": norm(), "bf16 few rows": matmul(8, False), "bf16 tile": matmul(200, False),
            "int8 decode, dynamic": matmul(2, True), "int8 few rows, dynamic": matmul(20, True)}, keep


@pytest.mark.parametrize("on", [1, 0])
def test_switch_covers_every_overlapped_launch(capi, monkeypatch, on):
    import torch
    rt = C.CDLL("libcudart.so.12")
    monkeypatch.setenv("B200DNN_PDL", str(on))
    kinds, keep = calls(capi, torch)
    for name, call in kinds.items():
        for _ in range(2):
            capi.check(call(torch.cuda.current_stream().cuda_stream))
            torch.cuda.synchronize()            # weights packed and seen complete
        g = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(g):
            st = torch.cuda.current_stream().cuda_stream
            for _ in range(3):
                capi.check(call(st))
        raw, n = C.c_void_p(g.raw_cuda_graph()), C.c_size_t(0)
        assert rt.cudaGraphGetEdges_v2(raw, None, None, None, C.byref(n)) == 0 and n.value >= 2
        ends, data = [(C.c_void_p * n.value)() for _ in range(2)], (C.c_uint8 * (8 * n.value))()      # cudaGraphEdgeData: ports, then the type
        assert rt.cudaGraphGetEdges_v2(raw, ends[0], ends[1], data, C.byref(n)) == 0
        overlapped = sum(data[8 * i + 2] == 1 for i in range(n.value))                               # cudaGraphDependencyTypeProgrammatic
        assert (overlapped > 0) == bool(on), (name, overlapped, n.value)
        torch.cuda.synchronize()
    capi.lib.b200dnn_clear_caches()

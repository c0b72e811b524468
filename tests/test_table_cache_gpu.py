"""The tables that MoE calls keep on the device are bounded in number: a call that finds the bound reached keeps those it has already asked for.  More layers than fit, as prompts and
as decode batches in turn (each form has tensor maps of its own), against the same calls with nothing kept."""
import pytest

from test_matmul_gpu import capi  # noqa: F401  (fixture)
from test_moe_few_gpu import layer

pytestmark = pytest.mark.gpu


def test_more_layers_than_tables(capi):
    import torch
    st = torch.cuda.current_stream().cuda_stream
    layers = [layer(capi, torch, 80, 64, 32, 2, 0, 1, seed=i) for i in range(72)]

    def run(i, T):
        _, out, keep = layers[i]
        x, logits, ex = keep[-3:]
        out.zero_()
        capi.check(capi.lib.b200dnn_moe_layer(x.data_ptr(), 64, logits.data_ptr(), T, 2, 0, 1, ex, 64, 32, 64, 0, capi.ACT["silu_and_mul"], out.data_ptr(), 64, st))
        assert capi.lib.b200dnn_stream_status(st) == capi.SUCCESS, capi.last_error()
        return out.clone()

    capi.lib.b200dnn_clear_caches()
    want = {}
    for i in range(len(layers)):
        for T in (80, 8):
            want[i, T] = run(i, T)
            assert want[i, T][:T].abs().max() > 0
        if i % 16 == 15:
            capi.lib.b200dnn_clear_caches()
    capi.lib.b200dnn_clear_caches()
    for T in (80, 8, 80):
        for i in range(len(layers)):
            assert torch.equal(run(i, T), want[i, T]), (i, T)
    for i in range(len(layers)):
        for T in (8, 80):
            assert torch.equal(run(i, T), want[i, T]), (i, T)
    capi.lib.b200dnn_clear_caches()

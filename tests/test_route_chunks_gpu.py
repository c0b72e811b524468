"""The two-launch routing of MoE layers of more than 64 tokens against the launches it stands for: the same layer, bit for bit, at the edges of its chunks of tokens, of its
1024 slots a pass and of its 256 experts, with ties, skew and logits that are all NaN beside others."""
import pytest

from test_matmul_gpu import capi  # noqa: F401  (fixture)
from test_moe_few_gpu import layer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,E,S,topk", [(65, 4, 0, 2), (96, 8, 1, 1), (1000, 255, 1, 16), (1025, 256, 0, 3), (8192, 60, 2, 4), (8193, 33, 0, 6), (20001, 7, 1, 7)])
@pytest.mark.parametrize("skew", [False, True])
def test_same_layer(capi, monkeypatch, T, E, S, topk, skew):
    import torch
    call, out, keep = layer(capi, torch, T, 64, 32, E, S, topk, skew=skew, seed=T)
    logits = keep[-2]
    logits[:, : E // 2] = logits[:, : E // 2].round()       # ties
    torch.cuda.synchronize()
    got = {}
    for chunks in ("0", "1"):
        monkeypatch.setenv("B200DNN_ROUTE_CHUNKS", chunks)
        out.zero_()
        capi.check(call())
        assert capi.lib.b200dnn_stream_status(torch.cuda.current_stream().cuda_stream) == capi.SUCCESS, capi.last_error()
        got[chunks] = out.clone()
    assert got["0"].abs().max() > 0 and torch.equal(got["0"], got["1"])
    capi.lib.b200dnn_clear_caches()


def test_tokens_without_a_choice(capi):
    """Rows of NaN logits reach no index outside the tables; the other tokens' results are what they are without them."""
    import torch
    call, out, keep = layer(capi, torch, 300, 64, 32, 8, 0, 1)
    capi.check(call())
    torch.cuda.synchronize()
    want = out.clone()
    keep[-2][7::50] = float("nan")
    torch.cuda.synchronize()
    capi.check(call())
    assert capi.lib.b200dnn_stream_status(torch.cuda.current_stream().cuda_stream) == capi.SUCCESS, capi.last_error()
    clean = torch.ones(300, dtype=torch.bool, device="cuda")
    clean[7::50] = False
    assert torch.equal(out[clean], want[clean])
    capi.lib.b200dnn_clear_caches()

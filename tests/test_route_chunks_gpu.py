"""The two-launch routing of MoE layers of more than 64 tokens against the launches it stands for: the same layer, bit for bit, at the edges of its chunks of tokens, of its
1024 slots a pass and of its 256 experts, with ties, skew and logits without a softmax beside others, in every form of the routing."""
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


@pytest.mark.parametrize("E", [8, 64, 100, 250, 300])
def test_routing_tables_without_a_choice(capi, E):
    """b200dnn_moe_route, and the general launches of a layer (more than 256 groups), with logits that have no softmax: experts and rows inside their tables, every row taken
    once, the other tokens as without them."""
    import torch
    torch.manual_seed(E)
    T, k = 100, 4
    logits = torch.randn(T, E, device="cuda")
    st = torch.cuda.current_stream().cuda_stream

    def route():
        ids, rows = (torch.full((T, k), -1, dtype=torch.int32, device="cuda") for _ in range(2))
        w, counts = torch.zeros(T, k, device="cuda"), torch.zeros(E, dtype=torch.int32, device="cuda")
        capi.check(capi.lib.b200dnn_moe_route(logits.data_ptr(), T, E, k, 1, ids.data_ptr(), w.data_ptr(), counts.data_ptr(), rows.data_ptr(), st))
        torch.cuda.synchronize()
        return ids, w, counts, rows

    want = route()
    bad = torch.zeros(T, dtype=torch.bool, device="cuda")
    bad[::7] = True
    logits[::7] = float("nan")
    logits[::14] = -float("inf")
    logits[7, 1:] = 0.0
    logits[7, 0] = float("inf")
    ids, w, counts, rows = route()
    assert int(ids.min()) >= 0 and int(ids.max()) < E and int(counts.sum()) == T * k
    assert torch.equal(rows.flatten().sort().values, torch.arange(T * k, dtype=torch.int32, device="cuda"))
    assert torch.equal(ids[~bad], want[0][~bad]) and torch.equal(w[~bad], want[1][~bad])
    call, out, keep = layer(capi, torch, T, 64, 32, E, 257 - min(E, 256), k)
    capi.check(call())
    torch.cuda.synchronize()
    clean = out.clone()
    keep[-2][::7] = float("nan")
    torch.cuda.synchronize()
    capi.check(call())
    assert capi.lib.b200dnn_stream_status(st) == capi.SUCCESS, capi.last_error()
    assert torch.equal(out[~bad], clean[~bad])
    capi.lib.b200dnn_clear_caches()

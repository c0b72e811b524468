"""The grouped GEMM for a few rows per expert (MoE layers of up to 64 tokens) against the tile kernel: the same layer, bit for bit (INT8 sums are exact and the epilogue's
operations the same; bf16 within the order of the f32 sums), at the edges of its row counts, of its 128-column tiles and of the routing, with tokens that name no expert, and its
bounded waits."""
import numpy as np
import pytest

from test_matmul_gpu import capi  # noqa: F401  (fixture)

pytestmark = pytest.mark.gpu


def layer(capi, torch, T, H, I, E, S, topk, act="silu_and_mul", bias=None, wdt="s8", skew=False, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    ex, keep = (capi.MoeExpert * (E + S))(), []
    for e in range(E + S):
        ex[e].ldb13, ex[e].ldb2 = 2 * I, H
        if wdt == "s8":
            w13, w2 = (torch.randint(-127, 128, s, dtype=torch.int8, device="cuda", generator=g) for s in ((H, 2 * I), (I, H)))
            s13, s2 = (torch.rand(n, device="cuda", generator=g) * 1e-3 + 1e-4 for n in (2 * I, H))
            ex[e].w13_scale, ex[e].w2_scale = s13.data_ptr(), s2.data_ptr()
            keep += [s13, s2]
        else:
            w13, w2 = (torch.randn(*s, device="cuda", generator=g).mul_(0.05).bfloat16() for s in ((H, 2 * I), (I, H)))
            ex[e].wei_dt = capi.DT["bf16"]
        ex[e].w13, ex[e].w2 = w13.data_ptr(), w2.data_ptr()
        keep += [w13, w2]
        if bias and e % 2 == 0:                          # an expert may have none
            b13, b2 = (torch.randn(n, device="cuda", generator=g).to(torch.float32 if bias == "f32" else torch.bfloat16) for n in (2 * I, H))
            ex[e].bias13, ex[e].bias13_dt, ex[e].bias2, ex[e].bias2_dt = b13.data_ptr(), capi.DT[bias], b2.data_ptr(), capi.DT[bias]
            keep += [b13, b2]
    x = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    logits = torch.randn(T, E, device="cuda", generator=g)
    if skew:
        logits[:, E - 1] += 50.0                         # every token asks for the last expert
    out = torch.zeros(T, H, dtype=torch.bfloat16, device="cuda")
    keep += [x, logits, ex]
    st = torch.cuda.current_stream().cuda_stream
    return (lambda: capi.lib.b200dnn_moe_layer(x.data_ptr(), H, logits.data_ptr(), T, E, S, topk, ex, H, I, H, 0, capi.ACT[act], out.data_ptr(), H, st)), out, keep


@pytest.mark.parametrize("T,H,I,E,S,topk,skew", [(1, 128, 32, 4, 0, 1, False), (16, 256, 96, 8, 1, 2, True), (17, 144, 160, 3, 0, 2, False), (33, 520, 64, 40, 2, 5, False),
                                                 (48, 200, 1056, 5, 0, 1, True), (64, 1030, 352, 70, 1, 8, False), (3, 4096, 32, 8, 0, 2, False)])
@pytest.mark.parametrize("kind", ["s8", "s8 bias f32", "s8 bias bf16 gelu", "s8 oai", "bf16", "bf16 bias f32"])
def test_against_the_tile_kernel(capi, monkeypatch, T, H, I, E, S, topk, skew, kind):
    import torch
    act = "gelu_and_mul" if "gelu" in kind else "swiglu_oai_mul" if "oai" in kind else "silu_and_mul"
    call, out, keep = layer(capi, torch, T, H, I, E, S, topk, act, "bf16" if "bias bf16" in kind else "f32" if "bias" in kind else None, kind.split()[0], skew, T + H)
    monkeypatch.setenv("B200DNN_MOE_FEW", "0")
    capi.check(call())
    assert capi.lib.b200dnn_stream_status(torch.cuda.current_stream().cuda_stream) == capi.SUCCESS, capi.last_error()
    want = out.clone()
    out.zero_()
    monkeypatch.setenv("B200DNN_MOE_FEW", "64")
    capi.check(call())
    assert capi.lib.b200dnn_stream_status(torch.cuda.current_stream().cuda_stream) == capi.SUCCESS, capi.last_error()
    assert want.abs().max() > 0
    if kind.startswith("s8"):
        assert torch.equal(out, want)
    else:                                                # two products of f32 sums with a rounding to bf16 between and behind them
        d = (out.float() - want.float()).abs()
        assert (d <= 2.0 ** -7 * want.float().abs() + 2.0 ** -7 * want.float().abs().max()).all()
    capi.lib.b200dnn_clear_caches()


@pytest.mark.parametrize("T", [9, 16, 64])
@pytest.mark.parametrize("topk,E,S", [(2, 4, 0), (8, 11, 1), (2, 300, 0)])
@pytest.mark.parametrize("wdt", ["s8", "bf16"])
def test_tokens_without_a_choice(capi, monkeypatch, T, topk, E, S, wdt):
    """Logits that are NaN or minus infinity throughout, or infinite once, name no expert, and all choices of such tokens may fall on one expert: more rows than there are
    tokens.  The other tokens keep their results, and (s8) all of them are those of the tile kernel; a few such tokens, and all of them."""
    import torch
    call, out, keep = layer(capi, torch, T, 136, 96, E, S, topk, wdt=wdt, skew=True, seed=T + topk)
    logits = keep[-2]
    st = torch.cuda.current_stream().cuda_stream

    def run(few):
        monkeypatch.setenv("B200DNN_MOE_FEW", few)
        out.zero_()
        capi.check(call())
        assert capi.lib.b200dnn_stream_status(st) == capi.SUCCESS, capi.last_error()
        return out.clone()

    want = run("64")
    assert want.abs().max() > 0
    inf = float("inf")
    for rows in (slice(1, None, 3), slice(None)):
        bad = torch.zeros(T, dtype=torch.bool, device="cuda")
        bad[rows] = True
        logits[rows] = -inf
        logits[rows][::3, E // 2] = float("nan")
        logits[rows][1::3] = float("nan")
        logits[rows][2::3, 0] = inf
        torch.cuda.synchronize()
        got, tile = run("64"), run("0")
        assert torch.equal(got[~bad], want[~bad])
        if wdt == "s8":
            assert torch.equal(got.view(torch.int16), tile.view(torch.int16))
    capi.lib.b200dnn_clear_caches()


def test_waits_run_out(capi, monkeypatch):
    import torch
    st = torch.cuda.current_stream().cuda_stream
    call, out, keep = layer(capi, torch, 9, 256, 96, 4, 0, 2)
    capi.check(call())
    assert capi.lib.b200dnn_stream_status(st) == capi.SUCCESS, capi.last_error()
    ref = out.clone()
    monkeypatch.setenv("B200DNN_TEST_NO_LOADS", "1")
    assert call() == capi.SUCCESS
    assert capi.lib.b200dnn_stream_status(st) == capi.FAILURE and "gave up waiting" in capi.last_error()
    monkeypatch.delenv("B200DNN_TEST_NO_LOADS")
    out.zero_()
    capi.check(call())
    assert capi.lib.b200dnn_stream_status(st) == capi.SUCCESS, capi.last_error()
    assert torch.equal(out, ref)
    capi.lib.b200dnn_clear_caches()

"""What a user of this library has it do, as cases that can be timed: the calls of a quantised decoder layer (projections in
INT8, 4-bit and bf16, attention, normalisation, mixture-of-experts blocks) through the C ABI, from one token to thousands.

  listed()          the fixed cases
  draw(rng)         one more case of the same ranges
  prepare(case, s)  inputs, weights, descriptors of one case, made on the GPU from the seed s
  run(state)        one call of the library's entry point; returns the outputs
  work(case)        bytes and operations that no implementation can do without
  tolerance(case)   how far another correct implementation's outputs may lie
"""
import ctypes as C
import math

import torch

from zendnn_b200 import capi

BF16, F32 = capi.DT["bf16"], capi.DT["f32"]


def listed():
    return [
        # ---- W8A8 projections (b200dnn_matmul, weights prepacked once at load time)
        # one token of one user through a square projection, activations quantised by the caller: the smallest call
        dict(name="w8a8_decode_1", kind="w8a8", M=1, K=4096, N=4096, src="s8", bias=False, act="none", out="bf16"),
        # a decode batch through a down projection, bf16 activations quantised inside the call
        dict(name="w8a8_decode_16_dyn", kind="w8a8", M=16, K=11008, N=4096, src="dyn", bias=False, act="none", out="bf16"),
        # a recommender- or vision-style layer: no size is a multiple of anything, u8 activations with a zero point, f32 out
        dict(name="w8a8_ragged_u8", kind="w8a8", M=500, K=1999, N=3001, src="u8", bias=True, act="relu", out="f32"),
        # a prompt through an up projection: dynamic quantisation, bias and GELU in the call
        dict(name="w8a8_prefill", kind="w8a8", M=2048, K=4096, N=14336, src="dyn", bias=True, act="gelu_tanh", out="bf16"),
        # ---- 4-bit weights (W4A8, groups of 128): a few users' tokens through an up projection
        dict(name="w4a8_decode_4", kind="w4a8", M=4, K=4096, N=11008, gs=128),
        # ---- the default data type, not quantised: a decode batch through an up projection
        dict(name="bf16_decode_8", kind="bf16", M=8, K=4096, N=11008, bias=False, act="none", out="bf16"),
        # ---- whole MoE layers (b200dnn_moe_layer), W8A8 experts
        # a prompt batch, eight large experts
        dict(name="moe_prefill_large_experts", kind="moe", T=4096, H=4096, I=14336, E=8, topk=2, shared=0, zipf=False, wdt="s8"),
        # a large batch over many small experts with skewed routing and shared experts
        dict(name="moe_prefill_fine_grained", kind="moe", T=16384, H=2048, I=1408, E=64, topk=6, shared=2, zipf=True, wdt="s8"),
        # a decode batch over the fine-grained experts: a few rows for each of them
        dict(name="moe_decode_fine_grained", kind="moe", T=32, H=2048, I=1408, E=64, topk=6, shared=2, zipf=True, wdt="s8"),
        # ---- attention (b200dnn_sdpa)
        # a prompt, causal
        dict(name="sdpa_prefill_causal", kind="sdpa", B=1, H=32, S=2048, KV=2048, D=128, mask="causal", layout="bhsd"),
        # a decode batch against its key/value cache
        dict(name="sdpa_decode", kind="sdpa", B=8, H=32, S=1, KV=3000, D=128, mask="none", layout="bhsd"),
        # ---- the normalisation in front of a W8A8 projection: residual add, RMSNorm, s8 rows out (b200dnn_normalization)
        dict(name="norm_add_rms_quant", kind="norm", rows=4096, cols=4096, form="fused_add_rms", quant=True),
    ]


# ------------------------------------------------------------------------------------------------ ranges
def _log(rng, lo, hi, step=1):
    """Log-uniform over [lo, hi], a multiple of step."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def _width(rng, lo, hi):
    """A layer width: mostly a multiple of 64 as models have it, sometimes any number (up to 8192)."""
    return _log(rng, lo, hi, 64) if rng.random() < 0.75 else _log(rng, lo, min(hi, 8192))


def _draw(rng):
    kind = rng.choice(["w8a8", "w8a8", "w8a8", "w4a8", "bf16", "bf16", "moe", "moe", "sdpa", "sdpa", "norm"])
    if kind == "w8a8":
        return dict(kind=kind, M=_log(rng, 1, 8192), K=_width(rng, 512, 14336), N=_width(rng, 512, 14336),
                    src=rng.choice(["s8", "u8", "dyn", "dyn"]), bias=rng.random() < 0.5,
                    act=rng.choice(["none", "none", "relu", "gelu_tanh", "swish"]), out=rng.choice(["bf16", "bf16", "f32"]))
    if kind == "w4a8":
        gs = rng.choice([32, 64, 128, 128])
        return dict(kind=kind, M=_log(rng, 1, 512), K=_log(rng, 1024, 14336, gs), N=_log(rng, 512, 14336, 8), gs=gs)
    if kind == "bf16":
        return dict(kind=kind, M=_log(rng, 1, 8192), K=_width(rng, 512, 14336), N=_width(rng, 512, 14336), bias=rng.random() < 0.5,
                    act=rng.choice(["none", "none", "relu", "gelu_tanh", "swish"]), out=rng.choice(["bf16", "bf16", "f32"]))
    if kind == "moe":
        E = rng.choice([8, 16, 32, 60, 64])
        return dict(kind=kind, T=_log(rng, 1, 16384), H=_log(rng, 1024, 4096, 64), I=_log(rng, 512, 14336, 32), E=E,
                    topk=rng.randint(1, 2) if E == 8 else rng.randint(2, 8), shared=rng.choice([0, 0, 1, 2]), zipf=rng.random() < 0.5,
                    wdt=rng.choice(["s8", "s8", "s8", "bf16"]))
    if kind == "sdpa":
        D, layout = rng.choice([64, 128, 128, 80]), rng.choice(["bhsd", "bshd"])
        if rng.random() < 0.5:      # a prompt
            S = _log(rng, 32, 4096)
            return dict(kind=kind, B=_log(rng, 1, 8), H=rng.choice([8, 12, 32, 40]), S=S, KV=S, D=D,
                        mask=rng.choice(["causal", "causal", "none", "pad"]), layout=layout)
        return dict(kind=kind, B=_log(rng, 1, 32), H=rng.choice([8, 12, 32, 40]), S=rng.choice([1, 1, 1, 4]), KV=_log(rng, 64, 8192), D=D,
                    mask=rng.choice(["none", "pad"]), layout=layout)
    return dict(kind=kind, rows=_log(rng, 1, 16384), cols=_width(rng, 512, 12288), form=rng.choice(["rms", "fused_add_rms", "fused_add_rms", "layer"]),
                quant=rng.random() < 0.5)


def _cost(case):
    w = work(case)
    return w["flops"] / 1e15 + w["bytes"] / 6e12


def draw(rng):
    """Sizes over the whole range, no case dearer than the dearest listed one, its weights no larger than theirs."""
    most = max(_cost(c) for c in listed())
    most_bytes = max(work(c)["bytes"] for c in listed())
    while True:
        case = _draw(rng)
        # the experts are all resident, whether a token meets them or not; inputs have to be made in a moment
        held = 3 * case["H"] * case["I"] * (case["E"] + case["shared"]) * (2 if case["wdt"] == "bf16" else 1) if case["kind"] == "moe" else 0
        if _cost(case) <= most and work(case)["bytes"] <= most_bytes and held <= most_bytes:
            return case


# ------------------------------------------------------------------------------------------------ inputs
def _randn(g, *shape, scale=1.0):
    return torch.randn(*shape, generator=g, device="cuda").mul_(scale).to(torch.bfloat16)


def _s8_weight(g, K, N):
    """[K, N] s8 from N(0, 0.02), one f32 scale per output channel."""
    w = torch.randn(K, N, generator=g, device="cuda").mul_(0.02)
    s = w.abs().amax(0).clamp_(min=1e-10) / 127.0
    return w.div_(s).round_().to(torch.int8), s


def _postops(case):
    return [] if case["act"] == "none" else [case["act"]]


def _matmul(case, g, st):
    M, K, N = case["M"], case["K"], case["N"]
    out_dt = BF16 if case["out"] == "bf16" else F32
    dst = torch.empty(M, N, dtype=torch.bfloat16 if case["out"] == "bf16" else torch.float32, device="cuda")
    bias = torch.randn(N, generator=g, device="cuda") if case["bias"] else None
    kw = dict(dst_dt=out_dt, bias=bias, postops=_postops(case), flags=capi.FLAG_STABLE_WEIGHTS)
    keep = [dst, bias]
    if case["kind"] == "bf16":
        src, w = _randn(g, M, K), _randn(g, K, N, scale=0.02)
        keep += [src, w]
        return capi.make_matmul(M, N, K, src, w, dst, src_dt=BF16, wei_dt=BF16, **kw), keep, dst
    # INT8: the float weight is quantised per channel and laid out by the library, once
    w = _randn(g, K, N, scale=0.02)
    packed = torch.empty(capi.lib.b200dnn_prepack_size(K, N, 0), dtype=torch.uint8, device="cuda")
    ws = torch.empty(N, dtype=torch.float32, device="cuda")
    capi.check(capi.lib.b200dnn_quant_prepack(w.data_ptr(), BF16, K, N, N, 0, 0, packed.data_ptr(), ws.data_ptr(), st))
    keep += [packed, ws]
    if case["src"] == "u8":
        src = torch.randint(0, 256, (M, K), generator=g, dtype=torch.uint8, device="cuda")
        scale = torch.full((1,), 0.02, device="cuda")
        zp = torch.full((1,), 128, dtype=torch.int32, device="cuda")
        keep += [src, scale, zp]
        kw.update(src_dt=capi.DT["u8"], src_scale=scale, src_zp=zp)
    elif case["src"] == "s8":
        x = torch.randn(M, K, generator=g, device="cuda")
        scale = x.abs().amax(1) / 127.0
        src = (x / scale[:, None]).round_().to(torch.int8)
        keep += [src, scale]
        kw.update(src_dt=capi.DT["s8"], src_scale=scale)
    else:
        src = _randn(g, M, K)
        keep += [src]
        kw.update(src_dt=BF16, dynamic_quant=True, src_scale=capi.quant(None, M, F32))
    return capi.make_matmul(M, N, K, src, packed, dst, wei_format="r", wei_scale=ws, **kw), keep, dst


def _w4a8(case, g):
    M, K, N, G = case["M"], case["K"], case["N"], case["K"] // case["gs"]
    src = _randn(g, M, K)
    w = torch.randint(0, 256, (K * N // 2,), generator=g, dtype=torch.uint8, device="cuda")     # two codes per byte
    ws = torch.rand(G, N, generator=g, device="cuda") * 4e-3 + 1e-3
    dst = torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    d = capi.make_matmul(M, N, K, src, w, dst, src_dt=BF16, wei_dt=capi.DT["s4"], dst_dt=BF16, dynamic_quant=True,
                         src_scale=capi.quant(None, M, F32), wei_scale=capi.quant(ws, G * N, F32))
    return d, [src, w, ws, dst], dst


def _moe(case, g, st):
    T, H, I, E, S = case["T"], case["H"], case["I"], case["E"], case["shared"]
    ex, keep = (capi.MoeExpert * (E + S))(), []
    for e in range(E + S):
        ex[e].ldb13, ex[e].ldb2 = 2 * I, H
        if case["wdt"] == "bf16":
            w13, w2 = _randn(g, H, 2 * I, scale=0.02), _randn(g, I, H, scale=0.02)
            ex[e].wei_dt = BF16
            keep.append((w13, w2))
        else:
            (w13, s13), (w2, s2) = _s8_weight(g, H, 2 * I), _s8_weight(g, I, H)
            ex[e].w13_scale, ex[e].w2_scale = s13.data_ptr(), s2.data_ptr()
            keep.append((w13, s13, w2, s2))
        ex[e].w13, ex[e].w2 = w13.data_ptr(), w2.data_ptr()
    x = _randn(g, T, H)
    logits = torch.randn(T, E, generator=g, device="cuda")
    if case["zipf"]:                # some experts are asked for far more often than others
        p = torch.arange(1, E + 1, device="cuda", dtype=torch.float64) ** -1.1
        logits = (logits + torch.log(p / p.sum())[torch.randperm(E, generator=g, device="cuda")].float()).contiguous()
    out = torch.empty(T, H, dtype=torch.bfloat16, device="cuda")
    args = (x.data_ptr(), H, logits.data_ptr(), T, E, S, case["topk"], ex, H, I, H, 0, capi.ACT["silu_and_mul"], out.data_ptr(), H, st)
    return args, [keep, x, logits, out, ex], out


def _sdpa(case, g):
    B, H, S, KV, D = case["B"], case["H"], case["S"], case["KV"], case["D"]
    bshd = case["layout"] == "bshd"

    def tensor(n):                  # [batch, head, seq, dim] or [batch, seq, head, dim] storage, seen as b, h, s, d
        t = _randn(g, B, n, H, D) if bshd else _randn(g, B, H, n, D)
        return t.transpose(1, 2) if bshd else t
    q, k, v = tensor(S), tensor(KV), tensor(KV)
    o = torch.empty((B, S, H, D) if bshd else (B, H, S, D), dtype=torch.bfloat16, device="cuda")
    oh = o.transpose(1, 2) if bshd else o
    d = capi.SdpaDesc()
    d.batch, d.num_heads, d.seq_len, d.kv_seq_len, d.head_dim = B, H, S, KV, D
    for name, t in (("q_stride", q), ("k_stride", k), ("v_stride", v), ("o_stride", oh)):
        setattr(d, name, (C.c_int64 * 4)(*t.stride()))
    d.qkv_dt = d.out_dt = BF16
    d.is_causal = int(case["mask"] == "causal")
    mask = None
    if case["mask"] == "pad":       # sequences of different lengths in one batch: keys past a sequence's end count for nothing
        ends = torch.randint((KV + 1) // 2, KV + 1, (B,), generator=g, device="cuda")
        mask = torch.zeros(B, 1, 1, KV, device="cuda")
        mask.masked_fill_(torch.arange(KV, device="cuda")[None, None, None, :] >= ends[:, None, None, None], -math.inf)
        d.mask_ndims, d.mask_dt, d.attn_mask = 4, F32, mask.data_ptr()
        d.mask_sizes, d.mask_strides = (C.c_int64 * 4)(B, 1, 1, KV), (C.c_int64 * 4)(KV, KV, KV, 1)
    d.query, d.key, d.value, d.output = q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr()
    return d, [q, k, v, mask, o], o


def _norm(case, g):
    R, N = case["rows"], case["cols"]
    x, gamma = _randn(g, R, N), torch.randn(N, generator=g, device="cuda")
    y = torch.empty(R, N, dtype=torch.bfloat16, device="cuda")
    d = capi.NormDesc()
    d.norm_type = capi.NORM[{"rms": "rms_norm", "fused_add_rms": "fused_add_rms_norm", "layer": "layer_norm"}[case["form"]]]
    d.batch, d.norm_size, d.epsilon, d.use_scale = R, N, 1e-6, 1
    d.src_dt = d.dst_dt = BF16
    d.gamma_dt = d.beta_dt = F32
    d.input, d.output, d.gamma = x.data_ptr(), y.data_ptr(), gamma.data_ptr()
    keep, out = [x, gamma, y], [y]
    if case["form"] == "layer":
        beta = torch.randn(N, generator=g, device="cuda")
        d.use_shift, d.beta = 1, beta.data_ptr()
        keep.append(beta)
    if case["form"] == "fused_add_rms":
        res = _randn(g, R, N)
        d.residual = res.data_ptr()
        out.append(res)
    if case["quant"]:               # the rows also leave as s8 codes with a scale each, for the projection behind
        q, s = torch.empty(R, N, dtype=torch.int8, device="cuda"), torch.empty(R, device="cuda")
        d.quant_dst, d.quant_ld, d.quant_scale = q.data_ptr(), N, s.data_ptr()
        out += [q, s]
    return d, keep + out, out


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    st = torch.cuda.current_stream().cuda_stream
    kind = case["kind"]
    # Raw constant weights are packed once and found again by their address.  This program has dropped earlier weights,
    # and the allocator may hand their addresses out again: so it drops the library's packed copies as well.
    capi.check(capi.lib.b200dnn_clear_caches())
    if kind in ("w8a8", "bf16"):
        desc, keep, out = _matmul(case, g, st)
    elif kind == "w4a8":
        desc, keep, out = _w4a8(case, g)
    elif kind == "moe":
        desc, keep, out = _moe(case, g, st)
    elif kind == "sdpa":
        desc, keep, out = _sdpa(case, g)
    else:
        desc, keep, out = _norm(case, g)
    torch.cuda.synchronize()        # the weights are in place before the first call
    return dict(kind=kind, desc=desc, stream=st, keep=keep, out=out)


def run(state):
    kind, desc, st = state["kind"], state["desc"], state["stream"]
    if kind == "moe":
        rc = capi.lib.b200dnn_moe_layer(*desc)
    elif kind == "sdpa":
        rc = capi.lib.b200dnn_sdpa(C.byref(desc), st)
    elif kind == "norm":
        rc = capi.lib.b200dnn_normalization(C.byref(desc), st)
    else:
        rc = capi.matmul(desc, st)
    capi.check(rc)
    return state["out"]


# ------------------------------------------------------------------------------------------------ what it costs, how exact it is
def work(case):
    kind = case["kind"]
    if kind in ("w8a8", "bf16"):
        M, K, N = case["M"], case["K"], case["N"]
        a = 2 if kind == "bf16" or case["src"] == "dyn" else 1
        b = 2 if kind == "bf16" else 1
        per_row = 4 * M if kind == "w8a8" and case["src"] == "s8" else 0
        return dict(bytes=M * K * a + K * N * b + M * N * (2 if case["out"] == "bf16" else 4) + per_row +
                    (4 * N if kind == "w8a8" else 0) + (4 * N if case["bias"] else 0), flops=2 * M * K * N)
    if kind == "w4a8":
        M, K, N = case["M"], case["K"], case["N"]
        return dict(bytes=2 * M * K + K * N // 2 + 4 * (K // case["gs"]) * N + 2 * M * N, flops=2 * M * K * N)
    if kind == "moe":
        T, H, I, S, k = case["T"], case["H"], case["I"], case["shared"], case["topk"]
        # experts that some token meets, on average: a token asks for expert e with probability q[e]
        w = [(e + 1) ** -1.1 if case["zipf"] else 1.0 for e in range(case["E"])]
        hit = sum(1 - (1 - min(1.0, k * p / sum(w))) ** T for p in w) + S
        per = 3 * H * I * (2 if case["wdt"] == "bf16" else 1) + (0 if case["wdt"] == "bf16" else 4 * (2 * I + H))
        return dict(bytes=hit * per + T * (4 * H + 4 * case["E"]), flops=2 * T * (k + S) * 3 * H * I)
    if kind == "sdpa":
        B, H, S, KV, D = case["B"], case["H"], case["S"], case["KV"], case["D"]
        pairs = S * (S + 1) // 2 if case["mask"] == "causal" else S * KV
        return dict(bytes=2 * B * H * D * (2 * S + 2 * KV) + (4 * B * KV if case["mask"] == "pad" else 0), flops=4 * B * H * pairs * D)
    R, N = case["rows"], case["cols"]
    per = 4 + (4 if case["form"] == "fused_add_rms" else 0) + (1 if case["quant"] else 0)
    return dict(bytes=R * N * per + 4 * N + (4 * N if case["form"] == "layer" else 0) + (4 * R if case["quant"] else 0), flops=5 * R * N)


def tolerance(case):
    kind = case["kind"]
    if kind == "w8a8" and case["out"] == "f32":
        # integer sums are exact; what follows is f32, but a token's codes may fall on the other side of a tie
        return dict(rel=1e-3) if case["src"] == "dyn" else dict(rel=1e-5)
    if kind == "bf16" and case["out"] == "f32":
        return dict(rel=1e-4)                       # f32 sums of exact products in another order
    if kind == "norm":
        return dict(rel=5e-3, max=0.02, differ=2e-3)    # bf16 rows within one rounding; codes beside a tie
    if kind == "moe":
        return dict(rel=1e-2, max=0.3)              # two products with a rounding and a quantisation between them
    return dict(rel=1e-2, max=0.1)                  # bf16 results

"""The fused attention kernels behind b200dnn_sdpa at the edges of their tiles and of the rule that chooses between them (few
query rows up to 16: split over the keys in blocks of 128; more: 128- and 256-row query tiles against 128-key blocks), against the
CPU oracle with the tolerance of the BMM form's tests (the kernels keep that form's steps and roundings)."""
import ctypes as C

import numpy as np
import pytest

from test_sdpa_gpu import capi, close, make, run, strides_of  # noqa: F401  (capi: fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,KV", [(1, 1), (1, 129), (16, 128), (17, 127), (8, 1025), (9, 1100), (127, 129), (128, 128), (129, 257), (257, 300), (300, 40)])
@pytest.mark.parametrize("D", [8, 72, 128])
@pytest.mark.parametrize("causal", [False, True])
def test_tile_edges(capi, oracle, S, KV, D, causal):
    rng = np.random.default_rng(S * 31 + KV + D)
    q, k, v = make(oracle, rng, 1, 3, S, KV, D)
    st, out = run(capi, q, k, v, causal=causal)
    assert st == capi.SUCCESS, capi.last_error()
    close(oracle, out, oracle.sdpa(q, k, v, causal=causal), v, (S, KV, D, causal))


@pytest.mark.parametrize("S", [3, 200])
def test_row_dependent_masks_and_rows_without_keys(capi, oracle, S):
    """f32 and bf16 masks that differ per query row (16-byte aligned rows and not), with rows that see no key."""
    for KV, bf16 in ((260, False), (263, False), (264, True), (261, True)):
        rng = np.random.default_rng(KV)
        q, k, v = make(oracle, rng, 2, 2, S, KV, 64)
        m = rng.standard_normal((2, 1, S, KV)).astype(np.float32)
        m[1, 0, S // 2] = -np.inf
        mask = oracle.f32_to_bf16(m) if bf16 else m
        st, out = run(capi, q, k, v, mask=mask)
        assert st == capi.SUCCESS, capi.last_error()
        ref = oracle.sdpa(q, k, v, oracle.bf16_to_f32(mask) if bf16 else m)
        close(oracle, out, ref, v, (S, KV, bf16))
        assert not out[1, :, S // 2].any()


def test_scores_that_grow_along_the_keys(capi, oracle):
    """The first sweep's reference stays the first block's maximum unless a later block leaves the range: keys whose scores grow
    by far more than that, block after block."""
    rng = np.random.default_rng(2)
    S = KV = 640
    q, k, v = make(oracle, rng, 1, 1, S, KV, 64)
    kf = oracle.bf16_to_f32(k) * (1.0 + np.arange(KV, dtype=np.float32)[None, None, :, None] / 40)
    k = oracle.f32_to_bf16(kf)
    st, out = run(capi, q, k, v, scale=2.0)
    assert st == capi.SUCCESS, capi.last_error()
    close(oracle, out, oracle.sdpa(q, k, v, scale=2.0), v, "growing scores")


@pytest.mark.parametrize("S", [4, 150])
def test_keys_and_values_shared_by_all_heads(capi, oracle, S):
    """A stride of 0 over the heads (one K / V for all of them), as host buffers cannot say it: device memory."""
    import torch
    B, H, KV, D = 2, 4, 300, 64
    rng = np.random.default_rng(S)
    q, _, _ = make(oracle, rng, B, H, S, KV, D)
    _, k, v = make(oracle, rng, B, 1, S, KV, D)
    dev = [torch.from_numpy(x.view(np.int16)).cuda() for x in (q, k, v)]
    out = torch.zeros((B, H, S, D), dtype=torch.int16, device="cuda")
    d = capi.SdpaDesc()
    d.batch, d.num_heads, d.seq_len, d.kv_seq_len, d.head_dim = B, H, S, KV, D
    d.q_stride = (C.c_int64 * 4)(*strides_of(q))
    d.o_stride = (C.c_int64 * 4)(*strides_of(q))
    d.k_stride = (C.c_int64 * 4)(KV * D, 0, D, 1)
    d.v_stride = (C.c_int64 * 4)(KV * D, 0, D, 1)
    d.qkv_dt = d.out_dt = capi.DT["bf16"]
    d.query, d.key, d.value, d.output = (t.data_ptr() for t in dev + [out])
    capi.check(capi.lib.b200dnn_sdpa(C.byref(d), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    rep = lambda x: np.ascontiguousarray(np.repeat(x, H, axis=1))  # noqa: E731
    close(oracle, out.cpu().numpy().view(np.uint16), oracle.sdpa(q, rep(k), rep(v)), v, S)


@pytest.mark.parametrize("S", [16, 20])
@pytest.mark.parametrize("masked", [False, True])
def test_few_heads_with_many_keys(capi, oracle, S, masked):
    """One head against 16384 keys: the three-step form where it can take all heads at once, the prompt kernel for another storage order."""
    rng = np.random.default_rng(S)
    B, H, KV, D = 1, 2, 16384, 128
    q, k, v = make(oracle, rng, B, H, S, KV, D)
    mask = None
    if masked:
        mask = np.zeros((1, 1, S, KV), dtype=np.float32)
        mask[..., KV - 700:] = np.finfo(np.float32).min
        mask[0, 0, 3] = -np.inf
    ref = oracle.sdpa(q, k, v, mask)
    st, out = run(capi, q, k, v, mask=mask)
    assert st == capi.SUCCESS, capi.last_error()
    close(oracle, out, ref, v, "one pitch")
    qs = np.ascontiguousarray(q.transpose(0, 2, 1, 3)).transpose(0, 2, 1, 3)      # [batch, seq, head, dim] storage
    st, out = run(capi, qs, k, v, mask=mask)
    assert st == capi.SUCCESS, capi.last_error()
    close(oracle, out, ref, v, "rows of the heads interleaved")


def test_few_heads_with_many_keys_in_a_graph(capi, oracle):
    """The same call captured and replayed on new inputs, with other calls on the stream in between."""
    import torch
    S, KV, D = 20, 16384, 128
    rng = np.random.default_rng(1)
    sets = [make(oracle, rng, 1, 1, S, KV, D) for _ in range(3)]
    dev = [torch.from_numpy(x.view(np.int16)).cuda() for x in sets[0]]
    out = torch.zeros((1, 1, S, D), dtype=torch.int16, device="cuda")

    def desc(q, k, v, o):
        d = capi.SdpaDesc()
        d.batch, d.num_heads, d.seq_len, d.kv_seq_len, d.head_dim = 1, 1, S, KV, D
        for name, x in (("q_stride", q), ("k_stride", k), ("v_stride", v), ("o_stride", o)):
            setattr(d, name, (C.c_int64 * 4)(*x.stride()))
        d.qkv_dt = d.out_dt = capi.DT["bf16"]
        d.query, d.key, d.value, d.output = (x.data_ptr() for x in (q, k, v, o))
        return d
    d = desc(*dev, out)
    stream = torch.cuda.Stream()
    other = [torch.from_numpy(x.view(np.int16)).cuda() for x in sets[2]]
    d_other = desc(*other, torch.zeros_like(out))
    with torch.cuda.stream(stream):
        capi.check(capi.lib.b200dnn_sdpa(C.byref(d), stream.cuda_stream))
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            capi.check(capi.lib.b200dnn_sdpa(C.byref(d), stream.cuda_stream))
        for s in sets[:2]:
            for t, x in zip(dev, s):
                t.copy_(torch.from_numpy(x.view(np.int16)))
            capi.check(capi.lib.b200dnn_sdpa(C.byref(d_other), stream.cuda_stream))
            out.zero_()
            g.replay()
            torch.cuda.synchronize()
            close(oracle, out.cpu().numpy().view(np.uint16), oracle.sdpa(*s), s[2], "replay")

// Launchers of the fused attention kernels (sdpa_flash.cuh): which form takes a call, tensor maps, grids.
#include <algorithm>
#include <cmath>
#include <cudaTypedefs.h>
#include "runtime.cuh"
#include "sdpa_flash.cuh"
#include "sdpa_flash_api.cuh"

namespace b200 {

namespace {

// [128 rows x 64 (128-byte swizzle) or 32 (no swizzle) elements] boxes of a bf16 tensor seen as (d, row, head, batch); an extent of
// one takes any stride
int32_t make_map_heads(CUtensorMap *m, const void *base, int64_t D, int64_t rows, int64_t H, int64_t B, int64_t st_row, int64_t st_h, int64_t st_b,
                       uint32_t inner = 64) {
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)rows, (cuuint64_t)H, (cuuint64_t)B};
  auto bytes = [&](int64_t st, int64_t n) { return (cuuint64_t)((n > 1 ? st : st_row) * 2); };
  cuuint64_t strides[3] = {(cuuint64_t)(st_row * 2), bytes(st_h, H), bytes(st_b, B)};
  cuuint32_t box[4] = {inner, 128, 1, 1}, estr[4] = {1, 1, 1, 1};
  CUresult r = rt().encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           inner == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  B2_CHECK(r == CUDA_SUCCESS, B200DNN_FAILURE, "cuTensorMapEncodeTiled (attention) failed with %d", (int)r);
  return B200DNN_SUCCESS;
}

int walks(int64_t stride, int64_t n) { return n > 1 && stride != 0 ? 1 : 0; }     // 0: broadcast

template <typename... P>
int32_t launch(void (*kern)(P...), unsigned grid, unsigned threads, size_t smem, unsigned cluster, cudaStream_t st, const P &...args) {
  B2_TRY(ensure_max_smem((const void *)kern, (int)smem));
  B2_TRY(launch_pdl_cluster(kern, grid, threads, smem, cluster, st, true, args...));
  B2_LAUNCHED();
  return B200DNN_SUCCESS;
}

// Few query rows: a cluster of CTAs per (batch, head), split over the keys.
int32_t launch_sdpa_decode(const SdpaCall &c, cudaStream_t st) {
  SdpaDecodeArgs a{};
  a.q = (const uint16_t *)c.q; a.out = (uint16_t *)c.out;
  a.qb = c.qs[0]; a.qh = c.qs[1]; a.qs = c.qs[2]; a.ob = c.os[0]; a.oh = c.os[1]; a.os = c.os[2];
  a.kb = walks(c.ks[0], c.B); a.kh = walks(c.ks[1], c.H); a.vb = walks(c.vs[0], c.B); a.vh = walks(c.vs[1], c.H);
  a.S = (int)c.S; a.KV = (int)c.KV; a.D = (int)c.D; a.H = (int)c.H;
  a.scale = c.scale; a.causal = c.causal;
  a.mask = SdpaMask{c.mask, c.mask_dt, c.mb, c.mh, c.mi};
  a.status = rt().status; a.test_no_loads = c.test_no_loads;
  const int64_t heads = c.B * c.H;
  const int db = c.D <= 64 ? 1 : 2;
  // CTAs per head: the busiest SM's keys, plus about 300 keys' worth of time (3 us) for the start and the exchange of each round of
  // CTAs that it runs one after the other (two are resident where their shared memory allows)
  auto chunk_of = [&](int s) { return (int)round_up((c.KV + s - 1) / s, 128); };
  auto smem_of = [&](int s) {
    const size_t scores = (size_t)c.S * (chunk_of(s) + 8) * 4, red = (size_t)kSdpaDecodeWarps * c.S * c.D * 4;
    return sdpa_decode_ring_bytes(db) + (scores > red ? scores : red) + 1024;
  };
  int split = 0;
  int64_t best = 0;
  for (int s = 1; s <= 8; s *= 2) {
    if (smem_of(s) > (size_t)220 * 1024) continue;
    const int64_t resident = smem_of(s) <= (size_t)112 * 1024 ? 2 : 1, per_sm = (heads * s + rt().sm_count - 1) / rt().sm_count;
    const int64_t cost = per_sm * chunk_of(s) + (per_sm + resident - 1) / resident * 300;
    if (split == 0 || cost <= best) { split = s; best = cost; }
  }
  if (split == 0 || heads * split > (1ll << 30)) return B200DNN_UNIMPLEMENTED;
  const size_t smem = smem_of(split);
  a.chunk = chunk_of(split);
  a.sc_stride = a.chunk + 8;             // rows start 8 banks apart: the fragments' eight-byte reads are free of conflicts
  CUtensorMap mk, mv;
  B2_TRY(make_map_heads(&mk, c.k, c.D, c.KV, a.kh ? c.H : 1, a.kb ? c.B : 1, c.ks[2], c.ks[1], c.ks[0], 32));
  B2_TRY(make_map_heads(&mv, c.v, c.D, c.KV, a.vh ? c.H : 1, a.vb ? c.B : 1, c.vs[2], c.vs[1], c.vs[0], 64));
  const unsigned grid = (unsigned)(heads * split);
  if (db == 1) {
    if (c.S <= 8) return launch(sdpa_decode_kernel<1, false>, grid, kSdpaDecodeThreads, smem, split, st, mk, mv, a);
    return launch(sdpa_decode_kernel<1, true>, grid, kSdpaDecodeThreads, smem, split, st, mk, mv, a);
  }
  if (c.S <= 8) return launch(sdpa_decode_kernel<2, false>, grid, kSdpaDecodeThreads, smem, split, st, mk, mv, a);
  return launch(sdpa_decode_kernel<2, true>, grid, kSdpaDecodeThreads, smem, split, st, mk, mv, a);
}

int32_t launch_sdpa_flash(const SdpaCall &c, cudaStream_t st) {
  SdpaFlashArgs a{};
  const int sms = rt().sm_count;
  const int64_t heads = c.B * c.H;
  a.S = (int)c.S; a.KV = (int)c.KV; a.D = (int)c.D; a.H = (int)c.H; a.n_bh = (int)heads;
  // 256 query rows per CTA, or 128 where that would leave SMs without work
  a.tiles = (c.S <= 128 || heads * ((c.S + 255) / 256) < sms) ? 1 : 2;
  a.n_qt = (int)((c.S + a.tiles * 128 - 1) / (a.tiles * 128));
  if (heads * a.n_qt >= (1ll << 31)) return B200DNN_UNIMPLEMENTED;
  // A CTA walks all keys of its rows, so a few heads with many keys leave most SMs idle (1 head x 17 queries x 16384 keys: 469 us with a mask),
  // where the three-step form spreads the keys over the device (122 us).  Both in microseconds, fitted to 1676 calls (1 to 32 heads, 4 to
  // 4096 queries, 512 to 131072 keys, with and without a mask): a wave of CTAs takes so much per 128 keys, the three-step form has its five
  // launches, K and V to pack and the scores to write and read.  The choice is 0.2 % off the better form on average, 26 % at worst; this
  // kernel always, 36 %.
  if (c.grouped) {
    const bool wide = c.D > 64, mask = c.mask != nullptr;
    const double blocks = (double)(((c.causal && c.S < c.KV ? c.S : c.KV) + 127) / 128), waves = (double)((heads * a.n_qt + sms - 1) / sms);
    const double block_us = a.tiles == 2 ? (mask ? 4.6 : 3.5) : (mask ? (wide ? 3.8 : 3.4) : (wide ? 2.3 : 2.0));
    const double h = (double)heads, s = (double)c.S, kv = (double)c.KV;
    const bool slower = 6.0 + waves * blocks * block_us > 31.0 + kv * (0.005 + h * (wide ? 0.0006 : 0.0004)) + 5e-6 * h * s * kv + (mask ? 0.002 : 0.001) * h * s;
    // (the three-step form sends tables from the call's pinned block, which a captured graph would read again when it is replayed)
    if (slower) {
      cudaStreamCaptureStatus cap = cudaStreamCaptureStatusActive;
      if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) cudaGetLastError();
      else if (cap == cudaStreamCaptureStatusNone) return B200DNN_UNIMPLEMENTED;
    }
  }
  // Longest query tiles of all heads first (under a causal mask their lengths differ by the sequence length) while every head's K
  // and V stay in the L2 together; head after head otherwise.
  a.bh_major = !c.causal || 4 * heads * c.KV * c.D > (64ll << 20);
  a.scale = c.scale; a.causal = c.causal;
  const double c_exact = (double)c.scale * 1.44269504088896340736;
  a.c = (float)c_exact;
  a.kappa = std::isnormal(a.c) ? (float)((c_exact / (double)a.c - 1.0) * 0.693147180559945309417) : 0.f;
  a.mask = SdpaMask{c.mask, c.mask_dt, c.mb, c.mh, c.mi};
  const int64_t mstep = c.mask_dt == B200DNN_F32 ? 4 : 8;
  a.mask_vec = (reinterpret_cast<uintptr_t>(c.mask) & 15) == 0 && c.mb % mstep == 0 && c.mh % mstep == 0 && c.mi % mstep == 0;
  a.kb = walks(c.ks[0], c.B); a.kh = walks(c.ks[1], c.H); a.vb = walks(c.vs[0], c.B); a.vh = walks(c.vs[1], c.H);
  a.out = (uint16_t *)c.out; a.ob = c.os[0]; a.oh = c.os[1]; a.os = c.os[2];
  const uintptr_t al = reinterpret_cast<uintptr_t>(c.out) | (uintptr_t)(c.os[2] * 2) | (c.H > 1 ? (uintptr_t)(c.os[1] * 2) : 0) | (c.B > 1 ? (uintptr_t)(c.os[0] * 2) : 0);
  a.out_align = (al & 31) == 0 ? 32 : ((al & 15) == 0 ? 16 : 2);
  a.status = rt().status; a.test_no_loads = c.test_no_loads;
  CUtensorMap mq, mk, mv;
  B2_TRY(make_map_heads(&mq, c.q, c.D, c.S, c.H, c.B, c.qs[2], c.qs[1], c.qs[0]));
  B2_TRY(make_map_heads(&mk, c.k, c.D, c.KV, a.kh ? c.H : 1, a.kb ? c.B : 1, c.ks[2], c.ks[1], c.ks[0]));
  B2_TRY(make_map_heads(&mv, c.v, c.D, c.KV, a.vh ? c.H : 1, a.vb ? c.B : 1, c.vs[2], c.vs[1], c.vs[0]));
  const int db = c.D <= 64 ? 1 : 2;
  // A CTA of one row tile has half the warps and half the tensor memory, so that two fit an SM where shared memory allows it: with one block of keys (two slots of
  // the ring are used) or a head dimension up to 64.  us before and after: 192 heads of 100 keys, head_dim 128, causal 13.8 -> 9.2; 160 of 90, 64, causal 11.4 -> 7.7;
  // 320 of 128, 128, causal 23.5 -> 17.6.  But one CTA per SM while there are SMs for all of them (two of one launch on an SM: 24 heads of 310 keys,
  // 64, with a mask 14.3 -> 18.5, one an SM 13.5).
  const bool one_block = a.tiles == 1 && (c.KV <= 128 || (c.causal && c.S <= 128));
  size_t smem = (size_t)(a.tiles + (one_block ? 2 : kFlashSlots)) * db * 16384 + 1024;
  if (heads * a.n_qt <= sms) smem = std::max(smem, (size_t)120 * 1024);
  const unsigned grid = (unsigned)(heads * a.n_qt), threads = 32u * (8 * a.tiles + 2);
  auto go = [&](auto plain, auto masked) { return launch(c.mask ? masked : plain, grid, threads, smem, 1, st, mq, mk, mv, a); };
  if (c.D <= 64) return go(sdpa_flash_kernel<4, false>, sdpa_flash_kernel<4, true>);
  if (c.D <= 80) return go(sdpa_flash_kernel<5, false>, sdpa_flash_kernel<5, true>);
  if (c.D <= 96) return go(sdpa_flash_kernel<6, false>, sdpa_flash_kernel<6, true>);
  return go(sdpa_flash_kernel<8, false>, sdpa_flash_kernel<8, true>);
}

}  // namespace

int32_t sdpa_fused(const SdpaCall &c, cudaStream_t st) {
  // both kernels read rows as 16-byte vectors (the copy engine's rule as well) and hold a head dimension of up to 128; the
  // row maximum is taken before the scale is applied
  if (c.D % 8 != 0 || c.D > 128 || !(c.scale > 0.f)) return B200DNN_UNIMPLEMENTED;
  auto ok = [](const void *p, const int64_t (&s)[3], int64_t B, int64_t H, bool broadcast) {
    if ((reinterpret_cast<uintptr_t>(p) & 15) != 0 || s[2] <= 0 || s[2] % 8 != 0) return false;
    if (H > 1 && (s[1] % 8 != 0 || s[1] < 0 || (s[1] == 0 && !broadcast))) return false;
    return B <= 1 || (s[0] % 8 == 0 && s[0] >= 0 && (s[0] != 0 || broadcast));
  };
  if (!ok(c.q, c.qs, c.B, c.H, false) || !ok(c.k, c.ks, c.B, c.H, true) || !ok(c.v, c.vs, c.B, c.H, true)) return B200DNN_UNIMPLEMENTED;
  if (c.B * c.H > (1ll << 28)) return B200DNN_UNIMPLEMENTED;
  if (c.S <= 16) {
    const int32_t rc = launch_sdpa_decode(c, st);
    if (rc != B200DNN_UNIMPLEMENTED) return rc;
  }
  return launch_sdpa_flash(c, st);
}

}  // namespace b200

// Fused attention kernels behind b200dnn_sdpa: softmax(Q K^T * scale + mask) V per (batch, head) without a score matrix in
// memory (reference operator: lowoha_operators/sdpa/lowoha_sdpa.hpp:48-55; steps of its BMM backend:
// bmm_sdpa/lowoha_sdpa_bmm.cpp).
//
// Both kernels keep the steps and roundings of that backend: f32 scores, f32 softmax with the FINAL row maximum and row sum,
// probabilities rounded to bf16 after the division, products with V accumulated in f32.  A one-sweep (online) softmax would
// round unnormalised probabilities instead and give other results; so the prompt kernel sweeps the keys twice: the first
// sweep takes row maximum and row sum, the second recomputes the scores and multiplies the normalised probabilities with V.
// The extra Q K^T costs half as much again on the tensor pipe and saves every rescale of the accumulator.
// Every exponent is formed with one rounding (see flash_frame).  Error of the f32 probabilities against double, mean / mean weighted by the
// probability / largest, for 2048 keys with scores of spread 1, 4 and 10 at scale 2^-3.5 (head_dim 128), in units of 1e-7:
//   three-step form                                                    0.94 / 0.79 / 5.3    3.5 / 1.9 / 24     9.4 / 2.4 / 62
//   distance from the maximum, exponential corrected for its argument   1.03 / 0.89 / 6.1    3.1 / 0.95 / 17    7.5 / 0.95 / 40      (before; first measured as
//                                                                       0.92 / 0.76 / 4.8    3.1 / 0.81 / 17    7.5 / 0.65 / 40)
//   here                                                               1.02 / 0.92 / 6.1    3.0 / 1.05 / 17    7.4 / 1.01 / 30
// (the last two from one run: their weighted means differ by no more than two measurements of one form do, all of it far below the rounding to bf16 behind).
// Results against double, head_dim 64 and 128, spread 1, 4, 10, with and without masks: 2.07e-3 to 2.36e-3 (bf16) in either form, within 1e-7 of one another.  With a mask of spread 1, before 1.3 / 1.1 / 10, 3.9 / 2.8 / 34 and 12 / 4.3 / 90, here 1.3 / 1.1 / 9, 3.4 / 2.2 / 25 and 10 / 3.2 / 57;
// with one of -1000 150 / 150 / 330 on both sides at spread 1.
#pragma once
#include "common.cuh"
#include "mbar.cuh"
#include "tc_gemm.cuh"

namespace b200 {

struct SdpaMask { const void *p; int32_t dt; int64_t mb, mh, mi; };   // element (b,h,i,j) at p + b*mb + h*mh + i*mi + j

struct SdpaFlashArgs {
  int S, KV, D, H;
  int n_bh;                 // batch * heads
  int n_qt;                 // query tiles of tiles * 128 rows
  int tiles;                // 128-row tiles per CTA: 1 or 2
  int bh_major;             // work order: all query tiles of a head first, else all heads of the longest query tile first
  float scale;              // > 0
  float c, kappa;           // scale log2 e in f32; (its relative error) ln 2
  int causal;
  SdpaMask mask; int mask_vec;   // mask_vec: every mask row starts on a 16-byte boundary
  int kb, kh, vb, vh;       // 0 where K / V are broadcast over the batch / the heads (stride 0), else 1
  uint16_t *out; int64_t ob, oh, os;
  int out_align;            // bytes every output row start is aligned to: 32, 16 or 2
  int32_t *status;
  int test_no_loads;        // test hook, as in SdpaDecodeArgs
};

constexpr int kFlashThreads = 32 * (16 + 2);      // softmax: two 128-row tiles x two halves of a key block x four lane quadrants; producer, MMAs
constexpr int kFlashSlots = 4;          // K / V ring

__device__ __forceinline__ float ex2f(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ uint64_t pk2(float lo, float hi) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ void upk2(uint64_t r, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(r)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) { uint64_t d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) { uint64_t d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }

// Exponentials of a row.  z: score (natural units with the mask added; without a mask the raw product, the scale is in c).  With M = fl(zmax c) the exponent
// x = z c - M is one fused operation and so one rounding, also where all scores share a large part.  M's own rounding moves every x of the row by the same amount and
// leaves with the row sum, as long as both sweeps use the same M; c = fl(scale log2 e) is off by a factor 1 + kappa, which a factor 1 + kappa ln2 x
// of the result makes good (for the row sum: the sum of 2^x x beside that of 2^x).  Rows whose M is so large that its rounding would leave the
// range of an exponential are shifted by r = zmax first (such scores are multiples of 16 or more, their distance is exact); r = 0 otherwise.
// Exponents stop at -127 (zero), so that an infinite one does not meet a zero in a product; a NaN passes.
constexpr float kLog2e = 1.44269504088896340736f, kLog2eLo = (float)(1.44269504088896340736 - (double)kLog2e), kLn2 = 0.693147180559945309417f;
constexpr float kFlashReach = 1.0f;         // the first sweep's frame follows the row maximum once a score's exponent passes this
struct FlashFrame { float r, M; };
__device__ __forceinline__ FlashFrame flash_frame(float m, float c) {
  const float p = __fmul_rn(m, c);
  const bool large = !(fabsf(p) <= 268435456.0f);
  return FlashFrame{large ? m : 0.f, large ? 0.f : p};
}
// what moving from one frame to another adds to every exponent
__device__ __forceinline__ float flash_shift(const FlashFrame &from, const FlashFrame &to, float c) {
  return fmaxf(__fmaf_rn(from.r - to.r, c, from.M - to.M), -1000.f);
}
__device__ __forceinline__ uint64_t flash_exponent2(uint64_t z2, uint64_t c2, uint64_t nM2) {
  float x0, x1;
  upk2(fma2(z2, c2, nM2), x0, x1);
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(x0) : "f"(-127.f));
  asm("max.NaN.f32 %0, %0, %1;" : "+f"(x1) : "f"(-127.f));
  return pk2(x0, x1);
}
__device__ __forceinline__ uint64_t ex2_pair(uint64_t x2) {
  float x0, x1;
  upk2(x2, x0, x1);
  return pk2(ex2f(x0), ex2f(x1));
}

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *map, int x, int y, int z, int w, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
               ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar) : "memory");
}
// A from tensor memory (bf16 pairs, one row per lane), B from shared memory
__device__ __forceinline__ void tc_mma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.b32 p, %4, 0;\nelect.sync _|q, 0xffffffff;\n"
               "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
               ::"r"(d_tmem), "r"(a_tmem), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
                 "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}

// MN-major, SWIZZLE_128B operand: 128-byte rows of 64 elements along N, one row per k.  Eight k rows are one 1 KiB group
// (stride byte offset 1024); the next 64 elements of N start `lead` bytes further (leading byte offset).
__device__ __forceinline__ uint64_t make_smem_desc_mn(uint32_t saddr, uint32_t lead) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lead >> 4) << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

// Prompt form: one CTA per (batch, head, 256 query rows), 576 threads (128 rows: 320).
//   warps 0-15      softmax: eight per 128-row tile, of which four take keys 0-63 of a block and four keys 64-127 (two threads per row), scores
//                   read from tensor memory 32 at a time (64 at once left no registers: 200 bytes spilled, 174 against 134 us with a padding mask)
//   next            TMA producer: Q once; K blocks of 128 keys (sweep 1); K and V blocks in turn (sweep 2)
//   last            MMA issuer
// Tensor memory: S0 S1 O0 O1, 128 columns each.  In sweep 1 the O columns are the second score buffer of their tile, so the
// tensor pipe runs a block ahead; in sweep 2 the normalised probabilities replace the scores in place as bf16 pairs and are the
// A operand of the product with V straight from tensor memory.  Sweep 2 goes in four streams, a tile's half of the keys each: as soon as its 64 probabilities a row
// are there, P V of these keys and the scores of the next block's 64 keys are issued, while the other streams are in their
// exponentials.  (Whole tiles of 128 keys waited for both halves and for the whole product: 3480 clocks a pair of blocks.)  One block of keys needs no second product: its
// scores stay in tensor memory.
// Bounds, per pair of 128 x 128 blocks (both row tiles): the exponentials, one per score and sweep at 16 a clock, 2048 clocks each, and the tensor pipe, 1024 in sweep 1 and
// 2560 in sweep 2 (64 columns at a time run at two thirds of the rate; head_dim 64: half of each); measured inside a CTA 2500 to 2700 and 3300 (head_dim 64: 2470).
// A share of the exponentials on the FMA pipe (a polynomial of degree six) was slower, 203 against 196 us: the pipes wait for one another, not for one of them.
// 32 heads x 2048, us before the streams and the one-rounding exponents and now: causal 63.8 -> 62.2, none 122 -> 117, padding mask 160 -> 130; head_dim 64, 240 heads x
// 1447 with padding 637 -> 527.  256 query rows per CTA, because K and V then pass the L2 half as often as with 128.
// KS: 16-element steps of the head dimension
template <int KS, bool MASK>
__global__ void __launch_bounds__(kFlashThreads, 1)
sdpa_flash_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                  const __grid_constant__ CUtensorMap map_v, const SdpaFlashArgs a) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[32];
  __shared__ float2 stats[2][2][128];                  // row maximum and row sum of each half
  __shared__ uint32_t tmem_base_slot;
  __shared__ volatile int s_err;
  constexpr int DB = (KS + 3) / 4;                     // 64-element blocks of the head dimension
  constexpr uint32_t kBox = 128 * 128;                 // [128 rows][64 elements]
  constexpr uint32_t kTile = DB * kBox;                // 128 rows of Q, K or V
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // (the same in every lane, and known to be)
  const int sw = 8 * a.tiles;                          // softmax warps; then the producer's and the MMAs'
  const uint32_t o_off = 128u * (uint32_t)a.tiles;     // tensor memory: scores of the tiles, then their outputs
  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t ring0 = smem0 + (uint32_t)a.tiles * kTile;
  const uint32_t bar0 = smem_u32(bars);
  const uint32_t q_full = bar0;
  auto kv_full = [&](int s) { return bar0 + 8u * (1 + s); };
  auto kv_empty = [&](int s) { return bar0 + 8u * (1 + kFlashSlots + s); };
  auto s_full = [&](int t, int b) { return bar0 + 8u * (1 + 2 * kFlashSlots + 2 * t + b); };
  auto s_free = [&](int t, int b) { return bar0 + 8u * (5 + 2 * kFlashSlots + 2 * t + b); };
  auto p_ready = [&](int t, int half) { return bar0 + 8u * (9 + 2 * kFlashSlots + 2 * t + half); };
  auto o_done = [&](int t) { return bar0 + 8u * (13 + 2 * kFlashSlots + t); };
  // (sweep 2 has barriers of its own: a phase of s_full may pass only when all warps of the tile have met the one before)
  auto s2_full = [&](int t, int half) { return bar0 + 8u * (15 + 2 * kFlashSlots + 2 * t + half); };

  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_q) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
    mbar_init(q_full, 1);
    for (int s = 0; s < kFlashSlots; ++s) { mbar_init(kv_full(s), 1); mbar_init(kv_empty(s), 1); }
    for (int t = 0; t < 2; ++t) {
      for (int b = 0; b < 2; ++b) { mbar_init(s_full(t, b), 1); mbar_init(s2_full(t, b), 1); mbar_init(s_free(t, b), 8); mbar_init(p_ready(t, b), 4); }
      mbar_init(o_done(t), 1);
    }
    s_err = 0;
    mbar_fence_init();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == sw + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(2u * o_off) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_slot;
  // (behind the allocation: a dependent's CTA on this SM can then not take tensor memory that this one still waits for)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // this CTA's work item
  int bh, qt;
  if (a.bh_major) { bh = blockIdx.x / a.n_qt; qt = a.n_qt - 1 - (blockIdx.x - bh * a.n_qt); }
  else { const int r = blockIdx.x / a.n_bh; bh = blockIdx.x - r * a.n_bh; qt = a.n_qt - 1 - r; }
  const int b = bh / a.H, h = bh - b * a.H;
  const int q0 = qt * a.tiles * 128;
  // key blocks that row tile t meets
  auto n_blocks = [&](int t) {
    const int r0 = q0 + t * 128;
    if (t >= a.tiles || r0 >= a.S) return 0;
    return (min(a.KV, a.causal ? r0 + 128 : a.KV) + 127) >> 7;
  };
  const int nb0 = n_blocks(0), nb1 = n_blocks(1), nmax = max(nb0, nb1);
  const bool keep = nmax == 1;        // one block of keys: its scores stay in tensor memory between the sweeps

  if (warp == sw) {
    // ------------------------------------------------------------------ producer
    if (lane == 0 && !a.test_no_loads) {
      const int active = nb1 > 0 ? 2 : 1;
      mbar_expect_tx(q_full, (uint32_t)active * kTile);
      for (int t = 0; t < active; ++t)
        for (int d = 0; d < DB; ++d)
          tma_load_4d(smem0 + (uint32_t)t * kTile + (uint32_t)d * kBox, &map_q, d * 64, q0 + t * 128, h, b, q_full);
      const int total = keep ? 2 : 3 * nmax;
      for (int u = 0; u < total; ++u) {
        const int slot = u % kFlashSlots;
        if (!mbar_wait(kv_empty(slot), ((uint32_t)(u / kFlashSlots) & 1u) ^ 1u)) { s_err = 1; report_status(a.status, 21); break; }
        const int w = u - nmax + (keep ? 1 : 0);           // (with one block: K, V)
        const bool is_v = w > 0 && (w & 1);
        const int blk = w < 0 ? u : (w >> 1);
        mbar_expect_tx(kv_full(slot), kTile);
        const CUtensorMap *m = is_v ? &map_v : &map_k;
        const int hh = is_v ? h * a.vh : h * a.kh, bb = is_v ? b * a.vb : b * a.kb;
        for (int d = 0; d < DB; ++d)
          tma_load_4d(ring0 + (uint32_t)slot * kTile + (uint32_t)d * kBox, m, d * 64, blk * 128, hh, bb, kv_full(slot));
      }
    }
  } else if (warp == sw + 1) {
    // ------------------------------------------------------------------ MMA issuer
    // (the whole warp walks the schedule: control flow and operands are the same in every lane)
    const uint32_t idesc_s = make_idesc_bf16(128), idesc_h = make_idesc_bf16(64);
    const uint32_t idesc_o = make_idesc_bf16(KS * 16) | (1u << 16);           // B (V) is N-major
    const uint64_t q_desc = make_smem_desc(smem0), k_desc = make_smem_desc(ring0), v_desc = make_smem_desc_mn(ring0, kBox);
    constexpr uint64_t kTileD = kTile >> 4, kBoxD = kBox >> 4;
    auto qk = [&](int t, uint32_t d_tmem, int slot, uint32_t bar) {
      const uint64_t qa = q_desc + (uint64_t)t * kTileD, ka = k_desc + (uint64_t)slot * kTileD;
#pragma unroll
      for (int k = 0; k < KS; ++k) tc_mma_bf16(d_tmem, qa + (k >> 2) * kBoxD + (k & 3) * 2, ka + (k >> 2) * kBoxD + (k & 3) * 2, idesc_s, k ? 1u : 0u);
      tc_commit(bar);
    };
    auto qk_half = [&](int t, int h2, int slot) {              // scores of 64 keys of a block, where that half of the tile's warps expects them
      const uint64_t qa = q_desc + (uint64_t)t * kTileD, ka = k_desc + (uint64_t)slot * kTileD + (uint64_t)h2 * (64 * 128 >> 4);
#pragma unroll
      for (int k = 0; k < KS; ++k)
        tc_mma_bf16(tmem + (uint32_t)t * 128u + (uint32_t)h2 * 64u, qa + (k >> 2) * kBoxD + (k & 3) * 2, ka + (k >> 2) * kBoxD + (k & 3) * 2, idesc_h, k ? 1u : 0u);
      tc_commit(s2_full(t, h2));
    };
    auto pv = [&](int t, int slot, bool first, int k0) {       // 64 keys: k0 = 0 or 4
      const uint64_t va = v_desc + (uint64_t)slot * kTileD + (uint64_t)(k0 * 128);
      const uint32_t pa = tmem + (uint32_t)t * 128u + (k0 ? 64u : 0u), od = tmem + o_off + (uint32_t)t * 128u;
#pragma unroll
      for (int k = 0; k < 4; ++k) tc_mma_bf16_ts(od, pa + (uint32_t)k * 8u, va + k * 128, idesc_o, (first && k0 + k == 0) ? 0u : 1u);
    };
    bool ok = mbar_wait_warp(q_full, 0);
    int u = 0;
    auto full = [&](int uu) { return mbar_wait_warp(kv_full(uu % kFlashSlots), (uint32_t)(uu / kFlashSlots) & 1u); };
    // sweep 1: scores only, two buffers per tile
    for (int j = 0; ok && j < nmax; ++j, ++u) {
      ok = full(u);
      if (!ok) break;
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        if (!ok || j >= (t ? nb1 : nb0)) continue;
        ok = mbar_wait_warp(s_free(t, j & 1), ((uint32_t)(j >> 1) & 1u) ^ 1u);
        if (!ok) break;
        tc_fence_after();
        qk(t, tmem + (uint32_t)t * 128u + ((j & 1) ? o_off : 0u), u % kFlashSlots, s_full(t, j & 1));
      }
      tc_commit(kv_empty(u % kFlashSlots));
    }
    // sweep 2: first scores, published to the two halves of a tile's warps
    if (ok && !keep) ok = full(u);
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int nb = t ? nb1 : nb0;
      if (!ok || keep || nb == 0) continue;
      ok = mbar_wait_warp(s_free(t, 0), ((uint32_t)((nb + 1) >> 1) & 1u) ^ 1u);
      if (!ok) break;
      tc_fence_after();
      qk_half(t, 0, u % kFlashSlots);
      qk_half(t, 1, u % kFlashSlots);
    }
    if (ok && !keep) { tc_commit(kv_empty(u % kFlashSlots)); ++u; }
    // then in turn for each tile and half: P V of its 64 keys, and the scores of the next block in place of P
    for (int j = 0; ok && j < nmax; ++j, u += 2) {
      ok = full(u) && (j + 1 >= nmax || full(u + 1));
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = i & 1, h2 = i >> 1, nb = t ? nb1 : nb0;
        if (!ok || j >= nb) continue;
        ok = mbar_wait_warp(p_ready(t, h2), (uint32_t)j & 1u);
        if (!ok) break;
        tc_fence_after();
        pv(t, u % kFlashSlots, j == 0, 4 * h2);
        if (j + 1 < nb) qk_half(t, h2, (u + 1) % kFlashSlots);
        else if (h2) tc_commit(o_done(t));
      }
      tc_commit(kv_empty(u % kFlashSlots));
      if (j + 1 < nmax) tc_commit(kv_empty((u + 1) % kFlashSlots));
    }
    if (!ok && lane == 0) { s_err = 1; report_status(a.status, 22); }
  } else {
    // ------------------------------------------------------------------ softmax
    // thread: one row, one half (64 keys) of every block
    const int t = warp >> 3, half = (warp >> 2) & 1, nb = t ? nb1 : nb0;
    const int row_in_tile = (warp & 3) * 32 + lane, row = q0 + t * 128 + row_in_tile;
    const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t ts0 = tmem + lane_off + (uint32_t)t * 128u + (uint32_t)half * 64u, to0 = ts0 + o_off;
    const float ninf = __int_as_float(0xff800000);
    const int n_keys = min(a.KV, a.causal ? row + 1 : a.KV);         // keys this row sees
    const int64_t moff = MASK ? (int64_t)b * a.mask.mb + (int64_t)h * a.mask.mh + (int64_t)min(row, a.S - 1) * a.mask.mi : 0;
    // a chunk of 32 scores; with a mask, scale and mask are applied here (vector loads where the mask's rows allow it: all lanes read the
    // same bytes when the mask does not depend on the query).  The mask is added as it is: the type's lowest finite value times log2(e)
    // would be an infinity, and a row that carries it throughout is a softmax over equal scores, not a row without keys
    auto mask_load = [&](float (&mk)[32], int j0) {
      const bool whole = a.mask_vec && j0 + 32 <= a.KV;
      if (a.mask.dt == DT_F32) {
        const float *mp = reinterpret_cast<const float *>(a.mask.p) + moff + j0;
        if (whole) {
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const float4 v = __ldg(reinterpret_cast<const float4 *>(mp + i));
            mk[i] = v.x; mk[i + 1] = v.y; mk[i + 2] = v.z; mk[i + 3] = v.w;
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) mk[i] = j0 + i < a.KV ? __ldg(mp + i) : 0.f;
        }
      } else {
        const uint16_t *mp = reinterpret_cast<const uint16_t *>(a.mask.p) + moff + j0;
        if (whole) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            const uint4 v = __ldg(reinterpret_cast<const uint4 *>(mp + i));
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) { mk[i + 2 * e] = __uint_as_float(w[e] << 16); mk[i + 2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u); }
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) mk[i] = j0 + i < a.KV ? bf16_bits_to_f32(__ldg(mp + i)) : 0.f;
        }
      }
    };
    auto mask_add = [&](uint32_t (&s)[32], const float (&mk)[32]) {
      const uint64_t sc2 = pk2(a.scale, a.scale);
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        float y0, y1;
        upk2(fma2(pk2(__uint_as_float(s[i]), __uint_as_float(s[i + 1])), sc2, pk2(mk[i], mk[i + 1])), y0, y1);
        s[i] = __float_as_uint(y0); s[i + 1] = __float_as_uint(y1);
      }
    };
    int n_vis = n_keys;
    // keys that a row does not see, where some row of the warp does not see all (a compare and a select per score otherwise: of 128 keys, all seen, 8 heads, head_dim 128
    // 7.29 -> 6.79 us; 32 heads x 2048 117 against 120 although the blocks in the middle did without before, in a copy of the code of their own)
    auto limit32 = [&](uint32_t (&s)[32], int j0) {
      if (!__any_sync(0xffffffffu, j0 + 32 > n_vis)) return;
#pragma unroll
      for (int i = 0; i < 32; ++i) if (j0 + i >= n_vis) s[i] = __float_as_uint(ninf);
    };
    float m = ninf, l = 0.f, lx = 0.f;            // the score whose frame it is (the row's largest, or one just below it), sums of 2^x and of 2^x x
    FlashFrame fr{0.f, 0.f};
    bool shifted = false;                       // some lane's frame has an r
    bool ok = true;
    uint32_t ph0 = 0, ph1 = 0;
    const float c = MASK ? kLog2e : a.c, kap = MASK ? kLog2eLo / kLog2e * kLn2 : a.kappa;
    const uint64_t c2 = pk2(c, c);
    auto shift32 = [&](uint32_t (&s)[32]) {
#pragma unroll
      for (int i = 0; i < 32; ++i) s[i] = __float_as_uint(__uint_as_float(s[i]) - fr.r);
    };
    // ---- sweep 1: row maximum and row sum of this half, 32 scores at a time.  The frame is that of the first scores until one lies far above it, so a
    // single score far above all others is met wherever it lies.  (fmaxf passes over a NaN; the sum does not)
    auto sum_half = [&](uint32_t ta, int k0) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t s[32];
        tc_ld32(ta + (uint32_t)q * 32u, s);
        float mk[MASK ? 32 : 1];
        if constexpr (MASK) mask_load(mk, k0 + q * 32);           // (in flight beside the scores)
        tc_wait_ld();
        if constexpr (MASK) mask_add(s, mk);
        limit32(s, k0 + q * 32);
        float mx = ninf, my = ninf;
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
          mx = fmaxf(mx, fmaxf(__uint_as_float(s[i]), __uint_as_float(s[i + 1])));
          my = fmaxf(my, fmaxf(__uint_as_float(s[i + 2]), __uint_as_float(s[i + 3])));
        }
        mx = fmaxf(mx, my);
        const bool move = mx > ninf && (m == ninf || !(__fmaf_rn(mx - fr.r, c, -fr.M) <= kFlashReach));
        if (__any_sync(0xffffffffu, move)) {
          if (move) {
            m = mx;
            const FlashFrame to = flash_frame(m, c);
            if (l != 0.f) {
              const float sh = flash_shift(fr, to, c), f = ex2f(sh);
              lx = f * __fmaf_rn(sh, l, lx);
              l *= f;
            }
            fr = to;
          }
          shifted = __any_sync(0xffffffffu, fr.r != 0.f);
        }
        if (shifted) shift32(s);
        const uint64_t nM2 = pk2(-fr.M, -fr.M);
        uint64_t acc[2] = {0ull, 0ull}, accx[2] = {0ull, 0ull};
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const uint64_t x2 = flash_exponent2(pk2(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1])), c2, nM2), e2 = ex2_pair(x2);
          acc[i & 1] = add2(acc[i & 1], e2);
          accx[i & 1] = fma2(e2, x2, accx[i & 1]);
        }
        float e0, e1;
        upk2(add2(acc[0], acc[1]), e0, e1);
        l += e0 + e1;
        upk2(add2(accx[0], accx[1]), e0, e1);
        lx += e0 + e1;
      }
    };
    for (int j = 0; ok && j < nb; ++j) {
      const int bf = j & 1, k0 = j * 128 + half * 64;
      ok = __all_sync(0xffffffffu, mbar_wait(s_full(t, bf), bf ? ph1 : ph0));      // one decision per warp: tensor-memory loads are warp-wide
      if (!ok) break;
      if (bf) ph1 ^= 1u; else ph0 ^= 1u;
      tc_fence_after();
      const uint32_t ta = bf ? to0 : ts0;
      sum_half(ta, k0);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(s_free(t, bf));
    }
    // ---- the two halves of a row together, each with its corrected sum, in the higher of the two frames
    l = __fmaf_rn(kap, lx, l);
    stats[t][half][row_in_tile] = make_float2(m, l);
    asm volatile("bar.sync %0, 256;" ::"r"(1 + t) : "memory");
    {
      const float2 o = stats[t][half ^ 1][row_in_tile];
      const float mn = fmaxf(m, o.x);
      fr = flash_frame(mn, c);
      const float sa = flash_shift(flash_frame(m, c), fr, c), sb = flash_shift(flash_frame(o.x, c), fr, c);
      l = ex2f(sa) * __fmaf_rn(kap * sa, l, l) + ex2f(sb) * __fmaf_rn(kap * sb, o.y, o.y);
      m = mn;
    }
    // ---- sweep 2: p = 2^x (1 + kappa ln2 x) / l.  A row without a score above -inf gives zeros (all its scores count as masked); a NaN
    // in the sum makes the whole row NaN
    const bool dead = m == ninf;
    if (dead) { n_vis = 0; fr = FlashFrame{0.f, 0.f}; }
    shifted = __any_sync(0xffffffffu, fr.r != 0.f);
    const float inv = dead ? 0.f : __fdiv_rn(1.0f, l), kinv = kap * inv;
    const uint64_t nM2 = pk2(-fr.M, -fr.M), inv2 = pk2(inv, inv), kinv2 = pk2(kinv, kinv);
    auto p_half = [&](int k0) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t s[32];
        tc_ld32(ts0 + (uint32_t)q * 32u, s);
        float mk[MASK ? 32 : 1];
        if constexpr (MASK) mask_load(mk, k0 + q * 32);           // (in flight beside the scores)
        tc_wait_ld();
        if constexpr (MASK) mask_add(s, mk);
        limit32(s, k0 + q * 32);
        if (shifted) shift32(s);
        uint32_t p[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const uint64_t x2 = flash_exponent2(pk2(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1])), c2, nM2);
          float x0, x1;
          upk2(mul2(ex2_pair(x2), fma2(x2, kinv2, inv2)), x0, x1);
          p[i] = pack_bf16x2(x0, x1);
        }
        tc_st16(ts0 + (uint32_t)q * 16u, p);      // (over scores of this half that have been read)
      }
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_ready(t, half));
    };
    for (int j = 0; ok && j < nb; ++j) {
      if (!keep) ok = __all_sync(0xffffffffu, mbar_wait(s2_full(t, half), (uint32_t)j & 1u));
      if (!ok) break;
      tc_fence_after();
      p_half(j * 128 + half * 64);
    }
    if (ok && nb > 0) ok = __all_sync(0xffffffffu, mbar_wait(o_done(t), 0));
    if (ok && nb > 0) {
      tc_fence_after();
      uint16_t *o = a.out + (int64_t)b * a.ob + (int64_t)h * a.oh + (int64_t)row * a.os;
      const int units = (a.D + 15) >> 4, u0 = half ? (units + 1) >> 1 : 0, u1 = half ? units : (units + 1) >> 1;     // the halves share the columns
      const uint32_t od = tmem + lane_off + o_off + (uint32_t)t * 128u;
      for (int d0 = u0 * 16; d0 < u1 * 16; d0 += 16) {
        uint32_t r[16], pk[8];
        tc_ld16(od + (uint32_t)d0, r);
        tc_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; ++i) pk[i] = pack_bf16x2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
        if (row < a.S) {
          if (a.out_align == 32 && d0 + 16 <= a.D) st_global_v8(o + d0, pk);
          else if (a.out_align >= 16) {
            *reinterpret_cast<uint4 *>(o + d0) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
            if (d0 + 16 <= a.D) *reinterpret_cast<uint4 *>(o + d0 + 8) = make_uint4(pk[4], pk[5], pk[6], pk[7]);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) if (d0 + i < a.D) o[d0 + i] = (uint16_t)(pk[i >> 1] >> ((i & 1) * 16));
          }
        }
        __syncwarp();
      }
    }
    if (!ok && lane == 0) { s_err = 1; report_status(a.status, 23); }
  }

  tc_fence_before();
  __syncthreads();
  if (s_err) {
    for (int i = 0; i < 64; ++i) __nanosleep(20000);     // copies still in flight land before shared memory is released
    __syncthreads();
  }
  if (warp == sw + 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2u * o_off) : "memory");
  }
}

// ---- few query rows (S <= 16) against many keys: bound by reading K and V once -----------------------------------------
// A cluster of C CTAs per (batch, head), each with a contiguous share of the keys; eight consumer warps and a producer warp.
//   0. the producer streams the share's K blocks and then its V blocks (128 keys each) through one shared-memory ring with TMA: the
//      first V blocks are on their way while the row maxima and sums of step 2 are exchanged, so HBM does not pause there, and the
//      bytes in flight per SM are the ring's (two CTAs of three slots), not a register budget.
//   1. scores: warp w takes keys 16 w .. 16 w + 15 of a block with mma.m16n8k16 (A: the query rows, in registers for the whole
//      call; B: eight keys).  K rows sit in 64-byte pieces ([128 keys][32 elements], no swizzle): a lane's fragment of key g is the
//      16 bytes at 8 t of a piece, the same assignment of d to fragment positions on both operands, so a quarter warp reads
//      128 contiguous bytes.  f32 scores (scaled, mask applied) stay in shared memory.
//   2. final row maximum and row sum over the cluster through distributed shared memory, p = bf16(e / sum).
//   3. p V: keys are the k dimension; V sits in 128-byte swizzled rows, a lane reads 16 bytes (8 columns) of four key rows (a
//      quarter warp: eight different bank groups) and pairs them with byte permutes.  Up to eight query rows: V^T p^T, columns
//      of V as the 16 MMA rows; more: p V with the query rows as MMA rows.
//   4. f32 partial outputs are added over warps and CTAs in a fixed order.
struct SdpaDecodeArgs {
  const uint16_t *q; uint16_t *out;
  int64_t qb, qh, qs, ob, oh, os;
  int kb, kh, vb, vh;      // 0 where K / V are broadcast over the batch / the heads, else 1
  int S, KV, D, H;
  int chunk;               // keys per CTA, a multiple of 128
  int sc_stride;           // f32 per score row in shared memory
  float scale;
  int causal;
  SdpaMask mask;
  int32_t *status;
  int test_no_loads;       // test hook: the producer issues no copies, so the waits expire
};
constexpr int kSdpaDecodeWarps = 8, kSdpaDecodeThreads = 32 * (kSdpaDecodeWarps + 1), kSdpaDecodeSlots = 3;

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t caddr) { float v; asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(caddr) : "memory"); return v; }

// shared memory: [ring][scores, later the partial outputs]
__host__ __device__ inline size_t sdpa_decode_ring_bytes(int db) { return (size_t)kSdpaDecodeSlots * db * 16384; }

// DB: 64-element blocks of the head dimension (1: D <= 64, 2: D <= 128); HI: more than eight query rows
template <int DB, bool HI>
__global__ void __launch_bounds__(kSdpaDecodeThreads, 2)
sdpa_decode_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const SdpaDecodeArgs a) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[2 * kSdpaDecodeSlots];
  __shared__ float wred[kSdpaDecodeWarps][16], cmax[16], csum[16], row_m[16], row_inv[16];
  __shared__ volatile int s_err;
  constexpr int NP = 2 * DB;                       // 32-element pieces of a key row
  constexpr uint32_t kSlot = DB * 16384;           // 128 keys
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  uint32_t csize, crank;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(csize));
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(crank));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u, bar0 = smem_u32(bars);
  float *sc = reinterpret_cast<float *>(smem_raw + (ring - smem_u32(smem_raw)) + sdpa_decode_ring_bytes(DB));
  auto full = [&](int s) { return bar0 + 8u * (uint32_t)s; };
  auto empty = [&](int s) { return bar0 + 8u * (uint32_t)(kSdpaDecodeSlots + s); };
  if (tid == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_k) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_v) : "memory");
    for (int s = 0; s < kSdpaDecodeSlots; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), kSdpaDecodeWarps); }
    s_err = 0;
    mbar_fence_init();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int bh = blockIdx.x / csize, b = bh / a.H, h = bh - b * a.H;
  const int k0 = (int)crank * a.chunk, k1 = min(a.KV, k0 + a.chunk);     // this CTA's keys (k1 <= k0: none)
  const int nblk = k1 > k0 ? (k1 - k0 + 127) >> 7 : 0;
  const int S = a.S, D = a.D;
  const float ninf = __int_as_float(0xff800000);
  bool ok = true;

  // The producer takes part in the barriers of step 2, so before them it may only wait for slots that the K blocks free: blocks up to
  // nblk + slots - 1; the others follow in step 3.
  auto produce = [&](int from, int to) {
    if (lane != 0 || a.test_no_loads) return;
    for (int u = from; u < to; ++u) {
      const int slot = u % kSdpaDecodeSlots;
      if (!mbar_wait(empty(slot), ((uint32_t)(u / kSdpaDecodeSlots) & 1u) ^ 1u)) { s_err = 1; report_status(a.status, 41); break; }
      const bool is_v = u >= nblk;
      const int key = k0 + (is_v ? u - nblk : u) * 128;
      const uint32_t dst = ring + (uint32_t)slot * kSlot;
      mbar_expect_tx(full(slot), kSlot);
      if (is_v) { for (int d = 0; d < DB; ++d) tma_load_4d(dst + (uint32_t)d * 16384u, &map_v, d * 64, key, h * a.vh, b * a.vb, full(slot)); }
      else { for (int i = 0; i < NP; ++i) tma_load_4d(dst + (uint32_t)i * 8192u, &map_k, i * 32, key, h * a.kh, b * a.kb, full(slot)); }
    }
  };
  const int n_early = min(2 * nblk, nblk + kSdpaDecodeSlots);
  if (warp == kSdpaDecodeWarps) { produce(0, n_early); __syncwarp(); }
  // ---- query fragments
  uint4 qlo[NP], qhi[HI ? NP : 1];
  if (warp < kSdpaDecodeWarps) {
    const uint16_t *qp = a.q + (int64_t)b * a.qb + (int64_t)h * a.qh;
#pragma unroll
    for (int i = 0; i < NP; ++i) {
      const int d = i * 32 + t * 8;
      qlo[i] = (g < S && d < D) ? __ldg(reinterpret_cast<const uint4 *>(qp + (int64_t)g * a.qs + d)) : make_uint4(0, 0, 0, 0);
      if constexpr (HI) qhi[i] = (g + 8 < S && d < D) ? __ldg(reinterpret_cast<const uint4 *>(qp + (int64_t)(g + 8) * a.qs + d)) : make_uint4(0, 0, 0, 0);
    }
    // ---- 1. scores
    float m_lo = ninf, m_hi = ninf;
    const int64_t moff = (int64_t)b * a.mask.mb + (int64_t)h * a.mask.mh;
    for (int u = 0; u < nblk; ++u) {
      const int slot = u % kSdpaDecodeSlots;
      // (one decision per warp; the other warps meet this one at the barriers below either way)
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(full(slot), (uint32_t)(u / kSdpaDecodeSlots) & 1u));
      if (!ok) { if (lane == 0) { s_err = 1; report_status(a.status, 42); } break; }
      const int kw = u * 128 + warp * 16;                    // this warp's first key, relative to k0
      uint4 kr[2][NP];
#pragma unroll
      for (int v = 0; v < 2; ++v)
#pragma unroll
        for (int i = 0; i < NP; ++i) kr[v][i] = ld_shared_v4(ring + (uint32_t)slot * kSlot + (uint32_t)(i * 8192 + (warp * 16 + v * 8 + g) * 64 + t * 16));
      __syncwarp();
      if (lane == 0) mbar_arrive(empty(slot));
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 0; i < NP; ++i) {
          uint4 hi = make_uint4(0, 0, 0, 0);
          if constexpr (HI) hi = qhi[i];
          mma_bf16_16816(acc, qlo[i].x, hi.x, qlo[i].y, hi.y, kr[v][i].x, kr[v][i].y);
          mma_bf16_16816(acc, qlo[i].z, hi.z, qlo[i].w, hi.w, kr[v][i].z, kr[v][i].w);
        }
        const int key = kw + v * 8 + 2 * t;
#pragma unroll
        for (int hb = 0; hb < (HI ? 2 : 1); ++hb) {
          const int row = g + 8 * hb;
          if (row < S) {
            float x[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int j = k0 + key + e;
              float y = __fmul_rn(acc[2 * hb + e], a.scale);
              if (a.mask.p && j < k1) y = __fadd_rn(y, load_as_f32(a.mask.p, a.mask.dt, moff + (int64_t)row * a.mask.mi + j));
              x[e] = (j < k1 && !(a.causal && j > row)) ? y : ninf;
            }
            *reinterpret_cast<float2 *>(sc + (size_t)row * a.sc_stride + key) = make_float2(x[0], x[1]);
            if (hb) m_hi = fmaxf(m_hi, fmaxf(x[0], x[1])); else m_lo = fmaxf(m_lo, fmaxf(x[0], x[1]));
          }
        }
      }
    }
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) { m_lo = fmaxf(m_lo, __shfl_xor_sync(0xffffffffu, m_lo, o)); m_hi = fmaxf(m_hi, __shfl_xor_sync(0xffffffffu, m_hi, o)); }
    if (t == 0) { wred[warp][g] = m_lo; wred[warp][g + 8] = m_hi; }
  }
  // ---- 2. row maximum and row sum over the cluster
  auto csync = [&]() { if (csize > 1) cluster_sync_all(); else __syncthreads(); };
  __syncthreads();
  if (tid < 16) {
    float v = wred[0][tid];
    for (int w = 1; w < kSdpaDecodeWarps; ++w) v = fmaxf(v, wred[w][tid]);
    cmax[tid] = v;
  }
  csync();
  if (tid < 16) {
    float v = cmax[tid];
    for (uint32_t r = 0; r < csize; ++r) if (r != crank) v = fmaxf(v, ld_cluster_f32(cluster_map(smem_u32(&cmax[tid]), r)));
    row_m[tid] = v;
  }
  __syncthreads();
  const int nk = nblk * 128;                               // (scores of keys past the end are -inf)
  if (warp < kSdpaDecodeWarps && ok) {
    // the warps share the rows; with fewer rows than warps each row is cut into 8 / S' parts (S' = rows rounded up to a power of two)
    const int parts = S >= 8 ? 1 : (S > 4 ? 1 : (S > 2 ? 2 : (S > 1 ? 4 : 8)));
    for (int row = warp / parts; row < S; row += kSdpaDecodeWarps / parts) {
      const float m = row_m[row];
      float sum = 0.f;
      float *sr = sc + (size_t)row * a.sc_stride;
      for (int j = ((warp % parts) * 32 + lane) * 2; j < nk; j += 64 * parts) {
        float2 x = *reinterpret_cast<float2 *>(sr + j);
        x.x = m == ninf ? 0.f : expf(x.x - m); x.y = m == ninf ? 0.f : expf(x.y - m);      // (no score above -inf: zeros)
        sum += x.x + x.y;
        *reinterpret_cast<float2 *>(sr + j) = x;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0) wred[warp % parts][row] = sum;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(kSdpaDecodeWarps * 32) : "memory");
    if (tid < S) {
      float v = wred[0][tid];
      for (int q = 1; q < parts; ++q) v += wred[q][tid];
      csum[tid] = v;
    }
  } else if (warp < kSdpaDecodeWarps) asm volatile("bar.sync 1, %0;" ::"n"(kSdpaDecodeWarps * 32) : "memory");
  csync();
  if (tid < 16) {
    float v = 0.f;
    if (tid < S) for (uint32_t r = 0; r < csize; ++r) v += csize > 1 ? ld_cluster_f32(cluster_map(smem_u32(&csum[tid]), r)) : csum[tid];
    row_inv[tid] = v > 0.f ? __fdiv_rn(1.0f, v) : 0.f;
  }
  __syncthreads();
  // ---- 3. p V
  constexpr int NA = HI ? 8 : 4;                           // accumulator tiles per 64 columns
  float acc[DB][NA][4];
#pragma unroll
  for (int s = 0; s < DB; ++s)
#pragma unroll
    for (int i = 0; i < NA; ++i) acc[s][i][0] = acc[s][i][1] = acc[s][i][2] = acc[s][i][3] = 0.f;
  if (warp == kSdpaDecodeWarps) { produce(n_early, 2 * nblk); __syncwarp(); }
  else {
    const float inv_lo = row_inv[g], inv_hi = row_inv[g + 8];
    for (int n = 0; n < nblk; ++n) {
      const int u = nblk + n, slot = u % kSdpaDecodeSlots;
      if (ok) ok = __all_sync(0xffffffffu, mbar_wait(full(slot), (uint32_t)(u / kSdpaDecodeSlots) & 1u));
      if (!ok) { if (lane == 0) { s_err = 1; report_status(a.status, 43); } break; }
      const int kw = n * 128 + warp * 16;
      uint4 vr[4][DB];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int row = warp * 16 + 2 * t + (r & 1) + (r >> 1) * 8;
#pragma unroll
        for (int s = 0; s < DB; ++s) vr[r][s] = ld_shared_v4(ring + (uint32_t)slot * kSlot + (uint32_t)(s * 16384 + row * 128 + ((g ^ (row & 7)) << 4)));
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty(slot));
      uint32_t p0 = 0, p1 = 0, p2 = 0, p3 = 0;             // probabilities of rows g (p0: keys 2t.., p2: 2t + 8..) and g + 8 (p1, p3)
      if (g < S) {
        const float *sr = sc + (size_t)g * a.sc_stride + kw + 2 * t;
        const float2 x = *reinterpret_cast<const float2 *>(sr), y = *reinterpret_cast<const float2 *>(sr + 8);
        p0 = pack_bf16x2(__fmul_rn(x.x, inv_lo), __fmul_rn(x.y, inv_lo)); p2 = pack_bf16x2(__fmul_rn(y.x, inv_lo), __fmul_rn(y.y, inv_lo));
      }
      if (HI && g + 8 < S) {
        const float *sr = sc + (size_t)(g + 8) * a.sc_stride + kw + 2 * t;
        const float2 x = *reinterpret_cast<const float2 *>(sr), y = *reinterpret_cast<const float2 *>(sr + 8);
        p1 = pack_bf16x2(__fmul_rn(x.x, inv_hi), __fmul_rn(x.y, inv_hi)); p3 = pack_bf16x2(__fmul_rn(y.x, inv_hi), __fmul_rn(y.y, inv_hi));
      }
#pragma unroll
      for (int s = 0; s < DB; ++s) {
        const uint32_t w0[4] = {vr[0][s].x, vr[0][s].y, vr[0][s].z, vr[0][s].w}, w1[4] = {vr[1][s].x, vr[1][s].y, vr[1][s].z, vr[1][s].w};
        const uint32_t w2[4] = {vr[2][s].x, vr[2][s].y, vr[2][s].z, vr[2][s].w}, w3[4] = {vr[3][s].x, vr[3][s].y, vr[3][s].z, vr[3][s].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          // columns 8 g + 2 i and 8 g + 2 i + 1 of this set, keys (2t, 2t + 1) and (2t + 8, 2t + 9)
          const uint32_t e0 = __byte_perm(w0[i], w1[i], 0x5410u), o0 = __byte_perm(w0[i], w1[i], 0x7632u);
          const uint32_t e1 = __byte_perm(w2[i], w3[i], 0x5410u), o1 = __byte_perm(w2[i], w3[i], 0x7632u);
          if constexpr (HI) {
            mma_bf16_16816(acc[s][(2 * i) % NA], p0, p1, p2, p3, e0, e1);
            mma_bf16_16816(acc[s][(2 * i + 1) % NA], p0, p1, p2, p3, o0, o1);
          } else mma_bf16_16816(acc[s][i], e0, o0, e1, o1, p0, p2);
        }
      }
    }
  }
  __syncthreads();                    // every warp has read its scores: the space takes the partial outputs
  // [8 warps][S][D] f32, then their sum in [0][S][D]
  float *red = sc;
  if (warp < kSdpaDecodeWarps) {
#pragma unroll
    for (int s = 0; s < DB; ++s)
#pragma unroll
      for (int i = 0; i < NA; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int row = HI ? g + 8 * (e >> 1) : 2 * t + (e & 1);
          const int d = HI ? s * 64 + (2 * t + (e & 1)) * 8 + i : s * 64 + g * 8 + 2 * i + (e >> 1);
          if (row < S && d < D) red[((size_t)warp * S + row) * D + d] = acc[s][i][e];
        }
  }
  __syncthreads();
  for (int i = tid; i < S * D; i += kSdpaDecodeThreads) {
    float v = red[i];
#pragma unroll
    for (int w = 1; w < kSdpaDecodeWarps; ++w) v += red[(size_t)w * S * D + i];
    red[i] = v;
  }
  csync();
  // ---- 4. sum over the cluster; the CTAs share the elements
  if (!s_err)
    for (int i = (int)crank * kSdpaDecodeThreads + tid; i < S * D; i += (int)csize * kSdpaDecodeThreads) {
      float v = 0.f;
      if (csize > 1) { for (uint32_t r = 0; r < csize; ++r) v += ld_cluster_f32(cluster_map(smem_u32(red + i), r)); }
      else v = red[i];
      const int row = i / D, d = i - row * D;
      a.out[(int64_t)b * a.ob + (int64_t)h * a.oh + (int64_t)row * a.os + d] = (uint16_t)(pack_bf16x2(v, 0.f) & 0xFFFFu);
    }
  if (csize > 1) cluster_sync_all();  // nobody leaves while a neighbour may still read its shared memory
  if (s_err) { for (int i = 0; i < 64; ++i) __nanosleep(20000); }      // copies still in flight land before shared memory is released
}

}  // namespace b200

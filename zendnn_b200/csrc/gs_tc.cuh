// W4A8 on the 5th-generation tensor cores: bf16 rows quantised per token to s8 x packed s4 weights with {G,N} scales, bf16 out, the contract of gs_gemm.cuh.  Exact
// integer sum per group, x weight scale and added in group order in f32 with one rounding (fused), x source scale once at the end: two
// roundings fewer per group than the scalar definition's product by product.
//
// As in skinny_gemm.cuh the operands change places: the MMA's M = 128 rows are 128 output columns, its N is a tile of BM rows of activations.
//   first warp     TMA: per block of 128 k one box of 8 KiB of codes ([128 columns][64 bytes], as they lie in memory); the last warp: the activations' box
//   warps 2-9      unpack: a thread takes one column's 64 bytes from the stage, two operations per four codes (a code goes to the high nibble of its
//                  byte, 16 x its value), and stores its 32 words to tensor memory, which is where the MMA takes its A operand from: no swizzle,
//                  no shared-memory round trip, and the activations are the only operand that shared memory feeds
//   warp 1         MMAs: kind::i8, K = 32 each; the sum of a group (32, 64 or a multiple of 128 k) has accumulator columns of its own
//   warps 10-      scale: a thread owns one output column and 8, 16 or 32 rows; per group it reads their sums, converts, multiplies by the column's
//                  scale (a ring that each thread fills for itself with cp.async) and adds, on packed f32x2 arithmetic
// Bound by what each warp does per block besides its work: a barrier's round trip, an issue of copies or MMAs, a fence take 50 to 150 clocks each, 300 ns a
// block where HBM would deliver one in 100.  So the unpackers work in two sets, the groups of a block share barriers, and codes and activations have a
// producer each (one set, one producer and a barrier per group: 840 ns).  M = 64, K = 4096, us, against gs_gemm_kernel with mma.sync: N = 11008 92 -> 21 (groups
// of 128), 232 -> 36 (32); N = 4096 41 -> 12; M = 512, N = 11008 381 -> 72.
// Few tiles: a cluster shares a tile's groups and adds f32 partial sums through distributed shared memory in the order of its ranks.
// Every wait is bounded, as in tc_gemm.cuh.
#pragma once
#include "common.cuh"
#include "mbar.cuh"
#include "tc_gemm.cuh"
#include "gs_gemm.cuh"

namespace b200 {

constexpr int kGsTcMaxStages = 20;
constexpr int kGsTcScaleSlots = 16;           // weight scales in flight per thread
constexpr int kGsTcMaxSplits = 8;

struct GsTcArgs {
  int M, N, k_blocks;         // k_blocks: blocks of 128 k (the last one may be short where GPB > 1)
  int group_blocks;           // blocks per group (GPB == 1)
  int G;
  int n_tiles, m_tiles, splits;
  int stages;
  const float *sa;            // [M]
  const float *sw;            // [G, N]
  int early;                  // codes and weight scales may be read before the kernel in front has finished
  int32_t *status;
  int test_no_loads;          // test hook, see TcGemmArgs
};

// BM: rows of a tile; GPB: groups per 128 k (4, 2, or 1: a group is a multiple of 128 k)
template <int BM, int GPB> struct GsTcShape {
  static constexpr int kScaleWarps = BM >= 64 ? 16 : 8;
  static constexpr int kCols = BM * 4 / kScaleWarps;          // accumulator columns (rows of the source) per thread
  static constexpr int kThreads = 32 * (11 + kScaleWarps);
  // groups that are published and scaled together: each barrier round of a warp costs 200 to 400 clocks, as much as the work on a group
  static constexpr int kSet = GPB == 1 ? 1 : (BM <= 32 ? GPB : (BM == 64 ? 2 : 1));
  // tensor memory: sums of kSets sets (BM columns a group) and unpacked weight blocks (32 columns each)
  static constexpr int kSets = BM == 128 ? 3 : (BM == 64 ? (GPB == 1 ? 4 : 3) : (kSet == 1 ? 8 : 8 / kSet));
  static constexpr int kWBufs = (512 - kSets * kSet * BM) / 32;
  static constexpr int kStage = 8192 + BM * 128;
  static constexpr int kTail = kScaleWarps * 32 * (kGsTcScaleSlots + 8) * 4;      // behind the ring: weight scales, outputs on their way
};

__device__ __forceinline__ void tc_mma_i8_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.b32 p, %4, 0;\nelect.sync _|q, 0xffffffff;\n"
               "@q tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n}"
               ::"r"(d_tmem), "r"(a_tmem), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
                 "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]),
                 "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]) : "memory");
}
__device__ __forceinline__ void tc_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
template <int N> __device__ __forceinline__ void tc_ld_n(uint32_t taddr, uint32_t (&r)[N]) {
  if constexpr (N == 8) tc_ld8(taddr, r);
  else if constexpr (N == 16) tc_ld16(taddr, r);
  else tc_ld32(taddr, r);
}

// waits of a role's warps end the role on expiry (the other roles run into their own limits)
template <int BM, int GPB>
__global__ void __launch_bounds__(GsTcShape<BM, GPB>::kThreads, 1)
gs_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const GsTcArgs a, const EpiParams epi) {
  using Sh = GsTcShape<BM, GPB>;
  constexpr int SW = Sh::kScaleWarps, NC = Sh::kCols, PG = Sh::kSet, NA = Sh::kSets, NW = Sh::kWBufs, NL = NC < 16 ? NC : 16;       // NL: sums read at a time
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[3 * kGsTcMaxStages + 2 * NA];
  __shared__ uint32_t tmem_base_slot;
  __shared__ volatile int s_err;
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const int S = a.stages;
  const uint32_t tail0 = smem0 + (uint32_t)S * Sh::kStage;
  const uint32_t bar0 = smem_u32(bars);
  auto codes = [&](int s) { return bar0 + 8u * (uint32_t)s; };                              // the stage's codes have landed
  auto ready = [&](int s) { return bar0 + 8u * (uint32_t)(kGsTcMaxStages + s); };           // its activations have landed and its codes are unpacked
  auto done = [&](int s) { return bar0 + 8u * (uint32_t)(2 * kGsTcMaxStages + s); };        // the MMAs of the block have read both
  auto acc_full = [&](int i) { return bar0 + 8u * (uint32_t)(3 * kGsTcMaxStages + i); };
  auto acc_free = [&](int i) { return bar0 + 8u * (uint32_t)(3 * kGsTcMaxStages + NA + i); };

  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
    for (int s = 0; s < S; ++s) { mbar_init(codes(s), 1); mbar_init(ready(s), 5); mbar_init(done(s), 1); }
    for (int i = 0; i < NA; ++i) { mbar_init(acc_full(i), 1); mbar_init(acc_free(i), SW); }
    s_err = 0;
    mbar_fence_init();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_slot, tmem_w = tmem + (uint32_t)(NA * PG * BM);
  // (behind the allocation: a dependent's CTA on this SM can then not take tensor memory that this one still waits for)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  // this CTA's tiles (rows of the source fastest: row tiles that share a column tile run together), and its share of the groups
  const int tiles = a.n_tiles * a.m_tiles;
  const int crank = a.splits > 1 ? (int)(blockIdx.x % (unsigned)a.splits) : 0;
  const int tile0 = (int)blockIdx.x / a.splits, tile_step = a.splits > 1 ? tiles : (int)gridDim.x;
  const int gb = GPB == 1 ? a.group_blocks : 1, units = a.k_blocks / gb;              // (a unit: blocks that hold whole groups)
  const int kb0 = (int)((long long)crank * units / a.splits) * gb, kb1 = (int)((long long)(crank + 1) * units / a.splits) * gb;
  const int g0 = GPB == 1 ? kb0 / gb : kb0 * GPB, g1 = GPB == 1 ? kb1 / gb : min(a.G, kb1 * GPB);

  if (warp == 0 || warp == Sh::kThreads / 32 - 1) {
    // ------------------------------------------------------------------ producers: codes, activations (a warp walks, one elected lane issues)
    const bool acts = warp != 0;
    int pre = 0;
    if (!acts && a.early && !a.test_no_loads && tile0 < tiles) {
      // the first ring of codes is requested before the activations exist
      pre = min(S, kb1 - kb0);
      const int y = (tile0 / a.m_tiles) * 16;
      if (elect_one())
        for (int i = 0; i < pre; ++i) {
          mbar_expect_tx(codes(i), 8192u);
          tma_load_2d(smem0 + (uint32_t)i * Sh::kStage, &map_w, (kb0 + i) * 128, y, codes(i));
        }
      __syncwarp();
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    bool ok = true;
    int s = 0; uint32_t ph = 0;
    for (int tile = tile0; tile < tiles && !a.test_no_loads; tile += tile_step) {
      const int nt = tile / a.m_tiles, y = nt * 16, m0 = (tile - nt * a.m_tiles) * BM;
      for (int kb = kb0; kb < kb1; ++kb) {
        const uint32_t dst = smem0 + (uint32_t)s * Sh::kStage;
        if (pre == 0 && !mbar_wait_warp(done(s), ph ^ 1u)) { ok = false; break; }
        if (elect_one()) {
          if (acts) {
            mbar_expect_tx(ready(s), (uint32_t)(BM * 128));
            tma_load_2d(dst + 8192u, &map_a, kb * 128, m0, ready(s));
          } else if (pre == 0) {
            mbar_expect_tx(codes(s), 8192u);
            tma_load_2d(dst, &map_w, kb * 128, y, codes(s));
          }
        }
        __syncwarp();
        if (pre > 0) --pre;
        if (++s == S) { s = 0; ph ^= 1u; }
      }
      if (!ok) break;
    }
    if (!ok && lane == 0) { s_err = 1; report_status(a.status, 51); }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (the warp walks, one elected lane issues)
    const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BM >> 3) << 17) | (8u << 24);      // s32 += s8 x s8, M = 128, N = BM
    int s = 0, b = 0, acc = 0; uint32_t ph = 0, aph = 0;
    bool ok = true;
    auto wait2 = [&](uint32_t bar, uint32_t parity, uint32_t bar2, uint32_t parity2) {        // both first tries in flight
      const uint32_t t1 = mbar_try_wait(bar, parity), t2 = mbar_try_wait(bar2, parity2);
      if (__all_sync(0xffffffffu, t1 & t2)) return true;
      return mbar_wait_warp(bar, parity) && mbar_wait_warp(bar2, parity2);
    };
    auto next_acc = [&]() { if (++acc == NA) { acc = 0; aph ^= 1u; } };
    for (int tile = tile0; tile < tiles; tile += tile_step) {
      int in_group = 0;
      for (int kb = kb0; kb < kb1; ++kb) {
        const uint64_t da = make_smem_desc(smem0 + (uint32_t)s * Sh::kStage + 8192u);
        const uint32_t wa = tmem_w + (uint32_t)(b * 32);
        if constexpr (GPB == 1) {
          ok = in_group ? mbar_wait_warp(ready(s), ph) : wait2(ready(s), ph, acc_free(acc), aph ^ 1u);
          if (!ok) break;
          tc_fence_after();
          const uint32_t d = tmem + (uint32_t)(acc * BM);
          const bool last = in_group == gb - 1;
#pragma unroll
          for (int k = 0; k < 4; ++k) tc_mma_i8_ts(d, wa + (uint32_t)(k * 8), da + (uint64_t)(k * 2), idesc, (in_group | k) ? 1u : 0u);
          tc_commit(done(s));
          if (last) tc_commit(acc_full(acc));
          if (last) { in_group = 0; next_acc(); } else ++in_group;
        } else {
          constexpr int KS = 4 / GPB;
#pragma unroll
          for (int h = 0; h < GPB / PG; ++h) {
            if (!ok || (h > 0 && kb * GPB + h * PG >= a.G)) continue;
            ok = h ? mbar_wait_warp(acc_free(acc), aph ^ 1u) : wait2(ready(s), ph, acc_free(acc), aph ^ 1u);
            if (!ok) continue;
            tc_fence_after();
            const bool last = h == GPB / PG - 1 || kb * GPB + (h + 1) * PG >= a.G;
            // (past the last group the stage holds zeros, and nobody reads the sums)
#pragma unroll
            for (int k = 0; k < PG * KS; ++k) {
              const int kk = h * PG * KS + k;
              tc_mma_i8_ts(tmem + (uint32_t)((acc * PG + k / KS) * BM), wa + (uint32_t)(kk * 8), da + (uint64_t)(kk * 2), idesc, k % KS ? 1u : 0u);
            }
            tc_commit(acc_full(acc));
            if (last) tc_commit(done(s));
            next_acc();
          }
          if (!ok) break;
        }
        if (++s == S) { s = 0; ph ^= 1u; }
        if (++b == NW) b = 0;
      }
      if (!ok) break;
    }
    if (!ok && lane == 0) { s_err = 1; report_status(a.status, 52); }
  } else if (warp < 10) {
    // ------------------------------------------------------------------ unpack: thread = column of the tile, two sets of four warps in turn
    const int q = warp & 3, col = q * 32 + lane, set = (warp - 2) >> 2;
    const uint32_t src = (uint32_t)((col >> 3) * 512 + (col & 7) * 32);
    // (the two 16-byte halves of a column's 32 bytes are read in opposite order by every other four columns: no bank conflicts)
    const uint32_t flip = (uint32_t)((col >> 2) & 1) * 16u;
    int s = set, b = set, sf = set; uint32_t ph = 0, phf = 0;            // sf, phf: the block whose tensor-memory words come next
    bool ok = true;
    const int mine = tile0 < tiles ? ((tiles - 1 - tile0) / tile_step + 1) * (kb1 - kb0) : 0;       // blocks of this CTA
    for (int n = set; n < mine; n += 2) {
      if (!mbar_wait_warp(codes(s), ph)) { ok = false; break; }
      const uint32_t p = smem0 + (uint32_t)s * Sh::kStage + src;
      const uint4 v0 = ld_shared_v4(p + flip), v1 = ld_shared_v4(p + (flip ^ 16u)), v2 = ld_shared_v4(p + 256u + flip), v3 = ld_shared_v4(p + 256u + (flip ^ 16u));
      const uint4 w0 = flip ? v1 : v0, w1 = flip ? v0 : v1, w2 = flip ? v3 : v2, w3 = flip ? v2 : v3;
      const uint32_t w[16] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w, w2.x, w2.y, w2.z, w2.w, w3.x, w3.y, w3.z, w3.w};
      uint32_t r[32];
#pragma unroll
      for (int i = 0; i < 16; ++i) { r[2 * i] = (w[i] << 4) & 0xF0F0F0F0u; r[2 * i + 1] = w[i] & 0xF0F0F0F0u; }
      if (n >= NW) {
        if (!mbar_wait_warp(done(sf), phf)) { ok = false; break; }
        if ((sf += 2) >= S) { sf -= S; phf ^= 1u; }
        tc_fence_after();
      }
      __syncwarp();
      tc_st32(tmem_w + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * 32), r);
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ready(s));
      if ((s += 2) >= S) { s -= S; ph ^= 1u; }
      if ((b += 2) >= NW) b -= NW;
    }
    if (!ok && lane == 0) { s_err = 1; report_status(a.status, 53); }
  } else {
    // ------------------------------------------------------------------ scale and add: thread = column of the tile, NC rows
    const int q = warp & 3, part = (warp - 10) >> 2, col = q * 32 + lane, tid = threadIdx.x - 320;
    const uint32_t ring = tail0 + (uint32_t)tid * 4u, outb = ring + (uint32_t)(kGsTcScaleSlots * SW * 32 * 4);
    constexpr uint32_t kSlot = SW * 32 * 4;
    // load side of the weight scales: a set of groups at a time, all slots but one set's ahead, across tiles
    constexpr int LA = kGsTcScaleSlots / PG - 1;
    if (!a.early) asm volatile("griddepcontrol.wait;" ::: "memory");
    int l_tile = tile0, l_g = g0, l_slot = 0;
    const float *l_p = nullptr;
    auto l_set = [&]() { l_p = a.sw + (int64_t)g0 * a.N + min((l_tile / a.m_tiles) * 128 + col, a.N - 1); };
    l_set();
    auto issue = [&]() {
      if (l_tile < tiles) {
#pragma unroll
        for (int j = 0; j < PG; ++j)
          if (j == 0 || l_g + j < g1) gs_cp_async<4>(ring + (uint32_t)(l_slot + j) * kSlot, l_p + (int64_t)j * a.N);
        l_p += (int64_t)PG * a.N;
        if ((l_g += PG) >= g1) { l_g = g0; l_tile += tile_step; l_set(); }
        l_slot = l_slot + PG == kGsTcScaleSlots ? 0 : l_slot + PG;
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll 1
    for (int i = 0; i < LA; ++i) issue();
    if (a.early) asm volatile("griddepcontrol.wait;" ::: "memory");
    const uint32_t tq = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(part * NC);
    const EpiCtx cx = epi_ctx(epi, 0);
    int acc = 0, c_slot = 0; uint32_t aph = 0;
    bool ok = true;
    for (int tile = tile0; tile < tiles && ok; tile += tile_step) {
      const int nt = tile / a.m_tiles, m0 = (tile - nt * a.m_tiles) * BM + part * NC, n = nt * 128 + col;
      uint64_t f2[NC / 2];
#pragma unroll
      for (int i = 0; i < NC / 2; ++i) f2[i] = 0ull;
      for (int g = g0; g < g1; g += PG) {
        issue();
        asm volatile("cp.async.wait_group %0;" ::"n"(LA) : "memory");
        uint64_t w2[PG];
#pragma unroll
        for (int j = 0; j < PG; ++j) {
          const float w = (j == 0 || g + j < g1) ? __uint_as_float(lds4(ring + (uint32_t)(c_slot + j) * kSlot)) : 0.f;
          w2[j] = f32x2_pack(w, w);
        }
        c_slot = c_slot + PG == kGsTcScaleSlots ? 0 : c_slot + PG;
        if (!mbar_wait_warp(acc_full(acc), aph)) { ok = false; break; }
        tc_fence_after();
        __syncwarp();
        const uint32_t ta = tq + (uint32_t)(acc * PG * BM);
        constexpr int NH = NC / NL;
#pragma unroll
        for (int c = 0; c < NH; ++c) {
          uint32_t r[PG][NL];
#pragma unroll
          for (int j = 0; j < PG; ++j) tc_ld_n<NL>(ta + (uint32_t)(j * BM + c * NL), r[j]);
          tc_wait_ld();
          if (c == NH - 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_free(acc));
          }
#pragma unroll
          for (int j = 0; j < PG; ++j)
#pragma unroll
            for (int i = 0; i < NL / 2; ++i)
              f2[c * NL / 2 + i] = f32x2_fma(f32x2_pack((float)(int32_t)r[j][2 * i], (float)(int32_t)r[j][2 * i + 1]), w2[j], f2[c * NL / 2 + i]);
        }
        if (++acc == NA) { acc = 0; aph ^= 1u; }
      }
      ok = __all_sync(0xffffffffu, ok) != 0;
      if (!ok) break;
      if (a.splits > 1) {
        // partial sums [row][128 columns] over the ring: every copy into it has been consumed
#pragma unroll
        for (int i = 0; i < NC / 2; ++i) {
          float x0, x1;
          f32x2_unpack(f2[i], x0, x1);
          const uint32_t at = smem0 + (uint32_t)(((part * NC + 2 * i) * 128 + col) * 4);
          asm volatile("st.shared.f32 [%0], %1;" ::"r"(at), "f"(x0) : "memory");
          asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + 512u), "f"(x1) : "memory");
        }
      } else {
        // eight rows at a time through words of its own in shared memory, so that the post-ops exist once
#pragma unroll
        for (int c = 0; c < NC / 8; ++c) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float x0, x1;
            f32x2_unpack(f2[c * 4 + i], x0, x1);
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(outb + (uint32_t)(2 * i) * kSlot), "f"(x0) : "memory");
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(outb + (uint32_t)(2 * i + 1) * kSlot), "f"(x1) : "memory");
          }
#pragma unroll 1
          for (int i = 0; i < 8; ++i) {
            const int m = m0 + c * 8 + i;
            if (m >= a.M || n >= a.N) continue;
            const float x = epi_finish(epi, cx, __fmul_rn(__uint_as_float(lds4(outb + (uint32_t)i * kSlot)), a.sa[m] * 0.0625f), m, n);
            reinterpret_cast<uint16_t *>(epi.dst)[(int64_t)m * epi.ldc + n] = f32_to_bf16_bits(x);
          }
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (!ok && lane == 0) { s_err = 1; report_status(a.status, 54); }
  }

  if (a.splits > 1) {
    tc_fence_before();
    cluster_sync_all();
    const bool healthy = __shfl_sync(0xffffffffu, s_err ? 0 : 1, 0) != 0;
    if (warp >= 10 && warp < 10 + SW && healthy) {
      const int nt = tile0 / a.m_tiles, m_first = (tile0 - nt * a.m_tiles) * BM, n4 = nt * 128 + lane * 4;
      const int rows = min(BM, a.M - m_first);
      const EpiCtx cx = epi_ctx(epi, 0);
      const bool whole = n4 + 4 <= a.N && ((reinterpret_cast<uintptr_t>(epi.dst) | (uintptr_t)(epi.ldc * 2)) & 7) == 0;
      for (int r = crank + a.splits * (warp - 10); r < rows && n4 < a.N; r += SW * a.splits) {
        const uint32_t own = smem0 + (uint32_t)(r * 512 + lane * 16);
        float x[4] = {0.f, 0.f, 0.f, 0.f};
        uint4 v[kGsTcMaxSplits];
#pragma unroll
        for (int j = 0; j < kGsTcMaxSplits; ++j) if (j < a.splits) v[j] = ld_cluster_v4(cluster_map(own, (uint32_t)j));
#pragma unroll
        for (int j = 0; j < kGsTcMaxSplits; ++j)
          if (j < a.splits) {
            const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = j ? __fadd_rn(x[i], __uint_as_float(w[i])) : __uint_as_float(w[i]);
          }
        const int m = m_first + r;
        const float s_row = a.sa[m] * 0.0625f;
        uint32_t y[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float z = n4 + i < a.N ? epi_finish(epi, cx, __fmul_rn(x[i], s_row), m, n4 + i) : 0.f;
          y[i] = f32_to_bf16_bits(z);
        }
        uint16_t *o = reinterpret_cast<uint16_t *>(epi.dst) + (int64_t)m * epi.ldc + n4;
        if (whole) *reinterpret_cast<uint2 *>(o) = make_uint2(y[0] | (y[1] << 16), y[2] | (y[3] << 16));
        else {
#pragma unroll
          for (int i = 0; i < 4; ++i) if (n4 + i < a.N) o[i] = (uint16_t)y[i];
        }
      }
    }
    cluster_sync_all();       // nobody leaves while a neighbour may still read its shared memory
  }
  tc_fence_before();
  __syncthreads();
  if (s_err) {
    for (int i = 0; i < 64; ++i) __nanosleep(20000);     // copies still in flight land before shared memory is released
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

}  // namespace b200

// tcgen05 W8A8 GEMM for sm_100a: the prefill-sized and grouped (MoE) form of the INT8 GEMM that
// the reference delegates to its backend (matmul/backends/aocl/aocl_kernel.cpp:1190-1301) and, for
// group_matmul_direct, to its tile micro-kernel (matmul/group_matmul/custom_kernel/ukernel/
// int8_microkernel.hpp:39-56) under a CPU scheduler (matmul/group_matmul/group_matmul_dispatch.cpp).
//
// One persistent CTA per SM, 608 threads, four roles:
//   warp 0     TMA producer: per K block of 128 bytes, one [128 x 128 B] box of A and one
//              [BN x 128 B] box of the packed weight into a ring of shared-memory stages
//              (SWIZZLE_128B, no multicast), completion on an mbarrier.
//   warp 1     MMA issuer: one lane issues tcgen05.mma.cta_group::1.kind::i8 (M=128, N=BN, K=32),
//              four per stage, accumulating s32 in tensor memory; tcgen05.commit releases the
//              stage and, after the last K block, publishes the accumulator.
//   warps 2-17 epilogue: tcgen05.ld the accumulator (one TMEM lane = one output row per thread, four
//              warps per lane quadrant, each taking a share of the tile's 32-column chunks), dequantise / bias /
//              post-ops (or gated activation) and store; results leave through a small per-warp
//              shared-memory block so that every store instruction writes whole 32-byte sectors of
//              16 rows.  Two accumulator buffers (2 x BN <= 512 TMEM columns) let the epilogue of tile i
//              overlap the MMAs of tile i+1.
//   warp 18    operand warp: runs one tile ahead of the epilogue and puts everything the epilogue needs
//              from global memory into double-buffered shared memory: the tile's coordinates and output
//              pointer, the per-column operands of its BN columns and the source scales of its 128 rows.
//              The epilogue warps then read only tensor memory and shared memory.
// Tile order: column-tile-major (CTAs running together share a weight tile through L2), or, when the
// activations are the large operand and a group's weight stays in L2, row-tile-major (n_fastest).
// Shared memory is the busiest resource (TMA writes the operands, the tensor core reads them back), so
// the epilogue keeps its own shared-memory traffic small.
// Grouped form: A is one [rows x K] matrix holding every expert's rows back to back; row offsets
// and the cumulative tile counts live in device memory, so no host round trip is needed after routing.
// Pair form (tc_gemm_kernel<false, true>, large plain and grouped GEMMs): clusters of two CTAs on neighbouring SMs
// work on one [256 x BN] tile with tcgen05.mma.cta_group::2.  Each CTA loads its own 128 rows of A and its own half
// (BN/2 rows) of the weight tile with plain, non-multicast TMA copies that complete on the leader CTA's barrier; the
// leader's MMA warp issues M256 MMAs for both, the tensor cores exchange the weight halves between the two shared
// memories themselves, and each CTA's epilogue warps finish the 128 rows whose accumulators sit in its own tensor
// memory.  Per MMA a CTA's shared memory takes half the weight bytes it takes in the single-CTA form, and shared-memory
// bandwidth (copy engine writing, tensor core reading) is what bounds the single-CTA form.
// Every wait is bounded: on expiry the kernel records a code in *status and leaves.
#pragma once
#include <cuda.h>
#include "common.cuh"
#include "mbar.cuh"
#include "pack_kernels.cuh"

namespace b200 {

constexpr int kTcBM = 128;
constexpr int kTcBK = 128;               // bytes of K per stage row (one 128-byte swizzle span)
#ifndef B200_TC_EPI_WARPS
#define B200_TC_EPI_WARPS 16
#endif
constexpr int kTcEpiWarps = B200_TC_EPI_WARPS;      // a multiple of 4: each warp may only read its own quadrant of TMEM lanes
constexpr int kTcEpiParts = kTcEpiWarps / 4;          // warps per lane quadrant, each taking a share of the tile's columns
constexpr int kTcThreads = 96 + 32 * kTcEpiWarps;   // producer warp + MMA warp + epilogue warps + operand warp
constexpr int kTcSmemBudget = 200 * 1024; // stage ring

struct TcGroupDesc {   // per expert, device memory (grouped form with caller-owned outputs)
  const void *wei_scale;
  const int32_t *colsum;
  const void *bias;
  void *dst;
  int64_t ldc;
};

struct TcGemmArgs {
  int n_groups;               // 1: plain GEMM
  int M_total;                // rows of A
  int N;                      // packed columns to produce (N, or 2*I in gated form)
  int k_blocks;               // Kp / 128
  int BN, stages;
  int n_tiles;                // ceil(N / BN)
  int m_tiles_plain;          // plain form: ceil(M / 128), or ceil(M / 256) in the pair form
  const int32_t *row_off;     // grouped: [n_groups+1] first row of each group (device)
  const int32_t *tile_prefix; // grouped: [n_groups+1] cumulative row tiles (128 rows each; 256 in the pair form) (device)
  const CUtensorMap *maps_b;  // grouped: one map per group (device memory); plain: null
  const TcGroupDesc *groups;  // grouped, optional: per-group epilogue pointers (local row index)
  int a_unsigned;
  int gated;                  // packed gate/up interleave: 0, 1 or 2 (see pack_kernels.cuh)
  int fast_act;               // FA_* code: which specialised epilogue loop to run
  int dbg;                    // timing experiments, only in builds with B200DNN_TIMING_EXPERIMENTS (results invalid):
                              // 1 no epilogue work, 2 tensor-memory loads only, 3 no stores; otherwise 0
  int shared_dst;             // every group writes epi.dst at its global row (set by the caller); plain GEMM: 1
  int tma_store;              // bf16 results of full 32-row blocks leave through TMA stores (map_c covers the shared destination)
  int test_no_loads;          // test hook: the producer issues no copies, so every wait on data runs out (bounded) and the
                              // kernel must leave with a status code and a usable context
  int k_splits;               // split form (tc_gemm_kernel<true>): the CTAs of a cluster each take a share of the K blocks of one
                              // tile and add their int32 partial sums through distributed shared memory (exact in any order)
  int n_fastest;              // tile order: 0 = all row tiles of a column tile first, 1 = all column tiles of a row tile first
  int pair;                   // pair form (tc_gemm_kernel<false, true>): row tiles are 256 rows, m_tiles_plain / tile_prefix count those
  int f16;                    // bf16 x bf16 form (tc_gemm_kernel<.., .., true>): kind::f16 MMAs, f32 accumulators, no scales
  int32_t *status;            // device word: 0 ok
  unsigned long long *stamps; // timing experiments only (builds with B200DNN_TIMING_EXPERIMENTS): 8 timer values per CTA; else null
};

#ifdef B200DNN_TIMING_EXPERIMENTS
#define TC_STAMP(i) do { if (a.stamps) { unsigned long long t_; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_)); \
                                          a.stamps[(size_t)blockIdx.x * 8 + (i)] = t_; } } while (0)
#else
#define TC_STAMP(i) do { } while (0)
#endif

// ---------------------------------------------------------------------------------------- PTX
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
// weight box from the block-interleaved layout: coordinates {byte 0, row-in-group 0, K block, row group}
__device__ __forceinline__ void tma_load_wt(uint32_t dst, const CUtensorMap *map, int kblock, int group, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
               ::"r"(dst), "l"(map), "r"(0), "r"(0), "r"(kblock), "r"(group), "r"(bar) : "memory");
}
// pair form: the copy lands in this CTA's shared memory, its bytes are counted on the barrier `bar` of the leader CTA
// (a shared::cluster address); no multicast
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_wt_pair(uint32_t dst, const CUtensorMap *map, int kblock, int group, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
               ::"r"(dst), "l"(map), "r"(0), "r"(0), "r"(kblock), "r"(group), "r"(bar) : "memory");
}
// MMAs and commits below are issued by a converged warp: the instruction is predicated on the elected lane (always the same one) inside its asm statement.  With a
// branch around them the operands no longer count as the same in every lane, and each MMA first moves them: a 128-byte block of K (a wait, four MMAs, a commit) took 370
// clocks whatever the tile, in a loop of its own; as it is, 227 with N = 16 and the tensor pipe's own 257 with N = 128.
// completion of the pair's MMAs, signalled on the barrier at the same offset in both CTAs
__device__ __forceinline__ void tc_commit_pair(uint32_t bar) {
  asm volatile("{\n.reg .pred q;\nelect.sync _|q, 0xffffffff;\n@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n}"
               ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void tc_mma_i8_pair(uint32_t d_tmem, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.b32 p, %4, 0;\nelect.sync _|q, 0xffffffff;\n"
               "@q tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n}"
               ::"r"(d_tmem), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
// arrive on a barrier of another CTA of the cluster (shared::cluster address from cluster_map)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("{\n.reg .pred q;\nelect.sync _|q, 0xffffffff;\n@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_mma_i8(uint32_t d_tmem, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.b32 p, %4, 0;\nelect.sync _|q, 0xffffffff;\n"
               "@q tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}"
               ::"r"(d_tmem), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// 32 contiguous bytes of one row in one instruction: every lane writes a whole sector of its own row, so the stores of a
// warp are full sectors without any exchange between the lanes.  The address must be 32-byte aligned.
__device__ __forceinline__ void st_global_v8(void *p, const uint32_t (&v)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
__device__ __forceinline__ uint32_t cluster_ctarank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
// every thread of every CTA of the cluster; the cluster's CTAs are scheduled together, so the wait ends once each thread
// has left its own (bounded) waits
__device__ __forceinline__ void cluster_sync_all() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_arrive_all() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait_all() {
  __syncwarp();
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_map(uint32_t saddr, uint32_t rank) {
  uint32_t r; asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank)); return r;
}
__device__ __forceinline__ uint4 ld_cluster_v4(uint32_t caddr) {
  uint4 v; asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(caddr) : "memory");
  return v;
}
__device__ __forceinline__ uint4 ld_shared_v4(uint32_t saddr) {
  uint4 v; asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(saddr) : "memory");
  return v;
}
__device__ __forceinline__ void st_shared_v4(uint32_t saddr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(saddr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// bf16 x bf16 -> f32, M x N x 16 (32 bytes of K per instruction, as kind::i8)
__device__ __forceinline__ void tc_mma_bf16_pair(uint32_t d_tmem, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.b32 p, %4, 0;\nelect.sync _|q, 0xffffffff;\n"
               "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n}"
               ::"r"(d_tmem), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
__device__ __forceinline__ void tc_mma_bf16(uint32_t d_tmem, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.b32 p, %4, 0;\nelect.sync _|q, 0xffffffff;\n"
               "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
               ::"r"(d_tmem), "l"(da), "l"(db), "r"(idesc), "r"(accumulate) : "memory");
}

// K-major, SWIZZLE_128B shared-memory operand descriptor: 8-row groups 1024 B apart
// (stride byte offset), leading byte offset unused for swizzled K-major, descriptor version 1.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// instruction descriptor, kind::i8: D = s32, A = u8|s8, B = s8, both K-major, M = 128, N = BN
__host__ __device__ inline uint32_t make_idesc_i8(int a_unsigned, int BN, int M = kTcBM) {
  return (2u << 4) | ((a_unsigned ? 0u : 1u) << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// instruction descriptor, kind::f16: D = f32, A = B = bf16, both K-major
__host__ __device__ inline uint32_t make_idesc_bf16(int BN, int M = kTcBM) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

struct TileCoord { int g, row0, rows, m_local0, nt; };

// Same mapping computed by a whole warp: the group of a row tile is the number of prefix entries
// tile_prefix[1..n_groups) that are <= the tile index (empty groups repeat a prefix value and are skipped).
// tile_m: rows of a tile (128, or 256 in the pair form); sub: this CTA's first row inside the tile (pair form: 128 for
// the second CTA).  rows may be 0 for the second CTA of a pair at the end of a group.
__device__ __forceinline__ TileCoord tc_tile_warp(const TcGemmArgs &a, int tile, int m_tiles, int lane, int tile_m = kTcBM, int sub = 0) {
  TileCoord t;
  int mt;
  if (a.n_fastest) { mt = tile / a.n_tiles; t.nt = tile - mt * a.n_tiles; }
  else { t.nt = tile / m_tiles; mt = tile - t.nt * m_tiles; }
  if (!a.tile_prefix) {
    t.g = 0; t.m_local0 = mt * tile_m + sub; t.row0 = t.m_local0; t.rows = max(0, min(kTcBM, a.M_total - t.row0));
    return t;
  }
  int g = 0;
  for (int base = 1; base < a.n_groups; base += 32) {
    const int i = base + lane;
    const bool le = i < a.n_groups && a.tile_prefix[i] <= mt;
    g += __popc(__ballot_sync(0xffffffffu, le));
  }
  t.g = g;
  t.m_local0 = (mt - a.tile_prefix[g]) * tile_m + sub;
  t.row0 = a.row_off[g] + t.m_local0;
  t.rows = max(0, min(kTcBM, a.row_off[g + 1] - t.row0));
  return t;
}

struct TileMeta {          // what the epilogue needs to know about a tile, written by the operand warp
  int row0, rows, m_dst0, nt;
  void *dst; int64_t ldc;
  int has_bias;
};

// ---- epilogue arithmetic ---------------------------------------------------------------------------
// Post-op structure resolved on the host so that the per-element loop carries no dispatch.
enum : int { FA_GENERIC = -1, FA_NONE = 0, FA_RELU, FA_GELU_TANH, FA_GELU_ERF, FA_SIGMOID, FA_SWISH, FA_TANH };

// sigmoid-family activations through one exp and one reciprocal.  gelu_tanh uses the identity
// 0.5*x*(1+tanh(u)) = x / (1 + exp(-2u)), which has no cancellation for very negative u.
// exp(-a) = 2^(-a log2 e); x / (1 + e) = x * rcp(1 + e): an infinite e gives 0 times x.
constexpr float kTcNegLog2e = -1.44269504088896340736f;
__device__ __forceinline__ float tc_ex2(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float tc_rcp(float x) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float fast_sigmoid_mul(float x, float arg) {
  return __fmul_rn(x, tc_rcp(__fadd_rn(1.0f, tc_ex2(__fmul_rn(arg, kTcNegLog2e)))));
}

template <int ACT>
__device__ __forceinline__ float tc_act(const EpiParams &epi, float x, int m, int n) {
  if (ACT == FA_NONE) return x;
  if (ACT == FA_RELU) return fmaxf(x, 0.0f);
  if (ACT == FA_GELU_TANH) {
    const float c = 0.79788458347320556640625f, f = 0.044715f;
    const float inner = __fmul_rn(__fmul_rn(c, x), __fmaf_rn(__fmul_rn(f, x), x, 1.0f));
    return fast_sigmoid_mul(x, 2.0f * inner);
  }
  if (ACT == FA_GELU_ERF) return po_gelu_erf(x);
  if (ACT == FA_SIGMOID) return fast_sigmoid_mul(1.0f, x);
  if (ACT == FA_SWISH) return fast_sigmoid_mul(x, x);
  if (ACT == FA_TANH) return tanhf(x);
  for (int i = 0; i < epi.n_po; ++i) x = apply_postop(epi.po[i], x, m, n);
  return x;
}

__device__ __forceinline__ uint32_t pack_bf16x2(float lo, float hi) {
  // one instruction; same round-to-nearest-even as the reference's bit trick for every finite value
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return d;
}

// two f32 operations per instruction, each rounded as the scalar one
__device__ __forceinline__ uint64_t tc_pack2(float lo, float hi) { uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ void tc_unpack2(uint64_t r, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(r)); }
__device__ __forceinline__ uint64_t tc_mul2(uint64_t a, uint64_t b) { uint64_t d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ uint64_t tc_fma2(uint64_t a, uint64_t b, uint64_t c) { uint64_t d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ uint64_t tc_add2(uint64_t a, uint64_t b) { uint64_t d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }

// x / (1 + exp(-arg)) of two elements, arg2 already times -log2(e): the operations of fast_sigmoid_mul
__device__ __forceinline__ uint64_t tc_sigmoid_mul2(uint64_t x2, uint64_t arg2) {
  float a0, a1, b0, b1;
  tc_unpack2(arg2, a0, a1);
  tc_unpack2(tc_add2(tc_pack2(1.0f, 1.0f), tc_pack2(tc_ex2(a0), tc_ex2(a1))), b0, b1);
  return tc_mul2(x2, tc_pack2(tc_rcp(b0), tc_rcp(b1)));
}
// gelu_tanh as in tc_act, 1 + (f x) x in one rounding: the factor 2 of its argument is in the constant (exact).  Largest error against double for x from -6
// to 6: 3.6e-6 of the result (20 rows; 4.4e-6 with a rounding between the product and the sum).
__device__ __forceinline__ uint64_t tc_gelu_tanh2(uint64_t x2) {
  const uint64_t c2 = tc_pack2(0.79788458347320556640625f, 0.79788458347320556640625f), f2 = tc_pack2(0.044715f, 0.044715f);
  const uint64_t inner = tc_mul2(tc_mul2(c2, x2), tc_fma2(tc_mul2(f2, x2), x2, tc_pack2(1.0f, 1.0f)));
  return tc_sigmoid_mul2(x2, tc_mul2(inner, tc_pack2(2.0f * kTcNegLog2e, 2.0f * kTcNegLog2e)));
}
__device__ __forceinline__ uint64_t tc_swish2(uint64_t x2) { return tc_sigmoid_mul2(x2, tc_mul2(x2, tc_pack2(kTcNegLog2e, kTcNegLog2e))); }

struct TileCols {          // per-tile column operands staged in shared memory
  float ws[256];
  float bias[256];
  int32_t comp[256];
};

// Coalesced store of a [32 rows x 32 bytes] block that a warp holds one row per lane (v[0], v[1] = the row's
// two 16-byte pieces).  The block goes through the warp's 1 KiB of shared memory (pieces swapped on every
// second group of four rows so that both the writes and the reads are free of bank conflicts) and leaves
// as two instructions that each write 16 rows x 32 contiguous bytes (whole sectors), instead of 32
// scattered 16-byte pieces per instruction.
// g_row0: address of the block's first row; rows_valid: how many of the 32 rows exist.
__device__ __forceinline__ void tc_staging_free(int lane) {
  if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  __syncwarp();
}
__device__ __forceinline__ void warp_store_rows32(uint8_t *sbuf, const uint4 &v0, const uint4 &v1, uint8_t *g_row0, int64_t pitch_bytes,
                                                  int rows_valid, int lane) {
  tc_staging_free(lane);
  const int sw = (lane >> 2) & 1;
  *reinterpret_cast<uint4 *>(sbuf + lane * 32 + ((0 ^ sw) << 4)) = v0;
  *reinterpret_cast<uint4 *>(sbuf + lane * 32 + ((1 ^ sw) << 4)) = v1;
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int R = 16 * j + (lane >> 1), p = lane & 1;
    const uint4 val = *reinterpret_cast<const uint4 *>(sbuf + R * 32 + ((p ^ ((R >> 2) & 1)) << 4));
    if (R < rows_valid) *reinterpret_cast<uint4 *>(g_row0 + (int64_t)R * pitch_bytes + p * 16) = val;
  }
  __syncwarp();
}
// [32 rows x 64 bytes] as two such blocks
__device__ __forceinline__ void warp_store_rows64(uint8_t *sbuf, const uint4 (&v)[4], uint8_t *g_row0, int64_t pitch_bytes,
                                                  int rows_valid, int lane) {
  warp_store_rows32(sbuf, v[0], v[1], g_row0, pitch_bytes, rows_valid, lane);
  warp_store_rows32(sbuf, v[2], v[3], g_row0 + 32, pitch_bytes, rows_valid, lane);
}

// A destination without 16-byte alignment (an odd N or ldc): every lane writes its own row as aligned 32-byte pieces, put together in registers from eight words and
// the last of the eight before them.  Three (bf16: four) steps of selects shift the words by the row's distance from a 32-byte boundary; where a run
// of columns begins or ends inside a piece, its elements are stored one by one.  (Through a staging block, four rows of eight words an instruction, as before: 32 instructions
// and twice as many partial sectors.)  M = 3027, K = 1280, N = 7295, INT8: f32 75.5 -> 45.4 us, bf16
// 49.9 -> 37.6; whole sectors at N = 7296 take 40.4 and 28.7.
struct RowCarry { uint32_t w[8]; bool have; };      // the eight words in front of the next ones; have: they are this run's, and not all of them are stored
template <int STEP, int N>
__device__ __forceinline__ void shift_words(const uint32_t (&x)[N], bool on, uint32_t (&y)[N - STEP]) {      // y[i] = on ? x[i] : x[i + STEP]
#pragma unroll
  for (int i = 0; i < N - STEP; ++i) y[i] = on ? x[i] : x[i + STEP];
}
// words from s on, or the first n words, of an aligned piece: at most one store of each size
__device__ __forceinline__ void put_words_from(uint8_t *base, const uint32_t (&o)[8], int s) {
  if (s & 1) *reinterpret_cast<uint32_t *>(base + 4 * s) = s < 4 ? (s < 2 ? o[1] : o[3]) : (s < 6 ? o[5] : o[7]);
  const int s2 = (s + 1) & ~1;
  if (s2 & 2) *reinterpret_cast<uint2 *>(base + 4 * s2) = s2 < 4 ? make_uint2(o[2], o[3]) : make_uint2(o[6], o[7]);
  const int s4 = (s2 + 2) & ~3;
  if (s4 <= 4) *reinterpret_cast<uint4 *>(base + 16) = make_uint4(o[4], o[5], o[6], o[7]);
  if (s4 == 0) *reinterpret_cast<uint4 *>(base) = make_uint4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ void put_words_to(uint8_t *base, const uint32_t (&o)[8], int n) {
  const int h = n & 4, k = n & 6;
  if (h) *reinterpret_cast<uint4 *>(base) = make_uint4(o[0], o[1], o[2], o[3]);
  if (n & 2) *reinterpret_cast<uint2 *>(base + 4 * h) = h ? make_uint2(o[4], o[5]) : make_uint2(o[0], o[1]);
  if (n & 1) *reinterpret_cast<uint32_t *>(base + 4 * k) = k < 4 ? (k < 2 ? o[0] : o[2]) : (k < 6 ? o[4] : o[6]);
}
// A piece of eight words from x (seven words in front, then eight of which the first belongs at p).  Elements, PER to a word and the first of them `off` in front of p, from
// lo to hi - 1 are written; edge: the element that shares its word with one outside, where off is 1.
template <int PER>
__device__ __forceinline__ void put_piece(uint8_t *p, const uint32_t (&x)[15], int off, int lo, int hi, uint16_t edge) {
  const int r = (int)((reinterpret_cast<uintptr_t>(p) >> 2) & 7);
  uint32_t t[14], u[12], q[8];
  shift_words<1>(x, (r & 1) != 0, t);
  shift_words<2>(t, (r & 2) != 0, u);
  shift_words<4>(u, (r & 4) != 0, q);
  uint8_t *base = p - 4 * r;
  const int e0 = -r * PER - off;                           // first element of the piece
  if (e0 >= lo && e0 + 8 * PER <= hi) st_global_v8(base, q);
  else if (lo == 0 && e0 + 8 * PER <= hi) {                // the run begins in this piece
    if (PER == 2 && off) *reinterpret_cast<uint16_t *>(p + 2) = edge;
    put_words_from(base, q, r + off);
  } else if (lo < 0 && hi == 0) {                          // and here it ends
    put_words_to(base, q, r);
    if (PER == 2 && off) *reinterpret_cast<uint16_t *>(p) = edge;
  } else if (e0 >= lo && e0 < hi) {                        // the last columns of the matrix
    const int n = hi - e0, k = n / PER;
    put_words_to(base, q, k);
    if (PER == 2 && (n & 1)) {
      const uint32_t w = k < 4 ? (k < 2 ? (k < 1 ? q[0] : q[1]) : (k < 3 ? q[2] : q[3])) : (k < 6 ? (k < 5 ? q[4] : q[5]) : (k < 7 ? q[6] : q[7]));
      *reinterpret_cast<uint16_t *>(base + 4 * k) = (uint16_t)w;
    }
  } else if (e0 < hi) {
#pragma unroll 1
    for (int i = 0; i < 8; ++i) {
      const int e = e0 + i * PER;
      const uint32_t lo4 = i < 4 ? (i < 2 ? (i < 1 ? q[0] : q[1]) : (i < 3 ? q[2] : q[3])) : (i < 6 ? (i < 5 ? q[4] : q[5]) : (i < 7 ? q[6] : q[7]));
      uint8_t *at = base + 4 * i;
      if constexpr (PER == 1) { if (e >= lo && e < hi) *reinterpret_cast<uint32_t *>(at) = lo4; }
      else {
        if (e >= lo && e < hi) *reinterpret_cast<uint16_t *>(at) = (uint16_t)lo4;
        if (e + 1 >= lo && e + 1 < hi) *reinterpret_cast<uint16_t *>(at + 2) = (uint16_t)(lo4 >> 16);
      }
    }
  }
}
// sixteen 4-byte columns at p, of which the first n exist (n > 0); last: the run ends here.  (Eight columns a piece: sixteen at once held 23 words, and small results paid for
// it, INT8, f32 out, 371 x 419, K = 768 5.8 us before rows left as pieces, 6.5 with, 5.7 now; 313 x 518, K = 896 8.2, 8.65, 8.2.)
__device__ __forceinline__ void row_put32(uint8_t *p, const uint32_t (&w)[16], int n, bool last, bool row_ok, RowCarry &c) {
  auto put = [&](uint8_t *at, const uint32_t *u, const uint32_t *v, int lo, int hi) {
    uint32_t x[15];
#pragma unroll
    for (int i = 0; i < 15; ++i) x[i] = i < 7 ? u[i + 1] : v[i - 7];
    if (row_ok) put_piece<1>(at, x, 0, lo, hi, 0);
  };
  const uint32_t none[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
  put(p, c.w, w, c.have ? -7 : 0, n);
  put(p + 32, w, w + 8, -7, n - 8);
#pragma unroll
  for (int i = 0; i < 8; ++i) c.w[i] = w[8 + i];
  c.have = true;
  if (last) {
    put(p + 64, w + 8, none, -7, n - 16);
    c.have = false;
  }
}
// the same for sixteen bf16 columns (eight words)
__device__ __forceinline__ void row_put16(uint8_t *p, const uint32_t (&w)[8], int n, bool last, bool row_ok, RowCarry &c) {
  const int odd = (int)((reinterpret_cast<uintptr_t>(p) >> 1) & 1);
  auto put = [&](uint8_t *at, const uint32_t (&v)[8], int lo, int hi, uint32_t edge) {
    uint32_t x[15];          // words of the destination: an odd element in front moves all of them by half a word
#pragma unroll
    for (int i = 0; i < 15; ++i) {
      const uint32_t cur = i < 7 ? c.w[i + 1] : v[i - 7], prev = i < 8 ? c.w[i] : v[i - 8];
      x[i] = odd ? __funnelshift_l(prev, cur, 16) : cur;
    }
    if (row_ok) put_piece<2>(at - 2 * odd, x, odd, lo, hi, (uint16_t)edge);
  };
  // (no columns left: this ends the run, and the word that its last element shares with one outside is the last of those before)
  put(p, w, c.have ? -16 : 0, n, n > 0 ? w[0] : c.w[7] >> 16);
#pragma unroll
  for (int i = 0; i < 8; ++i) c.w[i] = w[i];
  c.have = true;
  if (last || n < 16) {
    const uint32_t none[8] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
    put(p + 32, none, -16, n - 16, c.w[7] >> 16);
    c.have = false;
  }
}

// the last columns of a row that starts on 16 bytes, n of eight (sixteen) words: nothing to shift.  (M = 3000, K = 1024, N = 1000, bf16: 9.1 us, through the
// shifts above 9.5, through a staging block 9.3.)
template <int W>
__device__ __forceinline__ void put_tail_words(uint8_t *p, const uint32_t (&w)[W], int n) {
#pragma unroll
  for (int v = 0; v < W / 4; ++v) {
    if (n >= 4 * v + 4) *reinterpret_cast<uint4 *>(p + 16 * v) = make_uint4(w[4 * v], w[4 * v + 1], w[4 * v + 2], w[4 * v + 3]);
    else {
#pragma unroll
      for (int i = 0; i < 3; ++i) if (4 * v + i < n) *reinterpret_cast<uint32_t *>(p + 16 * v + 4 * i) = w[4 * v + i];
    }
  }
}

// The same [32 rows x 32 bytes] block as one TMA store: the lanes write their rows to the staging block (plain row-major) and one lane hands it
// to the copy engine.  Keeps the result off the load/store path.  The engine reads the block while the warp works on the next one: every
// use of the block waits for that first (tc_staging_free).
__device__ __forceinline__ void warp_tma_store_rows32(uint8_t *sbuf, const uint4 &v0, const uint4 &v1, const CUtensorMap *map,
                                                      int x_bytes, int row, int lane) {
  tc_staging_free(lane);
  *reinterpret_cast<uint4 *>(sbuf + lane * 32) = v0;
  *reinterpret_cast<uint4 *>(sbuf + lane * 32 + 16) = v1;
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncwarp();
  if (lane == 0) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];"
                 ::"l"(map), "r"(x_bytes), "r"(row), "r"(smem_u32(sbuf)) : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  }
}

struct EpiStore {          // where this warp's rows of the current tile go
  uint8_t *sbuf;           // the warp's staging block
  uint8_t *g_row0;         // address of (first row of the warp, column 0) in the destination
  int64_t pitch_bytes;
  int rows_valid;          // rows of the warp's 32 that exist in this tile
  bool coalesce;           // destination 16-byte aligned: use the staged path
  bool v8;                 // destination and pitch 32-byte aligned: every lane stores 32-byte pieces of its own row directly
  bool row_ok;             // this lane's row exists
  const CUtensorMap *map_c;  // non-null: full blocks go out as TMA stores, coordinates (byte column, row)
  int row_c;               // row coordinate of the warp's first row in map_c
};

// Sixteen columns of one output row.  Results leave, in this order of preference, as 32-byte stores of the lane's own
// row (destination 32-byte aligned), through the warp's staging block (16-byte aligned), or element by element.
// accumulator -> f32 before bias: the dequantising chain of the INT8 forms, or the f32 sum of the bf16 form as it is
template <bool F16>
__device__ __forceinline__ float tc_acc_f32(uint32_t r, int comp, float s_src, float w) {
  if constexpr (F16) return __uint_as_float(r);
  else return __fmul_rn(__fmul_rn((float)((int32_t)r - comp), s_src), w);
}

template <bool F16>
__device__ __forceinline__ float tc_acc_to_f32(uint32_t r) {
  if constexpr (F16) return __uint_as_float(r);
  else return (float)(int32_t)r;
}

template <int ACT>
__device__ __forceinline__ void tc_act16(const EpiParams &epi, float (&x)[16], int m, int n) {
#pragma unroll
  for (int i = 0; i < 16; ++i) x[i] = tc_act<ACT>(epi, x[i], m, n + i);
}

// (Only the activation depends on fast_act: the loads before it and the stores behind it exist once.  With the whole chunk
// instantiated per activation the split form spilled hundreds of registers.)
template <bool F16>
__device__ __forceinline__ void tc_epi_half(int fast_act, const EpiParams &epi, const EpiCtx &cx, const uint32_t (&r)[16], const TileCols &tc,
                                            int c0, int pc, int N, int m_dst, bool has_bias, const EpiStore &es, int lane, RowCarry &carry, bool last) {
  const bool has_zp = !F16 && epi.has_zp != 0;
  const bool full = pc + 16 <= N;
  if (!F16 && epi.dst_dt == DT_S32) {
    int32_t y[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) y[i] = has_zp ? (int32_t)r[i] - tc.comp[c0 + i] : (int32_t)r[i];
    if (es.v8 && full) {
      if (es.row_ok) {
        uint8_t *o = reinterpret_cast<uint8_t *>(cx.dst) + ((int64_t)m_dst * cx.ldc + pc) * 4;
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          uint32_t v[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = (uint32_t)y[8 * p + i];
          st_global_v8(o + 32 * p, v);
        }
      }
    } else if (es.coalesce && full) {
      uint4 v[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) v[p] = make_uint4(y[4 * p], y[4 * p + 1], y[4 * p + 2], y[4 * p + 3]);
      warp_store_rows64(es.sbuf, v, es.g_row0 + (size_t)pc * 4, es.pitch_bytes, es.rows_valid, lane);
    } else {
      uint32_t w[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) w[i] = (uint32_t)y[i];
      if (es.coalesce) { if (es.row_ok) put_tail_words(reinterpret_cast<uint8_t *>(cx.dst) + ((int64_t)m_dst * cx.ldc + pc) * 4, w, N - pc); }
      else if (pc < N) row_put32(reinterpret_cast<uint8_t *>(cx.dst) + ((int64_t)m_dst * cx.ldc + pc) * 4, w, min(16, N - pc), last || pc + 16 >= N, es.row_ok, carry);
    }
    return;
  }
  {
    // accumulator -> f32: compensation, x source scale, x weight scale, + bias, one rounding per operation, two columns per instruction.  (Scalar
    // arithmetic with selects for the operands that may be missing, 15.6 instructions an element in all, and a division per sigmoid: tiles of less than
    // 4096 bytes of K waited for them.  9472 x 8192 with bias and GELU, K = 2048: 139 -> 123 us, K = 4096: 213 -> 197; f32 out, K = 2048: 178 -> 147.)
    uint64_t x2[8];
    if (has_zp) {
#pragma unroll
      for (int i = 0; i < 16; i += 4) {
        const int4 k4 = *reinterpret_cast<const int4 *>(&tc.comp[c0 + i]);
        x2[i / 2] = tc_pack2((float)((int32_t)r[i] - k4.x), (float)((int32_t)r[i + 1] - k4.y));
        x2[i / 2 + 1] = tc_pack2((float)((int32_t)r[i + 2] - k4.z), (float)((int32_t)r[i + 3] - k4.w));
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) x2[i] = tc_pack2(tc_acc_to_f32<F16>(r[2 * i]), tc_acc_to_f32<F16>(r[2 * i + 1]));
    }
    if constexpr (!F16) {
      const uint64_t s2 = tc_pack2(cx.s_src, cx.s_src);
#pragma unroll
      for (int i = 0; i < 16; i += 4) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(&tc.ws[c0 + i]);
        x2[i / 2] = tc_mul2(tc_mul2(x2[i / 2], s2), w.x);
        x2[i / 2 + 1] = tc_mul2(tc_mul2(x2[i / 2 + 1], s2), w.y);
      }
    }
    if (has_bias) {
#pragma unroll
      for (int i = 0; i < 16; i += 4) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(&tc.bias[c0 + i]);
        x2[i / 2] = tc_add2(x2[i / 2], w.x);
        x2[i / 2 + 1] = tc_add2(x2[i / 2 + 1], w.y);
      }
    }
    if (fast_act == FA_GELU_TANH) {
#pragma unroll
      for (int i = 0; i < 8; ++i) x2[i] = tc_gelu_tanh2(x2[i]);
    } else if (fast_act == FA_SWISH) {
#pragma unroll
      for (int i = 0; i < 8; ++i) x2[i] = tc_swish2(x2[i]);
    }
    float x[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) tc_unpack2(x2[i], x[2 * i], x[2 * i + 1]);
    switch (fast_act) {
    case FA_NONE: case FA_GELU_TANH: case FA_SWISH: break;
    case FA_RELU: tc_act16<FA_RELU>(epi, x, m_dst, pc); break;
    case FA_GELU_ERF: tc_act16<FA_GELU_ERF>(epi, x, m_dst, pc); break;
    case FA_SIGMOID: tc_act16<FA_SIGMOID>(epi, x, m_dst, pc); break;
    case FA_TANH: tc_act16<FA_TANH>(epi, x, m_dst, pc); break;
    default: tc_act16<FA_GENERIC>(epi, x, m_dst, pc); break;
    }
    if (epi.dst_dt == DT_BF16) {
      uint32_t pk[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) pk[i] = pack_bf16x2(x[2 * i], x[2 * i + 1]);
      if (es.map_c && es.rows_valid == 32 && full) {
        warp_tma_store_rows32(es.sbuf, make_uint4(pk[0], pk[1], pk[2], pk[3]), make_uint4(pk[4], pk[5], pk[6], pk[7]), es.map_c, pc * 2, es.row_c, lane);
      } else if (es.v8 && full) {
        if (es.row_ok) st_global_v8(reinterpret_cast<uint8_t *>(cx.dst) + ((int64_t)m_dst * cx.ldc + pc) * 2, pk);
      } else if (es.coalesce && full) {
        warp_store_rows32(es.sbuf, make_uint4(pk[0], pk[1], pk[2], pk[3]), make_uint4(pk[4], pk[5], pk[6], pk[7]),
                          es.g_row0 + (size_t)pc * 2, es.pitch_bytes, es.rows_valid, lane);
      } else if (es.coalesce) {
        if (es.row_ok) {
          uint8_t *o = reinterpret_cast<uint8_t *>(cx.dst) + ((int64_t)m_dst * cx.ldc + pc) * 2;
          const int n = N - pc;
          put_tail_words(o, pk, n >> 1);
          if (n & 1) {
#pragma unroll
            for (int i = 0; i < 8; ++i) if (i == n >> 1 && n > 0) *reinterpret_cast<uint16_t *>(o + 4 * i) = (uint16_t)pk[i];
          }
        }
      } else {
        row_put16(reinterpret_cast<uint8_t *>(cx.dst) + ((int64_t)m_dst * cx.ldc + pc) * 2, pk, max(0, min(16, N - pc)), last, es.row_ok, carry);
      }
    } else {
      if (es.v8 && full) {
        if (es.row_ok) {
          uint8_t *o = reinterpret_cast<uint8_t *>(cx.dst) + ((int64_t)m_dst * cx.ldc + pc) * 4;
#pragma unroll
          for (int p = 0; p < 2; ++p) {
            uint32_t v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = __float_as_uint(x[8 * p + i]);
            st_global_v8(o + 32 * p, v);
          }
        }
      } else if (es.coalesce && full) {
        uint4 v[4];
#pragma unroll
        for (int p = 0; p < 4; ++p)
          v[p] = make_uint4(__float_as_uint(x[4 * p]), __float_as_uint(x[4 * p + 1]), __float_as_uint(x[4 * p + 2]), __float_as_uint(x[4 * p + 3]));
        warp_store_rows64(es.sbuf, v, es.g_row0 + (size_t)pc * 4, es.pitch_bytes, es.rows_valid, lane);
      } else {
        uint32_t w[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) w[i] = __float_as_uint(x[i]);
        if (es.coalesce) { if (es.row_ok) put_tail_words(reinterpret_cast<uint8_t *>(cx.dst) + ((int64_t)m_dst * cx.ldc + pc) * 4, w, N - pc); }
        else if (pc < N) row_put32(reinterpret_cast<uint8_t *>(cx.dst) + ((int64_t)m_dst * cx.ldc + pc) * 4, w, min(16, N - pc), last || pc + 16 >= N, es.row_ok, carry);
      }
    }
  }
}

// SPLIT: launched in clusters of a.k_splits CTAs, one tile per cluster (see TcGemmArgs::k_splits); plain, non-gated form only.
// PAIR: launched in clusters of two CTAs that share [256 x BN] tiles through cta_group::2 MMAs (see the head of this file).
// F16: the bf16 x bf16 form (kind::f16 MMAs over the same byte tiles, f32 accumulators); with SPLIT its f32 partial sums are
// added in a fixed order.
template <bool SPLIT, bool PAIR = false, bool F16 = false>
__global__ void __launch_bounds__(kTcThreads, 1)
tc_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b0,
               const __grid_constant__ CUtensorMap map_c, const TcGemmArgs a, const EpiParams epi) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[2 * 8 + 8];
  __shared__ __align__(16) TileCols cols[2];
  __shared__ __align__(16) float row_scale[2][kTcBM];
  __shared__ TileMeta meta[2];
  __shared__ __align__(128) uint8_t epi_stage[kTcEpiWarps][1024];
  __shared__ uint32_t tmem_base_slot;
  __shared__ volatile int s_err;

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // (the same in every lane, and known to be)
  if (threadIdx.x == 0) TC_STAMP(0);
  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  static_assert(!(SPLIT && PAIR), "the split form and the pair form are separate kernels");

  // pair form: this CTA holds its 128 rows of A and its half of the tile's weight rows
  const uint32_t a_bytes = kTcBM * kTcBK, b_bytes = (uint32_t)(PAIR ? a.BN / 2 : a.BN) * kTcBK, stage_bytes = a_bytes + b_bytes;
  const int S = a.stages;
  uint32_t crank = 0;
  if constexpr (SPLIT || PAIR) crank = cluster_ctarank();
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (8 + s); };
  auto tfull_bar = [&](int i) { return bar0 + 8u * (16 + i); };
  auto tempty_bar = [&](int i) { return bar0 + 8u * (18 + i); };
  auto cfull_bar = [&](int i) { return bar0 + 8u * (20 + i); };
  auto cempty_bar = [&](int i) { return bar0 + 8u * (22 + i); };

  if (threadIdx.x == 0) {
    // the copy engine reads the tensor maps from memory on first use: ask for them now
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
    if (!a.maps_b) asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b0) : "memory");
    if (a.tma_store) asm volatile("prefetch.tensormap [%0];" ::"l"(&map_c) : "memory");
    for (int s = 0; s < S; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    // pair form: the epilogue warps of both CTAs release the accumulator on the leader's barrier
    for (int i = 0; i < 2; ++i) { mbar_init(tfull_bar(i), 1); mbar_init(tempty_bar(i), PAIR ? 2 * kTcEpiWarps : kTcEpiWarps); }
    for (int i = 0; i < 2; ++i) { mbar_init(cfull_bar(i), 1); mbar_init(cempty_bar(i), kTcEpiWarps); }
    s_err = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    if constexpr (PAIR) {
      // the same warp of both CTAs allocates for the pair
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(512u) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(512u) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();   // the partner's barriers exist before anything of this CTA signals them
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  // programmatic dependent launch: the next kernel of the stream may take this CTA's SM as soon as it is free (not before this CTA has
  // its tensor memory, or a dependent's CTA could hold the columns that this one waits for); this kernel touches global memory
  // only after griddepcontrol.wait (the set-up before it uses none)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");   // everything before this launch in the stream is complete and visible
  if (threadIdx.x == 0) TC_STAMP(1);

  const int m_tiles = a.tile_prefix ? a.tile_prefix[a.n_groups] : a.m_tiles_plain;
  const int total_tiles = m_tiles * a.n_tiles;
  // persistent form: tiles blockIdx.x, blockIdx.x + gridDim.x, ... over all K blocks; split form: the cluster's one tile,
  // this CTA's share of the K blocks
  int tile0 = blockIdx.x, tile_step = gridDim.x, kb_begin = 0, kb_end = a.k_blocks;
  constexpr int tile_m = PAIR ? 2 * kTcBM : kTcBM;
  const int sub = PAIR ? (int)crank * kTcBM : 0;
  if constexpr (PAIR) { tile0 = blockIdx.x >> 1; tile_step = gridDim.x >> 1; }
  if constexpr (SPLIT) {
    tile0 = blockIdx.x / a.k_splits; tile_step = total_tiles;
    const int per = (a.k_blocks + a.k_splits - 1) / a.k_splits;
    kb_begin = (int)crank * per; kb_end = min(a.k_blocks, kb_begin + per);
  }

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    // (the whole warp walks the tiles and waits, one elected lane issues the copies)
    int stage = 0; uint32_t phase = 0;
    bool ok = true;
    for (int tile = tile0; tile < total_tiles && !a.test_no_loads; tile += tile_step) {
      // one decision for the whole warp (the lookup below uses warp-wide operations)
      if (!__shfl_sync(0xffffffffu, (ok && !s_err) ? 1 : 0, 0)) break;
      const TileCoord t = tc_tile_warp(a, tile, m_tiles, lane, tile_m, sub);
      const CUtensorMap *mb = a.maps_b ? a.maps_b + t.g : &map_b0;
      for (int kb = kb_begin; kb < kb_end; ++kb) {
        if (!mbar_wait_warp(empty_bar(stage), phase ^ 1u)) { if (lane == 0) { s_err = 1; report_status(a.status, 1); } ok = false; break; }
        const uint32_t sa = smem0 + (uint32_t)stage * stage_bytes;
        if (elect_one()) {
          if constexpr (PAIR) {
            // both CTAs' copies are counted on the leader's barrier; the leader expects the bytes of both
            const uint32_t lead_bar = cluster_map(full_bar(stage), 0);
            if (crank == 0) mbar_expect_tx(full_bar(stage), 2 * stage_bytes);
            tma_load_2d_pair(sa, &map_a, kb * kTcBK, t.row0, lead_bar);
            tma_load_wt_pair(sa + a_bytes, mb, kb, (t.nt * a.BN + (int)crank * (a.BN / 2)) >> 3, lead_bar);
          } else {
            mbar_expect_tx(full_bar(stage), stage_bytes);
            tma_load_2d(sa, &map_a, kb * kTcBK, t.row0, full_bar(stage));
            tma_load_wt(sa + a_bytes, mb, kb, (t.nt * a.BN) >> 3, full_bar(stage));
          }
        }
        __syncwarp();
        if (++stage == S) { stage = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    // (the whole warp walks the tiles: operands and control flow are the same in every lane, see the MMAs above)
    if (!PAIR || crank == 0) {      // pair form: the leader issues for both CTAs
      const uint32_t idesc = F16 ? make_idesc_bf16(a.BN, tile_m) : make_idesc_i8(a.a_unsigned, a.BN, tile_m);
      int stage = 0; uint32_t phase = 0; int acc = 0; uint32_t acc_phase = 0;
      auto commit = [&](uint32_t bar) { if constexpr (PAIR) tc_commit_pair(bar); else tc_commit(bar); };
      for (int tile = tile0; tile < total_tiles && __shfl_sync(0xffffffffu, s_err ? 0 : 1, 0); tile += tile_step) {
        if (!mbar_wait_warp(tempty_bar(acc), acc_phase ^ 1u)) { if (lane == 0) { s_err = 2; report_status(a.status, 2); } break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(acc * a.BN);
        bool ok = true;
        for (int kb = kb_begin; kb < kb_end; ++kb) {
          if (!mbar_wait_warp(full_bar(stage), phase)) { ok = false; break; }
          if (lane == 0 && kb == kb_begin && tile == tile0) TC_STAMP(2);
          tc_fence_after();
          const uint32_t sa = smem0 + (uint32_t)stage * stage_bytes;
          const uint64_t da = make_smem_desc(sa), db = make_smem_desc(sa + a_bytes);
#pragma unroll
          for (int k = 0; k < kTcBK / 32; ++k) {
            const uint32_t accum = ((kb - kb_begin) | k) ? 1u : 0u;
            if constexpr (PAIR && F16) tc_mma_bf16_pair(d_tmem, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, accum);
            else if constexpr (PAIR) tc_mma_i8_pair(d_tmem, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, accum);
            else if constexpr (F16) tc_mma_bf16(d_tmem, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, accum);
            else tc_mma_i8(d_tmem, da + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc, accum);
          }
          commit(empty_bar(stage));
          if (++stage == S) { stage = 0; phase ^= 1u; }
        }
        if (!ok) { if (lane == 0) { s_err = 3; report_status(a.status, 3); } break; }
        commit(tfull_bar(acc));
        if (lane == 0 && tile == tile0) TC_STAMP(3);
        if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      }
    }
  } else if (warp == 2 + kTcEpiWarps) {
    // ------------------------------------------------------------------ operand warp
    const int32_t zp = load_zp(epi);
    int cb = 0; uint32_t cphase = 0;
    for (int tile = tile0; tile < total_tiles; tile += tile_step) {
      if (!__shfl_sync(0xffffffffu, s_err ? 0 : 1, 0)) break;
      const TileCoord t = tc_tile_warp(a, tile, m_tiles, lane, tile_m, sub);
      const void *wsp = epi.wei_scale; const int32_t *csp = epi.colsum; const void *bp = epi.bias;
      void *dst = epi.dst; int64_t ldc = epi.ldc; int m_dst0 = t.row0;
      if (a.groups) {
        const TcGroupDesc gd = a.groups[t.g];
        wsp = gd.wei_scale; csp = gd.colsum; bp = gd.bias;
        if (gd.dst) { dst = gd.dst; ldc = gd.ldc; m_dst0 = t.m_local0; }   // else: shared dst, global row index
      }
      const int pc_tile = t.nt * a.BN;
      // All loads of a tile in flight at once: the types are decided outside the loops (decided inside, each load waited for the one before it and a
      // tile took 5800 clocks here, 3000 without scales -- the bound of every tile with less than 2048 bytes of K)
      float cw[8], cbv[8]; int32_t ck[8]; int n[8]; bool in[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int pc = pc_tile + lane + 32 * j;
        in[j] = lane + 32 * j < a.BN && pc < a.N;
        n[j] = in[j] ? (int)packed_to_logical(pc, a.gated, epi.gated_I) : 0;
        cw[j] = 1.0f; cbv[j] = 0.0f; ck[j] = 0;
      }
      auto load8 = [&](const void *p, int32_t dt, bool one, float (&v)[8]) {
        if (dt == DT_F32) {
#pragma unroll
          for (int j = 0; j < 8; ++j) if (in[j]) v[j] = reinterpret_cast<const float *>(p)[one ? 0 : n[j]];
        } else {
          uint16_t b[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) b[j] = in[j] ? reinterpret_cast<const uint16_t *>(p)[one ? 0 : n[j]] : (uint16_t)0;
#pragma unroll
          for (int j = 0; j < 8; ++j) if (in[j]) v[j] = bf16_bits_to_f32(b[j]);
        }
      };
      if (epi.wei_scale_n) load8(wsp, epi.wei_scale_dt, epi.wei_scale_n == 1, cw);
      if (bp) load8(bp, epi.bias_dt, false, cbv);
      if (zp) {
#pragma unroll
        for (int j = 0; j < 8; ++j) if (in[j]) ck[j] = csp[pc_tile + lane + 32 * j];
#pragma unroll
        for (int j = 0; j < 8; ++j) ck[j] *= zp;
      }
      float rs[4] = {1.0f, 1.0f, 1.0f, 1.0f};
      if (epi.src_scale_n) {
        if (epi.src_scale_dt == DT_F32) {
#pragma unroll
          for (int j = 0; j < 4; ++j) if (lane + 32 * j < t.rows) rs[j] = reinterpret_cast<const float *>(epi.src_scale)[epi.src_scale_n > 1 ? t.row0 + lane + 32 * j : 0];
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j) if (lane + 32 * j < t.rows) rs[j] = load_as_f32(epi.src_scale, epi.src_scale_dt, epi.src_scale_n > 1 ? t.row0 + lane + 32 * j : 0);
        }
      }
      // the buffer is free when the epilogue warps have left the tile that used it two tiles ago
      if (!mbar_wait_warp(cempty_bar(cb), cphase ^ 1u)) { if (lane == 0) { s_err = 6; report_status(a.status, 6); } break; }
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (lane + 32 * j < a.BN) { cols[cb].ws[lane + 32 * j] = cw[j]; cols[cb].bias[lane + 32 * j] = cbv[j]; cols[cb].comp[lane + 32 * j] = ck[j]; }
#pragma unroll
      for (int j = 0; j < 4; ++j) row_scale[cb][lane + 32 * j] = rs[j];
      if (lane == 0) {
        TileMeta m; m.row0 = t.row0; m.rows = t.rows; m.m_dst0 = m_dst0; m.nt = t.nt; m.dst = dst; m.ldc = ldc; m.has_bias = bp != nullptr;
        meta[cb] = m;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(cfull_bar(cb));
      if (++cb == 2) { cb = 0; cphase ^= 1u; }
    }
  } else {
    // ------------------------------------------------------------------ epilogue (warps 2..9)
    const int ew = warp - 2;                // 0..7
    const int q = warp & 3;                 // TMEM lane quadrant this warp may access
    const int part = ew >> 2;               // which share of the tile's columns this warp takes
    const int row_in_tile = q * 32 + lane;
    int acc = 0; uint32_t acc_phase = 0;
    int ob = 0; uint32_t ophase = 0;            // operand buffer of the current tile
    for (int tile = tile0; tile < total_tiles; tile += tile_step) {
      // everything from global memory was put into shared memory by the operand warp
      if (!mbar_wait_warp(cfull_bar(ob), ophase)) { if (lane == 0) { s_err = 5; report_status(a.status, 5); } break; }
      const TileMeta tm = meta[ob];
      const TileCols &tcols = cols[ob];
      const bool row_ok = row_in_tile < tm.rows;
      const int m_global = tm.row0 + row_in_tile;
      const int m_dst = tm.m_dst0 + row_in_tile;
      EpiCtx cx;
      cx.wei_scale = nullptr; cx.colsum = nullptr; cx.bias = nullptr; cx.dst = tm.dst; cx.ldc = tm.ldc;
      cx.s_src = row_scale[ob][row_in_tile];
      const int pc_tile = tm.nt * a.BN;
      if (!mbar_wait_warp(tfull_bar(acc), acc_phase)) { if (lane == 0) { s_err = 4; report_status(a.status, 4); } break; }
      if (warp == 2 && lane == 0 && tile == tile0) TC_STAMP(4);
      tc_fence_after();
      const bool has_bias = tm.has_bias != 0;
      EpiStore es;
      {
        const int esz = epi.dst_dt == DT_BF16 ? 2 : 4;
        es.sbuf = epi_stage[ew];
        es.pitch_bytes = tm.ldc * esz;
        es.g_row0 = reinterpret_cast<uint8_t *>(tm.dst) + (int64_t)(tm.m_dst0 + q * 32) * es.pitch_bytes;
        es.rows_valid = min(32, max(0, tm.rows - q * 32));
        es.coalesce = ((reinterpret_cast<uintptr_t>(tm.dst) | (uintptr_t)es.pitch_bytes) & 15) == 0;
        es.v8 = ((reinterpret_cast<uintptr_t>(tm.dst) | (uintptr_t)es.pitch_bytes) & 31) == 0;
        es.row_ok = row_ok;
        es.map_c = (a.tma_store && es.coalesce) ? &map_c : nullptr;
        es.row_c = tm.m_dst0 + q * 32;
      }
      const uint32_t taddr0 = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * a.BN);
      if constexpr (SPLIT) {
        // partial sums of this CTA's K blocks go to shared memory (the stage ring is free: every MMA that read it has
        // completed); [chunk][row][32 x int32], the eight 16-byte units of a row XOR-swizzled by the row
        const int nc = min(a.BN / 32, (a.N - pc_tile + 31) / 32);
        const int per = (a.BN / 32 + kTcEpiParts - 1) / kTcEpiParts;
        const int c_begin = part * per, c_end = min(nc, c_begin + per);
        for (int c = c_begin; c < c_end; ++c) {
          uint32_t r[32];
          if (kb_end > kb_begin) { tc_ld32(taddr0 + (uint32_t)(c * 32), r); tc_wait_ld(); }
          else {
#pragma unroll
            for (int i = 0; i < 32; ++i) r[i] = 0u;
          }
          const uint32_t base = smem0 + (uint32_t)((c * kTcBM + row_in_tile) * 128);
#pragma unroll
          for (int u = 0; u < 8; ++u)
            st_shared_v4(base + (uint32_t)((u ^ (row_in_tile & 7)) << 4), r[4 * u], r[4 * u + 1], r[4 * u + 2], r[4 * u + 3]);
        }
#ifdef B200DNN_TIMING_EXPERIMENTS
      } else if (a.dbg == 1) {
        // timing experiment: no epilogue work
#endif
      } else if (!a.gated) {
#ifdef B200DNN_TIMING_EXPERIMENTS
        if (a.dbg == 3) { es.coalesce = false; es.v8 = false; es.row_ok = false; es.map_c = nullptr; }
#endif
        // this warp's chunks: a contiguous share of the tile's 32-column chunks that lie inside N
        const int nc = min(a.BN / 32, (a.N - pc_tile + 31) / 32);
        const int per = (a.BN / 32 + kTcEpiParts - 1) / kTcEpiParts;
        const int c_begin = part * per, c_end = min(nc, c_begin + per);
        RowCarry carry;
        carry.have = false;
        for (int c = c_begin; c < c_end; ++c) {
#pragma unroll 1
          for (int h = 0; h < 2; ++h) {             // sixteen columns at a time: fewer values live at once
            uint32_t r[16];
            tc_ld16(taddr0 + (uint32_t)(c * 32 + 16 * h), r);
            tc_wait_ld();
#ifdef B200DNN_TIMING_EXPERIMENTS
            if (a.dbg == 2) { uint32_t x = 0;
#pragma unroll
              for (int i = 0; i < 16; ++i) x ^= r[i];
              if (x == 0x12345678u) report_status(a.status, 99); continue; }
#endif
            tc_epi_half<F16>(a.fast_act, epi, cx, r, tcols, c * 32 + 16 * h, pc_tile + c * 32 + 16 * h, a.N, m_dst, has_bias, es, lane, carry, c == c_end - 1 && h == 1);
          }
        }
      } else {
        // gated: packed columns [g(32) u(32)] -> 32 outputs; dst is [rows, I] bf16.  Sixteen outputs at a time: their
        // 32 bytes leave as one store of the lane's own row; the row maximum is taken on the bf16 bit patterns (two per
        // instruction; magnitudes order like integers, non-finite values do not count)
        uint32_t amax2 = 0u;
        for (int c = part; c < a.BN / 64; c += kTcEpiParts) {
          const int pc0 = pc_tile + c * 64;
          if (pc0 >= a.N) break;
          const int j0 = pc0 / 2;   // first output column of this pair of chunks
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t rg[16], ru[16];
            tc_ld16(taddr0 + (uint32_t)(c * 64 + 16 * h), rg);
            tc_ld16(taddr0 + (uint32_t)(c * 64 + 32 + 16 * h), ru);
            tc_wait_ld();
            const int cg = c * 64 + 16 * h, cu = cg + 32;
            const uint64_t s2 = tc_pack2(cx.s_src, cx.s_src);
            uint32_t pk[8], mag = 0u;
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              uint64_t g2[2], u2[2];
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                g2[j] = tc_pack2(tc_acc_to_f32<F16>(rg[i + 2 * j]), tc_acc_to_f32<F16>(rg[i + 2 * j + 1]));
                u2[j] = tc_pack2(tc_acc_to_f32<F16>(ru[i + 2 * j]), tc_acc_to_f32<F16>(ru[i + 2 * j + 1]));
              }
              if constexpr (!F16) {
                const ulonglong2 wg = *reinterpret_cast<const ulonglong2 *>(&tcols.ws[cg + i]), wu = *reinterpret_cast<const ulonglong2 *>(&tcols.ws[cu + i]);
                g2[0] = tc_mul2(tc_mul2(g2[0], s2), wg.x); g2[1] = tc_mul2(tc_mul2(g2[1], s2), wg.y);
                u2[0] = tc_mul2(tc_mul2(u2[0], s2), wu.x); u2[1] = tc_mul2(tc_mul2(u2[1], s2), wu.y);
              }
              if (has_bias) {
                const ulonglong2 bg = *reinterpret_cast<const ulonglong2 *>(&tcols.bias[cg + i]), bu = *reinterpret_cast<const ulonglong2 *>(&tcols.bias[cu + i]);
                g2[0] = tc_add2(g2[0], bg.x); g2[1] = tc_add2(g2[1], bg.y);
                u2[0] = tc_add2(u2[0], bu.x); u2[1] = tc_add2(u2[1], bu.y);
              }
#pragma unroll
              for (int j = 0; j < 2; ++j) {
                float z[2];
                if (epi.gated_act == ACT_SILU_MUL) tc_unpack2(tc_mul2(tc_swish2(g2[j]), u2[j]), z[0], z[1]);
                else {
                  float gv[2], uv[2];
                  tc_unpack2(g2[j], gv[0], gv[1]);
                  tc_unpack2(u2[j], uv[0], uv[1]);
#pragma unroll
                  for (int e = 0; e < 2; ++e) z[e] = gated_f32(epi.gated_act, gv[e], uv[e]);
                }
                pk[(i >> 1) + j] = pack_bf16x2(z[0], z[1]);
                mag = __vmaxu2(mag, pk[(i >> 1) + j] & 0x7FFF7FFFu);
              }
            }
            if (max(mag & 0xFFFFu, mag >> 16) >= 0x7F80u) {      // infinities and NaNs do not enter the maximum
              mag = 0u;
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const uint32_t m = pk[i] & 0x7FFF7FFFu;
                mag = __vmaxu2(mag, m & ~__vcmpgeu2(m, 0x7F807F80u));
              }
            }
            amax2 = __vmaxu2(amax2, mag);
            const int jc = j0 + 16 * h;
            if (es.map_c && es.rows_valid == 32) {
              warp_tma_store_rows32(es.sbuf, make_uint4(pk[0], pk[1], pk[2], pk[3]), make_uint4(pk[4], pk[5], pk[6], pk[7]), es.map_c,
                                    jc * 2, es.row_c, lane);
            } else if (es.v8) {
              if (row_ok) st_global_v8(reinterpret_cast<uint8_t *>(cx.dst) + ((int64_t)m_dst * cx.ldc + jc) * 2, pk);
            } else if (es.coalesce) {
              warp_store_rows32(es.sbuf, make_uint4(pk[0], pk[1], pk[2], pk[3]), make_uint4(pk[4], pk[5], pk[6], pk[7]),
                                es.g_row0 + (size_t)jc * 2, es.pitch_bytes, es.rows_valid, lane);
            } else if (row_ok) {
              uint16_t *o = reinterpret_cast<uint16_t *>(cx.dst) + (int64_t)m_dst * cx.ldc + jc;
#pragma unroll
              for (int i = 0; i < 16; ++i) o[i] = (uint16_t)(pk[i >> 1] >> ((i & 1) * 16));
            }
          }
        }
        if (row_ok && epi.row_absmax) {
          const uint32_t m16 = max(amax2 & 0xFFFFu, amax2 >> 16);
          atomicMax(epi.row_absmax + m_global, m16 << 16);     // the bf16 magnitude as float bits
        }
      }
      if (warp == 2 && lane == 0 && tile == tile0) TC_STAMP(5);
      tc_fence_before();
      __syncwarp();
      // this warp is done with the accumulator and with the tile's operand buffer
      if (lane == 0) {
        if constexpr (PAIR) mbar_arrive_cluster(cluster_map(tempty_bar(acc), 0)); else mbar_arrive(tempty_bar(acc));
        mbar_arrive(cempty_bar(ob));
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      if (++ob == 2) { ob = 0; ophase ^= 1u; }
    }
  }

  if constexpr (SPLIT) {
    // ------------------------------------------------------------------ sum over the cluster, then the epilogue
    cluster_sync_all();   // every CTA's partial sums are in its shared memory
    bool arrived = false;
    if (threadIdx.x == 0) TC_STAMP(6);
    const bool healthy = __shfl_sync(0xffffffffu, s_err ? 0 : 1, 0) != 0;   // one decision per warp: the barriers below are warp-wide
    if (warp >= 2 && warp < 2 + kTcEpiWarps && healthy && tile0 < total_tiles) {
      const int ew = warp - 2, q = warp & 3, part = ew >> 2, row_in_tile = q * 32 + lane;
      const TileMeta tm = meta[0];
      const TileCols &tcols = cols[0];
      const int m_dst = tm.m_dst0 + row_in_tile;
      EpiCtx cx;
      cx.wei_scale = nullptr; cx.colsum = nullptr; cx.bias = nullptr; cx.dst = tm.dst; cx.ldc = tm.ldc;
      cx.s_src = row_scale[0][row_in_tile];
      const int pc_tile = tm.nt * a.BN;
      const bool has_bias = tm.has_bias != 0;
      EpiStore es;
      const int esz = epi.dst_dt == DT_BF16 ? 2 : 4;
      es.sbuf = epi_stage[ew];
      es.pitch_bytes = tm.ldc * esz;
      es.g_row0 = reinterpret_cast<uint8_t *>(tm.dst) + (int64_t)(tm.m_dst0 + q * 32) * es.pitch_bytes;
      es.rows_valid = min(32, max(0, tm.rows - q * 32));
      es.coalesce = ((reinterpret_cast<uintptr_t>(tm.dst) | (uintptr_t)es.pitch_bytes) & 15) == 0;
      es.v8 = ((reinterpret_cast<uintptr_t>(tm.dst) | (uintptr_t)es.pitch_bytes) & 31) == 0;
      es.row_ok = row_in_tile < tm.rows;
      es.map_c = (a.tma_store && es.coalesce) ? &map_c : nullptr;
      es.row_c = tm.m_dst0 + q * 32;
      const int nc = min(a.BN / 32, (a.N - pc_tile + 31) / 32);
      // chunk c is finished by CTA c % k_splits; its warp parts share that CTA's chunks.  First all sums: the warp's 32
      // rows of a chunk are 4 KiB in a row, added over the CTAs with whole-warp contiguous reads (remote shared memory is
      // slow when every lane asks for a different line) and written back in place (only this CTA reads its own copy of a
      // chunk it finishes).
      for (int c = (int)crank + a.k_splits * part; c < nc; c += a.k_splits * kTcEpiParts) {
        const uint32_t blk = smem0 + (uint32_t)((c * kTcBM + q * 32) * 128) + (uint32_t)(lane * 16);
        uint4 sum[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) sum[i] = ld_shared_v4(blk + (uint32_t)(i * 512));
        for (int j = 0; j < a.k_splits; ++j) {
          if (j == (int)crank) continue;
          const uint32_t rb = cluster_map(blk, (uint32_t)j);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint4 v = ld_cluster_v4(rb + (uint32_t)(i * 512));
            if constexpr (F16) {
              // f32 partial sums: added in a fixed order (own share first, then the other CTAs by rank), so a result is
              // reproducible; it is not the unsplit kernel's sum bit for bit
              sum[i].x = __float_as_uint(__fadd_rn(__uint_as_float(sum[i].x), __uint_as_float(v.x)));
              sum[i].y = __float_as_uint(__fadd_rn(__uint_as_float(sum[i].y), __uint_as_float(v.y)));
              sum[i].z = __float_as_uint(__fadd_rn(__uint_as_float(sum[i].z), __uint_as_float(v.z)));
              sum[i].w = __float_as_uint(__fadd_rn(__uint_as_float(sum[i].w), __uint_as_float(v.w)));
            } else { sum[i].x += v.x; sum[i].y += v.y; sum[i].z += v.z; sum[i].w += v.w; }
          }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) st_shared_v4(blk + (uint32_t)(i * 512), sum[i].x, sum[i].y, sum[i].z, sum[i].w);
      }
      cluster_arrive_all();   // this warp reads no neighbour any more
      arrived = true;
      RowCarry carry;
      carry.have = false;
      for (int c = (int)crank + a.k_splits * part; c < nc; c += a.k_splits * kTcEpiParts) {
        const uint32_t base = smem0 + (uint32_t)((c * kTcBM + row_in_tile) * 128);
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          uint32_t r[16];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const uint4 v = ld_shared_v4(base + (uint32_t)(((u + 4 * h) ^ (row_in_tile & 7)) << 4));
            r[4 * u] = v.x; r[4 * u + 1] = v.y; r[4 * u + 2] = v.z; r[4 * u + 3] = v.w;
          }
          tc_epi_half<F16>(a.fast_act, epi, cx, r, tcols, c * 32 + 16 * h, pc_tile + c * 32 + 16 * h, a.N, m_dst, has_bias, es, lane, carry, h == 1);
        }
      }
    }
    // nobody leaves while a neighbour may still read its shared memory: arrive as soon as the own reads are done,
    // wait at the very end
    if (!arrived) cluster_arrive_all();
  }

  // ---------------------------------------------------------------------- teardown
  if (a.tma_store && warp >= 2 && warp < 2 + kTcEpiWarps && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  if constexpr (SPLIT) cluster_wait_all();
  tc_fence_before();
  __syncthreads();
  // pair form: neither CTA frees its tensor memory or leaves while the partner may still issue into it or signal its barriers
  if constexpr (PAIR) cluster_sync_all();
  if (s_err) {
    // give copies that may still be in flight time to land before shared memory is released
    for (int i = 0; i < 64; ++i) __nanosleep(20000);
    __syncthreads();
  }
  if (threadIdx.x == 0) TC_STAMP(7);
  if (warp == 1) {
    tc_fence_after();
    if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

}  // namespace b200

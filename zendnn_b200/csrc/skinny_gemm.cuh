// tcgen05 GEMM for few rows of activations (a decode batch), INT8 and bf16: stands in for the same reference paths as
// decode_gemm.cuh (matmul/backends/aocl/aocl_kernel.cpp:1190-1301, matmul/matmul_native/brgemm/kernel/int8/int8_gemv_bkc.cpp).
//
// Such a call is a stream of the weight, so the operands change places: the MMA's M = 128 rows are 128 output columns (one box of the
// packed weight per 128 bytes of K) and its N is the number of activation rows rounded up to 16.  The activation side of a stage is
// then MP x 128 bytes beside 16 KiB of weight, nearly the whole ring is weight in flight, and an accumulator holds no padding rows.
//   - One CTA per (128 columns, share of K); the CTAs of a cluster share a column tile and add their partial sums ([M][128] words
//     each) through distributed shared memory in the order of their ranks, every CTA finishing the rows m = rank (mod cluster).
//   - One CTA per SM with a ring as deep as shared memory allows: the bytes in flight are what the rate depends on (a ring of half the
//     size, M = 64, K = 4096, N = 11008 in INT8: 19.3 us).  (Kernels that allocate tensor memory got one CTA per SM whatever their ring.)
//   - warp 0 copies, warp 1 issues MMAs, warps 2-9 finish: a warp takes a whole row of the tile, four columns per lane, with 16-byte
//     reads of each share.
//   - Programmatic dependent launch: where the weight does not depend on the kernel before (see SkinnyArgs::early) its ring is
//     requested before griddepcontrol.wait and streams while, for instance, the activations are still being quantised.
// Bound by HBM behind a fixed cost of about 5 us (launch, the first copies' latency, the addition).  bf16, M = 8, K = 4096, N = 11008 (90 MB): 31.0 us
// in the 128-row tile kernel -> 19.2 us (4.7 TB/s).  INT8, M = 32, same sizes: 17.7 -> 13.5 us.
// Every wait is bounded, as in tc_gemm.cuh.
#pragma once
#include "common.cuh"
#include "mbar.cuh"
#include "tc_gemm.cuh"

namespace b200 {

constexpr int kSkinnyThreads = 320;
constexpr int kSkinnyMaxStages = 12;
constexpr int kSkinnyMaxM = 64;               // rows: tensor-memory columns of the accumulator, and the largest launch
constexpr int kSkinnyMaxSplits = 8;              // CTAs per cluster (the portable limit)
constexpr int kSkinnyRing = 216 * 1024;

struct SkinnyArgs {
  int M, N, k_blocks;       // k_blocks: 128-byte blocks of K
  int MP;                   // M rounded up to 16: the MMA's N
  int stages, splits;
  int a_unsigned;
  int fast_act;             // FA_* code of the tile kernel's epilogue, or FA_GENERIC for the post-op chain as it stands
  int early;                // the weight may be read before the kernel in front has finished
  int32_t *status;
  int test_no_loads;        // test hook, see TcGemmArgs
};

template <bool F16>
__global__ void __launch_bounds__(kSkinnyThreads, 1)
skinny_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const SkinnyArgs a, const EpiParams epi) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[2 * kSkinnyMaxStages + 1];
  __shared__ float row_scale[kSkinnyMaxM];
  __shared__ uint32_t tmem_base_slot;
  __shared__ volatile int s_err;
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t w_bytes = 128 * 128, a_bytes = (uint32_t)a.MP * 128u, stage_bytes = w_bytes + a_bytes;
  const int S = a.stages;
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (kSkinnyMaxStages + s); };
  const uint32_t tfull_bar = bar0 + 8u * (2 * kSkinnyMaxStages);
  constexpr uint32_t tmem_cols = kSkinnyMaxM;

  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_w) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
    for (int s = 0; s < S; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    mbar_init(tfull_bar, 1);
    s_err = 0;
    mbar_fence_init();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "n"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_slot;
  // (behind the allocation: a dependent's CTA on this SM can then not take tensor memory that this one still waits for)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

  const int tile = blockIdx.x / a.splits, crank = blockIdx.x - tile * a.splits;
  const int kb0 = (int)((long long)crank * a.k_blocks / a.splits), kb1 = (int)((long long)(crank + 1) * a.k_blocks / a.splits);

  // finishing warps: accumulator lane quadrant and share of the rows on the way out of tensor memory; then a warp takes whole rows, four
  // columns per lane
  const int q = warp & 3, part = (warp - 2) >> 2, col = q * 32 + lane, n4 = tile * 128 + lane * 4;
  float ws[4], bias[4]; int32_t comp[4];
  if (warp == 0) {
    // (the whole warp walks the blocks and waits, one elected lane issues)
    const int n_it = kb1 - kb0, pre = min(n_it, S);
    auto load_w = [&](int i, int slot) {
      mbar_expect_tx(full_bar(slot), stage_bytes);
      tma_load_wt(smem0 + (uint32_t)slot * stage_bytes, &map_w, kb0 + i, tile * 16, full_bar(slot));
    };
    auto load_a = [&](int i, int slot) { tma_load_2d(smem0 + (uint32_t)slot * stage_bytes + w_bytes, &map_a, (kb0 + i) * 128, 0, full_bar(slot)); };
    if (a.early && !a.test_no_loads && elect_one()) for (int i = 0; i < pre; ++i) load_w(i, i);
    __syncwarp();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (!a.test_no_loads) {
      if (elect_one()) for (int i = 0; i < pre; ++i) { if (!a.early) load_w(i, i); load_a(i, i); }
      __syncwarp();
      int slot = 0; uint32_t phase = 0;
      for (int i = pre; i < n_it; ++i) {
        if (!mbar_wait_warp(empty_bar(slot), phase)) { if (lane == 0) { s_err = 1; report_status(a.status, 31); } break; }
        if (elect_one()) { load_w(i, slot); load_a(i, slot); }
        __syncwarp();
        if (++slot == S) { slot = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    // the whole warp walks the blocks (operands stay in uniform registers)
    // A = weight (s8, or bf16), B = activations (u8 | s8, or bf16), both K-major; M = 128, N = MP
    const uint32_t idesc = F16 ? make_idesc_bf16(a.MP) : ((2u << 4) | (1u << 7) | ((a.a_unsigned ? 0u : 1u) << 10) | ((uint32_t)(a.MP >> 3) << 17) | (8u << 24));
    int slot = 0; uint32_t phase = 0;
    bool ok = true;
    for (int kb = kb0; kb < kb1; ++kb) {
      if (!mbar_wait_warp(full_bar(slot), phase)) { ok = false; break; }
      tc_fence_after();
      const uint32_t sw = smem0 + (uint32_t)slot * stage_bytes;
      const uint64_t dw = make_smem_desc(sw), da = make_smem_desc(sw + w_bytes);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if constexpr (F16) tc_mma_bf16(tmem, dw + (uint64_t)(k * 2), da + (uint64_t)(k * 2), idesc, ((kb - kb0) | k) ? 1u : 0u);
        else tc_mma_i8(tmem, dw + (uint64_t)(k * 2), da + (uint64_t)(k * 2), idesc, ((kb - kb0) | k) ? 1u : 0u);
      }
      tc_commit(empty_bar(slot));
      if (++slot == S) { slot = 0; phase ^= 1u; }
    }
    if (ok) tc_commit(tfull_bar);
    else if (lane == 0) { s_err = 1; report_status(a.status, 32); }
    __syncwarp();
  } else {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int m = threadIdx.x - 64; m < a.M; m += kSkinnyThreads - 64)
      row_scale[m] = epi.src_scale_n ? load_as_f32(epi.src_scale, epi.src_scale_dt, epi.src_scale_n > 1 ? m : 0) : 1.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int n = n4 + i;
      const bool in = n < a.N;
      ws[i] = (in && epi.wei_scale_n) ? load_as_f32(epi.wei_scale, epi.wei_scale_dt, epi.wei_scale_n > 1 ? n : 0) : 1.0f;
      bias[i] = (in && epi.bias) ? load_as_f32(epi.bias, epi.bias_dt, n) : 0.0f;
      comp[i] = (!F16 && in && epi.has_zp) ? load_zp(epi) * epi.colsum[n] : 0;
    }
    // the partial sums go to shared memory as [row][128 columns], over the ring (every product that read it has completed)
    const bool ok = mbar_wait_warp(tfull_bar, 0);
    if (ok) {
      tc_fence_after();
      for (int c = part; c * 16 < a.M; c += 2) {
        uint32_t r[16];
        tc_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(c * 16), r);
        tc_wait_ld();
        const uint32_t base = smem0 + (uint32_t)((c * 16 * 128 + col) * 4);
#pragma unroll
        for (int i = 0; i < 16; ++i) asm volatile("st.shared.u32 [%0], %1;" ::"r"(base + (uint32_t)(i * 512)), "r"(r[i]) : "memory");
      }
      tc_fence_before();
    } else if (lane == 0) { s_err = 1; report_status(a.status, 33); }
  }
  if (a.splits > 1) cluster_sync_all(); else __syncthreads();
  const bool healthy = __shfl_sync(0xffffffffu, s_err ? 0 : 1, 0) != 0;

  if (warp >= 2 && healthy && n4 < a.N) {
    const int esz = epi.dst_dt == DT_BF16 ? 2 : 4;
    const bool whole = n4 + 4 <= a.N && ((reinterpret_cast<uintptr_t>(epi.dst) | (uintptr_t)(epi.ldc * esz)) & (4 * esz - 1)) == 0;
    for (int m = crank + a.splits * (warp - 2); m < a.M; m += 8 * a.splits) {
      const uint32_t own = smem0 + (uint32_t)(m * 512 + lane * 16);
      uint4 v[kSkinnyMaxSplits];
#pragma unroll
      for (int j = 0; j < kSkinnyMaxSplits; ++j)
        if (j < a.splits) v[j] = a.splits > 1 ? ld_cluster_v4(cluster_map(own, (uint32_t)j)) : ld_shared_v4(own);
      uint32_t s[4] = {v[0].x, v[0].y, v[0].z, v[0].w};
#pragma unroll
      for (int j = 1; j < kSkinnyMaxSplits; ++j)
        if (j < a.splits) {
          const uint32_t w[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
#pragma unroll
          for (int i = 0; i < 4; ++i) s[i] = F16 ? __float_as_uint(__fadd_rn(__uint_as_float(s[i]), __uint_as_float(w[i]))) : s[i] + w[i];
        }
      uint8_t *o = reinterpret_cast<uint8_t *>(epi.dst) + ((int64_t)m * epi.ldc + n4) * esz;
      uint32_t y[4];
      if (!F16 && epi.dst_dt == DT_S32) {
#pragma unroll
        for (int i = 0; i < 4; ++i) y[i] = s[i] - (uint32_t)comp[i];
      } else {
        const float s_src = row_scale[m];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          float x = tc_acc_f32<F16>(s[i], comp[i], s_src, ws[i]);
          if (epi.bias) x = __fadd_rn(x, bias[i]);
          switch (a.fast_act) {
          case FA_NONE: break;
          case FA_RELU: x = tc_act<FA_RELU>(epi, x, m, n4 + i); break;
          case FA_GELU_TANH: x = tc_act<FA_GELU_TANH>(epi, x, m, n4 + i); break;
          case FA_SIGMOID: x = tc_act<FA_SIGMOID>(epi, x, m, n4 + i); break;
          case FA_SWISH: x = tc_act<FA_SWISH>(epi, x, m, n4 + i); break;
          default: if (n4 + i < a.N) for (int p = 0; p < epi.n_po; ++p) x = apply_postop(epi.po[p], x, m, n4 + i); break;
          }
          y[i] = epi.dst_dt == DT_BF16 ? (uint32_t)f32_to_bf16_bits(x) : __float_as_uint(x);
        }
      }
      if (esz == 2) {
        if (whole) *reinterpret_cast<uint2 *>(o) = make_uint2(y[0] | (y[1] << 16), y[2] | (y[3] << 16));
        else {
#pragma unroll
          for (int i = 0; i < 4; ++i) if (n4 + i < a.N) reinterpret_cast<uint16_t *>(o)[i] = (uint16_t)y[i];
        }
      } else if (whole) *reinterpret_cast<uint4 *>(o) = make_uint4(y[0], y[1], y[2], y[3]);
      else {
#pragma unroll
        for (int i = 0; i < 4; ++i) if (n4 + i < a.N) reinterpret_cast<uint32_t *>(o)[i] = y[i];
      }
    }
  }
  // nobody leaves while a neighbour may still read its shared memory
  if (a.splits > 1) cluster_sync_all(); else __syncthreads();
  if (s_err) {
    for (int i = 0; i < 64; ++i) __nanosleep(20000);     // copies still in flight land before shared memory is released
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(tmem_cols) : "memory");
  }
}

}  // namespace b200

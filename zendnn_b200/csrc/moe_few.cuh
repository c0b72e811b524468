// Grouped tcgen05 GEMM for a few rows per expert (MoE decode batches), INT8 and bf16: stands in for the tile micro-kernel under group_matmul_direct
// (matmul/group_matmul/custom_kernel/ukernel/int8_microkernel.hpp:39-56) where a layer has at most 64 tokens.
//
// As in skinny_gemm.cuh the operands change places: the MMA's M = 128 rows are 128 packed output columns of one expert, its N is the rows rounded up to 16.  The
// tile kernel's 128-row box of activations per 128 bytes of K, nearly all of it other experts' rows or padding, costs as many bytes from L2 to shared memory as
// the weight itself; here it is MP x 128 bytes beside 16 KiB of weight, and an accumulator holds no padding.
//   - One persistent CTA per SM over the tiles (MP rows of an expert, 128 packed columns); an expert's tiles are found on the device (tile_prefix).  MP holds all rows of an
//     expert that every token asks for once; a token whose logits name no expert (NaN) has the same one k times, and its expert more tiles.
//   - warp 0 copies, warp 1 issues MMAs, warps 2-9 finish; two accumulators and a ring that runs across tiles keep the weight stream going behind the epilogue.
//   - The accumulators pass through shared memory as [row][128 columns]; then a warp takes whole rows, four columns a lane, or (gated) two outputs, with the
//     arithmetic of the tile kernel's epilogue.
// Bound by HBM behind the launch, the ramp and one epilogue.  Layers, us in the tile kernel -> here: 1 token, 8 experts of 4096 x 14336, top 2: 115 -> 74; 3 tokens, bf16, 8
// of 1216 x 3968: 50 -> 33; 8 tokens, 60 of 1472 x 992, top 6: 63 -> 53; 32 tokens, 64 of 2048 x 1408, top 6, two shared: 82.2 -> 77.6.  Every wait is bounded, as in tc_gemm.cuh.
#pragma once
#include "common.cuh"
#include "mbar.cuh"
#include "tc_gemm.cuh"

namespace b200 {

constexpr int kMoeFewThreads = 320;
constexpr int kMoeFewMaxRows = 64;
constexpr int kMoeFewMaxStages = 12;
constexpr int kMoeFewSmem = 216 * 1024;

struct MoeFewArgs {
  int n_groups, n_tiles;          // experts; column tiles of 128 per expert
  int N, k_blocks;                // packed columns; 128-byte blocks of K
  int MP, stages;                 // rows of a tile, a multiple of 16; ring depth
  int gated;                      // packed gate/up interleave, see pack_kernels.cuh
  const int32_t *row_off, *tile_prefix;      // [n_groups + 1] first row of each expert; how many tiles of MP rows the experts in front have
  const CUtensorMap *maps_w;      // [n_groups], boxes of 128 packed rows
  const TcGroupDesc *groups;      // [n_groups] scales and biases
  int32_t *status;
  int test_no_loads;              // test hook, see TcGemmArgs
};

template <bool F16>
__global__ void __launch_bounds__(kMoeFewThreads, 1)
moe_few_kernel(const __grid_constant__ CUtensorMap map_a, const MoeFewArgs a, const EpiParams epi) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t bars[2 * kMoeFewMaxStages + 4];
  __shared__ float row_scale[2][kMoeFewMaxRows];
  __shared__ uint32_t tmem_base_slot;
  __shared__ volatile int s_err;
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t smem0 = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t w_bytes = 128 * 128, stage_bytes = w_bytes + (uint32_t)a.MP * 128u;
  const int S = a.stages;
  const uint32_t part0 = smem0 + (uint32_t)S * stage_bytes;           // [2][MP][128] words
  const uint32_t bar0 = smem_u32(bars);
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (kMoeFewMaxStages + s); };
  auto tfull_bar = [&](int i) { return bar0 + 8u * (2 * kMoeFewMaxStages + i); };
  auto tempty_bar = [&](int i) { return bar0 + 8u * (2 * kMoeFewMaxStages + 2 + i); };
  const uint32_t tmem_cols = a.MP <= 16 ? 32u : a.MP <= 32 ? 64u : 128u;

  if (threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
    for (int s = 0; s < S; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(tfull_bar(i), 1); mbar_init(tempty_bar(i), 8); }
    s_err = 0;
    mbar_fence_init();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_base_slot;
  // (behind the allocation: a dependent's CTA on this SM can then not take tensor memory that this one still waits for)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");

  const int total = a.tile_prefix[a.n_groups] * a.n_tiles;
  // a tile's expert (by a whole warp): the number of prefix entries up to its place among the row tiles; its first row and its rows, MP at most
  struct Rows { int g, row0, rows; };
  auto rows_of = [&](int tile) {
    const int mt = tile / a.n_tiles;
    int g = 0, first = 0;             // (first: the expert's first row tile, the last entry that does not lie beyond mt)
    for (int base = 1; base < a.n_groups; base += 32) {
      const int i = base + lane, p = i < a.n_groups ? a.tile_prefix[i] : 0x7fffffff;
      const unsigned up = __ballot_sync(0xffffffffu, p <= mt);
      g += __popc(up);
      if (up) first = __shfl_sync(0xffffffffu, p, 31 - __clz(up));
    }
    const int row0 = a.row_off[g] + (mt - first) * a.MP;
    return Rows{g, row0, min(a.MP, a.row_off[g + 1] - row0)};
  };

  if (warp == 0) {
    int slot = 0; uint32_t phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; ok && tile < total && !a.test_no_loads; tile += gridDim.x) {
      const Rows t = rows_of(tile);
      const int nt = tile % a.n_tiles, row0 = t.row0;
      const CUtensorMap *mw = a.maps_w + t.g;
      for (int kb = 0; kb < a.k_blocks; ++kb) {
        if (!mbar_wait_warp(empty_bar(slot), phase ^ 1u)) { if (lane == 0) { s_err = 1; report_status(a.status, 61); } ok = false; break; }
        const uint32_t sw = smem0 + (uint32_t)slot * stage_bytes;
        if (elect_one()) {
          mbar_expect_tx(full_bar(slot), stage_bytes);
          tma_load_wt(sw, mw, kb, nt * 16, full_bar(slot));
          tma_load_2d(sw + w_bytes, &map_a, kb * 128, row0, full_bar(slot));
        }
        __syncwarp();
        if (++slot == S) { slot = 0; phase ^= 1u; }
      }
    }
  } else if (warp == 1) {
    const uint32_t idesc = F16 ? make_idesc_bf16(a.MP) : make_idesc_i8(0, a.MP);      // A = weight, B = activations, both K-major; M = 128, N = MP
    int slot = 0, acc = 0; uint32_t phase = 0, acc_phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
      if (!mbar_wait_warp(tempty_bar(acc), acc_phase ^ 1u)) { ok = false; break; }
      tc_fence_after();
      const uint32_t d = tmem + (uint32_t)(acc * a.MP);
      for (int kb = 0; kb < a.k_blocks; ++kb) {
        if (!mbar_wait_warp(full_bar(slot), phase)) { ok = false; break; }
        tc_fence_after();
        const uint32_t sw = smem0 + (uint32_t)slot * stage_bytes;
        const uint64_t dw = make_smem_desc(sw), da = make_smem_desc(sw + w_bytes);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if constexpr (F16) tc_mma_bf16(d, dw + (uint64_t)(k * 2), da + (uint64_t)(k * 2), idesc, (kb | k) ? 1u : 0u);
          else tc_mma_i8(d, dw + (uint64_t)(k * 2), da + (uint64_t)(k * 2), idesc, (kb | k) ? 1u : 0u);
        }
        tc_commit(empty_bar(slot));
        if (++slot == S) { slot = 0; phase ^= 1u; }
      }
      if (!ok) break;
      tc_commit(tfull_bar(acc));
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
    }
    if (!ok && lane == 0) { s_err = 1; report_status(a.status, 62); }
  } else {
    const int q = warp & 3, part = (warp - 2) >> 2, col = q * 32 + lane, tid = threadIdx.x - 64;
    const int gc = (lane >> 4) * 64 + ((2 * lane) & 31);              // gated: this lane's first gate column of the tile (its up columns are 32 further)
    int acc = 0; uint32_t acc_phase = 0;
    for (int tile = blockIdx.x; tile < total; tile += gridDim.x) {
      const Rows t = rows_of(tile);
      const int nt = tile % a.n_tiles, row0 = t.row0, rows = t.rows;
      const TcGroupDesc gd = a.groups[t.g];
      // this lane's columns: four in a row, or two gate and two up columns
      float ws[4] = {1.f, 1.f, 1.f, 1.f}, bias[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int pc = nt * 128 + (a.gated ? gc + (i & 1) + (i >> 1) * 32 : lane * 4 + i);
        if (pc < a.N) {
          const int n = (int)packed_to_logical(pc, a.gated, epi.gated_I);
          if (epi.wei_scale_n) ws[i] = load_as_f32(gd.wei_scale, epi.wei_scale_dt, epi.wei_scale_n > 1 ? n : 0);
          if (gd.bias) bias[i] = load_as_f32(gd.bias, epi.bias_dt, n);
        }
      }
      if (tid < rows) row_scale[acc][tid] = epi.src_scale_n ? load_as_f32(epi.src_scale, epi.src_scale_dt, epi.src_scale_n > 1 ? row0 + tid : 0) : 1.0f;
      const uint32_t pbuf = part0 + (uint32_t)(acc * a.MP * 512);
      const bool ok = mbar_wait_warp(tfull_bar(acc), acc_phase);
      if (ok) {
        tc_fence_after();
        for (int c = part; c * 16 < a.MP; c += 2) {
          uint32_t r[16];
          tc_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * a.MP + c * 16), r);
          tc_wait_ld();
          const uint32_t base = pbuf + (uint32_t)((c * 16 * 128 + col) * 4);
#pragma unroll
          for (int i = 0; i < 16; ++i) asm volatile("st.shared.u32 [%0], %1;" ::"r"(base + (uint32_t)(i * 512)), "r"(r[i]) : "memory");
        }
        tc_fence_before();
      } else if (lane == 0) { s_err = 1; report_status(a.status, 63); }
      __syncwarp();
      if (lane == 0) mbar_arrive(tempty_bar(acc));
      // one decision for the eight warps: all of them meet here whether their wait ended well or not
      uint32_t all;
      asm volatile("{\n.reg .pred p, r;\nsetp.ne.u32 p, %1, 0;\nbarrier.cta.red.and.pred r, 1, 256, p;\nselp.u32 %0, 1, 0, r;\n}" : "=r"(all) : "r"((uint32_t)ok) : "memory");
      if (!all) break;
      for (int m = warp - 2; m < rows; m += 8) {
        const float s = row_scale[acc][m];
        uint16_t *o = reinterpret_cast<uint16_t *>(epi.dst) + (int64_t)(row0 + m) * epi.ldc;
        if (a.gated) {
          const uint32_t at = pbuf + (uint32_t)(m * 512 + gc * 4);
          uint32_t v[4];
          asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "r"(at) : "memory");
          asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v[2]), "=r"(v[3]) : "r"(at + 128u) : "memory");
          uint64_t g2 = tc_pack2(tc_acc_to_f32<F16>(v[0]), tc_acc_to_f32<F16>(v[1])), u2 = tc_pack2(tc_acc_to_f32<F16>(v[2]), tc_acc_to_f32<F16>(v[3]));
          if constexpr (!F16) {
            const uint64_t s2 = tc_pack2(s, s);
            g2 = tc_mul2(tc_mul2(g2, s2), tc_pack2(ws[0], ws[1]));
            u2 = tc_mul2(tc_mul2(u2, s2), tc_pack2(ws[2], ws[3]));
          }
          if (gd.bias) { g2 = tc_add2(g2, tc_pack2(bias[0], bias[1])); u2 = tc_add2(u2, tc_pack2(bias[2], bias[3])); }
          float z[2];
          if (epi.gated_act == ACT_SILU_MUL) tc_unpack2(tc_mul2(tc_swish2(g2), u2), z[0], z[1]);
          else {
            float gv[2], uv[2];
            tc_unpack2(g2, gv[0], gv[1]);
            tc_unpack2(u2, uv[0], uv[1]);
#pragma unroll
            for (int e = 0; e < 2; ++e) z[e] = gated_f32(epi.gated_act, gv[e], uv[e]);
          }
          const uint32_t pk = pack_bf16x2(z[0], z[1]);
          const int n = nt * 64 + 2 * lane;                           // (the width of an expert is a multiple of 32: a pair is inside or outside)
          const bool in = n * 2 < a.N;
          if (in) *reinterpret_cast<uint32_t *>(o + n) = pk;
          if (epi.row_absmax) {                                       // largest finite magnitude of the row, as the tile kernel takes it
            uint32_t lo = pk & 0x7FFFu, hi = (pk >> 16) & 0x7FFFu;
            lo = lo < 0x7F80u ? lo : 0u; hi = hi < 0x7F80u ? hi : 0u;
            const uint32_t top = __reduce_max_sync(0xffffffffu, in ? max(lo, hi) : 0u);
            if (lane == 0) atomicMax(epi.row_absmax + row0 + m, top << 16);
          }
        } else {
          const uint4 v = ld_shared_v4(pbuf + (uint32_t)(m * 512 + lane * 16));
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
          const int n = nt * 128 + lane * 4;
          uint16_t y[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float x = tc_acc_f32<F16>(w[i], 0, s, ws[i]);
            if (gd.bias) x = __fadd_rn(x, bias[i]);
            y[i] = f32_to_bf16_bits(x);
          }
          if (n + 4 <= a.N && ((reinterpret_cast<uintptr_t>(epi.dst) | (uintptr_t)(epi.ldc * 2)) & 7) == 0)
            *reinterpret_cast<uint2 *>(o + n) = make_uint2(y[0] | ((uint32_t)y[1] << 16), y[2] | ((uint32_t)y[3] << 16));
          else {
#pragma unroll
            for (int i = 0; i < 4; ++i) if (n + i < a.N) o[n + i] = y[i];
          }
        }
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (s_err) {
    for (int i = 0; i < 64; ++i) __nanosleep(20000);     // copies still in flight land before shared memory is released
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
  }
}

}  // namespace b200

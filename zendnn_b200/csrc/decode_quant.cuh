// Per-token quantisation inside the decode kernels: every CTA quantises the call's few bf16 rows itself, into the shared memory that its products read, instead of
// waiting for a kernel that does it once.  Codes and scales are those of the per-token kernels, bit for bit (the same functions, an abs-max in any order).
// What it saves is a launch and the chain behind it (load, reduce, store, launch, load); what it costs is the rows' bytes through L2 once per SM, so it
// pays for few elements: see the rule in b200dnn.cu.
#pragma once
#include "common.cuh"
#include "quant_kernels.cuh"

namespace b200 {

struct DecodeQuant {
  const uint16_t *src; int64_t ld;      // bf16 rows, 16-byte aligned; null: the rows are quantised already
  void *scale_out; int32_t scale_dt;    // where the caller wants the row scales (or null), and the type they are kept in
  int late;                             // the weight may not be read before the kernel in front has finished
};

// Called by THREADS threads (tid 0 .. THREADS - 1); sync() is a barrier of these.  rows: row r's codes at rows + r * stride; top: [16] words of shared memory, zeroed
// before a barrier that all of them have passed.  Every row has whole warps of its own, so that a row's maximum, scale and reciprocal are a warp's; NJ vectors of eight
// elements a lane stay in registers between the maximum and the codes, the others are read again.  (Bound by instruction issue: all SMs do the same work.  Vectors
// dealt out without regard to rows, with a division and a reciprocal each, took 0.11 us per 1000 elements.)
// ss gets the row scales; codes and scales may be read behind a barrier of the caller's.
template <int THREADS, int NJ, typename Sync>
__device__ __forceinline__ void decode_quant_rows(const DecodeQuant &q, uint8_t *rows, int stride, int M, int K, uint32_t *top, float *ss, int tid, bool publish, Sync sync) {
  const int lane = tid & 31, warp = tid >> 5, per_row = (THREADS / 32) / M;          // M <= 16 and no more rows than warps: see fused_quant_pays
  const int r = warp / per_row, step = per_row * 32, i0 = (warp - r * per_row) * 32 + lane, nv = r < M ? K >> 3 : 0;
  const uint4 *src = reinterpret_cast<const uint4 *>(q.src + (int64_t)min(r, M - 1) * q.ld);
  uint4 v[NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j) v[j] = i0 + j * step < nv ? __ldg(src + i0 + j * step) : make_uint4(0, 0, 0, 0);
  auto raise = [&](bool finite) {
    AbsMax<uint16_t> m;
    auto add = [&](const uint4 &x) { if (finite) m.add_finite(x); else m.add(x); };
#pragma unroll
    for (int j = 0; j < NJ; ++j) add(v[j]);
#pragma unroll 4
    for (int i = i0 + NJ * step; i < nv; i += step) add(__ldg(src + i));
    const uint32_t w = __reduce_max_sync(0xffffffffu, m.bits());
    if (lane == 0 && r < M) atomicMax(top + r, w);
    sync();
  };
  raise(false);
  if (__any_sync(0xffffffffu, lane < M && top[min(lane, 15)] >= 0x7F800000u)) {      // (the same in every warp) an infinity or a NaN: the finite elements alone
    sync();
    if (tid < 16) top[tid] = 0u;
    sync();
    raise(true);
  }
  const float scale = scale_from_absmax(__uint_as_float(top[min(r, 15)])), rinv = __frcp_rn(scale);
  uint2 *dst = reinterpret_cast<uint2 *>(rows + (size_t)r * stride);
#pragma unroll
  for (int j = 0; j < NJ; ++j) if (i0 + j * step < nv) dst[i0 + j * step] = quant_vec<uint16_t>(v[j], scale, rinv);
#pragma unroll 2
  for (int i = i0 + NJ * step; i < nv; i += step) dst[i] = quant_vec<uint16_t>(__ldg(src + i), scale, rinv);
  if (r < M && i0 == 0) {
    ss[r] = q.scale_dt == DT_BF16 ? bf16_bits_to_f32(f32_to_bf16_bits(scale)) : scale;
    if (publish && q.scale_out) {
      if (q.scale_dt == DT_BF16) reinterpret_cast<uint16_t *>(q.scale_out)[r] = f32_to_bf16_bits(scale);
      else reinterpret_cast<float *>(q.scale_out)[r] = scale;
    }
  }
}

}  // namespace b200

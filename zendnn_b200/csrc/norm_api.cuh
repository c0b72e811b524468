// normalization_direct: LayerNorm, RMSNorm, fused-add RMSNorm and inference BatchNorm, the operators on either side of the
// quantised GEMMs in a decoder layer (reference: lowoha_operators/normalization/lowoha_normalization.hpp:98-107, checks
// lowoha_normalization_utils.cpp:23-149, scalar definition kernel/reference_kernel.cpp:98-474).
//   LayerNorm        mean = sum(x)/n, var = sum((x-mean)^2)/n, y = (x-mean) * (1/sqrt(var+eps)) [* gamma] [+ beta]
//   RMSNorm          y = x * (1/sqrt(sum(x^2)/n + eps)) [* gamma]
//   fused-add RMS    residual <- round_to_src(residual + x) (in place); the sum of squares is taken over the unrounded sums,
//                    the output over the rounded residual (reference_kernel.cpp:437-462)
//   BatchNorm        y = (x - running_mean[c]) * (1/sqrt(running_var[c]+eps)) [* gamma[c]] [+ beta[c]], input [N, C, spatial]
// all in f32 with one rounding per operation; sums are block reductions here (the reference adds sequentially), so a result
// may differ from the reference's in the last f32 bit before the final rounding to the destination type.
// With no counterpart in the reference: the normalised row can leave, in the same pass, as per-token quantised s8 with its
// f32 scale (the arithmetic of reorder_direct's dynamic per-token quantisation applied to the row rounded to dst_dt), so that
// norm -> quantise -> W8A8 GEMM costs one read of the activations instead of a write and a second read.
// One CTA per row; the row is staged in shared memory as f32 (rows beyond the shared-memory budget are re-read from global
// memory).  HBM-bound: src + dst bytes per element.  Included at the end of b200dnn.cu.
#pragma once

namespace {

enum : int { NORM_LAYER = 0, NORM_BATCH = 1, NORM_RMS = 2, NORM_FUSED_ADD_RMS = 3 };
constexpr int kNormThreads = 256;
constexpr int kNormSmemElems = 48 * 1024;     // 192 KiB of staged f32

struct NormArgs {
  int type;
  int64_t batch, n;
  float eps;
  int use_scale, use_shift;
  int32_t src_dt, dst_dt, gamma_dt, beta_dt;
  const void *x; void *y; const void *gamma, *beta; void *residual;
  int8_t *q; int64_t q_ld; float *q_scale;     // optional fused per-token quantisation
  int staged;                                  // the row fits the shared-memory stage
};

__device__ __forceinline__ float norm_block_sum(float v, float *sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = 0.f;
  for (int i = 0; i < (int)(blockDim.x >> 5); ++i) r += sh[i];
  __syncthreads();
  return r;
}
__device__ __forceinline__ float norm_block_max(float v, float *sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = 0.f;
  for (int i = 0; i < (int)(blockDim.x >> 5); ++i) r = fmaxf(r, sh[i]);
  __syncthreads();
  return r;
}
__device__ __forceinline__ float norm_block_max_signed(float v, float *sh) {      // values may be negative (scores)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = sh[0];
  for (int i = 1; i < (int)(blockDim.x >> 5); ++i) r = fmaxf(r, sh[i]);
  __syncthreads();
  return r;
}
__device__ __forceinline__ float norm_round_to(float v, int32_t dt) {
  return dt == B200DNN_BF16 ? __uint_as_float(pack_bf16x2(v, 0.0f) << 16) : v;
}
__device__ __forceinline__ void norm_store(void *p, int32_t dt, int64_t i, float v) {
  if (dt == B200DNN_BF16) reinterpret_cast<uint16_t *>(p)[i] = (uint16_t)(pack_bf16x2(v, 0.0f) & 0xFFFFu);
  else reinterpret_cast<float *>(p)[i] = v;
}

__global__ void __launch_bounds__(kNormThreads) norm_rows_kernel(const NormArgs a) {
  extern __shared__ float row[];
  __shared__ float sh[kNormThreads / 32];
  const int64_t n = a.n;
  for (int64_t b = blockIdx.x; b < a.batch; b += gridDim.x) {
    const int64_t off = b * n;
    // ---- pass 1: stage the row (fused add: update the residual) and take the first sum
    float s1 = 0.f;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
      float v = load_as_f32(a.x, a.src_dt, off + i);
      if (a.type == NORM_FUSED_ADD_RMS) {
        const float sum = __fadd_rn(load_as_f32(a.residual, a.src_dt, off + i), v);
        s1 = __fmaf_rn(sum, sum, s1);
        norm_store(a.residual, a.src_dt, off + i, sum);
        v = norm_round_to(sum, a.src_dt);
      } else if (a.type == NORM_RMS) s1 = __fmaf_rn(v, v, s1);
      else s1 = __fadd_rn(s1, v);
      if (a.staged) row[i] = v;
    }
    s1 = norm_block_sum(s1, sh);
    float mean = 0.f, inv;
    if (a.type == NORM_LAYER) {
      mean = __fdiv_rn(s1, (float)n);
      float s2 = 0.f;
      for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
        const float d = __fadd_rn(a.staged ? row[i] : load_as_f32(a.x, a.src_dt, off + i), -mean);
        s2 = __fmaf_rn(d, d, s2);
      }
      s2 = norm_block_sum(s2, sh);
      inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(s2, (float)n), a.eps)));
    } else inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(s1, (float)n), a.eps)));
    // ---- pass 2: normalise, store; with the fused quantisation keep the rounded result staged and take its abs-max
    float amax = 0.f;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
      float v;
      if (a.staged) v = row[i];
      else if (a.type == NORM_FUSED_ADD_RMS) v = load_as_f32(a.residual, a.src_dt, off + i);
      else v = load_as_f32(a.x, a.src_dt, off + i);
      float y = __fmul_rn(__fadd_rn(v, -mean), inv);
      if (a.use_scale) y = __fmul_rn(y, load_as_f32(a.gamma, a.gamma_dt, i));
      if (a.use_shift && a.type == NORM_LAYER) y = __fadd_rn(y, load_as_f32(a.beta, a.beta_dt, i));
      if (a.y) norm_store(a.y, a.dst_dt, off + i, y);
      if (a.q) {
        y = norm_round_to(y, a.dst_dt);
        if (finite_f32(y)) amax = fmaxf(amax, fabsf(y));
        row[i] = y;
      }
    }
    if (a.q) {
      const float scale = scale_from_absmax(norm_block_max(amax, sh));     // (the barrier inside also publishes row[])
      for (int64_t i = threadIdx.x; i < n; i += blockDim.x) a.q[b * a.q_ld + i] = quant_sym(row[i], scale);
      if (threadIdx.x == 0) a.q_scale[b] = scale;
    }
    __syncthreads();      // row[] is reused by the next row of this CTA
  }
}

__device__ __forceinline__ float norm_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float norm_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }
// four parameters (f32 or bf16, 16-byte aligned array), group i4
__device__ __forceinline__ void norm_load4(const void *p, int32_t dt, int i4, float (&g)[4]) {
  if (dt == B200DNN_F32) {
    const float4 v = reinterpret_cast<const float4 *>(p)[i4];
    g[0] = v.x; g[1] = v.y; g[2] = v.z; g[3] = v.w;
  } else {
    const uint2 v = reinterpret_cast<const uint2 *>(p)[i4];
    g[0] = norm_lo(v.x); g[1] = norm_hi(v.x); g[2] = norm_lo(v.y); g[3] = norm_hi(v.y);
  }
}

// Parameters of the four columns c0 .. c0 + 3.  ANY: the columns start anywhere (c0 & 3 is the same for all vectors of a row) and may lie partly
// outside [0, n); f32 parameters come as two aligned float4, of which the wanted four are picked.
template <bool ANY>
__device__ __forceinline__ void norm_params4(const void *p, int32_t dt, int c0, int n, float (&g)[4]) {
  if constexpr (!ANY) norm_load4(p, dt, c0 >> 2, g);
  else {
    const int r = c0 & 3;
    if (dt == B200DNN_F32 && c0 >= 0 && c0 - r + 8 <= n) {
      const float4 *v = reinterpret_cast<const float4 *>(p) + (c0 >> 2);
      const float4 x = v[0], y = v[1];
      const float w[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
      float u[5];
#pragma unroll
      for (int e = 0; e < 5; ++e) u[e] = (r & 2) ? w[e + 2] : w[e];
#pragma unroll
      for (int e = 0; e < 4; ++e) g[e] = (r & 1) ? u[e + 1] : u[e];
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) g[e] = (unsigned)(c0 + e) < (unsigned)n ? load_as_f32(p, dt, c0 + e) : 0.f;
    }
  }
}

// a sum (or a largest value) over the CTA (sh: one word per warp, not used again before the next barrier)
template <bool MAX, int THREADS>
__device__ __forceinline__ float norm_row_reduce(float x, float *sh) {
  auto op = [](float p, float q) { return MAX ? fmaxf(p, q) : p + q; };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = op(x, __shfl_xor_sync(0xffffffffu, x, o));
  const int warps = (int)(blockDim.x >> 5);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = x;
  __syncthreads();
  float t = 0.f;
  if (THREADS <= 256) {
    for (int i = 0; i < warps; ++i) t = op(t, sh[i]);
  } else {
    t = (int)(threadIdx.x & 31) < warps ? sh[threadIdx.x & 31] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t = op(t, __shfl_xor_sync(0xffffffffu, t, o));
  }
  return t;
}

// eight bf16 of a tensor of `total` elements as a 16-byte vector; at the tensor's end (ANY) element by element
template <bool ANY>
__device__ __forceinline__ void norm_load_vec(const uint16_t *base, int64_t at, int64_t total, uint32_t (&w)[4]) {
  if (!ANY || at + 8 <= total) {
    const uint4 q = *reinterpret_cast<const uint4 *>(base + at);
    w[0] = q.x; w[1] = q.y; w[2] = q.z; w[3] = q.w;
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint32_t l = at + 2 * e < total ? base[at + 2 * e] : 0u, h = at + 2 * e + 1 < total ? base[at + 2 * e + 1] : 0u;
      w[e] = l | (h << 16);
    }
  }
}
// the elements of a vector that belong to the row: columns c0 .. c0 + 7 within [0, n)
template <bool ANY>
__device__ __forceinline__ void norm_store_vec(uint16_t *base, int64_t at, int c0, int n, const uint32_t (&w)[4]) {
  if (!ANY || (c0 >= 0 && c0 + 8 <= n)) *reinterpret_cast<uint4 *>(base + at) = make_uint4(w[0], w[1], w[2], w[3]);
  else {
#pragma unroll
    for (int e = 0; e < 8; ++e) if ((unsigned)(c0 + e) < (unsigned)n) base[at + e] = (uint16_t)(w[e >> 1] >> ((e & 1) * 16));
  }
}

// clears the elements of a vector outside the row (its first column is c0)
__device__ __forceinline__ void norm_clear_outside(uint32_t (&w)[4], int c0, int n) {
#pragma unroll
  for (int e = 0; e < 8; ++e)
    if ((unsigned)(c0 + e) >= (unsigned)n) w[e >> 1] &= (e & 1) ? 0x0000FFFFu : 0xFFFF0000u;
}

// One row of the full-width form, held by the CTA as the bf16 pairs it came in: v = input, r = residual (fused add); vector i holds the columns
// 8 i - shift .. 8 i - shift + 7 (shift = 0 unless ANY), and elements outside the row are zeros.  red: a buffer per reduction, used by one row in two
// (so one barrier each).  Same arithmetic as the generic kernel.
// FLOATS (aligned rows): the abs-max is taken on the values before they are rounded (rounding to bf16 is monotonic: the largest rounded magnitude is the rounded largest one)
// and rows are stored from row pointers; without, on the rounded words and through norm_store_vec.  The results are the same, what nvcc makes of either is not: see the rule.
template <int NV, int THREADS, bool ANY, bool FLOATS>
__device__ __forceinline__ void norm_row_vec(const NormArgs &a, int64_t b, int shift, uint32_t (&v)[NV][4], const uint32_t (&r)[NV][4], float (*red)[32]) {
  const int n = (int)a.n, nvec = FLOATS ? (int)(a.n >> 3) : (shift + n + 7) >> 3;
  auto lo = norm_lo; auto hi = norm_hi;
  const int64_t off = b * a.n - shift;          // element of vector 0
  uint4 *rv = a.residual ? reinterpret_cast<uint4 *>(reinterpret_cast<uint16_t *>(a.residual) + off) : nullptr;
  auto inside = [&](int c) { return (unsigned)c < (unsigned)n; };
  auto whole = [&](int c0) { return !ANY || (c0 >= 0 && c0 + 8 <= n); };
  float s1 = 0.f;
  if (a.type == NORM_FUSED_ADD_RMS) {
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = threadIdx.x + j * blockDim.x;
      if (i < nvec) {
        const uint32_t (&rw)[4] = r[j];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float s_lo = __fadd_rn(lo(rw[e]), lo(v[j][e])), s_hi = __fadd_rn(hi(rw[e]), hi(v[j][e]));
          s1 = __fmaf_rn(s_lo, s_lo, s1); s1 = __fmaf_rn(s_hi, s_hi, s1);
          v[j][e] = pack_bf16x2(s_lo, s_hi);
        }
        if constexpr (FLOATS) rv[i] = make_uint4(v[j][0], v[j][1], v[j][2], v[j][3]);
        else norm_store_vec<ANY>(reinterpret_cast<uint16_t *>(a.residual), off + (int64_t)i * 8, i * 8 - shift, n, v[j]);
      }
    }
  } else if (a.type == NORM_RMS) {
#pragma unroll
    for (int j = 0; j < NV; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) { s1 = __fmaf_rn(lo(v[j][e]), lo(v[j][e]), s1); s1 = __fmaf_rn(hi(v[j][e]), hi(v[j][e]), s1); }
  } else {
#pragma unroll
    for (int j = 0; j < NV; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) { s1 = __fadd_rn(s1, lo(v[j][e])); s1 = __fadd_rn(s1, hi(v[j][e])); }
  }
  s1 = norm_row_reduce<false, THREADS>(s1, red[0]);
  float mean = 0.f, inv;
  if (a.type == NORM_LAYER) {
    mean = __fdiv_rn(s1, (float)a.n);
    float s2 = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = threadIdx.x + j * blockDim.x, c0 = i * 8 - shift;
      if (i < nvec && whole(c0)) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float d0 = __fadd_rn(lo(v[j][e]), -mean), d1 = __fadd_rn(hi(v[j][e]), -mean);
          s2 = __fmaf_rn(d0, d0, s2); s2 = __fmaf_rn(d1, d1, s2);
        }
      } else if (ANY && i < nvec) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float d0 = inside(c0 + 2 * e) ? __fadd_rn(lo(v[j][e]), -mean) : 0.f, d1 = inside(c0 + 2 * e + 1) ? __fadd_rn(hi(v[j][e]), -mean) : 0.f;
          s2 = __fmaf_rn(d0, d0, s2); s2 = __fmaf_rn(d1, d1, s2);
        }
      }
    }
    s2 = norm_row_reduce<false, THREADS>(s2, red[1]);
    inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(s2, (float)a.n), a.eps)));
  } else inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(s1, (float)a.n), a.eps)));
  AbsMax<uint16_t> am;
  float top = 0.f;
  const bool layer = a.type == NORM_LAYER, shifted = a.use_shift && layer;
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int i = threadIdx.x + j * blockDim.x, c0 = i * 8 - shift;
    if (i < nvec) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {          // two halves of four elements
        float g[4] = {1.f, 1.f, 1.f, 1.f}, bt[4] = {0.f, 0.f, 0.f, 0.f};
        if (a.use_scale) norm_params4<ANY>(a.gamma, a.gamma_dt, c0 + 4 * h, n, g);
        if (shifted) norm_params4<ANY>(a.beta, a.beta_dt, c0 + 4 * h, n, bt);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const uint32_t w = v[j][2 * h + e];
          float y0 = lo(w), y1 = hi(w);
          if (layer) { y0 = __fadd_rn(y0, -mean); y1 = __fadd_rn(y1, -mean); }
          y0 = __fmul_rn(y0, inv); y1 = __fmul_rn(y1, inv);
          if (a.use_scale) { y0 = __fmul_rn(y0, g[2 * e]); y1 = __fmul_rn(y1, g[2 * e + 1]); }
          if (shifted) { y0 = __fadd_rn(y0, bt[2 * e]); y1 = __fadd_rn(y1, bt[2 * e + 1]); }
          v[j][2 * h + e] = pack_bf16x2(y0, y1);
          if constexpr (FLOATS) { if (a.q) top = fmaxf(top, fmaxf(fabsf(y0), fabsf(y1))); }      // (a NaN does not enter fmaxf, an infinity does)
        }
      }
      if (!whole(c0)) norm_clear_outside(v[j], c0, n);
      if constexpr (FLOATS) {
        if (a.y) reinterpret_cast<uint4 *>(reinterpret_cast<uint16_t *>(a.y) + off)[i] = make_uint4(v[j][0], v[j][1], v[j][2], v[j][3]);
      } else {
        if (a.q) am.add(make_uint4(v[j][0], v[j][1], v[j][2], v[j][3]));
        if (a.y) norm_store_vec<ANY>(reinterpret_cast<uint16_t *>(a.y), off + (int64_t)i * 8, c0, n, v[j]);
      }
    }
  }
  if (a.q) {
    float amax = norm_row_reduce<true, THREADS>(FLOATS ? top : am.finite() ? __uint_as_float(am.bits()) : __int_as_float(0x7F800000), red[2]);
    if constexpr (FLOATS) amax = __uint_as_float(pack_bf16x2(amax, 0.0f) << 16);
    if (!finite_f32(amax)) {
      // an infinite or NaN element (it quantises to 0): the maximum over the finite values instead
      AbsMax<uint16_t> fin;
#pragma unroll
      for (int j = 0; j < NV; ++j) fin.add_finite(make_uint4(v[j][0], v[j][1], v[j][2], v[j][3]));
      amax = norm_row_reduce<true, THREADS>(__uint_as_float(fin.bits()), red[3]);
    }
    const float scale = scale_from_absmax(amax);
    const float rinv = __frcp_rn(scale);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = threadIdx.x + j * blockDim.x, c0 = i * 8 - shift;
      if (i < nvec) {
        const uint2 codes = quant_vec<uint16_t>(make_uint4(v[j][0], v[j][1], v[j][2], v[j][3]), scale, rinv);
        int8_t *o = a.q + b * a.q_ld + c0;
        if (whole(c0)) *reinterpret_cast<uint2 *>(o) = codes;
        else {
#pragma unroll
          for (int e = 0; e < 8; ++e) if (inside(c0 + e)) o[e] = (int8_t)((e < 4 ? codes.x : codes.y) >> ((e & 3) * 8));
        }
      }
    }
    if (threadIdx.x == 0) a.q_scale[b] = scale;
  }
}

// The decoder-layer case at full width: bf16 rows of at most NV * 8 * blockDim elements in 16-byte aligned tensors, bf16 out.  One
// CTA per row; a thread keeps its NV vectors of eight elements in registers (as the bf16 pairs they are at every stage that
// is kept) between the passes, so the row is read once and every access is a 16-byte vector (8 bytes for the s8 codes).
// Bound by HBM without the quantised output and by instruction issue with it (3.05 of 4 instructions a cycle): all loads of a row (input and
// residual) are in flight before the first store, each reduction costs one barrier, and the launch overlaps the kernel in front.  4096 rows of 4096 with residual add and s8 codes
// (151 MB): 36.9 -> 28.3 us (5.3 TB/s); a ring of rows filled by bulk copies ahead of persistent CTAs took 35.7 us (four CTAs per SM where
// there are six here).
// ANY: rows of any length, one behind the other.  A row is covered by the aligned vectors of the tensor that it touches (the first and the last shared with
// its neighbours, of which it writes its own elements only); input, residual, result and codes then need no shifting, the parameters are picked out of two
// aligned loads.  Instruction issue again: 8903 x 844 LayerNorm with codes 59 (element by element) -> 30 us, 3000 x 7001 with residual add and codes 197 -> 57,
// 2000 x 12287 220 -> 55; the registers of two and four vectors a thread leave two CTAs an SM or more (one: 85 us for the last).
template <int NV, int THREADS, int CTAS, bool ANY, bool FLOATS = false>
__global__ void __launch_bounds__(THREADS, CTAS) norm_rows_vec_kernel(const NormArgs a) {
  __shared__ float red[2][4][32];
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int64_t total = a.batch * a.n;
  int parity = 0;
  for (int64_t b = blockIdx.x; b < a.batch; b += gridDim.x, parity ^= 1) {
    const int shift = ANY ? (int)((b * a.n) & 7) : 0, n = (int)a.n, nvec = FLOATS ? (int)(a.n >> 3) : (shift + n + 7) >> 3;
    const int64_t off = b * a.n - shift;
    uint32_t v[NV][4], r[NV][4];
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int i = threadIdx.x + j * blockDim.x;
      if constexpr (!ANY) {
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
        const uint4 x = i < nvec ? reinterpret_cast<const uint4 *>(reinterpret_cast<const uint16_t *>(a.x) + off)[i] : zero;
        const uint4 y = a.type == NORM_FUSED_ADD_RMS && i < nvec ? reinterpret_cast<const uint4 *>(reinterpret_cast<const uint16_t *>(a.residual) + off)[i] : zero;
        v[j][0] = x.x; v[j][1] = x.y; v[j][2] = x.z; v[j][3] = x.w;
        r[j][0] = y.x; r[j][1] = y.y; r[j][2] = y.z; r[j][3] = y.w;
        continue;
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) v[j][e] = r[j][e] = 0u;
      if (i < nvec) {
        norm_load_vec<ANY>(reinterpret_cast<const uint16_t *>(a.x), off + (int64_t)i * 8, total, v[j]);
        if (a.type == NORM_FUSED_ADD_RMS) norm_load_vec<ANY>(reinterpret_cast<const uint16_t *>(a.residual), off + (int64_t)i * 8, total, r[j]);
        if (ANY && (i == 0 || i == nvec - 1)) { norm_clear_outside(v[j], i * 8 - shift, n); norm_clear_outside(r[j], i * 8 - shift, n); }
      }
    }
    norm_row_vec<NV, THREADS, ANY, FLOATS>(a, b, shift, v, r, red[parity]);
  }
}

// BatchNorm: element-wise with per-channel constants
__global__ void norm_batch_kernel(const NormArgs a, const float *mean, const float *var, int64_t C, int64_t spatial) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.batch * C * spatial) return;
  const int64_t c = (i / spatial) % C;
  const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(var[c], a.eps)));
  float y = __fmul_rn(__fadd_rn(load_as_f32(a.x, a.src_dt, i), -mean[c]), inv);
  if (a.use_scale) y = __fmul_rn(y, load_as_f32(a.gamma, a.gamma_dt, c));
  if (a.use_shift) y = __fadd_rn(y, load_as_f32(a.beta, a.beta_dt, c));
  norm_store(a.y, a.dst_dt, i, y);
}

}  // namespace

extern "C" int32_t b200dnn_normalization(const b200dnn_norm_t *d, void *stream) {
  B2_CHECK(d, B200DNN_FAILURE, "null descriptor");
  B2_ENTER(stream);
  Runtime &R = rt();
  // ---- the reference's checks, in its order and words (lowoha_normalization_utils.cpp:23-149)
  const bool quant = d->quant_dst != nullptr || d->quant_scale != nullptr;
  B2_CHECK(d->input, B200DNN_FAILURE, "Normalization: Input pointer is null");
  B2_CHECK(d->output || quant, B200DNN_FAILURE, "Normalization: Output pointer is null");
  B2_CHECK(d->norm_type >= NORM_LAYER && d->norm_type <= NORM_FUSED_ADD_RMS, B200DNN_FAILURE, "Normalization: norm_type not specified");
  auto known = [](int32_t dt) { return dt == B200DNN_F32 || dt == B200DNN_BF16 || dt == 2 /* f16 */; };
  B2_CHECK(known(d->src_dt), B200DNN_FAILURE, "Normalization: Unsupported source data type");
  B2_CHECK(known(d->dst_dt), B200DNN_FAILURE, "Normalization: Unsupported destination data type");
  B2_CHECK(!((d->src_dt == 2 && d->dst_dt == B200DNN_BF16) || (d->src_dt == B200DNN_BF16 && d->dst_dt == 2)), B200DNN_FAILURE,
           "Normalization: f16/bf16 cross-mixing between src and dst is not supported");
  B2_CHECK(d->batch > 0, B200DNN_FAILURE, "Normalization: batch must be > 0");
  B2_CHECK(d->norm_size > 0, B200DNN_FAILURE, "Normalization: norm_size must be > 0");
  if (d->use_scale) {
    B2_CHECK(d->gamma, B200DNN_FAILURE, "Normalization: use_scale=true but gamma pointer is null");
    B2_CHECK(known(d->gamma_dt), B200DNN_FAILURE, "Normalization: Unsupported gamma data type (%d). Supported: f32, bf16, f16", d->gamma_dt);
  }
  const bool rms = d->norm_type == NORM_RMS || d->norm_type == NORM_FUSED_ADD_RMS;
  if (d->use_shift && !rms) {
    B2_CHECK(d->beta, B200DNN_FAILURE, "Normalization: use_shift=true but beta pointer is null");
    B2_CHECK(known(d->beta_dt), B200DNN_FAILURE, "Normalization: Unsupported beta data type (%d). Supported: f32, bf16, f16", d->beta_dt);
  }
  if (d->norm_type == NORM_FUSED_ADD_RMS)
    B2_CHECK(d->residual, B200DNN_FAILURE, "Normalization: FUSED_ADD_RMS_NORM requires a non-null writable residual buffer");
  if (d->norm_type == NORM_BATCH) {
    B2_CHECK(d->running_mean, B200DNN_FAILURE, "Normalization: BatchNorm inference requires running_mean (pre-computed from training)");
    B2_CHECK(d->running_var, B200DNN_FAILURE, "Normalization: BatchNorm inference requires running_var (pre-computed from training)");
    B2_CHECK(d->num_channels > 0, B200DNN_FAILURE, "Normalization: BatchNorm needs num_channels > 0");
  }
  B2_CHECK(d->epsilon > 0.0f, B200DNN_FAILURE, "Normalization: epsilon must be > 0, got %g", (double)d->epsilon);
  // ---- what this library leaves out
  auto f16 = [](int32_t dt) { return dt == 2; };
  B2_CHECK(!f16(d->src_dt) && !f16(d->dst_dt) && !(d->use_scale && f16(d->gamma_dt)) && !(d->use_shift && !rms && f16(d->beta_dt)),
           B200DNN_UNIMPLEMENTED, "Normalization: f16 buffers are not implemented");
  if (quant) {
    B2_CHECK(d->quant_dst && d->quant_scale, B200DNN_FAILURE, "Normalization: the fused quantisation needs both quant_dst and quant_scale");
    B2_CHECK(d->norm_type != NORM_BATCH, B200DNN_UNIMPLEMENTED, "Normalization: no fused quantisation for BatchNorm");
    B2_CHECK(d->quant_ld >= d->norm_size, B200DNN_FAILURE, "Normalization: quant_ld smaller than norm_size");
    B2_CHECK(d->norm_size <= kNormSmemElems, B200DNN_UNIMPLEMENTED, "Normalization: the fused quantisation stages the row (norm_size <= %d)", kNormSmemElems);
  }

  const int64_t batch = d->batch, n = d->norm_size;
  const int64_t elems = d->norm_type == NORM_BATCH ? batch * d->num_channels * n : batch * n;
  NormArgs a{};
  a.type = d->norm_type; a.batch = batch; a.n = n; a.eps = d->epsilon;
  a.use_scale = d->use_scale ? 1 : 0; a.use_shift = d->use_shift ? 1 : 0;
  a.src_dt = d->src_dt; a.dst_dt = d->dst_dt; a.gamma_dt = d->gamma_dt; a.beta_dt = d->beta_dt;
  const void *p;
  B2_TRY(stage_in(d->input, (size_t)elems * dt_size(d->src_dt), st, &p));
  a.x = p;
  const int64_t n_par = d->norm_type == NORM_BATCH ? d->num_channels : n;
  if (a.use_scale) { B2_TRY(stage_in(d->gamma, (size_t)n_par * dt_size(d->gamma_dt), st, &p)); a.gamma = p; }
  if (a.use_shift && !rms) { B2_TRY(stage_in(d->beta, (size_t)n_par * dt_size(d->beta_dt), st, &p)); a.beta = p; }
  Staged o_y, o_res, o_q, o_s;
  o_y.copy_back = o_res.copy_back = o_q.copy_back = o_s.copy_back = false;
  if (d->output) { B2_TRY(stage_out(d->output, (size_t)elems * dt_size(d->dst_dt), st, &o_y)); a.y = o_y.dev; }
  if (d->norm_type == NORM_FUSED_ADD_RMS) {
    // the residual is read and written: bring a host buffer over first
    B2_TRY(stage_out(d->residual, (size_t)elems * dt_size(d->src_dt), st, &o_res, true));
    a.residual = o_res.dev;
  }
  if (quant) {
    B2_TRY(stage_out(d->quant_dst, (size_t)((batch - 1) * d->quant_ld + n), st, &o_q, d->quant_ld != n));
    B2_TRY(stage_out(d->quant_scale, (size_t)batch * 4, st, &o_s));
    a.q = (int8_t *)o_q.dev; a.q_ld = d->quant_ld; a.q_scale = (float *)o_s.dev;
  }
  if (d->norm_type == NORM_BATCH) {
    const void *m, *v;
    B2_TRY(stage_in(d->running_mean, (size_t)d->num_channels * 4, st, &m));
    B2_TRY(stage_in(d->running_var, (size_t)d->num_channels * 4, st, &v));
    norm_batch_kernel<<<(unsigned)((elems + 255) / 256), 256, 0, st>>>(a, (const float *)m, (const float *)v, d->num_channels, n);
  } else {
    // full-width form: bf16 in and out in 16-byte aligned tensors, at most 16384 columns; rows that are no whole vectors (ANY) need codes laid out as the rows are
    auto al16 = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    const bool any = n % 8 != 0;
    const bool vec = d->src_dt == B200DNN_BF16 && d->dst_dt == B200DNN_BF16 && n <= 16384 - (any ? 14 : 0) &&
                     al16(a.x) && al16(a.y) && al16(a.residual) && (!a.use_scale || al16(a.gamma)) && (!(a.use_shift && !rms) || al16(a.beta)) &&
                     (!a.q || ((any ? a.q_ld == n : a.q_ld % 8 == 0) && (reinterpret_cast<uintptr_t>(a.q) & 7) == 0)) && env_int("B200DNN_NORM_VEC", 1) != 0;
    if (vec) {
      const int nvec = (int)((n + (any ? 14 : 0)) / 8);          // vectors that a row touches at most
      // One vector per thread where all rows are in flight at once (a row's latency counts): up to three rows an SM of 2048 columns, one of 8192.  us with two and one, residual add
      // and codes: 130 x 512 3.1, 2.5; 400 x 2048 3.5, 3.2; 130 x 4096 3.5, 2.9; 130 x 2999 5.3, 4.5; but 400 x 4096 4.4, 5.9; 900 x 1024 3.8, 4.5.
      // Else two while the CTA grows with the row (more CTAs in flight), and four for many long rows, which then pay less for what every thread does once per
      // row -- from where on depends on the registers a vector takes: two inputs with a residual, and an unaligned row's (any) instructions weigh more.  us with two
      // and four at 4096 rows: residual add and codes 4096 columns 28.5, 29.2; 6144 41.0, 41.3; 8192 53.8, 51.6, without codes 43.8, 44.5; LayerNorm and codes 2048
      // 15.8, 16.7; 4096 28.3, 27.2; 8192 55.6, 49.3; unaligned 2999 residual add 34.3, 33.7.  (More than 12288 columns need four.)
      const int from = any ? 256 : a.type != NORM_FUSED_ADD_RMS ? (batch < 2048 ? 769 : 512) : a.q ? 769 : 1537;
      const bool one_wave = nvec <= 1024 && batch <= (int64_t)R.sm_count * (nvec <= 256 ? 3 : 1);
      // Aligned rows of more than 512 vectors in fewer than 768 rows: an SM holds three CTAs of 512 threads with two vectors, four of 384, and four of 256 with four.  Launches overlap, so
      // that up to half of what the device holds runs as in an idle one, and more as if it were full.  us with two and four, residual add and codes: 230 x 6400 5.7, 5.1;
      // 360 x 6656 5.9, 6.6; 520 x 6400 8.6, 6.7; 520 x 8192 9.8, 8.5; 360 x 5120 5.9, 5.7; 640 x 5120 8.2, 8.8; 160 x 5120 4.0, 4.3.
      const int64_t sm = R.sm_count;
      const bool four = !any && nvec > 512 && nvec <= 1024 && batch <= 4 * sm && (nvec <= 768 ? batch > 2 * sm : batch > 3 * sm || (2 * batch > 3 * sm && batch <= 2 * sm));
      // (many rows with residual add and no codes: 8000 x 6400 68.7, 65.2; 2100 x 7168 23.0, 23.3; 8192 columns see above)
      const bool four_plain = !any && nvec > 768 && nvec <= 960 && batch >= 2560;
      const int per = one_wave ? 1 : nvec > 1536 || four || four_plain || (batch >= (any ? 2048 : 768) && nvec >= from) ? 4 : 2;
      // up to 1024 rows whole warps for each of an SM's four schedulers (700 x 2560: 160 threads 6.3 us, 256 5.4); beyond, idle warps cost more (4096 x 2560: 22.4, 19.9),
      // but one in eight does not (4100 x 6400 with residual add and codes: 224 threads 45.1, 256 44.3)
      int threads = (int)round_up((nvec + per - 1) / per, 32);
      if (batch < 1024 && threads > 128) threads = (int)round_up(threads, 128);
      if (!any && per == 4 && threads == 224) threads = 256;
      // 96 threads (16 CTAs an SM) or 128 (12), as above: 760 x 1536 3.9, 3.8; 1024 4.2, 5.6; 1300 6.4, 5.6; 2100 6.5, 7.4
      if (!any && per == 2 && threads == 96 && (batch <= 6 * sm || (batch > 8 * sm && batch <= 12 * sm))) threads = 128;
      const int nv = (nvec + threads - 1) / threads;
      // FLOATS for two vectors in up to 256 threads, with codes (but 2048 rows and more with residual add: 3000 x 1024 1.018 times as long, 4096 x 4096 1.005) or where at most half of the rows that the device holds (six CTAs of 256 threads an SM) are there, RMSNorm in 256 threads up to seven rows an SM.  us without and with:
      // 160 x 4096 residual add and codes 3.75, 3.61, RMSNorm 2.82, 2.74; 8000 x 1024 LayerNorm and codes 15.3, 15.0; 900 x 4096 RMSNorm 5.24, 5.09; but 2000 x 768 residual add
      // 1.055 times as long, 900 x 1920 1.05, 460 x 4096 1.025; one vector a thread 1 x 4096 2.62, 2.81, and two in more threads 420 x 4800 6.5, 7.2.
      const bool floats = (a.q && (a.type != NORM_FUSED_ADD_RMS || batch < 2048)) || batch * threads <= sm * 3 * 256 || (a.type == NORM_RMS && threads == 256 && batch <= 7 * sm);
      const long long cap = (long long)R.sm_count * 64;
      const unsigned grid = (unsigned)(batch < cap ? batch : cap);
      auto go = [&](auto kern) { return launch_pdl(kern, grid, (unsigned)threads, 0, st, true, a); };
      auto pick = [&](auto one, auto one_1024, auto two, auto two_512, auto two_768, auto four_128, auto four_256, auto four_512) {
        if (nv <= 1) return threads <= 256 ? go(one) : go(one_1024);
        if (nv <= 2) return threads <= 256 ? go(two) : threads <= 512 ? go(two_512) : go(two_768);
        return threads <= 128 ? go(four_128) : threads <= 256 ? go(four_256) : go(four_512);
      };
      B2_TRY(any ? pick(norm_rows_vec_kernel<1, 256, 4, true>, norm_rows_vec_kernel<1, 1024, 1, true>, norm_rows_vec_kernel<2, 256, 5, true>, norm_rows_vec_kernel<2, 512, 2, true>, norm_rows_vec_kernel<2, 768, 2, true>,
                        norm_rows_vec_kernel<4, 128, 8, true>, norm_rows_vec_kernel<4, 256, 4, true>, norm_rows_vec_kernel<4, 512, 2, true>)
                 : pick(norm_rows_vec_kernel<1, 256, 6, false>, norm_rows_vec_kernel<1, 1024, 1, false>, floats ? norm_rows_vec_kernel<2, 256, 6, false, true> : norm_rows_vec_kernel<2, 256, 6, false>, norm_rows_vec_kernel<2, 512, 3, false>, norm_rows_vec_kernel<2, 768, 2, false>,
                        norm_rows_vec_kernel<4, 128, 8, false>, norm_rows_vec_kernel<4, 256, 4, false>, norm_rows_vec_kernel<4, 512, 2, false>));
      B2_LAUNCHED();
      B2_CUDA(cudaGetLastError());
      return finish_out({&o_y, &o_res, &o_q, &o_s}, st);
    }
    a.staged = n <= kNormSmemElems ? 1 : 0;
    const size_t smem = a.staged ? (size_t)n * 4 : 0;
    B2_TRY(ensure_max_smem((const void *)norm_rows_kernel, (size_t)kNormSmemElems * 4));
    // short rows: fewer threads per row, more rows in flight per SM
    int threads = kNormThreads;
    while (threads > 32 && n < threads * 4) threads >>= 1;
    const long long cap = (long long)R.sm_count * 32;
    const unsigned grid = (unsigned)(batch < cap ? batch : cap);
    norm_rows_kernel<<<grid, threads, smem, st>>>(a);
  }
  B2_LAUNCHED();
  B2_CUDA(cudaGetLastError());
  return finish_out({&o_y, &o_res, &o_q, &o_s}, st);
}

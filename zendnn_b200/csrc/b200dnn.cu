// libb200dnn: extern "C" entry points (include/b200dnn.h) over the sm_100a kernels.
// Validation mirrors the INT8 rules of the reference's validator
// (matmul/lowoha_matmul_utils.cpp:180-420) for the supported subset; everything else returns
// unimplemented, never a different computation.
#include <cudaTypedefs.h>
#include <algorithm>
#include <chrono>

#include "runtime.cuh"
#include "common.cuh"
#include "matmul_validate.cuh"
#include "quant_kernels.cuh"
#include "pack_kernels.cuh"
#include "stream_gemm.cuh"
#include "decode_gemm.cuh"
#include "decode_ring.cuh"
#include "tc_gemm.cuh"
#include "skinny_gemm.cuh"
#include "moe_few.cuh"
#include "moe_kernels.cuh"
#include "sdpa_flash_api.cuh"

using namespace b200;

namespace {

cudaStream_t as_stream(void *s) { return reinterpret_cast<cudaStream_t>(s); }

// ------------------------------------------------------------------------------------ prepack
int32_t pack_into(const void *w_dev, int64_t K, int64_t N, int64_t ldb, int transB, int gated, void *dst_dev,
                  cudaStream_t st, PackedWeight *out) {
  const int64_t Kp = round_up(K, 128), Np = round_up(N, 128);
  const int64_t I = gated ? N / 2 : 0;
  if (gated) B2_CHECK(N % 2 == 0 && I % kGateGranule == 0, B200DNN_UNIMPLEMENTED,
                      "gated prepack needs N = 2*I with I a multiple of %d (N=%lld)", kGateGranule, (long long)N);
  uint8_t *base = reinterpret_cast<uint8_t *>(dst_dev);
  B2_CHECK((reinterpret_cast<uintptr_t>(base) & 255) == 0, B200DNN_FAILURE, "prepack destination must be 256-byte aligned");
  int32_t *colsum = reinterpret_cast<int32_t *>(base + kPackHeaderBytes);
  int8_t *wt = reinterpret_cast<int8_t *>(base + kPackHeaderBytes + Np * 4);
  pack_header_kernel<<<1, kPackHeaderBytes / 4, 0, st>>>(reinterpret_cast<PackHeader *>(base), K, N, Kp, Np, gated, I);
  B2_LAUNCHED();
  dim3 grid((unsigned)(Kp / 64), (unsigned)(Np / 32));
  pack_weight_kernel<<<grid, 256, 0, st>>>(reinterpret_cast<const int8_t *>(w_dev), ldb, transB, K, N, Kp, gated, I, wt);
  B2_LAUNCHED();
  pack_colsum_kernel<<<(unsigned)((Np + 7) / 8), 256, 0, st>>>(wt, Np, Kp, colsum);
  B2_LAUNCHED();
  B2_CUDA(cudaGetLastError());
  if (out) { out->colsum = colsum; out->wt = wt; out->K = K; out->N = N; out->Kp = Kp; out->Np = Np; out->gated = gated; out->I = I; }
  return B200DNN_SUCCESS;
}

PackedWeight view_of(const void *dev_base, const PackHeader &h) {
  PackedWeight pw;
  const uint8_t *b = reinterpret_cast<const uint8_t *>(dev_base);
  pw.colsum = reinterpret_cast<const int32_t *>(b + kPackHeaderBytes);
  pw.wt = reinterpret_cast<const int8_t *>(b + kPackHeaderBytes + h.Np * 4);
  pw.K = h.K; pw.N = h.N; pw.Kp = h.Kp; pw.Np = h.Np; pw.gated = h.gated; pw.I = h.I;
  return pw;
}

// A cache-owned packed weight was written on the stream of the call that first saw it: a call on another stream waits for that work.
// Until the work has been seen complete once the weight is `fresh` for every call: no kernel may read it ahead of its own
// griddepcontrol.wait.  (The order of the stream is no help there: a kernel that triggers its dependents before its own wait, as the
// GEMM kernels do, lets them start while the packing in front of it may still be on its way to memory.)  An event recorded during a
// stream capture cannot be asked, and each replay packs again: such a weight stays fresh.  Callers hold the cache mutex.
int32_t take_cached(PackedWeight &entry, cudaStream_t st, PackedWeight *pw) {
  if (!entry.complete && entry.ready) {
    if (!entry.captured) {
      RelaxedCapture relaxed;      // an event query is not a capturable call: allowed while this thread captures a graph
      if (cudaEventQuery(entry.ready) == cudaSuccess) entry.complete = true; else cudaGetLastError();
    }
    if (!entry.complete && st != entry.ready_stream) B2_CUDA(cudaStreamWaitEvent(st, entry.ready, 0));
  }
  *pw = entry;
  pw->fresh = !entry.complete;
  return B200DNN_SUCCESS;
}
int32_t mark_ready(PackedWeight &pw, cudaStream_t st) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) cudaGetLastError();
  B2_CUDA(cudaEventCreateWithFlags(&pw.ready, cudaEventDisableTiming));
  B2_CUDA(cudaEventRecord(pw.ready, st));
  pw.ready_stream = st; pw.complete = false; pw.captured = cap != cudaStreamCaptureStatusNone;
  return B200DNN_SUCCESS;
}

// Resolves the weight argument of a GEMM to a packed device buffer.  The caches belong to the device and are shared
// by all streams; the mutex is held while a new weight is packed (once per weight).
int32_t resolve_weight(const void *weight, int wei_format, int64_t K, int64_t N, int64_t ldb, int transB, int gated,
                       int weights_const, cudaStream_t st, PackedWeight *pw) {
  DeviceShared &D = *rt().shared;
  if (wei_format == 'r') {
    std::lock_guard<std::mutex> lk(D.cache_mu);
    if (is_device_ptr(weight)) {
      auto it = D.packed_registry.find(weight);
      if (it == D.packed_registry.end()) {
        PackHeader h;
        B2_CUDA(cudaMemcpyAsync(&h, weight, sizeof h, cudaMemcpyDeviceToHost, st));
        B2_CUDA(cudaStreamSynchronize(st));
        B2_CHECK(h.magic == kPackMagic, B200DNN_FAILURE, "mem_format_b='r' but the weight buffer was not written by b200dnn_prepack");
        it = D.packed_registry.emplace(weight, view_of(weight, h)).first;
      }
      *pw = it->second;
    } else {
      auto it = D.host_packed.find(weight);
      if (it == D.host_packed.end()) {
        PackHeader h; memcpy(&h, weight, sizeof h);
        B2_CHECK(h.magic == kPackMagic, B200DNN_FAILURE, "mem_format_b='r' but the weight buffer was not written by b200dnn_prepack");
        size_t bytes = pack_bytes(h.K, h.N);
        void *d = nullptr;
        B2_CUDA(cudaMalloc(&d, bytes));
        B2_CUDA(cudaMemcpyAsync(d, weight, bytes, cudaMemcpyHostToDevice, st));
        PackedWeight v = view_of(d, h); v.owned = d;
        B2_TRY(mark_ready(v, st));
        it = D.host_packed.emplace(weight, v).first;
      }
      B2_TRY(take_cached(it->second, st, pw));
    }
    B2_CHECK(pw->K == K && pw->N == N && pw->gated == gated, B200DNN_FAILURE,
             "prepacked weight is K=%lld N=%lld gated=%d, call asks for K=%lld N=%lld gated=%d", (long long)pw->K,
             (long long)pw->N, pw->gated, (long long)K, (long long)N, gated);
    return B200DNN_SUCCESS;
  }
  B2_CHECK(wei_format == 'n' || wei_format == 0, B200DNN_FAILURE, "mem_format_b must be 'n' or 'r'");
  auto key = std::make_tuple(weight, K, N, ldb, transB, gated);
  const bool cache = weights_const && env_int("ZENDNNL_MATMUL_WEIGHT_CACHE", 1) != 0;
  std::unique_lock<std::mutex> lk(D.cache_mu, std::defer_lock);
  if (cache) {
    lk.lock();
    auto it = D.wcache.find(key);
    if (it != D.wcache.end()) return take_cached(it->second, st, pw);
  }
  const int64_t wrows = transB ? N : K, wcols = transB ? K : N;
  const void *w_dev = nullptr;
  B2_TRY(stage_in(weight, span_bytes(wrows, wcols, ldb, B200DNN_S8), st, &w_dev));
  void *buf = nullptr;
  if (cache) B2_CUDA(cudaMalloc(&buf, pack_bytes(K, N)));
  else { buf = rt().ws.alloc(pack_bytes(K, N)); B2_CHECK(buf, B200DNN_FAILURE, "workspace allocation failed"); }
  B2_TRY(pack_into(w_dev, K, N, ldb, transB, gated, buf, st, pw));
  if (cache) { pw->owned = buf; B2_TRY(mark_ready(*pw, st)); D.wcache.emplace(key, *pw); }
  pw->fresh = true;
  return B200DNN_SUCCESS;
}

// ------------------------------------------------------------------------------------ quant helpers
template <bool EP>
int32_t launch_quant_rows_t(const RowQuantArgs &a, int32_t src_dt, int64_t rows, cudaStream_t st) {
  if (rows <= 0) return B200DNN_SUCCESS;
  // a warp per row takes aligned, non-grouped rows of up to 16 vectors a lane (bf16: 4096 elements)
  const int E = src_dt == B200DNN_BF16 ? 8 : 4;
  const bool aligned = a.n_groups == 0 && a.K % E == 0 && (reinterpret_cast<uintptr_t>(a.src) & 15) == 0 &&
                       (a.src_ld * (src_dt == B200DNN_BF16 ? 2 : 4)) % 16 == 0 &&
                       (!a.dst || ((reinterpret_cast<uintptr_t>(a.dst) % E) == 0 && a.dst_ld % E == 0));
  // rows whose abs-max is known: the streaming form (B200DNN_QUANT_STREAM=0 keeps the row-per-CTA kernel)
  if (aligned && a.absmax_bits && !a.gather && !a.scatter && rows >= 64 && a.K / E >= 64 &&
      (src_dt == B200DNN_BF16 || src_dt == B200DNN_F32) && env_int("B200DNN_QUANT_STREAM", 1) != 0) {
    // five CTAs of eight warps per SM are resident; rows are cut into segments (multiples of 128 vectors: four loads per
    // lane) until every warp has several items, so the last wave is short
    const int nvec = a.K / E;
    const long long warps = (long long)rt().sm_count * 5 * 8;
    int segs = 1;
    while (segs < 8 && rows * segs < 4 * warps && (nvec + segs) / (segs + 1) >= 128) ++segs;
    const int seg_len = (((nvec + segs - 1) / segs) + 31) & ~31;
    segs = (nvec + seg_len - 1) / seg_len;
    long long want = (rows * segs + 7) / 8;
    const unsigned grid = (unsigned)(want < rt().sm_count * 5 ? want : rt().sm_count * 5);
    // (eight loads in flight per lane measured slower: 110 against 92 us at configuration 4)
    if (src_dt == B200DNN_BF16) B2_TRY(launch_pdl(quant_known_absmax_kernel<uint16_t, 4>, grid, 256, 0, st, !EP, a, (int)rows, segs, seg_len));
    else B2_TRY(launch_pdl(quant_known_absmax_kernel<float, 4>, grid, 256, 0, st, !EP, a, (int)rows, segs, seg_len));
    B2_LAUNCHED();
    B2_CUDA(cudaGetLastError());
    return B200DNN_SUCCESS;
  }
  B2_CHECK(src_dt == B200DNN_BF16 || (!EP && src_dt == B200DNN_F32), B200DNN_UNIMPLEMENTED, "per-token quantisation takes f32 or bf16 input");
  // rows of any alignment (an odd K, say): vectors put together from words instead of element by element
  const bool any = !EP && !aligned && a.n_groups == 0 && !a.scatter && !a.absmax_bits && (!a.dst || (reinterpret_cast<uintptr_t>(a.dst) % E == 0 && a.dst_ld % E == 0));
  // A warp per row or a CTA per row.  A warp's chain is the longer one; it pays where the CTAs of two launches, which overlap, no longer fit the chip at
  // once (three a SM and launch), with nine to sixteen vectors a lane where those of one do not.  Device time, us, CTA and warp, bf16: K = 1024 400 rows
  // 1.8 and 1.9, 448 rows 2.3 and 1.9; K = 2048 128 rows 1.6 and 2.4, 512 rows 2.6 and 2.4, 4096 rows 8.3 and 4.5; K = 4096 128 rows 1.8 and 3.5, 1024
  // rows 3.6 and 3.8, 4096 rows 10.6 and 8.8; scattered to two places, K = 4096, 880 rows 4.0 and 4.7, 900 rows 4.8 and 4.7.  Vectors put together from words take a
  // warp longer still: K = 1021 640 rows 2.7 and 2.9, 4096 rows 8.5 and 6.4; K = 2045 1024 rows 3.9 and 5.2, K = 4093 4096 rows 15 and 25.
  // B200DNN_QUANT_WARP: -1 by these lines, 0 never, 1 whenever the row fits.
  const int nv = (a.K + 32 * E - 1) / (32 * E), qw = env_int("B200DNN_QUANT_WARP", -1), sms = rt().sm_count;      // nv: vectors a lane
  const long long line = any ? (nv <= 2 ? 3 : 7) * sms : nv <= 2 ? 64 : (nv <= 8 ? 3 : a.scatter ? 6 : 7) * sms;
  if ((aligned ? nv <= 16 : any && nv <= 4) && (qw < 0 ? rows >= line : qw != 0)) {
    unsigned grid = (unsigned)((rows + 7) / 8);
    if (EP && a.n_rows_dev && grid > (unsigned)(sms * 16)) grid = (unsigned)(sms * 16);   // the warps stride over the rows
#define B2_QW(T, NV) B2_TRY((launch_pdl(quant_per_token_warp_kernel<T, NV, EP>, grid, 256, 0, st, !EP, a, (int)rows)))
#define B2_QWA(T, NV) B2_TRY((launch_pdl(quant_per_token_warp_kernel<T, NV, false, true>, grid, 256, 0, st, true, a, (int)rows)))
    if (any) {      // (not in the expert-parallel forms)
      if (src_dt == B200DNN_BF16) { if (nv <= 2) B2_QWA(uint16_t, 2); else B2_QWA(uint16_t, 4); }
      else { if (nv <= 2) B2_QWA(float, 2); else B2_QWA(float, 4); }
    } else if (src_dt == B200DNN_BF16) { if (nv <= 2) B2_QW(uint16_t, 2); else if (nv <= 4) B2_QW(uint16_t, 4); else if (nv <= 8) B2_QW(uint16_t, 8); else B2_QW(uint16_t, 16); }
    else if constexpr (!EP) { if (nv <= 2) B2_QW(float, 2); else if (nv <= 4) B2_QW(float, 4); else if (nv <= 8) B2_QW(float, 8); else B2_QW(float, 16); }
#undef B2_QWA
#undef B2_QW
    B2_LAUNCHED();
    B2_CUDA(cudaGetLastError());
    return B200DNN_SUCCESS;
  }
  const int nvec = (a.K + E - 1) / E;
  const bool short_row = nvec <= 2 * kQuantThreads;     // the whole row fits two cached vectors per thread
  // few long rows (fewer than SMs): as many threads as keep a row in two vectors each, see quant_per_token_kernel
  const bool wide = !short_row && rows <= sms;
  unsigned grid_rows = (unsigned)rows;
  if (EP && a.n_rows_dev && grid_rows > (unsigned)(sms * 32)) grid_rows = (unsigned)(sms * 32);   // the CTAs stride over the rows
  // rows that do not all start on 16 bytes, or whose length is no multiple of a vector
  const bool src_any = !EP && !a.scatter && (a.K % E != 0 || (a.n_groups > 0 ? a.g_any != 0 : ((reinterpret_cast<uintptr_t>(a.src) | (uintptr_t)(a.src_ld * (16 / E))) & 15) != 0));
#define B2_QR(T, NV, FORM, THR, ANY) B2_TRY((launch_pdl(quant_per_token_kernel<T, NV, FORM, THR, ANY>, grid_rows, THR, 0, st, !EP, a)))
#define B2_QRF(T, NV, THR) do { \
    if constexpr (EP) B2_QR(T, NV, kRowsPeers, THR, false); \
    else if (a.n_groups > 0) { if (src_any) B2_QR(T, NV, kRowsGroups, THR, true); else B2_QR(T, NV, kRowsGroups, THR, false); } \
    else if (a.scatter) B2_QR(T, NV, kRowsScatter, THR, false); \
    else if (src_any) B2_QR(T, NV, kRowsPlain, THR, true); \
    else B2_QR(T, NV, kRowsPlain, THR, false); } while (0)
  if (src_dt == B200DNN_BF16) { if (short_row) B2_QRF(uint16_t, 2, kQuantThreads); else if (wide) B2_QRF(uint16_t, 2, 1024); else B2_QRF(uint16_t, kQuantRegVec, kQuantThreads); }
  else if constexpr (!EP) { if (short_row) B2_QRF(float, 2, kQuantThreads); else if (wide) B2_QRF(float, 2, 1024); else B2_QRF(float, kQuantRegVec, kQuantThreads); }
#undef B2_QRF
#undef B2_QR
  B2_LAUNCHED();
  B2_CUDA(cudaGetLastError());
  return B200DNN_SUCCESS;
}
int32_t launch_quant_rows(const RowQuantArgs &a, int32_t src_dt, int64_t rows, cudaStream_t st) {
  if (a.n_rows_dev || a.scatter_peer) return launch_quant_rows_t<true>(a, src_dt, rows, st);
  return launch_quant_rows_t<false>(a, src_dt, rows, st);
}

// ------------------------------------------------------------------------------------ GEMM launchers
int32_t launch_stream(const uint8_t *A, int64_t lda, bool a_unsigned, int M, int N, int K, const PackedWeight &pw,
                      const EpiParams &epi, cudaStream_t st) {
  Runtime &R = rt();
  StreamGemmArgs g{};
  g.A = A; g.lda = lda; g.M = M; g.N = N; g.K = K; g.Wt = pw.wt; g.Kp = (int)pw.Kp;
  g.chunks_total = (int)(pw.Kp / 64);
  // shape heuristic: enough CTAs to cover the SMs about twice, K range per CTA >= 1024 bytes
  int nb = env_int("B200DNN_STREAM_NB", 4);
  if (nb != 1 && nb != 2 && nb != 4 && nb != 8) nb = 4;
  g.nb = nb; g.kw = 8 / nb;
  const int tiles_n = (N + nb * 8 - 1) / (nb * 8);
  const int tiles_m = (M + 15) / 16;
  int ksplit = env_int("B200DNN_STREAM_KSPLIT", 0);
  if (ksplit <= 0) {
    ksplit = 1;
    while (tiles_n * tiles_m * ksplit < 2 * R.sm_count && g.chunks_total / (ksplit * 2) >= 16) ksplit *= 2;
  }
  if (ksplit > g.chunks_total) ksplit = g.chunks_total;
  g.chunks_per_cta = (g.chunks_total + ksplit - 1) / ksplit;
  ksplit = (g.chunks_total + g.chunks_per_cta - 1) / g.chunks_per_cta;
  const int kbytes = g.chunks_per_cta * 64;
  g.a_stride = (int)round_up(kbytes, 128) + 64;
  size_t smem = (size_t)16 * g.a_stride;
  if (smem < 4096) smem = 4096;
  B2_CHECK(smem <= 200 * 1024, B200DNN_FAILURE, "streaming kernel: K range per CTA too large (%d bytes)", kbytes);
  const size_t tiles = (size_t)tiles_n * tiles_m;
  if (ksplit > 1) {
    B2_CHECK(tiles <= R.n_counters, B200DNN_FAILURE, "streaming kernel: too many tiles for the split-K counters");
    g.partial = (int32_t *)R.ws.alloc(tiles * ksplit * 16 * nb * 8 * sizeof(int32_t));
    B2_CHECK(g.partial, B200DNN_FAILURE, "workspace allocation failed");
    g.counters = R.counters;
  }
  dim3 grid(tiles_n, ksplit, tiles_m);
  if (a_unsigned) {
    B2_TRY(ensure_max_smem((const void *)stream_gemm_kernel<true>, 200 * 1024));
    stream_gemm_kernel<true><<<grid, 256, smem, st>>>(g, epi);
  } else {
    B2_TRY(ensure_max_smem((const void *)stream_gemm_kernel<false>, 200 * 1024));
    stream_gemm_kernel<false><<<grid, 256, smem, st>>>(g, epi);
  }
  B2_LAUNCHED();
  B2_CUDA(cudaGetLastError());
  return B200DNN_SUCCESS;
}

// Shared memory of decode_gemm_kernel: staged rows, sums and epilogue operands of the CTA's column groups.
size_t decode_smem(int M, int N, int64_t Kp) {
  const int groups = (N + 7) / 8, grid = groups < rt().sm_count ? groups : rt().sm_count, local = (groups + grid - 1) / grid;
  return (size_t)(M > 8 ? 16 : 8) * (size_t)(Kp + 16) + (size_t)local * 512 + decode_epi_bytes(local);
}
// Decode-shape kernel (M <= 16): persistent, evenly split over all warps of the device.
// Returns unimplemented when the shape does not fit it (the caller then uses the tiled streaming kernel).
int32_t launch_decode(const uint8_t *A, int64_t lda, bool a_unsigned, int M, int N, int K, const PackedWeight &pw,
                      const EpiParams &epi, bool early_weights, cudaStream_t st, const DecodeQuant &dq = DecodeQuant{}) {
  Runtime &R = rt();
  DecodeGemmArgs g{};
  g.A = A; g.lda = lda; g.M = M; g.N = N; g.K = K; g.Wt = pw.wt; g.Kp = (int)pw.Kp;
  g.groups = (N + 7) / 8; g.blocks = (int)(pw.Kp / 128);
  g.a_stride = (int)pw.Kp + 16;
  g.rows_staged = M > 8 ? 16 : 8;
  const int grid = g.groups < R.sm_count ? g.groups : R.sm_count;
  g.max_local_groups = (g.groups + grid - 1) / grid;
  g.tune = env_int("B200DNN_DECODE_TUNE", 0);
  const size_t smem = decode_smem(M, N, pw.Kp);
  if (M > 16 || smem > 220 * 1024) return B200DNN_UNIMPLEMENTED;
  void (*kern)(DecodeGemmArgs, EpiParams, DecodeQuant) = dq.src ? decode_gemm_kernel<false, true> : a_unsigned ? decode_gemm_kernel<true> : decode_gemm_kernel<false>;
  B2_TRY(ensure_max_smem((const void *)kern));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid); cfg.blockDim = dim3(kDecodeWarps * 32); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = early_weights ? 1 : 0;
  B2_CUDA(cudaLaunchKernelEx(&cfg, kern, g, epi, dq));
  B2_LAUNCHED();
  return B200DNN_SUCCESS;
}

// Ring form of the decode GEMM (decode_ring.cuh).  unimplemented when the ring would be too shallow, or has fewer warps than rows to quantise.
template <int R>
int32_t launch_decode_ring(const uint8_t *A, int64_t lda, bool a_unsigned, int M, int N, int K, const PackedWeight &pw,
                           const EpiParams &epi, bool early_weights, cudaStream_t st, const DecodeQuant &dq) {
  Runtime &R_ = rt();
  DecodeRingArgs g{};
  g.A = A; g.lda = lda; g.M = M; g.N = N; g.K = K; g.Wt = pw.wt; g.Kp = (int)pw.Kp;
  g.groups = (N + 7) / 8; g.blocks = (int)(pw.Kp / 128);
  g.a_stride = (int)pw.Kp + 16;
  g.rows_staged = M > 8 ? 16 : M;
  const int grid = g.groups < R_.sm_count ? g.groups : R_.sm_count;
  g.max_local_groups = (g.groups + grid - 1) / grid;
  g.status = R_.status;
  g.test_no_loads = env_int("B200DNN_TEST_NO_LOADS", 0);   // see decode_ring.cuh; off unless a test sets it
  const size_t stage_bytes = (size_t)R * kRingWarps * 1024;
  const size_t fixed = ring_off_ring(g.rows_staged, g.a_stride, g.max_local_groups);
  const size_t budget = 227 * 1024;
  if (M > 16 || fixed + 3 * stage_bytes > budget || (dq.src && M > kRingWarps)) return B200DNN_UNIMPLEMENTED;
  int stages = (int)((budget - fixed) / stage_bytes);
  const int need = ((g.max_local_groups + R - 1) / R) * ((g.blocks + kRingWarps - 1) / kRingWarps);
  if (stages > kRingMaxStages) stages = kRingMaxStages;
  if (stages > need) stages = need;
  // three stages measured best: a deeper ring delays the activation loads behind its own requests
  const int cap = env_int("B200DNN_RING_STAGES", 3);
  if (cap > 1 && stages > cap) stages = cap;
  g.stages = stages;
  const size_t smem = fixed + (size_t)stages * stage_bytes;
  void (*kern)(DecodeRingArgs, EpiParams, DecodeQuant) = dq.src ? decode_ring_kernel<false, R, true> : a_unsigned ? decode_ring_kernel<true, R> : decode_ring_kernel<false, R>;
  B2_TRY(ensure_max_smem((const void *)kern));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid); cfg.blockDim = dim3((kRingWarps + 1) * 32); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = early_weights ? 1 : 0;
  B2_CUDA(cudaLaunchKernelEx(&cfg, kern, g, epi, dq));
  B2_LAUNCHED();
  return B200DNN_SUCCESS;
}

#ifdef B200DNN_TIMING_EXPERIMENTS
constexpr size_t kStampCtas = 4096;
unsigned long long *stamp_buffer() {
  static unsigned long long *p = nullptr;
  if (!p && cudaMalloc(&p, kStampCtas * 8 * sizeof(unsigned long long)) != cudaSuccess) p = nullptr;
  return p;
}
extern "C" __attribute__((visibility("default"))) int32_t b200dnn_debug_stamps(unsigned long long *host, int32_t ctas) {
  if (!stamp_buffer() || ctas < 0 || (size_t)ctas > kStampCtas) return B200DNN_FAILURE;
  return cudaMemcpy(host, stamp_buffer(), (size_t)ctas * 8 * sizeof(unsigned long long), cudaMemcpyDeviceToHost) == cudaSuccess ? B200DNN_SUCCESS : B200DNN_FAILURE;
}
#endif

// CTAs of a kernel that are resident at once when it is launched in clusters of s (clusters do not tile the GPCs perfectly); -1: none.
// Kept per device in *cache (0: not asked yet).  Several threads may ask at once: each stores the answer only when it has it, because a
// caller that met something else would split K another way, and f32 sums with it.
template <typename K>
int cluster_room(K kern, int threads, int smem, int s, std::atomic<int> *cache) {
  int room = cache->load(std::memory_order_relaxed);
  if (room != 0) return room;
  room = -1;
  if (ensure_max_smem((const void *)kern, smem) == B200DNN_SUCCESS) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(s * 64)); cfg.blockDim = dim3((unsigned)threads); cfg.dynamicSmemBytes = (size_t)smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)s; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0) room = n * s;
    else cudaGetLastError();
    if (env_int("B200DNN_DEBUG", 0)) fprintf(stderr, "b200dnn: clusters of %d (%d threads): %d resident CTAs\n", s, threads, room);
  }
  cache->store(room, std::memory_order_relaxed);
  return room;
}
int split_room(int s) { return cluster_room(tc_gemm_kernel<true>, kTcThreads, kTcSmemBudget + 1024, s, &rt().shared->split_room[s]); }

// ---- form and tile of a tcgen05 GEMM ------------------------------------------------------------------------------------------
// Microseconds of one launch, fitted to 375 plain GEMMs (M 65 to 8192, K and N 512 to 14336, INT8 and bf16) in every form and width, 23 times
// each: within 10 % (standard deviation).  A wave of tiles costs a part that grows with the width (the epilogue that nothing hides) and, per 128-byte block
// of K, the slower of a floor (the MMAs, or what a block costs beside them: barriers, issue) and its operands' way from L2 to shared memory at the
// measured 20.4 (17.5 in the pair form) TB/s; the last wave only what its tiles ask for.  Operands and result also have to pass DRAM.
// bf16: wide pair tiles keep the tensor pipe so busy that the clock gives way.  Choosing by it is 0.8 % off the best form and width on average;
// the rules before (waves times width + 16; pairs from two tiles per pair of SMs; a split model of its own) 9.5 %.  Largest differences, us: M = 3615,
// K = 5824, N = 576 in bf16 43.0 -> 28.4; M = 825, K = 1280, N = 10752 in INT8 22.9 -> 14.6; M = 4096, K = 14336, N = 4096 201 -> 161.
// Every plain call asks for it about forty times: terms of a form and width are in a table, divisions of 32 bits (the choice 0.19 -> 0.10 us of host time).
struct TcForm { double wave, per_kb, bytes; };      // us of a wave beside its blocks; of a block at least; of a block and tile in flight
struct TcForms {
  TcForm f[2][8];                                   // [one CTA a tile, a pair][width / 32 - 1]
  constexpr TcForms() : f{} {
    const double floor[2][8] = {{0.195, 0.20, 0.20, 0.20, 0.225, 0.24, 0.295, 0.315}, {0.205, 0.205, 0.206, 0.208, 0.217, 0.222, 0.26, 0.29}};
    for (int p = 0; p < 2; ++p)
      for (int i = 0; i < 8; ++i) {
        const int bn = 32 * (i + 1);
        f[p][i] = {p ? 0.63 + 1.9 * bn / 256.0 : 0.32 + 1.7 * bn / 256.0, floor[p][i], ((p ? 256 : 128) + bn) * 128.0 / (p ? 17.5e6 : 20.4e6)};
      }
  }
};
constexpr TcForms kTcForms;
inline double tc_dram_us(double bytes) { return 4.0 + bytes / 4.15e6; }
inline double tc_cost_us(bool pair, int bn, int splits, unsigned tiles, int k_blocks, double dram_us, bool f16, unsigned sms) {
  const TcForm &w = kTcForms.f[pair][bn / 32 - 1];
  const int kb = splits == 1 ? k_blocks : (k_blocks + splits - 1) / splits;
  const unsigned conc = pair ? sms / 2 : sms, ctas = tiles * (unsigned)splits, full = ctas / conc, last = ctas - full * conc;
  const double per_kb = pair && f16 && bn >= 224 && tiles > conc ? 1.08 * w.per_kb : w.per_kb;
  double t = pair ? 5.3 : 4.55;
  if (splits > 1) t += 1.6 + 0.77 / 128.0 * ((splits - 1) * bn);
  if (full) t += (double)full * (w.wave + kb * std::max(per_kb, w.bytes * (double)conc));
  if (last) t += w.wave + kb * std::max(per_kb, w.bytes * (double)last);
  return std::max(t, dram_us) + 0.15 * std::min(t, dram_us);
}

struct TcChoice { int pair, bn, splits; };

// Knobs: B200DNN_TC_PAIR -1 (default) by cost, 0 never, 1 whenever the shape allows; B200DNN_TC_BN, B200DNN_TC_KSPLIT (1 never, 2 to 4 that many).
TcChoice tc_choose(long long M, int N, int k_blocks, bool f16) {
  const int mode = env_int("B200DNN_TC_PAIR", -1), forced_bn = env_int("B200DNN_TC_BN", 0), forced = env_int("B200DNN_TC_KSPLIT", 0);
  const double dram_us = tc_dram_us((double)k_blocks * 128.0 * (double)(M + N) + 2.0 * (double)M * N);
  const unsigned sms = (unsigned)rt().sm_count, m128 = (unsigned)((M + 127) / 128), m256 = (m128 + 1) / 2;
  TcChoice best{0, forced_bn > 0 ? forced_bn : 128, 1};
  double best_us = 1e30;
  auto consider = [&](int pair, int bn, int s, unsigned tiles) {
    const double us = tc_cost_us(pair != 0, bn, s, tiles, k_blocks, dram_us, f16, sms);
    if (us < best_us) { best_us = us; best = {pair, bn, s}; }
  };
  const bool pair_ok = N >= 128 && mode != 0 && forced < 2, single_ok = !(mode == 1 && N >= 128) || forced >= 2;
  for (int bn = 256; bn >= 32; bn -= 32) {
    const bool width = forced_bn > 0 ? bn == forced_bn : true;
    if (!width) continue;
    const unsigned n_tiles = (unsigned)(N + bn - 1) / (unsigned)bn, tiles = m128 * n_tiles;
    if (pair_ok && bn >= 64) consider(1, bn, 1, m256 * n_tiles);
    if (!single_ok) continue;
    if (forced < 2) consider(0, bn, 1, tiles);
    if (forced == 1 || (forced_bn <= 0 && bn != 64 && bn != 128 && bn != 256)) continue;
    // clusters of 2 to 4 CTAs share a tile, each with K blocks of its own and at least one 32-column chunk to finish; the int32 partial sums are added
    // through distributed shared memory, so the result is the same bit for bit.  All clusters are resident at once, with room for two more where they
    // are of three: those do not tile the GPCs, and behind another kernel the last ones wait (M = 100, K = 7168 behind the quantisation, in two and three
    // shares, us: 45 tiles 15.3 and 20.8, 44 tiles 15.3 and 18.0, 43 tiles 15.2 and 15.4, 42 tiles 15.1 and 14.3).
    for (int s = 2; s <= 4; ++s) {
      if (bn / 32 < s || (forced >= 2 && s != forced) || (forced < 2 && tiles * s > sms)) continue;
      const int per = (k_blocks + s - 1) / s;
      if (per * (s - 1) >= k_blocks || per < 2) continue;
      if (forced < 2 && (int)(tiles * s) + (s == 3 ? 6 : 0) > split_room(s)) continue;
      consider(0, bn, s, tiles);
    }
  }
  if (best_us > 1e29 && forced_bn <= 0) consider(0, 128, 1, m128 * ((unsigned)(N + 127) / 128u));        // (a knob that fits no form)
  return best;
}

// Tile width of a grouped GEMM whose row tiles (128 rows, or 256 in the pair form) are counted already.  Gated: whole 64-column gate/up blocks in every
// CTA's part of a tile.
int pick_bn(int m_tiles, int N, int k_blocks, int gated, int pair, bool f16) {
  const int forced = env_int("B200DNN_TC_BN", 0);
  if (forced > 0) return forced;
  const int step = gated ? (pair ? 128 : 64) : 32;
  int best = 0;
  double best_us = 0.0;
  for (int bn = 256; bn >= (gated ? step : 64); bn -= step) {
    const double us = tc_cost_us(pair != 0, bn, 1, (unsigned)m_tiles * ((unsigned)(N + bn - 1) / (unsigned)bn), k_blocks, tc_dram_us(0.0), f16, (unsigned)rt().sm_count);
    if (best == 0 || us < best_us) { best = bn; best_us = us; }
  }
  return best;
}

// Rows of a row tile of a grouped GEMM over about `rows` rows: 256 (pair form, two CTAs per tile) for large problems, else 128.
int tc_tile_rows(long long rows, int N) {
  const int mode = env_int("B200DNN_TC_PAIR", -1);
  if (mode == 0 || N < 128) return kTcBM;
  if (mode == 1) return 2 * kTcBM;
  // worth it once every CTA pair has several tiles: the pair form wastes up to 255 rows at the end of a group
  const long long tiles = ((rows + 255) / 256) * ((N + 255) / 256);
  return tiles >= 2LL * (rt().sm_count / 2) ? 2 * kTcBM : kTcBM;
}

// The epilogue's FA_* code of a post-op chain.
int fast_act_code(const EpiParams &epi) {
  if (epi.n_po == 0) return FA_NONE;
  if (epi.n_po != 1) return FA_GENERIC;
  switch (epi.po[0].type) {
  case PO_RELU: return FA_RELU;
  case PO_GELU_TANH: return FA_GELU_TANH;
  case PO_GELU_ERF: return FA_GELU_ERF;
  case PO_SIGMOID: return FA_SIGMOID;
  case PO_SWISH: return FA_SWISH;
  case PO_TANH: return FA_TANH;
  default: return FA_GENERIC;
  }
}

// Plain or grouped tcgen05 GEMM (plain: form and tile are chosen here; grouped: args.pair and m_tiles_hint, its bound on row tiles, are given).
// A: [M_total, lda] device, 16-byte aligned rows.  bf16 form (args.f16): K and lda count
// bytes (two per element) and pw0 holds a bf16 pack.
int32_t launch_tc(const uint8_t *A, int64_t lda, bool a_unsigned, int M_total, int N, int K, const PackedWeight &pw0,
                  TcGemmArgs args, const EpiParams &epi, int m_tiles_hint, cudaStream_t st) {
  Runtime &R = rt();
  CUtensorMap map_a, map_b, map_c;
  B2_TRY(make_map_2d(&map_a, A, (uint64_t)K, (uint64_t)M_total, (uint64_t)lda, kTcBM));
  args.M_total = M_total; args.N = N; args.k_blocks = (int)(pw0.Kp / 128);
  args.a_unsigned = a_unsigned ? 1 : 0; args.gated = pw0.gated; args.status = R.status;
  args.fast_act = fast_act_code(epi);
  args.test_no_loads = env_int("B200DNN_TEST_NO_LOADS", 0);   // see tc_gemm.cuh; off unless a test sets it
  args.stamps = nullptr;
#ifdef B200DNN_TIMING_EXPERIMENTS
  args.dbg = env_int("B200DNN_TC_DBG", 0);    // parts of the epilogue switched off: results are invalid
  if (env_int("B200DNN_TC_STAMPS", 0)) args.stamps = stamp_buffer();
#else
  args.dbg = 0;
#endif
  const bool plain = args.n_groups <= 1 && !args.maps_b && !args.groups && !args.tile_prefix && !pw0.gated;
  args.k_splits = 1;
  if (plain) {
    const TcChoice c = tc_choose(M_total, N, args.k_blocks, args.f16 != 0);
    args.pair = c.pair; args.BN = c.bn; args.k_splits = c.splits;
    args.n_groups = 1; args.m_tiles_plain = m_tiles_hint = (M_total + (c.pair ? 255 : 127)) / (c.pair ? 256 : 128);
  } else args.BN = pick_bn(m_tiles_hint, N, args.k_blocks, pw0.gated, args.pair, args.f16 != 0);
  B2_CHECK(args.BN % 32 == 0 && args.BN >= 32 && args.BN <= 256 && (!pw0.gated || args.BN % 64 == 0), B200DNN_FAILURE,
           "bad tile width %d", args.BN);
  B2_CHECK(!args.pair || (args.BN % 32 == 0 && args.BN >= 64 && (!pw0.gated || args.BN % 128 == 0)), B200DNN_FAILURE,
           "bad tile width %d for the pair form", args.BN);
  args.n_tiles = (N + args.BN - 1) / args.BN;
  // Tile order.  Sweeping the row tiles under one column tile keeps that weight slice hot and re-reads the
  // activations once per column tile.  When the weight of a group is small enough to stay in L2 and the
  // activations are the larger operand (many rows, as in a fine-grained MoE), the column tiles of one row tile
  // run together instead: activations are read once, the weight is re-read from L2.
  // Which one moves fewer DRAM bytes is estimated from what the L2 can keep (ncu on the down projection of a
  // Mixtral-like layer, 14336 x 4096 per expert: column-tile-major read the 117 MB of activations once per wave of tiles,
  // 1.43 GB for 0.59 GB of operands; row-tile-major finishes an expert in about one wave).
  {
    const long long kL2 = 96ll << 20;                                   // what a sweep can count on, of 126 MB
    const long long w_group = (long long)pw0.Kp * pw0.Np, groups = args.n_groups > 0 ? args.n_groups : 1;
    const long long w_all = w_group * groups, a_bytes = (long long)M_total * K;
    const long long conc = R.sm_count / (args.pair ? 2 : 1);           // tiles in flight
    const long long tiles_all = (long long)m_tiles_hint * args.n_tiles;
    const long long waves = (tiles_all + conc - 1) / conc;
    // column-tile-major: the activations survive between the waves only if they fit beside the weight slices in flight
    const long long a_reads = (a_bytes + w_all / (args.n_tiles > 0 ? args.n_tiles : 1) <= kL2) ? 1 : (waves < args.n_tiles ? waves : args.n_tiles);
    const long long traffic_col = w_all + a_bytes * a_reads;
    // row-tile-major: a group's weight is read again for every wave of that group's row tiles unless it stays in L2
    const long long tiles_group = ((long long)m_tiles_hint + groups - 1) / groups * args.n_tiles;
    const long long w_reads = (w_group <= kL2 / 2) ? 1 : (tiles_group + conc - 1) / conc;
    const long long traffic_row = a_bytes + w_all * w_reads;
    args.n_fastest = env_int("B200DNN_TC_ORDER", traffic_row < traffic_col ? 1 : 0);
  }
  const int stage_bytes = kTcBM * kTcBK + (args.pair ? args.BN / 2 : args.BN) * kTcBK;   // per CTA
  int stages = kTcSmemBudget / stage_bytes;
  if (stages > 8) stages = 8;
  int forced_stages = env_int("B200DNN_TC_STAGES", 0);
  if (forced_stages > 0 && forced_stages <= stages) stages = forced_stages;
  args.stages = stages;
  B2_TRY(make_map_wt(&map_b, pw0.wt, (uint64_t)pw0.Kp, (uint64_t)pw0.Np, (uint32_t)(args.pair ? args.BN / 2 : args.BN)));
  const size_t smem = (size_t)stages * stage_bytes + 1024;
  B2_TRY(ensure_max_smem((const void *)tc_gemm_kernel<false>, kTcSmemBudget + 1024));   // the kernel also has static shared memory
  long long tiles = (long long)m_tiles_hint * args.n_tiles;
  int grid = (int)(tiles < R.sm_count ? (tiles > 0 ? tiles : 1) : R.sm_count);
  // bf16 results into one shared destination (plain GEMM, or a grouped GEMM whose groups all write epi.dst at their
  // global row): whole 32-row blocks leave as TMA stores.  Measured: 9 % faster for short-K plain GEMMs, no gain for long K.  The gated form keeps the
  // load/store path, one 32-byte store of a lane's own row: neither is the faster (60 MoE layers, 32 to 16384 tokens, one call after the other in either form:
  // 0.2 % apart on average; eight experts of 14336, 4096 tokens 1323 us in both, 64 of 1408, 16384 tokens 1300 and 1289 with TMA stores).
  // B200DNN_TC_TMA_STORE: 0 never, 1 always, 2 (default) all but the gated form.
  {
    const int64_t cols = pw0.gated ? epi.gated_I : N;
    const bool can = args.shared_dst && epi.dst_dt == B200DNN_BF16 && epi.dst && cols * 2 >= 32 &&
                     ((reinterpret_cast<uintptr_t>(epi.dst) | (uintptr_t)(epi.ldc * 2)) & 15) == 0 &&
                     (env_int("B200DNN_TC_TMA_STORE", 2) == 1 || (env_int("B200DNN_TC_TMA_STORE", 2) == 2 && !pw0.gated));
    args.tma_store = can ? 1 : 0;
    if (can) B2_TRY(make_map_store(&map_c, epi.dst, (uint64_t)cols * 2, (uint64_t)M_total, (uint64_t)epi.ldc * 2));
    else map_c = map_a;
  }
  // Both forms are launched with the programmatic-serialisation attribute: the kernel waits (griddepcontrol.wait) for
  // everything before it in the stream before it touches global memory, so the ordering is that of a plain launch; what
  // overlaps with the tail of the previous kernel is the launch itself.
  {
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = dim3(kTcThreads); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (env_int("B200DNN_PDL", 1) != 0) {
      attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[na].val.programmaticStreamSerializationAllowed = 1;
      ++na;
    }
    if (args.pair) {
      // clusters of two CTAs, one [256 x BN] tile at a time per cluster, persistent over the tiles
      B2_TRY(ensure_max_smem((const void *)tc_gemm_kernel<false, true>, kTcSmemBudget + 1024));
      attr[na].id = cudaLaunchAttributeClusterDimension;
      attr[na].val.clusterDim.x = 2; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = 1;
      ++na;
      const long long pairs = tiles < R.sm_count / 2 ? (tiles > 0 ? tiles : 1) : R.sm_count / 2;
      cfg.gridDim = dim3((unsigned)(2 * pairs));
      cfg.attrs = attr; cfg.numAttrs = na;
      if (args.f16) {
        B2_TRY(ensure_max_smem((const void *)tc_gemm_kernel<false, true, true>, kTcSmemBudget + 1024));
        B2_CUDA(cudaLaunchKernelEx(&cfg, tc_gemm_kernel<false, true, true>, map_a, map_b, map_c, args, epi));
      } else B2_CUDA(cudaLaunchKernelEx(&cfg, tc_gemm_kernel<false, true>, map_a, map_b, map_c, args, epi));
    } else if (args.k_splits > 1) {
      // one cluster of k_splits CTAs per tile; the partial sums need BN * 512 bytes of the stage ring
      B2_CHECK((size_t)args.BN * 512 <= (size_t)stages * stage_bytes, B200DNN_FAILURE, "split form: stage ring smaller than the partial sums");
      B2_TRY(ensure_max_smem((const void *)tc_gemm_kernel<true>, kTcSmemBudget + 1024));
      attr[na].id = cudaLaunchAttributeClusterDimension;
      attr[na].val.clusterDim.x = (unsigned)args.k_splits; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = 1;
      ++na;
      cfg.gridDim = dim3((unsigned)(tiles * args.k_splits));
      cfg.attrs = attr; cfg.numAttrs = na;
      if (args.f16) {
        B2_TRY(ensure_max_smem((const void *)tc_gemm_kernel<true, false, true>, kTcSmemBudget + 1024));
        B2_CUDA(cudaLaunchKernelEx(&cfg, tc_gemm_kernel<true, false, true>, map_a, map_b, map_c, args, epi));
      } else B2_CUDA(cudaLaunchKernelEx(&cfg, tc_gemm_kernel<true>, map_a, map_b, map_c, args, epi));
    } else {
      cfg.gridDim = dim3((unsigned)grid);
      cfg.attrs = attr; cfg.numAttrs = na;
      if (args.f16) {
        B2_TRY(ensure_max_smem((const void *)tc_gemm_kernel<false, false, true>, kTcSmemBudget + 1024));
        B2_CUDA(cudaLaunchKernelEx(&cfg, tc_gemm_kernel<false, false, true>, map_a, map_b, map_c, args, epi));
      } else B2_CUDA(cudaLaunchKernelEx(&cfg, tc_gemm_kernel<false>, map_a, map_b, map_c, args, epi));
    }
  }
  B2_LAUNCHED();
  B2_CUDA(cudaGetLastError());
  return B200DNN_SUCCESS;
}

int skinny_room(int s) { return cluster_room(skinny_gemm_kernel<false>, kSkinnyThreads, kSkinnyRing + 1024, s, &rt().shared->skinny_room[s]); }

// Few rows (skinny_gemm.cuh).  A: [M, lda] device bytes, 16-byte aligned rows; K and lda count bytes; early: see SkinnyArgs.
int32_t launch_skinny(const uint8_t *A, int64_t lda, bool a_unsigned, bool f16, int M, int N, int K, const PackedWeight &pw, const EpiParams &epi,
                      int fast_act, bool early, cudaStream_t st) {
  Runtime &R = rt();
  SkinnyArgs g{};
  g.M = M; g.N = N; g.k_blocks = (int)(pw.Kp / 128); g.MP = (M + 15) & ~15;
  g.a_unsigned = a_unsigned ? 1 : 0; g.fast_act = fast_act; g.early = early ? 1 : 0; g.status = R.status;
  g.test_no_loads = env_int("B200DNN_TEST_NO_LOADS", 0);
  B2_CHECK(M >= 1 && g.MP <= kSkinnyMaxM, B200DNN_FAILURE, "skinny form: %d rows", M);
  // Shares of K: the fewest microseconds by a model of the stream (6.5 TB/s over the device, at most 65 GB/s an SM) plus the additions
  // through distributed shared memory, among the choices that are resident at once.  Fitted to 200 measured (M, K, N, shares): within 0.4 % of the
  // best on average, 8 % at worst.  (With 100 GB/s an SM it took too few shares: bf16, M = 33, K = 3520, N = 8384: 17.5 us with one, 15.3 with two;
  // M = 33, K = N = 4096: 12.7 with two, 11.0 with four.)
  const int tiles = (N + 127) / 128;
  int best = 1;
  double best_us = 1e30;
  const int forced = env_int("B200DNN_SKINNY_SPLIT", 0);
  for (int s = 1; s <= kSkinnyMaxSplits; ++s) {
    if (s > 1 && (g.k_blocks < 4 * s || (long long)tiles * s > skinny_room(s))) continue;
    if (forced > 0 && s != forced) continue;
    const long long ctas = (long long)tiles * s, room = R.sm_count;
    const long long live = ctas < room ? ctas : room;
    const double rate = std::min(6.5e6 / (double)live, 6.5e4);           // bytes per microsecond and CTA
    const double us = (double)((g.k_blocks + s - 1) / s) * (128 * 128 + g.MP * 128) / rate * (double)((ctas + room - 1) / room) + 0.15 * s;
    if (us < best_us) { best_us = us; best = s; }
  }
  g.splits = best;
  const int stage_bytes = 128 * 128 + g.MP * 128;
  int stages = kSkinnyRing / stage_bytes;
  const int per = (g.k_blocks + best - 1) / best;
  if (stages > kSkinnyMaxStages) stages = kSkinnyMaxStages;
  if (stages > per) stages = per;
  g.stages = stages;
  size_t smem = (size_t)stages * stage_bytes;
  if (smem < (size_t)g.MP * 512) smem = (size_t)g.MP * 512;      // the partial sums lie over the ring
  smem += 1024;
  CUtensorMap map_a, map_w;
  B2_TRY(make_map_2d(&map_a, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda, (uint32_t)g.MP));
  B2_TRY(make_map_wt(&map_w, pw.wt, (uint64_t)pw.Kp, (uint64_t)pw.Np, 128));
  auto kern = f16 ? skinny_gemm_kernel<true> : skinny_gemm_kernel<false>;
  B2_TRY(ensure_max_smem((const void *)kern, kSkinnyRing + 1024));
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(tiles * best)); cfg.blockDim = dim3(kSkinnyThreads); cfg.dynamicSmemBytes = smem; cfg.stream = st;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (env_int("B200DNN_PDL", 1) != 0) {
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  if (best > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = (unsigned)best; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = 1;
    ++na;
  }
  cfg.attrs = attr; cfg.numAttrs = na;
  B2_CUDA(cudaLaunchKernelEx(&cfg, kern, map_a, map_w, g, epi));
  B2_LAUNCHED();
  return B200DNN_SUCCESS;
}

// Does the few-row kernel beat the tile kernel?  col_bytes: bytes of a weight column.  Up to 24 rows over 1400 shapes (M 1 to 64, K 512 to 14336, N 512
// to 50176, bf16 and INT8) the choice was 0.7 % off the better of the two on average; above 24 rows, over 840 shapes (M 17 to 64, K 512 to 14336, N 512 to
// 28672, device time), it is 0.3 % off in INT8 and 0.2 % in bf16, 12 % at worst.  (With the lines fitted to an earlier tile kernel, and none of more than 48
// INT8 rows: 3.0 and 1.1 %, 75 % at worst: K = 14336, N = 512, M = 56 12.8 us in tiles, 7.3 here; bf16, K = 1024, N = 11008, M = 64 7.4 and 10.9.)
//   - Column tiles for at most one wave of CTAs: always up to 24 rows (bf16, K = 4096, N = 1024, M = 16: 6.6 us against 12.5); with more rows the
//     fixed cost of handling them (about 0.04 us a row) must be less than what the tile kernel loses by not sharing K (about 0.9 us a KiB
//     of column).  Above 48 rows and 40 tiles that takes 4096 bytes (K = 2048, N = 9472, M = 64 in INT8: 7.5 in tiles, 9.2 here).  With tiles for more than half the
//     SMs no CTA shares K and the rows are paid in full: columns of 3072 to 8191 bytes (4096 x 11008, M = 48: 11.2 and 13.3), and above 48 rows shorter ones
//     too, go to the tile kernel.
//   - More column tiles than SMs: the kernel is not persistent, so its last wave must be well filled (K = 8192, N = 20480 is 160 tiles: 71
//     against 60 us for 8 rows; N = 50176 is 392 and K = 4096: 69 against 107), and every tile pays for its rows again (K = 4096, N = 28672:
//     8 rows 44 against 56, 32 rows 48 against 45).  Columns of at most 512 bytes are one short burst each: 12.9 against 17.1 (N = 50176).
bool few_rows_pay(int M, int N, int64_t col_bytes) {
  const long long tiles = (N + 127) / 128, sms = rt().sm_count, waves = (tiles + sms - 1) / sms;
  if (waves == 1) {
    if (M <= 24) return true;
    if (col_bytes < 32ll * ((M + 15) & ~15)) return false;
    if (M <= 32) return true;
    if (2 * tiles <= sms) return M <= 48 || tiles <= 40 || col_bytes >= 4096;
    return col_bytes >= 8192 || (M <= 48 && col_bytes < 3072);
  }
  if (M <= 24 && col_bytes <= 512) return true;
  return 3 * tiles >= 2 * waves * sms && (M <= 8 || (M <= 24 && col_bytes >= 3072));
}

// the stream has been drained: report a kernel that gave up on one of its bounded waits
int32_t check_tc_status(cudaStream_t st) {
  B2_CUDA(cudaStreamSynchronize(st));
  return read_status();
}

int32_t fill_epi(const b200dnn_matmul_t *d, EpiParams *e) {
  memset(e, 0, sizeof *e);
  e->dst_dt = d->dst_dt; e->ldc = d->ldc;
  e->bias_dt = d->bias_dt;
  e->n_po = d->n_postops;
  return B200DNN_SUCCESS;
}

}  // namespace

namespace {
// matmul_direct's transA: the source arrives as [K, lda] (element (m, k) at k * lda + m) and is transposed into the
// workspace as [M, pitch]; 32 x 32 tiles through shared memory, elements of 1, 2 or 4 bytes.
template <typename T>
__global__ void transpose_src_kernel(const T *src, int64_t lda, int M, int K, T *dst, int64_t pitch) {
  __shared__ T tile[32][33];
  const int k0 = blockIdx.y * 32, m0 = blockIdx.x * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int k = k0 + r, m = m0 + threadIdx.x;
    if (k < K && m < M) tile[r][threadIdx.x] = src[(int64_t)k * lda + m];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int m = m0 + r, k = k0 + threadIdx.x;
    if (m < M && k < K) dst[(int64_t)m * pitch + k] = tile[threadIdx.x][r];
  }
}

// Rows that are not 16-byte aligned, copied to a pitch the copy engine takes (16-byte multiple, zero-padded): 16 bytes per thread, counted in bytes.
// Launched with overlap: the launch hides behind the kernel in front, and the GEMM behind it may start early (the trigger comes after the wait, so
// whatever such a GEMM reads before its own wait was written by work that is complete).
__global__ void __launch_bounds__(256) repitch_rows_kernel(const uint8_t *src, int64_t src_ld, uint8_t *dst, int pitch, int rows, int cols) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int segs = pitch >> 4;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)rows * segs) return;
  const int r = (int)(i / segs), k = (int)(i - (int64_t)r * segs) * 16;
  *reinterpret_cast<uint4 *>(dst + (int64_t)r * pitch + k) = ld16_any(src + (int64_t)r * src_ld + k, cols - k);
}
// rows of `cols` bytes, `ld` apart -> workspace rows, *pitch apart
int32_t repitch_rows(const uint8_t *src, int64_t ld, int rows, int cols, cudaStream_t st, const uint8_t **out, int64_t *pitch) {
  *pitch = round_up(cols, 16);
  uint8_t *tmp = (uint8_t *)rt().ws.alloc((size_t)rows * *pitch);
  B2_CHECK(tmp, B200DNN_FAILURE, "workspace allocation failed");
  B2_TRY(launch_pdl(repitch_rows_kernel, (unsigned)(((int64_t)rows * (*pitch / 16) + 255) / 256), 256u, 0, st, true, src, ld, tmp, (int)*pitch, rows, cols));
  B2_LAUNCHED();
  *out = tmp;
  return B200DNN_SUCCESS;
}

int32_t untranspose_source(const b200dnn_matmul_t *d, b200dnn_matmul_t *t, cudaStream_t st) {
  const int M = d->M, K = d->K;
  B2_CHECK(d->src && M > 0 && K > 0, B200DNN_FAILURE, "null src or non-positive dimension");
  B2_CHECK(d->lda >= M, B200DNN_FAILURE, "transA: lda smaller than M");
  const size_t esz = dt_size(d->src_dt);
  B2_CHECK(esz == 1 || esz == 2 || esz == 4, B200DNN_UNIMPLEMENTED, "transA: source dtype %d", d->src_dt);
  const void *src = nullptr;
  B2_TRY(stage_in(d->src, span_bytes(K, M, d->lda, d->src_dt), st, &src));
  const int64_t pitch = round_up(K, (int64_t)(16 / esz));
  void *buf = rt().ws.alloc((size_t)M * pitch * esz);
  B2_CHECK(buf, B200DNN_FAILURE, "workspace allocation failed");
  if (pitch != K) B2_CUDA(cudaMemsetAsync(buf, 0, (size_t)M * pitch * esz, st));
  dim3 grid((unsigned)((M + 31) / 32), (unsigned)((K + 31) / 32)), block(32, 8);
  if (esz == 1) transpose_src_kernel<uint8_t><<<grid, block, 0, st>>>((const uint8_t *)src, d->lda, M, K, (uint8_t *)buf, pitch);
  else if (esz == 2) transpose_src_kernel<uint16_t><<<grid, block, 0, st>>>((const uint16_t *)src, d->lda, M, K, (uint16_t *)buf, pitch);
  else transpose_src_kernel<uint32_t><<<grid, block, 0, st>>>((const uint32_t *)src, d->lda, M, K, (uint32_t *)buf, pitch);
  B2_LAUNCHED();
  B2_CUDA(cudaGetLastError());
  *t = *d;
  t->transA = 0; t->src = buf; t->lda = pitch;
  return B200DNN_SUCCESS;
}
}  // namespace

#include "gs_api.cuh"
#include "bf16_api.cuh"
#include "woq_api.cuh"

// =========================================================================================== C ABI
extern "C" {

const char *b200dnn_last_error(void) { return err_text().c_str(); }
int32_t b200dnn_version(void) { return 100; }
int32_t b200dnn_device_count(void) { return device_count(); }
int64_t b200dnn_launch_count(void) { return launch_counter().load(); }

size_t b200dnn_prepack_size(int64_t K, int64_t N, int32_t gated) {
  (void)gated;
  if (K <= 0 || N <= 0) return 0;
  return (pack_bytes(K, N) + 63) & ~size_t(63);
}

int32_t b200dnn_prepack(const void *weight, int64_t K, int64_t N, int64_t ldb, int32_t transB, int32_t gated, void *dst,
                        void *stream) {
  B2_ENTER(stream);
  B2_CHECK(weight && dst && K > 0 && N > 0, B200DNN_FAILURE, "prepack: null pointer or non-positive dimension");
  B2_CHECK(ldb >= (transB ? K : N), B200DNN_FAILURE, "prepack: ldb=%lld too small", (long long)ldb);
  const void *w_dev = nullptr;
  B2_TRY(stage_in(weight, span_bytes(transB ? N : K, transB ? K : N, ldb, B200DNN_S8), st, &w_dev));
  Staged out;
  B2_TRY(stage_out(dst, pack_bytes(K, N), st, &out));
  PackedWeight pw;
  B2_TRY(pack_into(w_dev, K, N, ldb, transB, gated, out.dev, st, &pw));
  {
    DeviceShared &D = *rt().shared;
    std::lock_guard<std::mutex> lk(D.cache_mu);
    if (!out.copy_back && !out.sync) D.packed_registry[dst] = pw;
    else {
      auto it = D.host_packed.find(dst);
      if (it != D.host_packed.end()) { if (it->second.owned) cudaFree(it->second.owned); if (it->second.ready) cudaEventDestroy(it->second.ready); D.host_packed.erase(it); }
    }
  }
  return finish_out({&out}, st);
}

int32_t b200dnn_quant_per_token(const void *src, int32_t src_dt, int64_t M, int64_t K, int64_t src_ld, void *dst,
                                int64_t dst_ld, void *scale, int32_t scale_dt, void *stream) {
  B2_ENTER(stream);
  B2_CHECK(src && scale, B200DNN_FAILURE, "dynamic quantisation needs src and a scale buffer");
  B2_CHECK(M > 0 && K > 0 && src_ld >= K && (!dst || dst_ld >= K), B200DNN_FAILURE, "bad shape or stride");
  B2_CHECK(scale_dt == B200DNN_F32 || scale_dt == B200DNN_BF16, B200DNN_UNIMPLEMENTED, "scale dtype must be f32 or bf16");
  const void *s_dev = nullptr;
  B2_TRY(stage_in(src, span_bytes(M, K, src_ld, src_dt), st, &s_dev));
  Staged o_q, o_s;
  B2_TRY(stage_out(dst, span_bytes(M, K, dst_ld, B200DNN_S8), st, &o_q, dst && dst_ld != K));
  B2_TRY(stage_out(scale, (size_t)M * dt_size(scale_dt), st, &o_s));
  RowQuantArgs a{};
  a.src = s_dev; a.src_ld = src_ld; a.dst = (int8_t *)o_q.dev; a.dst_ld = dst_ld; a.scale = o_s.dev; a.scale_dt = scale_dt;
  a.K = (int32_t)K; a.gather_div = 1;
  B2_TRY(launch_quant_rows(a, src_dt, M, st));
  return finish_out({&o_q, &o_s}, st);
}

int32_t b200dnn_quant_per_token_asym(const void *src, int32_t src_dt, int64_t M, int64_t K, int64_t src_ld, void *dst,
                                     int64_t dst_ld, float *scale, int32_t *zero_point, void *stream) {
  B2_ENTER(stream);
  B2_CHECK(src && scale && zero_point, B200DNN_FAILURE, "asymmetric dynamic quantisation needs src, a scale buffer and a zero-point buffer");
  B2_CHECK(M > 0 && K > 0 && src_ld >= K && (!dst || dst_ld >= K), B200DNN_FAILURE, "bad shape or stride");
  B2_CHECK(src_dt == B200DNN_BF16 || src_dt == B200DNN_F32, B200DNN_UNIMPLEMENTED, "source must be f32 or bf16");
  const void *s_dev = nullptr;
  B2_TRY(stage_in(src, span_bytes(M, K, src_ld, src_dt), st, &s_dev));
  Staged o_q, o_s, o_z;
  B2_TRY(stage_out(dst, span_bytes(M, K, dst_ld, B200DNN_U8), st, &o_q, dst && dst_ld != K));
  B2_TRY(stage_out(scale, (size_t)M * 4, st, &o_s));
  B2_TRY(stage_out(zero_point, (size_t)M * 4, st, &o_z));
  if (src_dt == B200DNN_BF16)
    quant_per_token_asym_kernel<uint16_t><<<(unsigned)M, kQuantThreads, 0, st>>>((const uint16_t *)s_dev, src_ld, (int)K, (uint8_t *)o_q.dev, dst_ld, (float *)o_s.dev, (int32_t *)o_z.dev);
  else
    quant_per_token_asym_kernel<float><<<(unsigned)M, kQuantThreads, 0, st>>>((const float *)s_dev, src_ld, (int)K, (uint8_t *)o_q.dev, dst_ld, (float *)o_s.dev, (int32_t *)o_z.dev);
  B2_LAUNCHED();
  B2_CUDA(cudaGetLastError());
  return finish_out({&o_q, &o_s, &o_z}, st);
}

int32_t b200dnn_group_quant_per_token(int32_t num_groups, const void *const *src, int32_t src_dt, const int32_t *M,
                                      const int32_t *K, const int64_t *src_ld, void *const *dst, const int64_t *dst_ld,
                                      void *const *scale, int32_t scale_dt, void *stream) {
  B2_ENTER(stream);
  B2_CHECK(num_groups > 0 && src && M && K && src_ld && dst && dst_ld && scale, B200DNN_FAILURE, "null argument");
  // groups of one row length share a launch; the reference lets K differ per group (reorder/lowoha_reorder.cpp:279-400):
  // one launch per distinct K
  std::vector<Staged> outs;
  outs.reserve(2 * num_groups);
  std::vector<const void *> s_dev(num_groups); std::vector<void *> d_dev(num_groups), sc_dev(num_groups);
  std::vector<int> distinct_k;
  for (int g = 0; g < num_groups; ++g) {
    if (M[g] <= 0) { s_dev[g] = nullptr; d_dev[g] = nullptr; sc_dev[g] = nullptr; continue; }
    B2_CHECK(K[g] > 0 && (!dst[g] || dst_ld[g] >= K[g]), B200DNN_FAILURE, "group %d: bad K or destination stride", g);
    B2_CHECK(src[g] && scale[g] && src_ld[g] >= K[g], B200DNN_FAILURE, "group %d: null pointer or bad stride", g);
    B2_TRY(stage_in(src[g], span_bytes(M[g], K[g], src_ld[g], src_dt), st, &s_dev[g]));
    Staged a, b;
    B2_TRY(stage_out(dst[g], span_bytes(M[g], K[g], dst_ld[g], B200DNN_S8), st, &a, dst[g] && dst_ld[g] != K[g]));
    B2_TRY(stage_out(scale[g], (size_t)M[g] * dt_size(scale_dt), st, &b));
    d_dev[g] = a.dev; sc_dev[g] = b.dev; outs.push_back(a); outs.push_back(b);
    if (std::find(distinct_k.begin(), distinct_k.end(), K[g]) == distinct_k.end()) distinct_k.push_back(K[g]);
  }
  if (distinct_k.empty()) return B200DNN_SUCCESS;
  for (int Kc : distinct_k) {
    // groups of another row length have no rows in this launch
    std::vector<int32_t> row_off(num_groups + 1, 0);
    for (int g = 0; g < num_groups; ++g) row_off[g + 1] = row_off[g] + ((M[g] > 0 && K[g] == Kc) ? M[g] : 0);
    const size_t tb = sizeof(void *) * num_groups;
    std::vector<uint8_t> host(3 * tb + 2 * sizeof(int64_t) * num_groups + sizeof(int32_t) * (num_groups + 1));
    uint8_t *h = host.data();
    memcpy(h, s_dev.data(), tb); memcpy(h + tb, d_dev.data(), tb); memcpy(h + 2 * tb, sc_dev.data(), tb);
    memcpy(h + 3 * tb, src_ld, sizeof(int64_t) * num_groups);
    memcpy(h + 3 * tb + sizeof(int64_t) * num_groups, dst_ld, sizeof(int64_t) * num_groups);
    memcpy(h + 3 * tb + 2 * sizeof(int64_t) * num_groups, row_off.data(), sizeof(int32_t) * (num_groups + 1));
    void *tab_dev = nullptr;
    B2_TRY(upload_blob(h, host.size(), st, &tab_dev));
    uint8_t *tab = (uint8_t *)tab_dev;
    RowQuantArgs a{};
    a.n_groups = num_groups; a.K = Kc; a.scale_dt = scale_dt; a.gather_div = 1;
    a.g_src = (const void *const *)tab; a.g_dst = (void *const *)(tab + tb); a.g_scale = (void *const *)(tab + 2 * tb);
    a.g_src_ld = (const int64_t *)(tab + 3 * tb); a.g_dst_ld = (const int64_t *)(tab + 3 * tb + sizeof(int64_t) * num_groups);
    a.row_off = (const int32_t *)(tab + 3 * tb + 2 * sizeof(int64_t) * num_groups);
    for (int g = 0; g < num_groups; ++g)
      if (row_off[g + 1] > row_off[g] && ((reinterpret_cast<uintptr_t>(s_dev[g]) | (uintptr_t)(src_ld[g] * dt_size(src_dt))) & 15) != 0) a.g_any = 1;
    B2_TRY(launch_quant_rows(a, src_dt, row_off[num_groups], st));
  }
  bool any = false;
  for (auto &s : outs) { if (s.copy_back) { B2_CUDA(cudaMemcpyAsync(s.host, s.dev, s.bytes, cudaMemcpyDeviceToHost, st)); any = true; } else if (s.sync) any = true; }
  if (any) B2_CUDA(cudaStreamSynchronize(st));
  return B200DNN_SUCCESS;
}

int32_t b200dnn_quant_dynamic(const void *src, int32_t src_dt, int64_t M, int64_t N, int64_t src_ld, int32_t per_channel,
                              void *dst, int64_t dst_ld, float *scale, void *stream) {
  B2_ENTER(stream);
  B2_CHECK(src && scale && M > 0 && N > 0 && src_ld >= N && (!dst || dst_ld >= N), B200DNN_FAILURE, "bad argument");
  B2_CHECK(src_dt == B200DNN_BF16 || src_dt == B200DNN_F32, B200DNN_UNIMPLEMENTED, "source must be f32 or bf16");
  const void *s_dev = nullptr;
  B2_TRY(stage_in(src, span_bytes(M, N, src_ld, src_dt), st, &s_dev));
  const int64_t ns = per_channel ? N : 1;
  Staged o_q, o_s;
  B2_TRY(stage_out(dst, span_bytes(M, N, dst_ld, B200DNN_S8), st, &o_q, dst && dst_ld != N));
  B2_TRY(stage_out(scale, (size_t)ns * 4, st, &o_s));
  uint32_t *amax = (uint32_t *)rt().ws.alloc((size_t)ns * 4);
  B2_CHECK(amax, B200DNN_FAILURE, "workspace allocation failed");
  B2_CUDA(cudaMemsetAsync(amax, 0, (size_t)ns * 4, st));
  dim3 grid((unsigned)((N + 255) / 256), (unsigned)(M < 64 ? 1 : (M / 64 > 256 ? 256 : M / 64)));
  if (src_dt == B200DNN_BF16) absmax_cols_kernel<uint16_t><<<grid, 256, 0, st>>>((const uint16_t *)s_dev, M, N, src_ld, per_channel, amax);
  else absmax_cols_kernel<float><<<grid, 256, 0, st>>>((const float *)s_dev, M, N, src_ld, per_channel, amax);
  B2_LAUNCHED();
  scales_from_absmax_kernel<<<(unsigned)((ns + 255) / 256), 256, 0, st>>>(amax, ns, (float *)o_s.dev);
  B2_LAUNCHED();
  if (dst) {
    dim3 g2((unsigned)((N + 255) / 256), (unsigned)(M > 1024 ? 1024 : M));
    if (src_dt == B200DNN_BF16)
      quant_static_kernel<uint16_t><<<g2, 256, 0, st>>>((const uint16_t *)s_dev, M, N, src_ld, (const float *)o_s.dev, ns, nullptr, 0, o_q.dev, B200DNN_S8, dst_ld);
    else
      quant_static_kernel<float><<<g2, 256, 0, st>>>((const float *)s_dev, M, N, src_ld, (const float *)o_s.dev, ns, nullptr, 0, o_q.dev, B200DNN_S8, dst_ld);
    B2_LAUNCHED();
  }
  B2_CUDA(cudaGetLastError());
  return finish_out({&o_q, &o_s}, st);
}

int32_t b200dnn_quant_static(const void *src, int32_t src_dt, int64_t M, int64_t N, int64_t src_ld, const float *scale,
                             int64_t n_scale, const int32_t *zp, int64_t n_zp, void *dst, int32_t dst_dt, int64_t dst_ld,
                             void *stream) {
  B2_ENTER(stream);
  B2_CHECK(src && dst && scale && M > 0 && N > 0 && src_ld >= N && dst_ld >= N, B200DNN_FAILURE, "bad argument");
  B2_CHECK((n_scale == 1 || n_scale == N) && (!zp || n_zp == 1 || n_zp == N), B200DNN_UNIMPLEMENTED, "scale / zero-point granularity");
  B2_CHECK((src_dt == B200DNN_BF16 || src_dt == B200DNN_F32) && (dst_dt == B200DNN_S8 || dst_dt == B200DNN_U8), B200DNN_UNIMPLEMENTED, "dtype combination");
  const void *s_dev, *sc_dev, *zp_dev = nullptr;
  B2_TRY(stage_in(src, span_bytes(M, N, src_ld, src_dt), st, &s_dev));
  B2_TRY(stage_in(scale, (size_t)n_scale * 4, st, &sc_dev));
  if (zp) B2_TRY(stage_in(zp, (size_t)n_zp * 4, st, &zp_dev));
  Staged o;
  B2_TRY(stage_out(dst, span_bytes(M, N, dst_ld, dst_dt), st, &o, dst_ld != N));
  dim3 g2((unsigned)((N + 255) / 256), (unsigned)(M > 1024 ? 1024 : M));
  if (src_dt == B200DNN_BF16)
    quant_static_kernel<uint16_t><<<g2, 256, 0, st>>>((const uint16_t *)s_dev, M, N, src_ld, (const float *)sc_dev, n_scale, (const int32_t *)zp_dev, n_zp, o.dev, dst_dt, dst_ld);
  else
    quant_static_kernel<float><<<g2, 256, 0, st>>>((const float *)s_dev, M, N, src_ld, (const float *)sc_dev, n_scale, (const int32_t *)zp_dev, n_zp, o.dev, dst_dt, dst_ld);
  B2_LAUNCHED();
  B2_CUDA(cudaGetLastError());
  return finish_out({&o}, st);
}

int32_t b200dnn_dequant_static(const void *src, int32_t src_dt, int64_t M, int64_t N, int64_t src_ld, const float *scale,
                               int64_t n_scale, const int32_t *zp, int64_t n_zp, void *dst, int32_t dst_dt, int64_t dst_ld,
                               void *stream) {
  B2_ENTER(stream);
  B2_CHECK(src && dst && scale && M > 0 && N > 0 && src_ld >= N && dst_ld >= N, B200DNN_FAILURE, "bad argument");
  B2_CHECK((n_scale == 1 || n_scale == N) && (!zp || n_zp == 1 || n_zp == N), B200DNN_UNIMPLEMENTED, "scale / zero-point granularity");
  B2_CHECK((src_dt == B200DNN_S8 || src_dt == B200DNN_U8) && (dst_dt == B200DNN_F32 || dst_dt == B200DNN_BF16), B200DNN_UNIMPLEMENTED, "dtype combination");
  const void *s_dev, *sc_dev, *zp_dev = nullptr;
  B2_TRY(stage_in(src, span_bytes(M, N, src_ld, src_dt), st, &s_dev));
  B2_TRY(stage_in(scale, (size_t)n_scale * 4, st, &sc_dev));
  if (zp) B2_TRY(stage_in(zp, (size_t)n_zp * 4, st, &zp_dev));
  Staged o;
  B2_TRY(stage_out(dst, span_bytes(M, N, dst_ld, dst_dt), st, &o, dst_ld != N));
  dim3 g2((unsigned)((N + 255) / 256), (unsigned)(M > 1024 ? 1024 : M));
  dequant_static_kernel<<<g2, 256, 0, st>>>(s_dev, src_dt, M, N, src_ld, (const float *)sc_dev, n_scale, (const int32_t *)zp_dev, n_zp, o.dev, dst_dt, dst_ld);
  B2_LAUNCHED();
  B2_CUDA(cudaGetLastError());
  return finish_out({&o}, st);
}

int32_t b200dnn_gated_act(void *buf, int32_t dt, int64_t M, int64_t N, int64_t ldc, int32_t act, void *stream) {
  B2_ENTER(stream);
  B2_CHECK(buf && M > 0 && N > 0 && N % 2 == 0 && ldc >= N, B200DNN_FAILURE, "bad argument");
  B2_CHECK(act >= 1 && act <= 3, B200DNN_FAILURE, "unknown gated activation %d", act);
  B2_CHECK(dt == B200DNN_BF16 || dt == B200DNN_F32, B200DNN_UNIMPLEMENTED, "gated activation on f32 or bf16 only");
  Staged o;
  B2_TRY(stage_out(buf, span_bytes(M, N, ldc, dt), st, &o, true));
  if (dt == B200DNN_BF16) gated_act_kernel<uint16_t><<<(unsigned)M, 256, 0, st>>>((uint16_t *)o.dev, N, ldc, act);
  else gated_act_kernel<float><<<(unsigned)M, 256, 0, st>>>((float *)o.dev, N, ldc, act);
  B2_LAUNCHED();
  B2_CUDA(cudaGetLastError());
  return finish_out({&o}, st);
}

int32_t b200dnn_moe_weighted_reduce(const void *const *row_ptrs, const float *topk_weights, int32_t T, int32_t topk,
                                    int32_t D, int32_t skip_weighted, int32_t dt, void *out, int64_t ld_out, void *stream) {
  B2_ENTER(stream);
  B2_CHECK(row_ptrs && out && T > 0 && topk > 0 && D > 0 && ld_out >= D, B200DNN_FAILURE, "bad argument");
  B2_CHECK(skip_weighted || topk_weights, B200DNN_FAILURE, "topk_weights is null");
  B2_CHECK(dt == B200DNN_BF16 || dt == B200DNN_F32, B200DNN_UNIMPLEMENTED, "weighted reduce on f32 or bf16 only");
  const size_t nslot = (size_t)T * topk;
  // row_ptrs is a host array (the reference's contract).  Rows in host memory are gathered into one pinned slab and
  // sent with one copy (a copy per row costs microseconds each: 8192 of them at 4096 tokens x top-2).
  std::vector<const void *> dev_rows(nslot);
  const bool rows_on_device = is_device_ptr(row_ptrs[0]);
  if (rows_on_device) {
    for (size_t i = 0; i < nslot; ++i) { B2_CHECK(row_ptrs[i], B200DNN_FAILURE, "row_ptrs[%zu] is null", i); dev_rows[i] = row_ptrs[i]; }
  } else {
    const size_t rb = (size_t)D * dt_size(dt), pitch = (rb + 15) & ~size_t(15);
    uint8_t *slab = (uint8_t *)rt().ws.alloc(nslot * pitch);
    uint8_t *pin = rt().pinned_slab(nslot * pitch);
    B2_CHECK(slab && pin, B200DNN_FAILURE, "staging allocation failed");
    for (size_t i = 0; i < nslot; ++i) {
      B2_CHECK(row_ptrs[i], B200DNN_FAILURE, "row_ptrs[%zu] is null", i);
      memcpy(pin + i * pitch, row_ptrs[i], rb);
      dev_rows[i] = slab + i * pitch;
    }
    B2_CUDA(cudaMemcpyAsync(slab, pin, nslot * pitch, cudaMemcpyHostToDevice, st));
    B2_CUDA(cudaStreamSynchronize(st));   // the pinned slab is reused by the next call
  }
  void *tab = nullptr;
  B2_TRY(upload_blob(dev_rows.data(), nslot * sizeof(void *), st, &tab));
  const void *w_dev = nullptr;
  if (!skip_weighted) B2_TRY(stage_in(topk_weights, nslot * 4, st, &w_dev));
  Staged o;
  B2_TRY(stage_out(out, span_bytes(T, D, ld_out, dt), st, &o, ld_out != D));
  ReduceArgs a{};
  a.row_ptrs = (const void *const *)tab; a.w = (const float *)w_dev; a.skip_weighted = skip_weighted;
  a.nslots = topk; a.D = D; a.dt = dt; a.out = o.dev; a.ld_out = ld_out;
  moe_reduce_kernel<<<(unsigned)T, 256, (sizeof(void *) + 4) * topk, st>>>(a);
  B2_LAUNCHED();
  B2_CUDA(cudaGetLastError());
  return finish_out({&o}, st);
}

}  // extern "C"

// Router and stable-rank launches: the fast forms when the sizes allow, the general kernels otherwise.
int32_t launch_route_topk(const float *logits, int T, int E, int topk, int renorm, int32_t *ids, float *w, cudaStream_t st) {
  const unsigned blocks = (unsigned)(((size_t)T * 32 + 255) / 256);
  if (E <= 32) route_topk_warp_kernel<1><<<blocks, 256, 0, st>>>(logits, T, E, topk, renorm, ids, w);
  else if (E <= 64) route_topk_warp_kernel<2><<<blocks, 256, 0, st>>>(logits, T, E, topk, renorm, ids, w);
  else if (E <= 128) route_topk_warp_kernel<4><<<blocks, 256, 0, st>>>(logits, T, E, topk, renorm, ids, w);
  else if (E <= 256) route_topk_warp_kernel<8><<<blocks, 256, 0, st>>>(logits, T, E, topk, renorm, ids, w);
  else route_topk_kernel<<<(unsigned)((T + 127) / 128), 128, 0, st>>>(logits, T, E, topk, renorm, ids, w);
  B2_LAUNCHED();
  return B200DNN_SUCCESS;
}
int32_t launch_expert_rank(const int32_t *ids, int nslots, int nkeys, int32_t *rank, int32_t *counts, cudaStream_t st) {
  const int nchunks = (nslots + kRankChunk - 1) / kRankChunk;
  if (nkeys > kRankMaxKeys || nchunks < 4) {
    expert_rank_kernel<<<(unsigned)nkeys, 1024, 0, st>>>(ids, nslots, rank, counts);
    B2_LAUNCHED();
    return B200DNN_SUCCESS;
  }
  int32_t *cc = (int32_t *)rt().ws.alloc((size_t)nchunks * nkeys * 4);
  B2_CHECK(cc, B200DNN_FAILURE, "workspace allocation failed");
  rank_count_kernel<<<(unsigned)nchunks, kRankChunk, 0, st>>>(ids, nslots, nkeys, cc);
  B2_LAUNCHED();
  rank_scan_kernel<<<(unsigned)((nkeys * 32 + 255) / 256), 256, 0, st>>>(cc, nchunks, nkeys, counts);
  B2_LAUNCHED();
  rank_assign_kernel<<<(unsigned)nchunks, kRankChunk, (size_t)32 * nkeys * 4, st>>>(ids, nslots, nkeys, cc, rank);
  B2_LAUNCHED();
  return B200DNN_SUCCESS;
}

// Few rows on the tensor cores (skinny_gemm.cuh).  Up to 16 rows against the decode kernel, us: K = 4096, N = 11008 12.7 -> 12.2, K = 14336,
// N = 4096 31.0 -> 16.0, but K = N = 4096 7.2 -> 7.6 (its fixed cost is higher), and with more column tiles than SMs K = 4096, N = 50176
// 37.3 -> 41.0: there only rows that the decode kernel has no room for.  From 17 to 64 rows against the tile kernel: few_rows_pay.
bool skinny_decode(int M, int N, int K, int64_t Kp) {
  return M > 8 && (long long)K * N >= (24ll << 20) && ((N + 127) / 128 <= rt().sm_count || decode_smem(M, N, Kp) > 220 * 1024);
}

// decode kernel: 0 tiled only, 1 register-batch form, 2 ring form, 3..5 ring with that many groups per stage;
// default: ring for M <= 2 and weights of 24 MB or more (measured faster there: 10.9 against 11.5 us at 45 MB, but
// 5.9 against 5.7 us at 16.8 MB), register-batch form otherwise
int decode_form(int M, int N, int K) { return env_int("B200DNN_DECODE_KERNEL", (M <= 2 && (long long)K * N >= (24ll << 20)) ? 2 : 1); }

// Dynamic quantisation inside the decode kernel (decode_quant.cuh): aligned bf16 rows that the decode kernels take, few enough elements, and no
// overlap of the results with the source (every CTA reads all of it, while others may already write).  The line, by the elements that every SM quantises: a kernel of its own
// costs 0.3 to 5 us, all SMs quantising every row about 0.06 us per 1000 elements, part of it behind a weight that is long in coming -- if that may be read before the kernel in front
// has finished (STABLE_WEIGHTS); where it may not, only the kernel of its own has it read meanwhile.  From 37 MB on a weight came from HBM in these measurements (three in turn pass the L2),
// and its stream hides more.  us, kernel of its own and fused, weights in place: M = 1, K = 11008, N = 4096 15.8, 11.7; M = 4, K = N = 4096 7.6, 7.3, N = 11008 14.9, 12.7; M = 3, K = 11008,
// N = 4096 15.5, 14.4; M = 8, K = N = 2048 6.1, 5.8; but M = 8, K = 4096, N = 8192 10.7, 12.1; M = 4, K = 8192, N = 4096 10.8, 11.7; M = 10, K = 2048, N = 1024 5.4, 5.9; weights that wait:
// M = 4, K = N = 4096 7.6, 7.6; M = 4, K = 8192, N = 4096 10.9, 12.6; M = 4, K = 2048, N = 14336 8.8, 9.3.  Over 874 (549) sizes the slowest call is 2 (3) % behind a kernel of its
// own, and 6.4 (4.6) % are gained on average.  B200DNN_FUSED_QUANT: 0 never, 1 whenever the rows allow it, -1 by the line.
bool fused_quant_pays(const b200dnn_matmul_t *d, const void *src, const PackedWeight &pw) {
  const int M = d->M, N = d->N, K = d->K;
  if (M > 16 || d->force_kernel != 0 || d->src_dt != B200DNN_BF16 || K % 8 != 0 || d->lda % 8 != 0 || (reinterpret_cast<uintptr_t>(src) & 15) != 0) return false;
  const int form = decode_form(M, N, K);
  if (skinny_decode(M, N, K, pw.Kp) || decode_smem(M, N, pw.Kp) > 220 * 1024 || form == 0 || (form >= 2 && M > kRingWarps)) return false;      // (a warp per row at least)
  const int mode = env_int("B200DNN_FUSED_QUANT", -1);
  const bool hbm = (long long)K * N >= 37000000;
  const int most = (d->flags & B200DNN_FLAG_STABLE_WEIGHTS) == 0 ? (M <= 2 || K <= 1024 ? 16384 : N < 8192 ? 12288 : 0)
                   : M <= 2 ? 32768 : hbm ? (N <= 6144 ? 45056 : K <= 4096 ? 32768 : 24576) : N <= 768 ? 24576 : 16384;
  if (mode == 0 || (mode < 0 && M * K > most)) return false;
  auto apart = [](const void *p, size_t n, const void *q, size_t m) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p), b = reinterpret_cast<uintptr_t>(q);
    return !p || !q || a + n <= b || b + m <= a;
  };
  const size_t in = span_bytes(M, K, d->lda, d->src_dt);
  return apart(d->src, in, d->dst, span_bytes(M, N, d->ldc, d->dst_dt)) && apart(d->src, in, d->src_scale.buff, (size_t)M * 4);
}

extern "C" {

int32_t b200dnn_moe_route(const float *logits, int32_t T, int32_t E, int32_t topk, int32_t renorm, int32_t *ids,
                          float *weights, int32_t *expert_counts, int32_t *slot_to_row, void *stream) {
  B2_ENTER(stream);
  B2_CHECK(logits && ids && T > 0 && E > 0 && topk > 0 && topk <= E && topk <= kMaxTopk, B200DNN_FAILURE, "bad argument");
  const void *l_dev;
  B2_TRY(stage_in(logits, (size_t)T * E * 4, st, &l_dev));
  const size_t ns = (size_t)T * topk;
  Staged o_ids, o_w, o_cnt, o_s2r;
  B2_TRY(stage_out(ids, ns * 4, st, &o_ids));
  B2_TRY(stage_out(weights, ns * 4, st, &o_w));
  B2_TRY(stage_out(expert_counts, (size_t)E * 4, st, &o_cnt));
  B2_TRY(stage_out(slot_to_row, ns * 4, st, &o_s2r));
  float *w_dev = (float *)o_w.dev;
  if (!w_dev) { w_dev = (float *)rt().ws.alloc(ns * 4); B2_CHECK(w_dev, B200DNN_FAILURE, "workspace allocation failed"); }
  B2_TRY(launch_route_topk((const float *)l_dev, T, E, topk, renorm, (int32_t *)o_ids.dev, w_dev, st));
  if (expert_counts || slot_to_row) {
    int32_t *cnt = (int32_t *)o_cnt.dev;
    if (!cnt) { cnt = (int32_t *)rt().ws.alloc((size_t)E * 4); B2_CHECK(cnt, B200DNN_FAILURE, "workspace allocation failed"); }
    int32_t *rank = (int32_t *)rt().ws.alloc(ns * 4);
    int32_t *off = (int32_t *)rt().ws.alloc((size_t)(E + 1) * 4);
    B2_CHECK(rank && off, B200DNN_FAILURE, "workspace allocation failed");
    B2_TRY(launch_expert_rank((const int32_t *)o_ids.dev, (int)ns, E, rank, cnt, st));
    if (slot_to_row) {
      expert_offsets_kernel<<<1, 32, 0, st>>>(cnt, E, 0, T, off);
      B2_LAUNCHED();
      int32_t *row_tok = (int32_t *)rt().ws.alloc(ns * 4);
      float *sw = (float *)rt().ws.alloc(ns * 4);
      B2_CHECK(row_tok && sw, B200DNN_FAILURE, "workspace allocation failed");
      build_maps_kernel<<<(unsigned)((ns + 255) / 256), 256, 0, st>>>((const int32_t *)o_ids.dev, rank, w_dev, off, T, topk, E, 0,
                                                                     (int32_t *)o_s2r.dev, sw, row_tok);
      B2_LAUNCHED();
    }
  }
  B2_CUDA(cudaGetLastError());
  return finish_out({&o_ids, &o_w, &o_cnt, &o_s2r}, st);
}

// -------------------------------------------------------------------------------------------- matmul
int32_t b200dnn_matmul(const b200dnn_matmul_t *d, void *stream) {
  B2_CHECK(d, B200DNN_FAILURE, "null descriptor");
  B2_ENTER(stream);
  b200dnn_matmul_t untransposed;
  if (d->transA) { B2_TRY(untranspose_source(d, &untransposed, st)); d = &untransposed; }
  if (is_woq_matmul(d)) return matmul_woq(d, st);               // bf16 source x s4|u4 weights, no dynamic quantisation
  if (is_group_scaled(d)) return matmul_group_scaled(d, st);   // per-group scales and W4A8: own validation and kernel
  if (is_bf16_matmul(d)) return matmul_bf16(d, st);             // bf16 x bf16: own validation, the kernel's bf16 form
  Runtime &R = rt();
  const int M = d->M, N = d->N, K = d->K;
  B2_TRY(validate_matmul_desc(d));
  const bool dyn = d->dynamic_quant != 0;

  // ---- operands on the device
  PackedWeight pw;
  B2_TRY(resolve_weight(d->weight, d->wei_format, K, N, d->ldb, d->transB, 0, d->weights_const, st, &pw));
  EpiParams epi;
  fill_epi(d, &epi);
  const void *src_dev = nullptr;
  B2_TRY(stage_in(d->src, span_bytes(M, K, d->lda, d->src_dt), st, &src_dev, &R.small));
  const uint8_t *A = (const uint8_t *)src_dev; int64_t lda = d->lda; bool a_unsigned = d->src_dt == B200DNN_U8;
  Staged o_scale;
  DecodeQuant dq{};
  if (dyn && fused_quant_pays(d, src_dev, pw)) {
    const int32_t sdt = d->src_scale.buff ? d->src_scale.dt : B200DNN_F32;
    B2_TRY(stage_out(const_cast<void *>(d->src_scale.buff), (size_t)M * dt_size(sdt), st, &o_scale));
    dq = DecodeQuant{(const uint16_t *)src_dev, d->lda, o_scale.dev, sdt};
    A = nullptr; a_unsigned = false;
    epi.src_scale_dt = B200DNN_F32; epi.src_scale_n = M;      // (the kernel has them in shared memory)
  } else if (dyn) {
    const int64_t Kq = round_up(K, 16);
    int8_t *q = (int8_t *)R.ws.alloc((size_t)M * Kq);
    B2_CHECK(q, B200DNN_FAILURE, "workspace allocation failed");
    const int32_t sdt = d->src_scale.buff ? d->src_scale.dt : B200DNN_F32;
    B2_TRY(stage_out(const_cast<void *>(d->src_scale.buff), (size_t)M * dt_size(sdt), st, &o_scale));
    void *sc = o_scale.dev;
    if (!sc) { sc = R.ws.alloc((size_t)M * 4); B2_CHECK(sc, B200DNN_FAILURE, "workspace allocation failed"); }
    RowQuantArgs qa{};
    qa.src = src_dev; qa.src_ld = d->lda; qa.dst = q; qa.dst_ld = Kq; qa.scale = sc; qa.scale_dt = sdt; qa.K = K; qa.gather_div = 1;
    B2_TRY(R.small.flush(st, false));
    B2_TRY(launch_quant_rows(qa, d->src_dt, M, st));
    A = (const uint8_t *)q; lda = Kq; a_unsigned = false;
    epi.src_scale = sc; epi.src_scale_dt = sdt; epi.src_scale_n = M > 1 ? M : 1;
  } else if (d->src_scale.count > 0) {
    const void *p;
    B2_TRY(stage_in(d->src_scale.buff, (size_t)d->src_scale.count * dt_size(d->src_scale.dt), st, &p, &R.small));
    epi.src_scale = p; epi.src_scale_dt = d->src_scale.dt; epi.src_scale_n = (int32_t)d->src_scale.count;
  }
  if (d->wei_scale.count > 0) {
    const void *p;
    B2_TRY(stage_in(d->wei_scale.buff, (size_t)d->wei_scale.count * dt_size(d->wei_scale.dt), st, &p, &R.small));
    epi.wei_scale = p; epi.wei_scale_dt = d->wei_scale.dt; epi.wei_scale_n = (int32_t)d->wei_scale.count;
  }
  if (d->src_zp.buff) {
    B2_CHECK(d->src_zp.dt == B200DNN_S32 || d->src_zp.dt == B200DNN_S8 || d->src_zp.dt == B200DNN_U8, B200DNN_UNIMPLEMENTED, "src zero-point dtype");
    const void *p;
    B2_TRY(stage_in(d->src_zp.buff, dt_size(d->src_zp.dt), st, &p, &R.small));
    epi.src_zp = p; epi.src_zp_dt = d->src_zp.dt; epi.has_zp = 1;
  }
  epi.colsum = pw.colsum;
  if (d->bias) {
    const void *p;
    B2_TRY(stage_in(d->bias, (size_t)N * dt_size(d->bias_dt), st, &p, &R.small));
    epi.bias = p;
  }
  for (int i = 0; i < d->n_postops; ++i) {
    const b200dnn_postop_t &p = d->postops[i];
    epi.po[i].type = p.type; epi.po[i].dt = p.dt; epi.po[i].ld = p.ld; epi.po[i].alpha = p.alpha; epi.po[i].beta = p.beta;
    epi.po[i].buff = nullptr;
    if (p.type == PO_BINARY_ADD || p.type == PO_BINARY_MUL) {
      const void *b;
      B2_TRY(stage_in(p.buff, p.ld ? span_bytes(M, N, p.ld, p.dt) : (size_t)N * dt_size(p.dt), st, &b, &R.small));
      epi.po[i].buff = b;
    }
  }
  Staged o_dst;
  B2_TRY(stage_out(d->dst, span_bytes(M, N, d->ldc, d->dst_dt), st, &o_dst, d->ldc != N));
  epi.dst = o_dst.dev;
  // requantised integer destination: the GEMM writes f32 into the workspace, one more pass scales, shifts, clamps and rounds
  const bool requant = d->dst_dt == B200DNN_S8 || d->dst_dt == B200DNN_U8;
  const void *dst_scale_dev = nullptr, *dst_zp_dev = nullptr;
  if (requant) {
    float *tmp = (float *)R.ws.alloc((size_t)M * N * 4);
    B2_CHECK(tmp, B200DNN_FAILURE, "workspace allocation failed");
    epi.dst = tmp; epi.ldc = N; epi.dst_dt = B200DNN_F32;
    if (d->dst_scale.buff) B2_TRY(stage_in(d->dst_scale.buff, 4, st, &dst_scale_dev, &R.small));
    if (d->dst_zp.buff) B2_TRY(stage_in(d->dst_zp.buff, 4, st, &dst_zp_dev, &R.small));
  }
  B2_TRY(R.small.flush(st, o_dst.copy_back || o_dst.sync));

  // ---- kernel choice: weight-streaming kernel for decode-sized M, tcgen05 otherwise
  // Rows that the copy engine cannot read in place (K or lda not a multiple of 16) are copied to such a pitch first: one pass over the
  // activations, against a weight stream per 16 rows in the tiled streaming kernel (M = 500, K = 1999, N = 3001: 86 us with it).
  if (d->force_kernel == 0 && M > 16 && ((lda % 16 != 0) || (reinterpret_cast<uintptr_t>(A) & 15) != 0)) {
    B2_TRY(repitch_rows(A, lda, M, K, st, &A, &lda));
  }
  const bool tc_ok = (lda % 16 == 0) && ((reinterpret_cast<uintptr_t>(A) & 15) == 0);
  int which = d->force_kernel;
  if (which == 0) which = (M <= 16 || !tc_ok) ? 1 : 2;
  // the weight may be read before the kernel in front has finished: that kernel is this call's quantisation, which itself waited for
  // everything before it, or the caller says that its weights are in place (and the library's own copy of them is: see take_cached)
  const bool early = !pw.fresh && ((dyn && !dq.src) || (d->flags & B200DNN_FLAG_STABLE_WEIGHTS) != 0);
  const bool skinny = M <= 16 ? skinny_decode(M, N, K, pw.Kp) : M <= kSkinnyMaxM && few_rows_pay(M, N, K);
  const bool few_rows = d->force_kernel == 0 && !dq.src && tc_ok && skinny;
  B2_CHECK(few_rows || which == 1 || which == 3 || tc_ok, B200DNN_FAILURE, "tcgen05 kernel needs a 16-byte aligned source with lda %% 16 == 0");
  if (few_rows) {
    B2_TRY(launch_skinny(A, lda, a_unsigned, false, M, N, K, pw, epi, M <= 16 && epi.n_po > 0 ? FA_GENERIC : fast_act_code(epi), early, st));
  } else if (which == 1 || which == 3) {
    int32_t rc = B200DNN_UNIMPLEMENTED;
    const int dk = decode_form(M, N, K);
    dq.late = early ? 0 : 1;
    const bool pdl = (early || dq.src) && env_int("B200DNN_PDL", 1) != 0;
    if (which == 1 && M <= 16 && dk >= 2) {
      // groups per stage: split the CTA's groups into equal sets of at most five
      const int groups = (N + 7) / 8, grid = groups < rt().sm_count ? groups : rt().sm_count;
      const int local = (groups + grid - 1) / grid, sets = (local + 4) / 5;
      int r = dk > 2 ? dk : (local + sets - 1) / sets;
      if (r <= 2) rc = launch_decode_ring<2>(A, lda, a_unsigned, M, N, K, pw, epi, pdl, st, dq);
      else if (r == 3) rc = launch_decode_ring<3>(A, lda, a_unsigned, M, N, K, pw, epi, pdl, st, dq);
      else if (r == 4) rc = launch_decode_ring<4>(A, lda, a_unsigned, M, N, K, pw, epi, pdl, st, dq);
      else rc = launch_decode_ring<5>(A, lda, a_unsigned, M, N, K, pw, epi, pdl, st, dq);
    }
    if (which == 1 && M <= 16 && dk != 0 && rc == B200DNN_UNIMPLEMENTED) rc = launch_decode(A, lda, a_unsigned, M, N, K, pw, epi, pdl, st, dq);
    if (rc == B200DNN_UNIMPLEMENTED) rc = launch_stream(A, lda, a_unsigned, M, N, K, pw, epi, st);
    B2_TRY(rc);
  } else {
    TcGemmArgs ta{};
    ta.shared_dst = 1;
    B2_TRY(launch_tc(A, lda, a_unsigned, M, N, K, pw, ta, epi, 0, st));
  }
  if (requant) {
    const int64_t n = (int64_t)M * N;
    requant_dst_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>((const float *)epi.dst, M, N, (const float *)dst_scale_dev,
                                                                    (const int32_t *)dst_zp_dev, o_dst.dev, d->dst_dt, d->ldc);
    B2_LAUNCHED();
    B2_CUDA(cudaGetLastError());
  }
  return finish_out({&o_dst, &o_scale}, st);   // calls that synchronise read the status word there
}

int32_t b200dnn_stream_status(void *stream) {
  B2_ENTER(stream);
  B2_CUDA(cudaStreamSynchronize(st));
  return read_status();
}

int32_t b200dnn_phase_timing(void *stream, int32_t enable) {
  B2_ENTER(stream);
  rt().timing = enable != 0;
  rt().n_tev = 0;
  return B200DNN_SUCCESS;
}

int32_t b200dnn_phase_times(void *stream, float *ms, int32_t n, int32_t *calls) {
  B2_ENTER(stream);
  B2_CHECK(ms && n > 0, B200DNN_FAILURE, "bad argument");
  B2_CUDA(cudaStreamSynchronize(st));
  Runtime &R = rt();
  for (int i = 0; i < n; ++i) ms[i] = 0.f;
  int n_calls = 0;
  for (size_t i = 0; i < R.n_tev; ++i) {
    if (R.tphase[i] < 0) { ++n_calls; continue; }      // a call starts here
    if (i == 0) continue;
    float t = 0.f;
    B2_CUDA(cudaEventElapsedTime(&t, R.tev[i - 1], R.tev[i]));
    if (R.tphase[i] < n) ms[R.tphase[i]] += t;
  }
  if (n_calls > 0) for (int i = 0; i < n; ++i) ms[i] /= (float)n_calls;
  if (calls) *calls = n_calls;
  R.n_tev = 0;
  return B200DNN_SUCCESS;
}

int32_t b200dnn_clear_caches(void) {
  if (device_count() <= 0) return B200DNN_SUCCESS;
  int cur = 0;
  cudaGetDevice(&cur);
  for (int dev = 0; dev < 64; ++dev) {
    DeviceShared *D;
    { std::lock_guard<std::mutex> lk(devices_mu()); D = device_slot(dev); }
    if (!D) continue;
    cudaSetDevice(dev);
    cudaDeviceSynchronize();
    {
      std::lock_guard<std::mutex> lk(D->cache_mu);
      for (auto &kv : D->wcache) { if (kv.second.owned) cudaFree(kv.second.owned); if (kv.second.ready) cudaEventDestroy(kv.second.ready); }
      D->wcache.clear();
      for (auto &kv : D->woq_cache) { if (kv.second.owned) cudaFree(kv.second.owned); if (kv.second.ready) cudaEventDestroy(kv.second.ready); }
      D->woq_cache.clear();
      for (auto &kv : D->host_packed) { if (kv.second.owned) cudaFree(kv.second.owned); if (kv.second.ready) cudaEventDestroy(kv.second.ready); }
      D->host_packed.clear();
      D->packed_registry.clear();
    }
    std::lock_guard<std::mutex> lk(D->ctx_mu);
    for (auto &kv : D->ctxs) { std::lock_guard<std::mutex> lk2(kv.second->mu); kv.second->release_buffers(); }
  }
  cudaSetDevice(cur);
  return B200DNN_SUCCESS;
}

}  // extern "C"

#include "moe_api.cuh"
#include "moe_ep.cuh"
#include "group_api.cuh"
#include "nshard_api.cuh"
#include "norm_api.cuh"
#include "sdpa_api.cuh"
#include "quant_prepack_api.cuh"

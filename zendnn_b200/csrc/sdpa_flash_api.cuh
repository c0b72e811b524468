// Host interface of the fused attention kernels (sdpa_flash.cu), called by b200dnn_sdpa with device pointers.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace b200 {

struct SdpaCall {
  int64_t B, H, S, KV, D;
  const void *q, *k, *v; void *out;
  int64_t qs[3], ks[3], vs[3], os[3];      // strides in elements: batch, head, row (the head dimension is dense)
  float scale; int causal;
  const void *mask; int32_t mask_dt; int64_t mb, mh, mi;   // element (b,h,i,j) at b*mb + h*mh + i*mi + j; null: none
  int test_no_loads;
  int grouped;             // the caller has the three-step form for all heads at once: it may be the faster one (see sdpa_fused)
};

// Enqueues one kernel, or returns unimplemented when the call does not fit (the caller then takes the BMM form).
int32_t sdpa_fused(const SdpaCall &c, cudaStream_t st);

}  // namespace b200

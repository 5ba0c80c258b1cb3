// What the kernels of the generalized delta rule share (tpx_delta.cu, tpx_delta_chunk.cu).
#pragma once
#include "tpx_hybrid.cuh"

namespace tpx {

__device__ __forceinline__ void dl_cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ float dl_sigmoid(float v) { return __fdividef(1.0f, 1.0f + __expf(-v)); }

struct DeltaFastParams {
  const uint16_t* proj;
  const float *wraw, *a_bias, *norm_w;
  const int *start, *dev_len;
  float* state;
  uint16_t* out;
  long long ldp, ldo;
  int S, past, H, dim;
  float eps;
};

int delta_chunk(const DeltaFastParams& p, int64_t B, cudaStream_t st);  // heads of 64

}  // namespace tpx

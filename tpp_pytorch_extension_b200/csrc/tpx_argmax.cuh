// Index of the largest value of each row, the first among equals, a NaN counting as the largest: torch.argmax over the last dimension.
#pragma once
#include "tpx_common.cuh"

namespace tpx {

// A decode step's logits are a few rows of some ten thousand values, fresh in L2, and nothing else runs beside this kernel: bound by latency. A CTA of 1024
// threads per row asks for 16-byte pieces eight at a time; values are compared as whole numbers of the same order, and positions only where a
// thread meets a larger one, its own coming in rising order. 5 rows of 32000 fp32 logits: 17.3 us with 256 threads and a value at a time, now 4.5; of bf16
// logits 5.1 us with positions and NaN tests at every value, now 4.6.
constexpr int kArgmaxThreads = 1024;

__device__ __forceinline__ uint32_t argmax_key(float v) {
  const uint32_t u = __float_as_uint(v + 0.0f);  // -0 equals 0
  return v != v ? 0xffffffffu : (u & 0x80000000u) ? ~u : u | 0x80000000u;
}

template <typename T>
__global__ void __launch_bounds__(kArgmaxThreads) argmax_kernel(const T* x, long long n, long long* __restrict__ out) {
  constexpr int V = 16 / sizeof(T), Q = 8;  // values of a piece, pieces on the way
  __shared__ uint32_t sk[32];
  __shared__ long long si[32];
  pdl_trigger();
  pdl_wait();
  x += (size_t)blockIdx.x * n;
  uint32_t key = 0;
  long long at = 0x7fffffffffffffffLL;
  auto take = [&](float v, long long i) {
    const uint32_t k = argmax_key(v);
    if (k > key) key = k, at = i;
  };
  const long long nv = (reinterpret_cast<uintptr_t>(x) & 15) == 0 ? n / V : 0;
  for (long long i0 = threadIdx.x; i0 < nv; i0 += Q * kArgmaxThreads) {
    uint4 w[Q];
#pragma unroll
    for (int q = 0; q < Q; q++)
      if (i0 + q * kArgmaxThreads < nv) w[q] = reinterpret_cast<const uint4*>(x)[i0 + q * kArgmaxThreads];
#pragma unroll
    for (int q = 0; q < Q; q++) {
      const long long i = i0 + q * kArgmaxThreads;
      if (i >= nv) break;
      const uint32_t ww[4] = {w[q].x, w[q].y, w[q].z, w[q].w};
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if constexpr (sizeof(T) == 4) {
          take(__uint_as_float(ww[j]), i * V + j);
        } else {
          take(__uint_as_float(ww[j] << 16), i * V + 2 * j);
          take(__uint_as_float(ww[j] & 0xffff0000u), i * V + 2 * j + 1);
        }
      }
    }
  }
  for (long long i = nv * V + threadIdx.x; i < n; i += kArgmaxThreads) {
    if constexpr (sizeof(T) == 4) take(x[i], i);
    else take(bf16_bits_to_f32(x[i]), i);
  }
  auto reduce = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const uint32_t k = __shfl_xor_sync(0xffffffffu, key, o);
      const long long i = __shfl_xor_sync(0xffffffffu, at, o);
      if (k > key || (k == key && i < at)) key = k, at = i;
    }
  };
  reduce();
  if ((threadIdx.x & 31) == 0) sk[threadIdx.x >> 5] = key, si[threadIdx.x >> 5] = at;
  __syncthreads();
  if (threadIdx.x < 32) {
    key = sk[threadIdx.x], at = si[threadIdx.x];
    reduce();
    if (threadIdx.x == 0) out[blockIdx.x] = at;
  }
}

}  // namespace tpx

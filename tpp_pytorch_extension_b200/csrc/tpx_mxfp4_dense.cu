// MXFP4 linear for many tokens: the weight unpacked to bf16 for this call, then the bf16 kernel on CTA pairs.
//
// Serves the same calls as tpx_qlinear_tcp2.cu (fc_plain / fc_gate_up / fc_add of src/csrc/llm/fused_llm_infer.cpp on MXFP4
// weights). A quarter of an E2M1 code times its power-of-two scale is exact in bf16, and the activations enter as they are, where the block-scaled
// kernel multiplies two 8-bit terms per activation: half of its MMA work carries the remainders, so that it ends at 1050 TFLOP/s
// where the bf16 pair kernel reaches 1300-1450 beside the unpacking.
// What it costs is one pass over the weight, 2.5 bytes per value (a gate/up pair of 14336 x 4096: 54 us), hence a
// least number of tokens. A pair's rows are unpacked in turn (gate i, up i), so that one lane of the epilogue holds both.
#include <cuda_fp4.h>

#include "tpx_bf16_pair.cuh"
#include "tpx_mxfp4_dense.cuh"
#include "../../include/tpx_b200.h"

namespace tpx {

// One CTA per packed 128 x 128 tile (8 KB of codes and 512 bytes of scales, the layout of repack_mxfp4_tc_kernel): a thread
// turns 4 bytes of each of eight rows into 16-byte stores, sixteen neighbouring threads write 256 consecutive bytes. Bound by HBM
// (all loads of a thread are in flight before the first store).
__global__ void __launch_bounds__(256) unpack_mxfp4_bf16_kernel(const uint8_t* __restrict__ wq, const uint8_t* __restrict__ sfa, int KS, int nw, long long N,
                                                                int K, uint16_t* __restrict__ out) {
  pdl_trigger();
  const long long tile = blockIdx.x;  // (tn * KS + ks) * nw + d
  const int d = (int)(tile % nw);
  const long long tk = tile / nw, tn = tk / KS;
  const int c = threadIdx.x & 15, r0 = threadIdx.x >> 4, k = (int)(tk % KS) * 128 + c * 8;
  uint32_t q[8];
  float s[8];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int r = r0 + 16 * i;
    q[i] = __ldg(reinterpret_cast<const uint32_t*>(wq + tile * 8192 + r * 64 + c * 4));
    const uint32_t e = __ldg(sfa + tile * 512 + (r % 32) * 16 + (r / 32) * 4 + c / 4);
    // 2^(e - 129), a quarter of the scale: six times 2^127 is beyond bf16, and the smallest product, 2^-130, is exact as a subnormal. The
    // multiplying kernel's epilogue takes the sums four times. 255 is the format's NaN.
    s[i] = __uint_as_float(e == 255 ? 0x7fc00000u : e > 2 ? (e - 2) << 23 : 0x00100000u << e);
  }
  pdl_wait();  // `out` may still be read by an earlier grid
  if (k >= K) return;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const long long n = tn * 128 + r0 + 16 * i;
    if (n >= N) continue;
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const __half2_raw h = __nv_cvt_fp4x2_to_halfraw2((__nv_fp4x2_storage_t)((q[i] >> (8 * j)) & 0xff), __NV_E2M1);
      o[j] = bp_pack(__half2float(__ushort_as_half(h.x)) * s[i], __half2float(__ushort_as_half(h.y)) * s[i]);
    }
    *reinterpret_cast<uint4*>(out + (n * nw + d) * K + k) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

struct DensePlan {
  size_t off_w, off_x, total;
};
static DensePlan dense_plan(int64_t M, int64_t N, int64_t K, bool pair) {
  DensePlan d;
  const int64_t rows = pair ? 2 * N : N;
  auto up = [](size_t b) { return (b + 1023) & ~(size_t)1023; };
  d.off_w = up(bf_pair_scratch_bytes(M, rows, K));
  d.off_x = d.off_w + up((size_t)rows * K * 2);
  d.total = d.off_x + up((size_t)M * K * 2);  // the normed input, where there is a norm
  return d;
}

// Below the least number of tokens the unpacking costs more than the faster MMAs save. Weights of more than 256 MiB in bf16 stay
// packed, so that the scratch stays bounded. TPX_MXFP4_DENSE=0 never, =1 from 129 tokens on.
// (14336 x 4096 pair, packed against unpacked: 2048 tokens 433 / 375 us, 4096: 873 / 732, 8192: 1792 / 1355; one weight, 4096 x 14336: 222 / 211,
// 441 / 405, 901 / 762; 6144 x 4096: 116 / 114, 171 / 174, 370 / 320; 8192 x 2048: 80 / 81, 114 / 109, 255 / 215. The line leaves out N and K: where
// tiles end just past a round the unpacked form loses up to 10 % above it, 2560 x 2048 at 4096 tokens 56 / 61, and elsewhere it would win below.)
constexpr int64_t kDenseMinTokens = 4096, kDenseMinTokensPair = 2048;
constexpr int64_t kDenseMaxBytes = 256ll << 20;
bool mxfp4_dense_serves(int64_t M, int64_t N, int64_t K, bool pair) {
  const int k = knobs().mx_dense;
  if (k == 0 || M <= 128 || M >= (1 << 24) || K % 64 || N % 32) return false;
  if ((pair ? 2 : 1) * N * K * 2 > kDenseMaxBytes) return false;
  return k > 0 || M >= (pair ? kDenseMinTokensPair : kDenseMinTokens);
}
size_t mxfp4_dense_scratch_bytes(int64_t M, int64_t N, int64_t K, bool pair) { return dense_plan(M, N, K, pair).total; }

bool mxfp4_dense_takes(const uint16_t* x, int64_t M, int64_t N, int64_t K, bool pair, const TcParams& base, size_t scratch_bytes, const TcNorm* norm) {
  if (!mxfp4_dense_serves(M, N, K, pair) || scratch_bytes < mxfp4_dense_scratch_bytes(M, N, K, pair)) return false;
  if (((uintptr_t)base.bias | (uintptr_t)base.mul_in | (uintptr_t)base.res | (uintptr_t)base.y) & 15) return false;
  if (norm && (norm->pre || (norm->gamma && ((uintptr_t)norm->gamma & 15)))) return false;
  if (norm && norm->gamma) return true;  // read once, by the norm
  // tiles are read once per 256 features: only from the device's own memory
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, x) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return at.type == cudaMemoryTypeDevice;
}

int mxfp4_dense_run(const uint8_t* wq, const uint8_t* sfa, bool pair, const uint16_t* x, int64_t M, int64_t N, int64_t K, const TcParams& base,
                    void* scratch, size_t scratch_bytes, cudaStream_t st, const TcNorm* norm) {
  const DensePlan d = dense_plan(M, N, K, pair);
  TPX_REQUIRE(scratch && scratch_bytes >= d.total, TPX_ERR_SCRATCH, "qlinear_mxfp4_tc: scratch of %zu bytes needed, %zu given", d.total, scratch_bytes);
  unsigned char* sc = reinterpret_cast<unsigned char*>(scratch);
  uint16_t* w = reinterpret_cast<uint16_t*>(sc + d.off_w);
  if (norm && norm->gamma) {
    uint16_t* xn = reinterpret_cast<uint16_t*>(sc + d.off_x);
    const int rc = tpx_rmsnorm(x, norm->gamma, norm->gamma_f32, norm->eps, M, K, xn, st);
    if (rc) return rc;
    x = xn;
  }
  const int nw = pair ? 2 : 1, KS = tc_padded_ks(K, pair);
  const unsigned tiles = (unsigned)((N + 127) / 128 * KS * nw);
  TPX_CUDA_OK(launch_pdl(unpack_mxfp4_bf16_kernel, dim3(tiles), dim3(256), 0, st, wq, sfa, KS, nw, (long long)N, (int)K, w));
  BfParams p = {};
  p.t = base;
  p.glu = pair;
  p.quarter = 1;
  p.t.err = reinterpret_cast<unsigned*>(sc + kTcCounterBytes - 4);
  return bf_pair_run(p, w, x, M, nw * N, K, K, K, scratch, d.off_w, st);
}

}  // namespace tpx

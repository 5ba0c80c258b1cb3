// int8 linear of few tokens (tpx_qlinear_i8_rows.cu): what its launch takes, and the quantised activations it reads.
#pragma once
#include "tpx_tc_ptx.cuh"

namespace tpx {

// The quantised activations of a token tile and k step (128 values) are one run of memory, fetched by one untiled copy: TOK rows of 128
// bytes, their 16-byte units in the order of the 128-byte swizzle, then the scales of the step's blocks, [1 or 2][TOK] (a block that
// spans several steps: with its last one). As plain rows of K bytes the 16 pieces of a step lay a power of two apart, and all CTAs
// asking for them at once was what bounded the kernel (11008 x 4096, 16 tokens: 20 us, 19.4 without any weight traffic).
struct I8Act {
  int TOK, ksteps, B, bytes;  // bytes per (token tile, step)
  __host__ __device__ I8Act(int tok, int ks, int block) : TOK(tok), ksteps(ks), B(block), bytes(tok * 128 + (block == 64 ? 2 : 1) * tok * 4) {}
  __device__ __forceinline__ uint8_t* step(uint8_t* xq, int tok, int k) const { return xq + ((size_t)(tok / TOK) * ksteps + k / 128) * bytes; }
  __device__ __forceinline__ uint8_t* value(uint8_t* xq, int tok, int k) const {  // up to the next 16 values
    const int r = tok % TOK;
    return step(xq, tok, k) + r * 128 + (((k % 128) / 16) ^ (r & 7)) * 16 + k % 16;
  }
  __device__ __forceinline__ float* scale(uint8_t* xq, int tok, int blk) const {
    const int k = blk * B + B - 1;
    return reinterpret_cast<float*>(step(xq, tok, k) + TOK * 128) + (B == 64 ? blk & 1 : 0) * TOK + tok % TOK;
  }
};

// The same for up to 32 tokens in blocks of 64, one tile of TOK = 16 or 32, which the kernel for few tokens reads where the call is its: the TOK rows of 64 bytes of
// one block, then the other's, in the order of the 64-byte swizzle, then the scales [2][TOK]. The 16 bytes that a lane of that kernel's MMAs takes from a token are one unit, and a
// warp's 32 units (8 tokens) one run of 512 bytes; places are found without a division (1 us of a linear of 32 tokens).
struct I8Act64 {
  static constexpr int B = 64;
  uint32_t TOK;
  static __host__ __device__ constexpr bool serves(int tok, int block) { return tok <= 32 && block == B; }
  static __host__ __device__ constexpr uint32_t bytes(uint32_t tok) { return tok * 136; }  // per step
  __device__ __forceinline__ uint8_t* value(uint8_t* xq, int tok, int k) const {
    const uint32_t u = k;
    return xq + (u / 128 * bytes(TOK) + (u % 128 / 64 * TOK + tok) * 64 + ((u % 64 / 16) ^ (((uint32_t)tok >> 1) & 3)) * 16 + u % 16);
  }
  __device__ __forceinline__ float* scale(uint8_t* xq, int tok, int blk) const {
    return reinterpret_cast<float*>(xq + ((uint32_t)blk / 2 * bytes(TOK) + TOK * 128)) + (blk & 1) * TOK + tok;
  }
};

// Eight values of a quantisation block that as many neighbouring lanes have as `lanes` says -> eight int8; returns the block's scale.
__device__ __forceinline__ float i8_quantize8(const float (&f)[8], int lanes, uint2& out) {
  float amax = 0.0f;
#pragma unroll
  for (int j = 0; j < 8; j++) amax = fmaxf(amax, fabsf(f[j]));
  for (int o = 1; o < lanes; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float scale = (float)((double)amax / 127.0);
  const float iscale = scale != 0.0f ? 1.0f / scale : 0.0f;
  uint32_t o2[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    uint32_t word = 0;
#pragma unroll
    for (int e = 0; e < 4; e++) {
      float r = nearbyintf(f[4 * h + e] * iscale);
      r = fminf(fmaxf(r, -127.0f), 127.0f);
      word |= ((uint32_t)(uint8_t)(int8_t)(int)r) << (8 * e);
    }
    o2[h] = word;
  }
  out = make_uint2(o2[0], o2[1]);
  return scale;
}
__device__ __forceinline__ void i8_unpack_bf16(uint4 v, float (&f)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; j++) {
    f[2 * j] = bf16_bits_to_f32((uint16_t)(w[j] & 0xffff));
    f[2 * j + 1] = bf16_bits_to_f32((uint16_t)(w[j] >> 16));
  }
}
// piece i of the norm's weight
__device__ __forceinline__ void i8_gamma(const void* gamma, int gamma_f32, int i, float (&g)[8]) {
  if (gamma_f32) {
    const float4 g0 = reinterpret_cast<const float4*>(gamma)[2 * i], g1 = reinterpret_cast<const float4*>(gamma)[2 * i + 1];
    g[0] = g0.x; g[1] = g0.y; g[2] = g0.z; g[3] = g0.w; g[4] = g1.x; g[5] = g1.y; g[6] = g1.z; g[7] = g1.w;
  } else {
    i8_unpack_bf16(reinterpret_cast<const uint4*>(gamma)[i], g);
  }
}

struct I8RowsParams {
  TcParams t;                // epilogue fields (bias, act, mul_in, res, res_scale, y, M, N)
  const int8_t* w[2];        // plain int8 weight [Np][Kp]; of a pair: gate, up
  const float* swT[2];       // [K/64][Np]
  uint8_t* xq;               // I8Act64
  const uint16_t* x;         // or, if not null: bf16 activations, to be quantised (behind an RMSNorm if gamma is set) and left in xq as well
  const void* gamma;
  int gamma_f32;
  float eps;
  int nkb, Kp, Np, tiles;  // k blocks; N / 16
};

bool i8_rows_serves(int64_t M, int64_t N, int64_t K, int64_t block, bool pair);
bool i8_rows_quantizes(const void* x, const void* y, int64_t M, int64_t N, int64_t K);  // whether the launch takes x instead of xq
int i8_rows_launch(I8RowsParams p, bool pair, cudaStream_t st);  // sets t.cluster

}  // namespace tpx

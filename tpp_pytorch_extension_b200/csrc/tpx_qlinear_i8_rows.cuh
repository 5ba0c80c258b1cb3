// int8 linear of few tokens (tpx_qlinear_i8_rows.cu): what its launch takes, and the quantised activations it reads.
#pragma once
#include "tpx_tc_ptx.cuh"

namespace tpx {

// Quantised activations, blocks of 64 values: [K/64][Mp][64] int8, then the scales [K/64][Mp]. The 16 bytes that a lane of the kernel's MMAs
// takes from a token are one piece, and a warp's 32 pieces (8 tokens) are one run of 512 bytes.
struct I8Rows {
  int Mp, nkb, B;  // tokens, padded to what a kernel reads; k blocks; B = 64, the scale block, as in I8Act
  __host__ __device__ I8Rows(int M, int64_t K) : Mp(M <= 8 ? 8 : M <= 16 ? 16 : 32), nkb((int)(K / 64)), B(64) {}
  __host__ __device__ size_t bytes() const { return (size_t)nkb * Mp * 68; }
  __device__ __forceinline__ uint8_t* value(uint8_t* xq, int tok, int k) const { return xq + ((size_t)(k / 64) * Mp + tok) * 64 + k % 64; }
  __device__ __forceinline__ float* scale(uint8_t* xq, int tok, int blk) const {
    return reinterpret_cast<float*>(xq + (size_t)nkb * Mp * 64) + (size_t)blk * Mp + tok;
  }
};

struct I8RowsParams {
  TcParams t;                // epilogue fields (bias, act, mul_in, res, res_scale, y, M, N)
  const int8_t* w[2];        // plain int8 weight [Np][Kp]; of a pair: gate, up
  const float* swT[2];       // [K/64][Np]
  const uint8_t* xq;         // I8Rows
  int nkb, Mp, Kp, Np, tiles;  // tiles: N / 16
};

bool i8_rows_serves(int64_t M, int64_t N, int64_t block, bool pair);
int i8_rows_launch(I8RowsParams p, bool pair, cudaStream_t st);  // sets t.cluster

}  // namespace tpx

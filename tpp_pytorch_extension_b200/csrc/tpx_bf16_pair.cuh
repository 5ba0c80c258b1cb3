// Parameter block of the bf16 linear's kernels (tpx_linear_bf16.cu, tpx_linear_bf16_pair.cu).
#pragma once
#include "tpx_hybrid.cuh"
#include "tpx_tc_ptx.cuh"

namespace tpx {

// Epilogue of tpx_linear: fp32 bias, row stride, fp32 or bf16 result, activation from a column on; gated units from pairs of
// columns; or the residual sum with the norm of its next reader.
struct BfEx {
  const float *bias, *ap;
  void* y;
  long long ldy;
  int on, out_f32, act, act_from;
  uint16_t* z;
  const float *res, *add, *nw, *nb;
  float* x_out;
  uint16_t* h;
  long long ldz, ldr, ldh;
  float limit, nalpha;
};

struct BfParams {
  TcParams t;   // epilogue fields (bias, act, mul_in, res, res_scale, y, M, N, err)
  int ksteps;   // k steps of 64 (K rounded up)
  int TN, TM;   // feature tiles, token tiles
  int split;    // 1: the CTAs share all pipeline stages of all tiles evenly; a tile cut between CTAs is put together by the last of them
  BfEx ex;
};

int bf_make_map(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows);
// many tokens on CTA pairs (tpx_linear_bf16_pair.cu): whether it takes this call, and the call
bool bf_pair_serves(const BfParams& p, int64_t M, int64_t N, int64_t K);
int bf_pair_run(BfParams& p, const void* w, const void* x, int64_t M, int64_t N, int64_t K, int64_t ldw, int64_t ldx, cudaStream_t st);

}  // namespace tpx

// MXFP4 linear of up to 16 tokens (tpx_qlinear_mx_rows.cu).
#pragma once
#include "tpx_tc_ptx.cuh"

namespace tpx {

bool mx_rows_serves(int64_t M, int64_t N, int64_t K, bool pair);
size_t mx_rows_scratch_bytes(int64_t M, int64_t K);  // 16-byte aligned
// wq, sfa: the packed weight, KS its padded k steps; b: the epilogue's fields
int mx_rows_run(const uint8_t* wq, const uint8_t* sfa, bool pair, const uint16_t* x, int64_t M, int64_t N, int64_t K, int KS, TcParams b, void* scratch,
                cudaStream_t st, const TcNorm* norm);

}  // namespace tpx

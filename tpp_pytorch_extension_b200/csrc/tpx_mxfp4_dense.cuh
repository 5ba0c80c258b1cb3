// MXFP4 linear for many tokens on a weight unpacked to bf16: tpx_mxfp4_dense.cu
#pragma once
#include "tpx_tc_ptx.cuh"

namespace tpx {
// whether shapes are taken (then the call's scratch is mxfp4_dense_scratch_bytes), whether a call is, the call
bool mxfp4_dense_serves(int64_t M, int64_t N, int64_t K, bool pair);
size_t mxfp4_dense_scratch_bytes(int64_t M, int64_t N, int64_t K, bool pair);
bool mxfp4_dense_takes(const uint16_t* x, int64_t M, int64_t N, int64_t K, bool pair, const TcParams& base, size_t scratch_bytes, const TcNorm* norm);
int mxfp4_dense_run(const uint8_t* wq, const uint8_t* sfa, bool pair, const uint16_t* x, int64_t M, int64_t N, int64_t K, const TcParams& base,
                    void* scratch, size_t scratch_bytes, cudaStream_t st, const TcNorm* norm);
}  // namespace tpx

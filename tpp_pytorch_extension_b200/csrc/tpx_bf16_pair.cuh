// Shared by the linears of tpx_linear_bf16.cu, tpx_linear_bf16_pair.cu, tpx_linear_f32.cu and tpx_linear_f32_pair.cu: parameter
// blocks, the walk of CTA pairs over output tiles, sums of cut tiles.
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
  int quarter;  // (bf16 pair kernel, plain epilogue) the weight holds a quarter of its values (tpx_mxfp4_dense.cu)
  int glu;      // (with `quarter`) features 2i and 2i+1 are gate and up of unit i: y = act(gate + bias) * up, rows of N / 2
  int ctas;     // (one-CTA kernel) 0: whole tiles; else so many CTAs share all pipeline stages of all tiles evenly, a tile cut between CTAs is put together by the last of them
  int pieces;   // (pair kernels: see BpWork) pieces that each tile of the last round is cut into along k; up to 1: not cut
  BfEx ex;
};

struct F32Epi {
  const float* bias;
  void* y;
  long long ldy;
  int out_f32, act, act_from;
  const float* ap;
  float* z;  // gated units
  const float *res, *add, *nw, *nb;
  float *x_out, *h;
  long long ldz, ldr, ldh;
  float limit, nalpha;
};
// 32-bit linear: many rows on the tensor cores (tpx_linear_f32_pair.cu); rows m0 .. m0 + rows - 1 of a call on the CUDA cores
// (tpx_linear_f32.cu), with `flags` only the columns that the tensor cores left out: all if flags[0], else those of slabs of
// `slab` columns whose flag is set
bool f32_pair_serves(const TpxLinear& a);
int f32_pair_run(const TpxLinear& a, const F32Epi& e, cudaStream_t st);
int f32_fma_run(const TpxLinear& a, const F32Epi& e, int64_t m0, int64_t rows, const unsigned* flags, int64_t slab, cudaStream_t st);

// few tokens (tpx_linear_bf16_rows.cu)
bool bf_rows_serves(int64_t M, int64_t N, int64_t K, int64_t ldw);
int bf_rows_run(const BfParams& b, const void* w, const void* x, int64_t M, int64_t N, int64_t K, int64_t ldw, int64_t ldx, cudaStream_t st);
int bf_make_map(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows);
// many tokens on CTA pairs (tpx_linear_bf16_pair.cu): whether it takes this call, its scratch, the call
bool bf_pair_serves(const BfParams& p, int64_t M, int64_t N, int64_t K);
size_t bf_pair_scratch_bytes(int64_t M, int64_t N, int64_t K);
int bf_pair_run(BfParams& p, const void* w, const void* x, int64_t M, int64_t N, int64_t K, int64_t ldw, int64_t ldx, void* scratch,
                size_t scratch_bytes, cudaStream_t st);
// pieces that the tiles of the last round are cut into (1: not cut), clusters of the launch, and the bytes of the pieces
int bf_pair_split(int64_t M, int64_t N, int64_t K, double us_per_step);
int bf_pair_clusters(int64_t M, int64_t N, int split);
size_t bf_pair_split_bytes();

constexpr int kBpEpiWarps = 16;                 // four per 32-lane quarter of tensor memory
constexpr int kBpEpiCols = 1024 / kBpEpiWarps;  // features per warp
constexpr int kBpGroup = 16;  // token tiles walked side by side (bf16, 16384 x 14336 x 4096: 1210 us, with 8: 1231, with 4: 1270)

// What a cluster works on: k steps [g0, g1) of tile (tn, tm). Tiles are dealt out in turn, in blocks of kBpGroup token tiles (inside
// a block the token tiles of one feature tile are neighbours). p.pieces = S > 1: the tiles of the last, partly filled round are
// cut along k into S pieces for as many clusters.
struct BpWork {
  int T, ks, G, cid, TN, TM, S, W;  // W: tiles in front of the cut ones
  int tile, piece, g0, g1, tn, tm;
  __device__ __forceinline__ BpWork(const BfParams& p)
      : T(p.TN * p.TM), ks(p.ksteps), G((int)gridDim.x / 2), cid((int)blockIdx.x / 2), TN(p.TN), TM(p.TM), S(p.pieces > 1 ? p.pieces : 1) {
    W = T / G * G;
    tile = cid - G;
    piece = 0;
  }
  __device__ __forceinline__ bool next() {
    tile += G;
    g0 = 0;
    g1 = ks;
    if (tile >= W) {
      const int at = tile - W;  // beyond the range on the call after the last
      tile = W + at / S;
      if (at >= G || tile >= T) return false;
      piece = at % S;
      g0 = piece * ks / S;
      g1 = (piece + 1) * ks / S;
    }
    const int per = kBpGroup * TN, first = tile / per * kBpGroup, in = tile % per;
    const int side = min(kBpGroup, TM - first);
    tn = in / side;
    tm = first + in % side;
    return true;
  }
  __device__ __forceinline__ bool whole() const { return S == 1 || tile < W; }
  __device__ __forceinline__ int cluster_of(int j) const { return (tile - W) * S + j; }
};

// Partial sums of one epilogue warp of one CTA: [kBpEpiCols][32 lanes].
__device__ __forceinline__ float* bp_part(const BfParams& p, int cta, int ew) {
  return p.t.partial + ((size_t)cta * kBpEpiWarps + ew) * kBpEpiCols * 32;
}
// Called by all epilogue warps of a CTA behind their partial sums: whether this CTA is the last of the tile's (its half of the rows).
__device__ __forceinline__ bool bp_last(const BfParams& p, const BpWork& k, int crank, int* flag) {
  __threadfence();
  asm volatile("bar.sync 1, %0;" ::"n"(kBpEpiWarps * 32) : "memory");
  if (threadIdx.x == 64) {
    unsigned* c = p.t.counters + (k.tile - k.W) * 2 + crank;
    const bool last = atomicAdd(c, 1u) == (unsigned)(k.S - 1);
    if (last) *c = 0;
    *flag = last;
  }
  asm volatile("bar.sync 1, %0;" ::"n"(kBpEpiWarps * 32) : "memory");
  const bool last = *flag != 0;
  __threadfence();
  return last;
}
// The tile's pieces, added in the order of k; all columns of a piece are in flight at once, each load a round trip to L2.
__device__ __forceinline__ void bp_sum(const BfParams& p, const BpWork& k, int crank, int ew, int lane, float (&v)[kBpEpiCols]) {
#pragma unroll
  for (int j = 0; j < kBpEpiCols; j++) v[j] = 0.0f;
  for (int s = 0; s < k.S; s++) {
    const float* q = bp_part(p, k.cluster_of(s) * 2 + crank, ew) + lane;
    float t[kBpEpiCols];
#pragma unroll
    for (int j = 0; j < kBpEpiCols; j++) t[j] = __ldcg(q + j * 32);
#pragma unroll
    for (int j = 0; j < kBpEpiCols; j++) v[j] += t[j];
  }
}

__device__ __forceinline__ void bp_tma_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t cluster_bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(map), "r"(c0), "r"(c1), "r"(cluster_bar)
      : "memory");
}
__device__ __forceinline__ void bp_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
      "  tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p; }" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void bp_commit_both(uint32_t bar) {  // arrives on the barrier at this offset in both CTAs
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"((uint16_t)3)
               : "memory");
}
__device__ __forceinline__ void bp_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ bool bp_wait_cluster(uint32_t bar, uint32_t parity) {  // arrivals come from both CTAs; one verdict per warp
  uint32_t ok = 0;
  for (unsigned spins = 0; spins < kTcSpinLimit && !ok; spins++) {
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
  }
  return __all_sync(0xffffffffu, ok != 0);
}

// Eight consecutive values; the caller guarantees 16-byte alignment.
__device__ __forceinline__ void bp_ld8(const uint16_t* p, float (&o)[8]) {
  const uint4 v = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; j++) {
    o[2 * j] = __uint_as_float(w[j] << 16);
    o[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
  }
}
__device__ __forceinline__ void bp_ld8(const float* p, float (&o)[8]) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
}
__device__ __forceinline__ uint32_t bp_pack(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ void bp_st8(uint16_t* p, const float (&v)[8]) {
  *reinterpret_cast<uint4*>(p) = make_uint4(bp_pack(v[0], v[1]), bp_pack(v[2], v[3]), bp_pack(v[4], v[5]), bp_pack(v[6], v[7]));
}
__device__ __forceinline__ void bp_st8(float* p, const float (&v)[8]) {
  reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
  reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
}

}  // namespace tpx

// What the kernels for few tokens share (tpx_qlinear_i8_rows.cu, tpx_qlinear_mx_rows.cu, tpx_linear_bf16_rows.cu): weights copied by each warp into a ring of its own, activations
// straight from L2, tiles of 16 features.
#pragma once
#include "tpx_tc_ptx.cuh"

namespace tpx {

__device__ __forceinline__ void rows_copy16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ uint4 rows_lds16(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
// What the kernel before this one wrote: not __ldg, which may be moved in front of the wait for that kernel.
__device__ __forceinline__ uint4 rows_ldg16(const void* a) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(a) : "memory");
  return v;
}
__device__ __forceinline__ float2 rows_ldg8(const void* a) {
  float2 v;
  asm volatile("ld.global.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(a) : "memory");
  return v;
}
// Piece q (8 values) of a norm's weight on its way into L2. It may be what the kernel before this one writes, so that it is read behind the wait for that kernel;
// from HBM, beside the weight's stream, that took 0.5 us of every linear behind a norm.
__device__ __forceinline__ void rows_prefetch_gamma(const void* gamma, int f32, int q) {
  if ((q & (f32 ? 3 : 7)) == 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(gamma) + (size_t)q * (f32 ? 32 : 16)));
}
__device__ __forceinline__ float rows_lds4(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

// a float of the shared memory of member c of the cluster, at the address that it has here
__device__ __forceinline__ float rows_ld_member(uint32_t a, int c) {
  float v;
  asm volatile("{ .reg .b32 r; mapa.shared::cluster.u32 r, %1, %2; ld.shared::cluster.f32 %0, [r]; }" : "=f"(v) : "r"(a), "r"(c) : "memory");
  return v;
}

// Whether every CTA may read x for itself: x is in the memory of a device, and no CTA's y lands in it while another still reads.
inline bool rows_shared_x(const void* x, size_t x_bytes, const void* y, size_t y_bytes) {
  const uintptr_t a = (uintptr_t)x, b = (uintptr_t)y;
  if (a < b + y_bytes && b < a + x_bytes) return false;
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, x) == cudaSuccess) return at.type == cudaMemoryTypeDevice;
  (void)cudaGetLastError();
  return false;
}

// Feature tiles per CTA: one round of CTAs where that takes at most seven each, else the fewest rounds.
inline int rows_tiles(int64_t tiles) {
  const int sms = sm_count();
  int64_t tf = (tiles + sms - 1) / sms;
  if (tf > 7) {
    const int64_t rounds = (tiles + 7 * sms - 1) / (7 * sms);
    tf = (tiles + rounds * sms - 1) / (rounds * sms);
  }
  return tf < 1 ? 1 : (int)tf;
}

// How a CTA's T tiles of 16 features (of a pair: gate and up tiles in turn) and MG groups of 8 tokens are shared by its W warps: KG groups take the
// blocks of k in turn, each of H warps with N of the tiles, MOST being as many as a warp has registers for.
template <int T_, int MG_, int W_, int MOST>
struct RowsSplit {
  static constexpr int T = T_, MG = MG_, W = W_, H = T <= MOST ? 1 : T <= 2 * MOST ? 2 : 4;
  static constexpr int KG = W / H, N = (T + H - 1) / H;
  static constexpr int SURE = N - (H * N - T);  // tiles that the last of the H warps has
  static_assert(SURE > 0, "parts");
  static constexpr int RP = 16 * T + 4;  // a token's row of sums: 4 banks past a multiple of 16, so that lanes' stores do not meet
  static constexpr size_t PARTS = (size_t)(KG == 16 ? 8 : KG) * MG * 8 * RP * 4;
};

// Sums of a CTA's (or cluster's) groups, the epilogue and the store. acc: a lane's sums, [tile][tokens][row g, row g + 8] of tokens 2t, 2t + 1.
template <class C, bool DUAL>
__device__ __forceinline__ void rows_finish(float2 (&acc)[C::N][C::MG][2], unsigned char* smem, const TcParams& p, int tile0, int tile_own, int csize,
                                            int crank) {
  constexpr int T = C::T, MG = C::MG, KG = C::KG, N = C::N, RP = C::RP, TF = DUAL ? T / 2 : T;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, first = warp / KG * N;
  // the groups' sums, in their order
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  float* part_sums = reinterpret_cast<float*>(smem);
  constexpr int GS = KG == 16 ? 8 : KG;  // sums that are left per output
  if constexpr (KG == 16) {  // the upper eight warps hand theirs to the lower eight, which keeps the buffer small
    auto at = [&](int w) { return part_sums + (((size_t)w * T * MG) * 32 + lane) * 4; };
    if (warp >= 8)
#pragma unroll
      for (int j = 0; j < T * MG; j++) {
        const float2* v = acc[j / MG][j % MG];
        *reinterpret_cast<float4*>(at(warp - 8) + j * 128) = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
      }
    __syncthreads();
    if (warp < 8)
#pragma unroll
      for (int j = 0; j < T * MG; j++) {
        const float4 v = *reinterpret_cast<const float4*>(at(warp) + j * 128);
        float2* o = acc[j / MG][j % MG];
        o[0].x += v.x, o[0].y += v.y, o[1].x += v.z, o[1].y += v.w;
      }
    __syncthreads();
  }
  if (KG < 16 || warp < 8)
#pragma unroll
    for (int j = 0; j < N; j++)
#pragma unroll
      for (int m = 0; m < MG; m++) {
        if (j >= C::SURE && first + j >= T) continue;
        float* o = part_sums + ((size_t)(warp % GS) * MG * 8 + m * 8 + 2 * t) * RP + (first + j) * 16 + g;
        o[0] = acc[j][m][0].x;
        o[RP] = acc[j][m][0].y;
        o[8] = acc[j][m][1].x;
        o[RP + 8] = acc[j][m][1].y;
      }
  __syncthreads();
  constexpr int R = 16 * TF;
  const int skip = (tile_own - tile0) * 16, outs = R * p.M;
  // element idx of the CTA's outputs: its sums over the groups of this CTA; those of a pair's second weight 16 places on
  auto place = [&](int idx) { return part_sums + (size_t)(idx / R) * RP + (DUAL ? (idx % R / 16) * 32 + idx % 16 : idx % R); };
  auto group_sum = [&](const float* s) {
    float v = 0.0f;
#pragma unroll
    for (int w = 0; w < GS; w++) v += s[(size_t)w * MG * 8 * RP];
    return v;
  };
  auto finish = [&](int idx, float v, float u) {
    const int tok = idx / R, n = tile0 * 16 + idx % R;
    if (idx % R < skip) return;
    const size_t o = (size_t)tok * p.N + n;
    if (p.bias) v += bf16_bits_to_f32(p.bias[n]);
    if (p.act) v = apply_act(v, p.act);
    if (DUAL) v *= u;
    if (p.mul_in) v *= bf16_bits_to_f32(p.mul_in[o]);
    if (p.res) v += bf16_bits_to_f32(p.res[o]) * p.res_scale;
    p.y[o] = f32_to_bf16_bits(v);
  };
  if (csize == 1) {
    for (int idx = threadIdx.x; idx < outs; idx += C::W * 32) {
      const float* s = place(idx);
      finish(idx, group_sum(s), DUAL ? group_sum(s + 16) : 0.0f);
    }
    return;
  }
  // each member sums over its own groups, then takes its turn at adding the members' sums over distributed shared memory
  for (int idx = threadIdx.x; idx < outs; idx += C::W * 32) {
    float* s = place(idx);
    const float v = group_sum(s), u = DUAL ? group_sum(s + 16) : 0.0f;
    s[0] = v;
    if (DUAL) s[16] = u;
  }
  tc_cluster_sync();
  for (int idx = crank * C::W * 32 + threadIdx.x; idx < outs; idx += csize * C::W * 32) {
    const uint32_t at = tc_smem_u32(place(idx));
    float v = 0.0f, u = 0.0f;
    for (int c = 0; c < csize; c++) {
      v += rows_ld_member(at, c);
      if (DUAL) u += rows_ld_member(at + 64, c);
    }
    finish(idx, v, u);
  }
  tc_cluster_sync();  // nobody leaves before all have read
}

template <class P>
inline int rows_launch(void (*kernel)(P), int ctas, int cluster, int threads, size_t smem, cudaStream_t st, const P& p) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(ctas * cluster));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = knobs().pdl;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  count_launch();
  TPX_CUDA_OK(cudaLaunchKernelEx(&cfg, kernel, p));
  return TPX_OK;
}

}  // namespace tpx

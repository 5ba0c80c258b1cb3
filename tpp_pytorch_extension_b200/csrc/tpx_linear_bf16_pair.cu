// bf16 linear for many tokens on CTA pairs: tcgen05.mma.cta_group::2 kind::f16, M = 256 tokens x N = 256 features per pair.
//
// Serves the same calls as tpx_linear_bf16.cu (fc_plain on unquantized weights, the linears of the hybrid decoders) beyond
// 128 tokens. There a CTA multiplied 128 features by 256 tokens with three stages in flight, fetched 48 KB per 64 values of
// k, and its lanes held features, so that every result left as a 2-byte store.
// Here tokens are the rows of the MMA: a cluster of two CTAs computes 256 tokens x 256 features, each CTA holding its own 128
// tokens of x and HALF of the weight tile (the hardware reads both halves for both CTAs), 32 KB per 64 values of k, seven
// stages deep. A lane of the epilogue owns one token and consecutive features: 16-byte loads and stores, gated units without
// an exchange between lanes. Two accumulators of 256 columns fill tensor memory: the sixteen epilogue warps of a CTA work
// under the next tile's MMAs. Clusters walk the tiles in blocks of sixteen token tiles, so that the tiles in flight at a time
// share their operands through L2.
//   warp 0: TMA producer (both CTAs; copies complete on the first CTA's barrier)   warp 1: MMA issuer (first CTA)
//   warps 2-17: epilogue, four per 32-lane quarter of tensor memory
#include "tpx_bf16_pair.cuh"

namespace tpx {

struct BpCfg {
  static constexpr int HALF_BYTES = 128 * 128;  // 128 rows x 64 bf16
  static constexpr int STAGE_BYTES = 2 * HALF_BYTES;
  static constexpr int STAGES = 7;
  static constexpr int EPI_WARPS = 16;             // four per 32-lane quarter of tensor memory
  static constexpr int EPI_COLS = 1024 / EPI_WARPS;  // features per warp
  static constexpr int THREADS = 64 + 32 * EPI_WARPS;
  static constexpr int GROUP = 16;  // token tiles walked side by side (16384 x 14336 x 4096: 1210 us, with 8: 1231, with 4: 1270)
  static constexpr size_t SMEM = (size_t)STAGES * STAGE_BYTES + 1024;
};

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
__device__ __forceinline__ bool bp_wait_cluster(uint32_t bar, uint32_t parity) {  // arrivals come from both CTAs
  for (unsigned spins = 0; spins < kTcSpinLimit; spins++) {
    uint32_t ok;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    if (ok) return true;
  }
  return false;
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

// Features n .. n+7 of one token.
__device__ __forceinline__ void bp_finish8(const BfParams& p, long long row, int n, float (&x)[8]) {
  float t[8];
  if (!p.ex.on) {
    const TcParams& c = p.t;
    const size_t o = (size_t)row * c.N + n;
    if (c.bias) {
      bp_ld8(c.bias + n, t);
#pragma unroll
      for (int j = 0; j < 8; j++) x[j] += t[j];
    }
    switch (c.act) {
      case TPX_ACT_GELU:
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] = 0.5f * x[j] * (1.0f + erff(x[j] * 0.70710678118654752f));
        break;
      case TPX_ACT_SILU:
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] = __fdividef(x[j], 1.0f + __expf(-x[j]));
        break;
      case TPX_ACT_RELU:
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] = fmaxf(x[j], 0.0f);
        break;
      default: break;
    }
    if (c.mul_in) {
      bp_ld8(c.mul_in + o, t);
#pragma unroll
      for (int j = 0; j < 8; j++) x[j] *= t[j];
    }
    if (c.res) {
      bp_ld8(c.res + o, t);
#pragma unroll
      for (int j = 0; j < 8; j++) x[j] += t[j] * c.res_scale;
    }
    bp_st8(c.y + o, x);
    return;
  }
  const BfEx& e = p.ex;
  if (e.bias) {
    bp_ld8(e.bias + n, t);
#pragma unroll
    for (int j = 0; j < 8; j++) x[j] += t[j];
  }
  if (e.x_out) {
    if (e.add) {
      bp_ld8(e.add + n, t);
#pragma unroll
      for (int j = 0; j < 8; j++) x[j] += t[j];
    }
    bp_ld8(e.res + row * e.ldr + n, t);
#pragma unroll
    for (int j = 0; j < 8; j++) x[j] += t[j];
    bp_st8(e.x_out + row * e.ldr + n, x);
    float w[8];
    bp_ld8(e.nw + n, w);
    bp_ld8(e.nb + n, t);
#pragma unroll
    for (int j = 0; j < 8; j++) x[j] = fmaf(tanhf(e.nalpha * x[j]), w[j], t[j]);
    bp_st8(e.h + row * e.ldh + n, x);
    return;
  }
  if (e.act && n >= e.act_from) {
    if (e.act == TPX_ACT_CLAMPED_GLU) {
      float u[4];
#pragma unroll
      for (int j = 0; j < 4; j++) u[j] = hy_clamped_glu_fast(x[2 * j], x[2 * j + 1], e.limit);
      *reinterpret_cast<uint2*>(e.z + row * e.ldz + (n - e.act_from) / 2) = make_uint2(bp_pack(u[0], u[1]), bp_pack(u[2], u[3]));
      return;
    }
    const float a0 = e.ap ? e.ap[0] : 0.0f, a1 = e.ap ? e.ap[1] : 0.0f;
#pragma unroll
    for (int j = 0; j < 8; j++) x[j] = hy_act(x[j], e.act, a0, a1);
  }
  if (e.out_f32) bp_st8(reinterpret_cast<float*>(e.y) + row * e.ldy + n, x);
  else bp_st8(reinterpret_cast<uint16_t*>(e.y) + row * e.ldy + n, x);
}

// Tile t of the walk: blocks of GROUP token tiles, inside a block the token tiles of one feature tile are neighbours.
__device__ __forceinline__ void bp_tile(const BfParams& p, int t, int& tn, int& tm) {
  const int per = BpCfg::GROUP * p.TN;
  const int g0 = t / per * BpCfg::GROUP, in = t % per;
  const int rows = min(BpCfg::GROUP, p.TM - g0);
  tn = in / rows;
  tm = g0 + in % rows;
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(BpCfg::THREADS, 1)
linear_bf16_pair_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, BfParams p) {
  using C = BpCfg;
  extern __shared__ unsigned char bp_smem_raw[];
  __shared__ __align__(8) unsigned long long bar_full[C::STAGES], bar_empty[C::STAGES];
  __shared__ __align__(8) unsigned long long acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_holder;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_base = (tc_smem_u32(bp_smem_raw) + 1023u) & ~1023u;
  const int crank = (int)tc_cluster_rank();  // 0: issues the MMAs and owns the barriers the copies complete on
  const int T = p.TN * p.TM, G = gridDim.x / 2, cid = blockIdx.x / 2;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; s++) {
      tc_mbar_init(tc_smem_u32(&bar_full[s]), 1);
      tc_mbar_init(tc_smem_u32(&bar_empty[s]), 1);
    }
    for (int b = 0; b < 2; b++) {
      tc_mbar_init(tc_smem_u32(&acc_full[b]), 1);
      tc_mbar_init(tc_smem_u32(&acc_empty[b]), 2 * C::EPI_WARPS);  // the epilogue warps of both CTAs
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {  // the same warp of both CTAs: the allocation covers both SMs at the same address
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(&tmem_holder)), "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_cluster_sync();  // the partner's barriers and tensor memory exist before anything is sent to them
  tc_fence_after();
  const uint32_t tmem = tmem_holder;
  pdl_trigger();

  if (warp == 0) {
    // ------------------------------------------------------------ producer (both CTAs)
    pdl_wait();
    int s = 0;
    uint32_t phase = 1;  // parity to wait for on bar_empty: the first round over the ring finds every stage free
    bool dead = false;
    for (int t = cid; t < T && !dead; t += G) {
      int tn, tm;
      bp_tile(p, t, tn, tm);
      const int row = tm * 256 + crank * 128, col = tn * 256 + crank * 128;
      for (int g = 0; g < p.ksteps; g++) {
        if (!tc_wait(tc_smem_u32(&bar_empty[s]), phase)) {
          if (tc_elect()) atomicExch(p.t.err, 2u);
          dead = true;
          break;
        }
        if (tc_elect()) {
          const uint32_t st = smem_base + (uint32_t)s * C::STAGE_BYTES;
          const uint32_t lbar = tc_mapa(tc_smem_u32(&bar_full[s]), 0u);  // the first CTA's barrier
          if (crank == 0) tc_mbar_expect_tx(tc_smem_u32(&bar_full[s]), 2u * C::STAGE_BYTES);
          bp_tma_2d(st, &tmX, g * 64, row, lbar);
          bp_tma_2d(st + C::HALF_BYTES, &tmW, g * 64, col, lbar);
        }
        __syncwarp();
        if (++s == C::STAGES) s = 0, phase ^= 1u;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (first CTA only)
    if (crank == 0) {
      // kind::f16: D = F32 (1), A = B = BF16 (1), both K-major, N = 256, M = 256 over the pair
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(256 >> 3) << 17) | ((256u >> 4) << 24);
      const uint64_t desc0 = tc_smem_desc(smem_base);
      int s = 0, i = 0;
      uint32_t phase = 0;
      bool dead = false;
      for (int t = cid; t < T && !dead; t += G, i++) {
        const int buf = i & 1;
        if (i >= 2) {  // both CTAs' epilogue warps have drained this accumulator
          if (!bp_wait_cluster(tc_smem_u32(&acc_empty[buf]), (uint32_t)((i / 2 - 1) & 1))) {
            if (tc_elect()) atomicExch(p.t.err, 3u);
            break;
          }
          tc_fence_after();
        }
        for (int g = 0; g < p.ksteps; g++) {
          if (!tc_wait(tc_smem_u32(&bar_full[s]), phase)) {
            if (tc_elect()) atomicExch(p.t.err, 4u);
            dead = true;
            break;
          }
          tc_fence_after();
          if (tc_elect()) {
            const uint64_t desc = desc0 + (uint64_t)(s * (C::STAGE_BYTES >> 4));  // descriptors count 16-byte units
#pragma unroll
            for (int j = 0; j < 4; j++)
              bp_mma(tmem + buf * 256, desc + (uint64_t)(2 * j), desc + (uint64_t)((C::HALF_BYTES >> 4) + 2 * j), idesc, (g | j) ? 1u : 0u);
            bp_commit_both(tc_smem_u32(&bar_empty[s]));
            if (g == p.ksteps - 1) bp_commit_both(tc_smem_u32(&acc_full[buf]));
          }
          __syncwarp();
          if (++s == C::STAGES) s = 0, phase ^= 1u;
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2 .. 17 of both CTAs)
    const int sub = warp & 3;  // tensor-memory lanes 32*sub .. 32*sub+31 belong to this warp
    const int c_first = ((warp - 2) >> 2) * C::EPI_COLS;
    const uint32_t lane_base = ((uint32_t)(sub * 32)) << 16;
    pdl_wait();  // residual and multiplier inputs belong to earlier grids
    int i = 0;
    for (int t = cid; t < T; t += G, i++) {
      const int buf = i & 1;
      if (!tc_wait(tc_smem_u32(&acc_full[buf]), (uint32_t)((i / 2) & 1))) {
        if (lane == 0) atomicExch(p.t.err, 6u);
        break;
      }
      tc_fence_after();
      int tn, tm;
      bp_tile(p, t, tn, tm);
      const long long row = (long long)tm * 256 + crank * 128 + sub * 32 + lane;
      const int n0 = tn * 256 + c_first;
#pragma unroll 1
      for (int c = 0; c < C::EPI_COLS && n0 + c < p.t.N; c += 16) {
        uint32_t a[16];
        tc_ld_x16(tmem + lane_base + (uint32_t)(buf * 256 + c_first + c), a);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (row < p.t.M) {
#pragma unroll
          for (int h = 0; h < 2; h++) {
            float x[8];
#pragma unroll
            for (int j = 0; j < 8; j++) x[j] = __uint_as_float(a[h * 8 + j]);
            if (n0 + c + h * 8 < p.t.N) bp_finish8(p, row, n0 + c + h * 8, x);
          }
        }
        __syncwarp();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) bp_arrive_cluster(tc_mapa(tc_smem_u32(&acc_empty[buf]), 0u));
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_cluster_sync();  // nobody leaves, and tensor memory is not freed, while the partner may still use this CTA's memory
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// The epilogue moves eight values at a time: every row it touches has to start on a 16-byte boundary.
bool bf_pair_serves(const BfParams& p, int64_t M, int64_t N, int64_t K) {
  (void)K;
  if (M <= 128 || N % 8) return false;
  uintptr_t at = 0;
  int64_t ld = 0;
  if (!p.ex.on) {
    at = (uintptr_t)p.t.bias | (uintptr_t)p.t.mul_in | (uintptr_t)p.t.res | (uintptr_t)p.t.y;
  } else {
    const BfEx& e = p.ex;
    at = (uintptr_t)e.bias | (uintptr_t)e.res | (uintptr_t)e.add | (uintptr_t)e.x_out | (uintptr_t)e.h;
    if (e.x_out) at |= (uintptr_t)e.nw | (uintptr_t)e.nb, ld |= e.ldr | e.ldh;
    else at |= (uintptr_t)e.y, ld |= e.ldy;
    if (e.act == TPX_ACT_CLAMPED_GLU) at |= (uintptr_t)e.z, ld |= e.ldz | e.act_from;
    else if (e.act) ld |= e.act_from;
  }
  return at % 16 == 0 && ld % 8 == 0;
}

int bf_pair_run(BfParams& p, const void* w, const void* x, int64_t M, int64_t N, int64_t K, int64_t ldw, int64_t ldx, cudaStream_t st) {
  using C = BpCfg;
  p.split = 0;
  p.t.M = (int)M; p.t.N = (int)N; p.t.K = (int)K;
  p.ksteps = (int)((K + 63) / 64);
  p.TN = (int)((N + 255) / 256);
  p.TM = (int)((M + 255) / 256);
  CUtensorMap mw, mx;
  int rc = bf_make_map(&mw, w, (uint64_t)N, (uint64_t)K, (uint64_t)ldw, 128);
  if (rc) return rc;
  rc = bf_make_map(&mx, x, (uint64_t)M, (uint64_t)K, (uint64_t)ldx, 128);
  if (rc) return rc;
  static bool opted[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16 || !opted[dev]) {
    TPX_CUDA_OK(cudaFuncSetAttribute(linear_bf16_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM));
    if (dev >= 0 && dev < 16) opted[dev] = true;
  }
  const long long T = (long long)p.TN * p.TM;
  const long long pairs = sm_count() / 2;
  const int grid = 2 * (int)(T < pairs ? T : pairs);
  TPX_CUDA_OK(launch_pdl(linear_bf16_pair_kernel, dim3((unsigned)grid), dim3(C::THREADS), C::SMEM, st, mw, mx, p));
  return TPX_OK;
}

}  // namespace tpx

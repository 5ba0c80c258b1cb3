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
  static constexpr int THREADS = 64 + 32 * kBpEpiWarps;
  static constexpr size_t SMEM = (size_t)STAGES * STAGE_BYTES + 1024;
};

__device__ __forceinline__ void bp_activate8(int act, float (&x)[8]) {
  switch (act) {
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
}

// Units n .. n+7 of one token from sixteen features (BfParams::glu; the features are a multiple of 64).
__device__ __forceinline__ void bp_finish_glu8(const BfParams& p, long long row, int n, const float (&v)[16]) {
  const TcParams& c = p.t;
  const size_t o = (size_t)row * (c.N / 2) + n;
  float x[8], t[8];
#pragma unroll
  for (int j = 0; j < 8; j++) x[j] = v[2 * j];
  if (c.bias) {
    bp_ld8(c.bias + n, t);
#pragma unroll
    for (int j = 0; j < 8; j++) x[j] += t[j];
  }
  bp_activate8(c.act, x);
#pragma unroll
  for (int j = 0; j < 8; j++) x[j] *= v[2 * j + 1];
  if (c.res) {
    bp_ld8(c.res + o, t);
#pragma unroll
    for (int j = 0; j < 8; j++) x[j] += t[j] * c.res_scale;
  }
  bp_st8(c.y + o, x);
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
    bp_activate8(c.act, x);
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

// QUARTER: BfParams::quarter as a constant (as a factor read from the parameters it took 1 us of a 13 us call in spilled registers)
template <bool QUARTER>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(BpCfg::THREADS, 1)
linear_bf16_pair_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, BfParams p) {
  using C = BpCfg;
  extern __shared__ unsigned char bp_smem_raw[];
  __shared__ __align__(8) unsigned long long bar_full[C::STAGES], bar_empty[C::STAGES];
  __shared__ __align__(8) unsigned long long acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_holder;
  __shared__ int last_piece;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_base = (tc_smem_u32(bp_smem_raw) + 1023u) & ~1023u;
  const int crank = (int)tc_cluster_rank();  // 0: issues the MMAs and owns the barriers the copies complete on

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; s++) {
      tc_mbar_init(tc_smem_u32(&bar_full[s]), 1);
      tc_mbar_init(tc_smem_u32(&bar_empty[s]), 1);
    }
    for (int b = 0; b < 2; b++) {
      tc_mbar_init(tc_smem_u32(&acc_full[b]), 1);
      tc_mbar_init(tc_smem_u32(&acc_empty[b]), 2 * kBpEpiWarps);  // the epilogue warps of both CTAs
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
    for (BpWork k(p); !dead && k.next();) {
      const int row = k.tm * 256 + crank * 128, col = k.tn * 256 + crank * 128;
      for (int g = k.g0; g < k.g1; g++) {
        if (!tc_wait_warp(tc_smem_u32(&bar_empty[s]), phase)) {
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
      for (BpWork k(p); !dead && k.next(); i++) {
        const int buf = i & 1;
        if (i >= 2) {  // both CTAs' epilogue warps have drained this accumulator
          if (!bp_wait_cluster(tc_smem_u32(&acc_empty[buf]), (uint32_t)((i / 2 - 1) & 1))) {
            if (tc_elect()) atomicExch(p.t.err, 3u);
            break;
          }
          tc_fence_after();
        }
        for (int g = k.g0; g < k.g1; g++) {
          if (!tc_wait_warp(tc_smem_u32(&bar_full[s]), phase)) {
            if (tc_elect()) atomicExch(p.t.err, 4u);
            dead = true;
            break;
          }
          tc_fence_after();
          if (tc_elect()) {
            const uint64_t desc = desc0 + (uint64_t)(s * (C::STAGE_BYTES >> 4));  // descriptors count 16-byte units
#pragma unroll
            for (int j = 0; j < 4; j++)
              bp_mma(tmem + buf * 256, desc + (uint64_t)(2 * j), desc + (uint64_t)((C::HALF_BYTES >> 4) + 2 * j), idesc,
                     (g > k.g0 || j) ? 1u : 0u);
            bp_commit_both(tc_smem_u32(&bar_empty[s]));
            if (g == k.g1 - 1) bp_commit_both(tc_smem_u32(&acc_full[buf]));
          }
          __syncwarp();
          if (++s == C::STAGES) s = 0, phase ^= 1u;
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2 .. 17 of both CTAs)
    const int sub = warp & 3;  // tensor-memory lanes 32*sub .. 32*sub+31 belong to this warp
    const int c_first = ((warp - 2) >> 2) * kBpEpiCols;
    const uint32_t lane_base = ((uint32_t)(sub * 32)) << 16;
    pdl_wait();  // residual and multiplier inputs belong to earlier grids
    int i = 0;
    bool dead = false;  // a warp that gave up still meets the others at their barriers
    for (BpWork k(p); k.next(); i++) {
      const int buf = i & 1;
      if (!dead && !tc_wait_warp(tc_smem_u32(&acc_full[buf]), (uint32_t)((i / 2) & 1))) {
        if (lane == 0) atomicExch(p.t.err, 6u);
        dead = true;
      }
      tc_fence_after();
      const long long row = (long long)k.tm * 256 + crank * 128 + sub * 32 + lane;
      const int n0 = k.tn * 256 + c_first;
      const bool whole = k.whole();
      float* part = bp_part(p, blockIdx.x, warp - 2) + lane;
      auto finish = [&](int c, float (&v)[16]) {
        if (QUARTER) {
#pragma unroll
          for (int j = 0; j < 16; j++) v[j] *= 4.0f;
        }
        if (QUARTER && p.glu) {
          if (row < p.t.M && n0 + c < p.t.N) bp_finish_glu8(p, row, (n0 + c) / 2, v);
          return;
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
          float x[8];
#pragma unroll
          for (int j = 0; j < 8; j++) x[j] = v[h * 8 + j];
          if (row < p.t.M && n0 + c + h * 8 < p.t.N) bp_finish8(p, row, n0 + c + h * 8, x);
        }
      };
#pragma unroll 1
      for (int c = 0; c < kBpEpiCols && n0 + c < p.t.N && !dead; c += 16) {
        uint32_t a[16];
        float v[16];
        tc_ld_x16(tmem + lane_base + (uint32_t)(buf * 256 + c_first + c), a);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] = __uint_as_float(a[j]);
        if (whole) finish(c, v);
        else {
#pragma unroll
          for (int j = 0; j < 16; j++) part[(c + j) * 32] = v[j];
        }
        __syncwarp();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) bp_arrive_cluster(tc_mapa(tc_smem_u32(&acc_empty[buf]), 0u));
      if (!whole && bp_last(p, k, crank, &last_piece)) {
        float sum[kBpEpiCols];
        bp_sum(p, k, crank, warp - 2, lane, sum);
#pragma unroll
        for (int c = 0; c < kBpEpiCols; c += 16) {
          float v[16];
#pragma unroll
          for (int j = 0; j < 16; j++) v[j] = sum[c + j];
          finish(c, v);
        }
      }
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

// The last round of tiles leaves clusters idle where it is at most half full: its tiles are then cut along k into up to four pieces,
// if the k steps saved are worth more than 1.2 us per piece (written to L2 by one CTA, read by another) and 2 us.
int bf_pair_split(int64_t M, int64_t N, int64_t K, double us_per_step) {
  const int64_t T = ((M + 255) / 256) * ((N + 255) / 256), ks = (K + 63) / 64, G = sm_count() / 2;
  const int64_t R = T % G;
  if (R == 0) return 1;
  int best = 1;
  double gain = 0.0;
  for (int S = 2; S <= 4 && S * R <= G && S * 4 <= ks; S++) {
    const double g = (double)(ks - (ks + S - 1) / S) * us_per_step - 1.2 * S - 2.0;
    if (g > gain) gain = g, best = S;
  }
  return best;
}
int bf_pair_clusters(int64_t M, int64_t N, int split) {
  const int64_t T = ((M + 255) / 256) * ((N + 255) / 256), G = sm_count() / 2;
  return (int)(T >= G ? G : T * split);
}
size_t bf_pair_split_bytes() { return (size_t)(sm_count() / 2) * 2 * 128 * 256 * 4; }

constexpr double kBpUsPerStep = 0.27;
size_t bf_pair_scratch_bytes(int64_t M, int64_t N, int64_t K) {
  return kTcCounterBytes + (bf_pair_split(M, N, K, kBpUsPerStep) > 1 ? bf_pair_split_bytes() : 0);
}

int bf_pair_run(BfParams& p, const void* w, const void* x, int64_t M, int64_t N, int64_t K, int64_t ldw, int64_t ldx, void* scratch,
                size_t scratch_bytes, cudaStream_t st) {
  using C = BpCfg;
  p.pieces = bf_pair_split(M, N, K, kBpUsPerStep);
  if (p.pieces > 1 && scratch_bytes < kTcCounterBytes + bf_pair_split_bytes()) p.pieces = 1;
  p.t.counters = reinterpret_cast<unsigned*>(scratch);
  p.t.partial = reinterpret_cast<float*>(reinterpret_cast<unsigned char*>(scratch) + kTcCounterBytes);
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
    TPX_CUDA_OK(cudaFuncSetAttribute(linear_bf16_pair_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM));
    TPX_CUDA_OK(cudaFuncSetAttribute(linear_bf16_pair_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM));
    if (dev >= 0 && dev < 16) opted[dev] = true;
  }
  const int grid = 2 * bf_pair_clusters(M, N, p.pieces);
  TPX_CUDA_OK(launch_pdl(p.quarter ? linear_bf16_pair_kernel<true> : linear_bf16_pair_kernel<false>, dim3((unsigned)grid), dim3(C::THREADS), C::SMEM, st, mw, mx, p));
  return TPX_OK;
}

}  // namespace tpx

// 32-bit linear for many rows on the tensor cores: every fp32 operand is the sum of three bf16 terms (x = h + m + l, each the
// rounding of what the terms before it left; 3 x 8 significand bits with signed remainders hold all 24), and a product of two
// operands is taken as the sum of six products of terms: hh, hm, mh, mm, hl, lh. bf16 products are exact in fp32. The three left out
// (ml, lm, ll) are together at most 2^-24 of the product (|m| <= 2^-8 |x|, |l| <= 2^-17 |x|).
// Operands are multiplied by 2^24 before they are cut, sums by 2^-48 behind: the last bit of any fp32 value, subnormal ones
// included, is then at least 2^-125, which bf16 terms (multiples of 2^-133) and their products hold. (Without it an operand of 2^-120
// lost eight bits.) Operands of 2^30 and more are left to the CUDA cores, so that no sum of products of terms can overflow.
//
// Sums: the tensor core's own accumulation is kept short. 64 values of k (24 MMAs, the small terms first) accumulate in tensor
// memory; then sixteen epilogue warps pull the accumulator and add it to fp32 registers with rounding to nearest, while the
// next 64 values multiply into the other accumulator. A sum over K = 4096 so has 64 rounded additions where a loop of
// fused multiply-adds has 4096: against 64 bits the result is closer than that of linear_f32_kernel.
// Bounds: 6 bf16 products per fp32 product, i.e. a sixth of the bf16 rate; 96 KB per 64 values of k and CTA leave room for two
// stages, and 3072 cycles of MMAs per stage hide the copies.
// The terms are made per call in the scratch: all of x (up to kFpRows rows at a time), the weights in slabs small enough to
// stay in L2 between the kernel that writes them and the one that reads them. For an infinity, a NaN or a value of 2^30 and more the
// split kernels raise a flag: the tensor-core kernel then leaves that slab alone and linear_f32_kernel computes it.
#include "tpx_bf16_pair.cuh"

namespace tpx {

constexpr int64_t kFpRows = 2048;             // rows of x at a time
constexpr int64_t kFpSlabBytes = 48ll << 20;  // terms of a slab of weight rows
constexpr int kFpFlags = 128;                 // x, then one per slab

constexpr float kFpScale = 16777216.0f, kFpUnscale = 1.0f / (kFpScale * kFpScale);  // 2^24, 2^-48
constexpr float kFpLargest = 1073741824.0f;                                        // 2^30: K products stay below K 2^108
constexpr int64_t kFpMostK = 1 << 19;

constexpr double kFpUsPerStep = 1.7;

struct FpCfg {
  static constexpr int HALF_BYTES = 128 * 128;  // 128 rows x 64 terms
  static constexpr int STAGE_BYTES = 6 * HALF_BYTES;
  static constexpr int STAGES = 2;
  static constexpr int THREADS = 64 + 32 * kBpEpiWarps;
  static constexpr size_t SMEM = (size_t)STAGES * STAGE_BYTES + 1024;
};

// Eight values of a row per thread: src [rows][K], rows ld apart -> terms [3][rows][K].
__global__ void __launch_bounds__(256) split3_kernel(const float* __restrict__ src, long long ld, long long rows, int K, uint16_t* __restrict__ dst,
                                                     unsigned* __restrict__ flag) {
  pdl_trigger();
  pdl_wait();
  const int kv = K / 8;
  const long long n = rows * kv, plane = rows * K;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n; i += (long long)gridDim.x * 256) {
    const long long r = i / kv;
    const int k = (int)(i - r * kv) * 8;
    float v[8];
    bp_ld8(src + r * ld + k, v);
    float m[8], l[8];
    bool odd = false;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const bool bad = !(fabsf(v[j]) < kFpLargest);
      odd |= bad;
      v[j] *= kFpScale;
      const float r1 = bad ? 0.0f : v[j] - __bfloat162float(__float2bfloat16_rn(v[j]));
      m[j] = __bfloat162float(__float2bfloat16_rn(r1));
      l[j] = r1 - m[j];
    }
    if (odd) *flag = 1u;
    uint16_t* d = dst + r * K + k;
    bp_st8(d, v);
    bp_st8(d + plane, m);
    bp_st8(d + 2 * plane, l);
  }
}

// Features n .. n+7 of one token.
__device__ __forceinline__ void fp_finish8(const F32Epi& e, long long row, int n, float (&x)[8]) {
  float t[8];
  if (e.bias) {
    bp_ld8(e.bias + n, t);
#pragma unroll
    for (int j = 0; j < 8; j++) x[j] += t[j];
  }
  if (e.x_out) {
    bp_ld8(e.res + row * e.ldr + n, t);
#pragma unroll
    for (int j = 0; j < 8; j++) x[j] += t[j];
    if (e.add) {
      bp_ld8(e.add + n, t);
#pragma unroll
      for (int j = 0; j < 8; j++) x[j] += t[j];
    }
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
      for (int j = 0; j < 4; j++) u[j] = hy_clamped_glu(x[2 * j], x[2 * j + 1], e.limit);
      *reinterpret_cast<float4*>(e.z + row * e.ldz + (n - e.act_from) / 2) = make_float4(u[0], u[1], u[2], u[3]);
      return;
    }
    const float a0 = e.ap ? e.ap[0] : 0.0f, a1 = e.ap ? e.ap[1] : 0.0f;
#pragma unroll
    for (int j = 0; j < 8; j++) x[j] = hy_act(x[j], e.act, a0, a1);
  }
  if (e.out_f32) bp_st8(reinterpret_cast<float*>(e.y) + row * e.ldy + n, x);
  else bp_st8(reinterpret_cast<uint16_t*>(e.y) + row * e.ldy + n, x);
}

// p: tiles of this launch (rows 0 .. M-1 of the x terms, weight rows 0 .. N-1 of the slab); rows0, n0: where they lie in the call.
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(FpCfg::THREADS, 1)
linear_f32_pair_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, BfParams p, F32Epi e, long long row0,
                       int n00, const unsigned* __restrict__ flag_x, const unsigned* __restrict__ flag_w) {
  using C = FpCfg;
  extern __shared__ unsigned char fp_smem_raw[];
  __shared__ __align__(8) unsigned long long bar_full[C::STAGES], bar_empty[C::STAGES];
  __shared__ __align__(8) unsigned long long acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_holder;
  __shared__ int last_piece;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_base = (tc_smem_u32(fp_smem_raw) + 1023u) & ~1023u;
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
  pdl_wait();
  const bool skip = *flag_x != 0 || *flag_w != 0;  // the same in every thread of the grid

  if (skip) {
  } else if (warp == 0) {
    // ------------------------------------------------------------ producer (both CTAs)
    int s = 0;
    uint32_t phase = 1;
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
#pragma unroll
          for (int t = 0; t < 3; t++) {  // rows beyond a plane's end belong to the next: results of those rows are dropped
            bp_tma_2d(st + t * C::HALF_BYTES, &tmX, g * 64, t * p.t.M + row, lbar);
            bp_tma_2d(st + (3 + t) * C::HALF_BYTES, &tmW, g * 64, t * p.t.N + col, lbar);
          }
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
      constexpr int XT[6] = {0, 2, 1, 0, 1, 0}, WT[6] = {2, 0, 1, 1, 0, 0};  // terms h = 0, m = 1, l = 2
      int s = 0, i = 0;
      uint32_t phase = 0;
      bool dead = false;
      for (BpWork k(p); !dead && k.next();) {
        for (int g = k.g0; g < k.g1; g++, i++) {
          const int buf = i & 1;
          if (i >= 2) {  // both CTAs' epilogue warps have drained this accumulator
            if (!bp_wait_cluster(tc_smem_u32(&acc_empty[buf]), (uint32_t)((i / 2 - 1) & 1))) {
              if (tc_elect()) atomicExch(p.t.err, 3u);
              dead = true;
              break;
            }
          }
          if (!tc_wait_warp(tc_smem_u32(&bar_full[s]), phase)) {
            if (tc_elect()) atomicExch(p.t.err, 4u);
            dead = true;
            break;
          }
          tc_fence_after();
          if (tc_elect()) {
            const uint64_t desc = desc0 + (uint64_t)(s * (C::STAGE_BYTES >> 4));  // descriptors count 16-byte units
#pragma unroll
            for (int t = 0; t < 6; t++) {
#pragma unroll
              for (int j = 0; j < 4; j++)
                bp_mma(tmem + buf * 256, desc + (uint64_t)(XT[t] * (C::HALF_BYTES >> 4) + 2 * j),
                       desc + (uint64_t)((3 + WT[t]) * (C::HALF_BYTES >> 4) + 2 * j), idesc, (t | j) ? 1u : 0u);
            }
            bp_commit_both(tc_smem_u32(&bar_empty[s]));
            bp_commit_both(tc_smem_u32(&acc_full[buf]));
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
    int i = 0;
    bool dead = false;  // a warp that gave up still meets the others at their barriers
    for (BpWork k(p); k.next();) {
      float acc[kBpEpiCols] = {};
      for (int g = k.g0; g < k.g1; g++, i++) {
        const int buf = i & 1;
        if (!dead && !tc_wait_warp(tc_smem_u32(&acc_full[buf]), (uint32_t)((i / 2) & 1))) {
          if (lane == 0) atomicExch(p.t.err, 6u);
          dead = true;
        }
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < kBpEpiCols; c += 16) {
          uint32_t a[16];
          tc_ld_x16(tmem + lane_base + (uint32_t)(buf * 256 + c_first + c), a);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 16; j++) acc[c + j] += __uint_as_float(a[j]);
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) bp_arrive_cluster(tc_mapa(tc_smem_u32(&acc_empty[buf]), 0u));
      }
      const long long row = (long long)k.tm * 256 + crank * 128 + sub * 32 + lane;
      const int n0 = k.tn * 256 + c_first;
      if (!k.whole()) {
        float* part = bp_part(p, blockIdx.x, warp - 2) + lane;
#pragma unroll
        for (int c = 0; c < kBpEpiCols; c++) part[c * 32] = acc[c];
        if (!bp_last(p, k, crank, &last_piece)) continue;
        bp_sum(p, k, crank, warp - 2, lane, acc);
      }
#pragma unroll
      for (int c = 0; c < kBpEpiCols; c += 8) {
        float x[8];
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] = acc[c + j] * kFpUnscale;
        if (!dead && row < p.t.M && n0 + c < p.t.N) fp_finish8(e, row0 + row, n00 + n0 + c, x);
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

// ---------------------------------------------------------------- host side
struct FpPlan {
  int64_t rows, slab;  // rows of x and of the weight at a time
  size_t off_flags, off_x, off_w, total;
};

static FpPlan fp_plan(int64_t M, int64_t N, int64_t K) {
  FpPlan pl;
  pl.rows = M < kFpRows ? M : kFpRows;
  pl.slab = kFpSlabBytes / (6 * K) / 256 * 256;
  if (pl.slab < 256) pl.slab = 256;
  if ((N + pl.slab - 1) / pl.slab > kFpFlags - 1) pl.slab = ((N + kFpFlags - 2) / (kFpFlags - 1) + 255) / 256 * 256;
  if (pl.slab > N) pl.slab = N;
  size_t o = kTcCounterBytes + bf_pair_split_bytes();
  auto bump = [&](size_t bytes) { size_t r = o; o += (bytes + 255) & ~(size_t)255; return r; };
  pl.off_flags = bump(kFpFlags * sizeof(unsigned));
  pl.off_x = bump((size_t)pl.rows * K * 6);
  pl.off_w = bump((size_t)pl.slab * K * 6);
  pl.total = o;
  return pl;
}

// From 48 rows on and where the CUDA cores would take 40 us or more (they do 15 TFLOP/s); rows in whole 16-byte units of eight values.
static bool fp_shape(int64_t M, int64_t N, int64_t K) {
  return M >= 48 && K % 8 == 0 && K <= kFpMostK && N % 8 == 0 && 2.0 * M * N * K >= 6e8;
}
size_t f32_pair_scratch_bytes(int64_t M, int64_t N, int64_t K) { return fp_shape(M, N, K) ? fp_plan(M, N, K).total : 0; }

bool f32_pair_serves(const TpxLinear& a) {
  if (!fp_shape(a.M, a.N, a.K) || !a.scratch || ((uintptr_t)a.scratch & 255) || a.scratch_bytes < fp_plan(a.M, a.N, a.K).total) return false;
  uintptr_t at = (uintptr_t)a.w | (uintptr_t)a.x | (uintptr_t)a.bias | (uintptr_t)a.res | (uintptr_t)a.add | (uintptr_t)a.x_out | (uintptr_t)a.h;
  int64_t ld = a.ldx | a.ldw;
  if (a.x_out) at |= (uintptr_t)a.norm_w | (uintptr_t)a.norm_b, ld |= a.ldr | a.ldh;
  else at |= (uintptr_t)a.y, ld |= a.ldy;
  if (a.act == TPX_ACT_CLAMPED_GLU) at |= (uintptr_t)a.z, ld |= a.ldz | a.act_from;
  else if (a.act) ld |= a.act_from;
  return at % 16 == 0 && ld % 8 == 0;
}

int f32_pair_run(const TpxLinear& a, const F32Epi& e, cudaStream_t st) {
  using C = FpCfg;
  const FpPlan pl = fp_plan(a.M, a.N, a.K);
  unsigned char* sc = reinterpret_cast<unsigned char*>(a.scratch);
  unsigned* flags = reinterpret_cast<unsigned*>(sc + pl.off_flags);
  uint16_t *xt = reinterpret_cast<uint16_t*>(sc + pl.off_x), *wt = reinterpret_cast<uint16_t*>(sc + pl.off_w);
  static bool opted[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16 || !opted[dev]) {
    TPX_CUDA_OK(cudaFuncSetAttribute(linear_f32_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM));
    if (dev >= 0 && dev < 16) opted[dev] = true;
  }
  auto split = [&](const float* src, int64_t ld, int64_t rows, uint16_t* dst, unsigned* flag) {
    const int64_t blocks = (rows * (a.K / 8) + 255) / 256, most = 8ll * sm_count();
    return launch_pdl(split3_kernel, dim3((unsigned)(blocks < most ? blocks : most)), dim3(256), 0, st, src, (long long)ld, (long long)rows, (int)a.K,
                      dst, flag);
  };
  for (int64_t m0 = 0; m0 < a.M; m0 += pl.rows) {
    const int64_t rows = a.M - m0 < pl.rows ? a.M - m0 : pl.rows;
    TPX_CUDA_OK(cudaMemsetAsync(flags, 0, kFpFlags * sizeof(unsigned), st));
    TPX_CUDA_OK(split((const float*)a.x + m0 * a.ldx, a.ldx, rows, xt, flags));
    CUtensorMap mx;
    int rc = bf_make_map(&mx, xt, (uint64_t)rows * 3, (uint64_t)a.K, (uint64_t)a.K, 128);
    if (rc) return rc;
    int slab = 0;
    for (int64_t n0 = 0; n0 < a.N; n0 += pl.slab, slab++) {
      const int64_t n = a.N - n0 < pl.slab ? a.N - n0 : pl.slab;
      TPX_CUDA_OK(split((const float*)a.w + n0 * a.ldw, a.ldw, n, wt, flags + 1 + slab));
      CUtensorMap mw;
      rc = bf_make_map(&mw, wt, (uint64_t)n * 3, (uint64_t)a.K, (uint64_t)a.K, 128);
      if (rc) return rc;
      BfParams p = {};
      p.t.M = (int)rows; p.t.N = (int)n; p.t.K = (int)a.K;
      p.t.counters = reinterpret_cast<unsigned*>(sc);
      p.t.partial = reinterpret_cast<float*>(sc + kTcCounterBytes);
      p.t.err = reinterpret_cast<unsigned*>(sc + kTcCounterBytes - 4);
      p.ksteps = (int)((a.K + 63) / 64);
      p.TN = (int)((n + 255) / 256);
      p.TM = (int)((rows + 255) / 256);
      p.pieces = bf_pair_split(rows, n, a.K, kFpUsPerStep);
      const int grid = 2 * bf_pair_clusters(rows, n, p.pieces);
      TPX_CUDA_OK(launch_pdl(linear_f32_pair_kernel, dim3((unsigned)grid), dim3(C::THREADS), C::SMEM, st, mw, mx, p, e, (long long)m0, (int)n0,
                             flags, flags + 1 + slab));
    }
    rc = f32_fma_run(a, e, m0, rows, flags, pl.slab, st);  // what could not be split
    if (rc) return rc;
  }
  return TPX_OK;
}

}  // namespace tpx

extern "C" size_t tpx_linear_f32_scratch_bytes(int64_t M, int64_t N, int64_t K) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  return tpx::f32_pair_scratch_bytes(M, N, K);
}

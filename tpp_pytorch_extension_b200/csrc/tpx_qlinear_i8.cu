// int8 linear on the tcgen05 tensor cores, with the reference's own arithmetic, for any number of tokens.
//
// Replaces TppBlockedQInt8LinearW (src/csrc/fused_gemm.h:1075-1341): activations are quantised on the fly to int8 with
// one scale per (token, K block) (quantize_int8sym, :1249), every K block is an int8 x int8 -> int32 product
// (:1134-1137, :1197-1198) and the output accumulates tmp * s_x[token, block] * s_w[block, feature]
// (DequantTPP, :1200-1204). Here:
//   quantize_act_i8_*_kernel  x bf16 [M][K] -> int8 and scales as the GEMM's stages hold them (I8Act; padding tokens zero)
//   qlinear_i8_kernel<TOK, BS>   A = 128 weight rows (int8, TMA, 128-byte swizzle), B = TOK tokens, tcgen05.mma kind::i8,
//                            one int32 accumulator per K block in tensor memory (a ring of them); the four epilogue
//                            warps pull each finished block, scale it and add it to fp32 registers
// Difference to the reference, inside the parity tolerance: the running output is kept in fp32, where the reference
// rounds it to bf16 after every K block. Blocks of 64 and few tokens: tpx_qlinear_i8_rows.cu, the same arithmetic.
//
// Work split: one output tile (128 features x TOK tokens, TOK = 16, 32, 64 or, for more than 64 tokens, 128) per CTA;
// when tiles are few, a thread-block cluster per tile cuts K between its CTAs, which add their parts over distributed
// shared memory. (Sharing the k units of all tiles evenly between the CTAs, 86 tiles of 11008 features on 148 SMs, brought nothing
// up to 64 tokens: a CTA's chain of copy, MMA, drain is short enough, and putting cut tiles together costs what it saves.)
#include "tpx_qlinear_i8_rows.cuh"

namespace tpx {

constexpr int kI8MaxStages = 8;

struct I8Params {
  TcParams t;          // epilogue fields (bias, act, mul_in, res, res_scale, y, M, N, err, cluster)
  const float* swT;    // [K/B][Np] weight scales, feature-contiguous
  const uint8_t* xq;   // quantised activations (I8Act)
  int ksteps;          // k steps of 128 (K padded)
  int Np;              // features padded to 128
  int nblk;            // scale blocks of the real K (the k padding of the last step has none)
  int tilesN;          // feature tiles; CTA (or cluster) t works on feature tile t % tilesN, token tile t / tilesN
};

__device__ __forceinline__ void i8_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{ .reg .pred p; setp.ne.b32 p, %4, 0;\n"
      "  tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p; }" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ float i8_ld_shared(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float4 i8_ld_shared4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  return v;
}

// Blocks of 512 values: a warp per (token row of the padded tile, block), sixteen consecutive values per lane; scale = max|x| / 127 in
// double as the reference does (src/csrc/qtypes.cpp:153-197), q = clamp(rint(x / scale)). Bound by latency: with a thread per block, which
// went round its 512 values on its own, 16 tokens of 4096 values took 67.6 us with the linear, now 8.5.
constexpr int kQbWarps = 4;
__global__ void __launch_bounds__(kQbWarps * 32) quantize_act_i8_block512_kernel(const uint16_t* __restrict__ x, int M, int K, int rows, I8Act L,
                                                                                uint8_t* __restrict__ xq) {
  pdl_trigger();
  pdl_wait();
  const int nb = K / 512, lane = threadIdx.x & 31;
  const int64_t idx = (int64_t)blockIdx.x * kQbWarps + threadIdx.x / 32;
  if (idx >= (int64_t)rows * nb) return;
  const int tok = (int)(idx / nb), blk = (int)(idx % nb), k = blk * 512 + lane * 16;
  float f[16];
  float amax = 0.0f;
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const uint4 v = tok < M ? reinterpret_cast<const uint4*>(x + (size_t)tok * K + k)[h] : make_uint4(0, 0, 0, 0);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      f[8 * h + 2 * j] = bf16_bits_to_f32((uint16_t)(w[j] & 0xffff));
      f[8 * h + 2 * j + 1] = bf16_bits_to_f32((uint16_t)(w[j] >> 16));
    }
  }
#pragma unroll
  for (int i = 0; i < 16; i++) amax = fmaxf(amax, fabsf(f[i]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const float scale = (float)((double)amax / 127.0);
  const float iscale = scale != 0.0f ? 1.0f / scale : 0.0f;
  uint32_t o[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    uint32_t word = 0;
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const float r = fminf(fmaxf(nearbyintf(f[4 * q + e] * iscale), -127.0f), 127.0f);
      word |= ((uint32_t)(uint8_t)(int8_t)(int)r) << (8 * e);
    }
    o[q] = word;
  }
  *reinterpret_cast<uint4*>(L.value(xq, tok, k)) = make_uint4(o[0], o[1], o[2], o[3]);
  if (lane == 0) *L.scale(xq, tok, blk) = scale;
}

// The same quantisation for blocks of up to 256 values, optionally behind an RMSNorm of the row
// (y = bf16(x * rsqrt(mean(x^2) + eps) * gamma), llama_rms_norm of the reference, rows of up to 8192 values then): eight consecutive
// values per thread and vector, the B/8 threads of a block reduce its maximum with shuffles. With the norm a CTA has a whole row in
// VECS vectors per thread, without it a row is spread over gridDim.y CTAs: the kernel is latency, and one CTA that goes round
// over a row of 11008 values took 9 us.
constexpr int kQaThreads = 256;
template <int VECS, class LAYOUT>
__global__ void __launch_bounds__(kQaThreads) quantize_act_i8_row_kernel(const uint16_t* __restrict__ x, const void* __restrict__ gamma,
                                                                         int gamma_f32, float eps, int M, int K, LAYOUT L, uint8_t* __restrict__ xq) {
  __shared__ float red[kQaThreads / 32];
  pdl_trigger();
  pdl_wait();
  const int tok = blockIdx.x;
  const int nv = K / 8;
  const int lanes = L.B / 8;  // threads per scale block: 8, 16 or 32
  const bool live = tok < M;
  const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)tok * K);
  float f[VECS][8];
  float ss = 0.0f;
#pragma unroll
  for (int q = 0; q < VECS; q++) {
    const int i = threadIdx.x + (blockIdx.y * VECS + q) * kQaThreads;
    i8_unpack_bf16(live && i < nv ? xr[i] : make_uint4(0, 0, 0, 0), f[q]);
#pragma unroll
    for (int j = 0; j < 8; j += 2) ss += f[q][j] * f[q][j] + f[q][j + 1] * f[q][j + 1];
  }
  if (gamma) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int w = 0; w < kQaThreads / 32; w++) tot += red[w];
    const float inv = rsqrtf(tot / (float)K + eps);
#pragma unroll
    for (int q = 0; q < VECS; q++) {
      const int i = threadIdx.x + q * kQaThreads;
      if (i >= nv) continue;
      float g[8];
      i8_gamma(gamma, gamma_f32, i, g);
#pragma unroll
      for (int j = 0; j < 8; j++) f[q][j] = bf16_bits_to_f32(f32_to_bf16_bits(f[q][j] * inv * g[j]));
    }
  }
#pragma unroll
  for (int q = 0; q < VECS; q++) {
    const int i = threadIdx.x + (blockIdx.y * VECS + q) * kQaThreads;
    uint2 o2;
    const float scale = i8_quantize8(f[q], lanes, o2);
    if (i < nv) {
      *reinterpret_cast<uint2*>(L.value(xq, tok, i * 8)) = o2;
      if ((i % lanes) == 0) *L.scale(xq, tok, i / lanes) = live ? scale : 0.0f;
    }
  }
}

// Interchange tensors of remap_and_quantize_qint8 (q [N/16][K/B][B/4][16][4], scales [N/16][K/B][16]) -> plain int8
// weight [Np][Kp] (zero padding) and feature-contiguous scales [K/B][Np].
__global__ void repack_qint8_tc_kernel(const int8_t* __restrict__ q, const float* __restrict__ scales, int64_t N, int64_t K, int64_t B,
                                       int64_t Np, int64_t Kp, int8_t* __restrict__ wq, float* __restrict__ swT) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx < Np * (Kp / 4)) {
    const int64_t n = idx / (Kp / 4), k = (idx % (Kp / 4)) * 4;
    uint32_t w = 0;
    if (n < N && k < K) w = *reinterpret_cast<const uint32_t*>(q + ((((n / 16) * (K / B) + k / B) * (B / 4) + (k % B) / 4) * 16 + (n % 16)) * 4);
    *reinterpret_cast<uint32_t*>(wq + n * Kp + k) = w;
  }
  const int64_t nb = K / B;
  if (idx < nb * Np) {
    const int64_t blk = idx / Np, n = idx % Np;
    swT[idx] = n < N ? scales[((n / 16) * nb + blk) * 16 + (n % 16)] : 0.0f;
  }
}

// BS: k32 steps per scale block (block / 32)
template <int TOK, int BS>
struct I8Cfg {
  static constexpr int A_BYTES = 128 * 128;   // 128 features x 128 k values
  static constexpr int B_BYTES = TOK * 128;   // TOK tokens x 128 k values
  // Scales of the blocks of a step travel with it: read from global memory group by group they cost the epilogue a memory
  // latency per 256 k values.
  static constexpr int ROWS = BS == 2 ? 2 : 1;  // scale rows per step (a block that spans several steps: its row with each of them)
  static constexpr int SX_BYTES = ROWS * TOK * 4, SW_BYTES = ROWS * 128 * 4;  // behind the activations, in this order
  static constexpr int STAGE_BYTES = (A_BYTES + B_BYTES + SW_BYTES + SX_BYTES + 1023) / 1024 * 1024;
  static constexpr int STAGES_FIT = (227 * 1024 - 3072) / STAGE_BYTES;   // as many stages as shared memory holds: the bytes in
  static constexpr int STAGES = STAGES_FIT > kI8MaxStages ? kI8MaxStages : STAGES_FIT;  // flight bound the stream, not the MMAs
  static constexpr int GROUP = TOK >= 128 ? 2 : 4;  // accumulators per group
  static constexpr int NBUF = 512 / TOK > 16 ? 16 : 512 / TOK;  // int32 accumulators (one per K block) in tensor memory
  static constexpr int NGRP = NBUF / GROUP;
  // K blocks that are handed to the epilogue per barrier round trip: 256 k values, or one larger block; their k steps
  static constexpr int GS = BS >= 8 ? 1 : (8 / BS < GROUP ? 8 / BS : GROUP);
  static constexpr int SG = GS * BS / 4;
  static constexpr int ALIGN = BS > 4 ? BS / 4 : 1;  // k steps per scale block when a block spans several
  // Draining a K block (tensor memory -> int32 -> * s_x * s_w -> fp32 sum) is a chain of dependent scalar instructions;
  // with one warp per 32-row quarter it, not the MMAs, bounds the kernel as soon as there are many tokens. Every quarter
  // has EPI_SPLIT warps, each owning TW = TOK / EPI_SPLIT tokens (columns) of the tile.
  static constexpr int EPI_SPLIT = TOK >= 64 ? 4 : TOK / 16;
  static constexpr int TW = TOK / EPI_SPLIT;
  static constexpr int THREADS = 64 + 128 * EPI_SPLIT;
  static constexpr int TMEM_COLS = NBUF * TOK < 32 ? 32 : NBUF * TOK;
  static constexpr size_t SMEM = (size_t)STAGES * STAGE_BYTES + 1024;
  static_assert(NBUF * TOK <= 512, "tensor memory");
  static_assert(SG >= 1 && SG <= STAGES, "a group's stages are held until it is drained");
  static_assert(128 * TOK * 4 <= STAGES * STAGE_BYTES, "the partial tile of a cluster member fits in the stages");
};

// One warp copies and one issues MMAs, for tens of steps of a few hundred cycles: everything in their loops that depends on the
// block size is a constant, loop state is the same in all lanes, and only the issue itself is under an elected lane. (With the
// bookkeeping of blocks and groups per MMA in one thread, the empty loops alone took 0.35 us per step.) 11008 x 4096, block 64, with the
// quantisation of x, before and after this form: 1 token 27.4 / 16.3 us, 32: 30.1 / 18.8, 64: 38.0 / 26.3, 128: 81 / 43. What is left is a
// chain per 256 k values (copies, eight MMAs, drain) that no single part of sets the pace: leaving one out takes 1 to 2 us off.
template <int TOK, int BS>
__global__ void __launch_bounds__(I8Cfg<TOK, BS>::THREADS, 1)
qlinear_i8_kernel(const __grid_constant__ CUtensorMap tmW, I8Params p) {
  using C = I8Cfg<TOK, BS>;
  extern __shared__ unsigned char i8_smem_raw[];
  __shared__ __align__(8) unsigned long long bar_full[C::STAGES], bar_empty[C::STAGES];
  __shared__ __align__(8) unsigned long long d_full[C::NGRP], d_free[C::NGRP];
  __shared__ uint32_t tmem_holder;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_base = (tc_smem_u32(i8_smem_raw) + 1023u) & ~1023u;
  const int csize = p.t.cluster;
  const int crank = csize > 1 ? (int)tc_cluster_rank() : 0;
  const int tile = (int)(blockIdx.x / csize) % p.tilesN;  // feature tile
  const int tm = (int)(blockIdx.x / csize) / p.tilesN;    // token tile
  // K range of this CTA in k steps, whole scale blocks
  const int groups = p.ksteps / C::ALIGN;
  const int ks0 = (int)((long long)crank * groups / csize) * C::ALIGN, ks1 = (int)((long long)(crank + 1) * groups / csize) * C::ALIGN;
  const int nsteps = ks1 - ks0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; s++) {
      tc_mbar_init(tc_smem_u32(&bar_full[s]), 1);
      tc_mbar_init(tc_smem_u32(&bar_empty[s]), 4 * C::EPI_SPLIT);
    }
    for (int b = 0; b < C::NGRP; b++) {
      tc_mbar_init(tc_smem_u32(&d_full[b]), 1);
      tc_mbar_init(tc_smem_u32(&d_free[b]), 4 * C::EPI_SPLIT);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem_u32(&tmem_holder)),
                 "r"((uint32_t)C::TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_holder;
  pdl_trigger();

  constexpr int TW = C::TW;
  if (warp == 0) {
    // ------------------------------------------------------------ producer
    constexpr uint32_t kScales = C::A_BYTES + C::B_BYTES + C::SX_BYTES;
    auto first_row = [](int ks) { return BS == 2 ? 2 * ks : ks / C::ALIGN; };
    auto rows = [&](int ks) { return min(C::ROWS, max(0, p.nblk - first_row(ks))); };  // the k padding of the last step has no scales
    auto fetch_w = [&](int s, int ks) {
      if (tc_elect()) {
        const uint32_t st = smem_base + (uint32_t)s * C::STAGE_BYTES, bar = tc_smem_u32(&bar_full[s]);
        const int n = rows(ks);
        tc_mbar_expect_tx(bar, kScales + n * 512);
        tc_tma_2d(st, &tmW, ks * 128, tile * 128, bar);
        const float* src = p.swT + (size_t)first_row(ks) * p.Np + tile * 128;
#pragma unroll
        for (int r = 0; r < C::ROWS; r++)
          if (r < n) tc_bulk_g2s(st + kScales + r * 512, src + (size_t)r * p.Np, 512, bar);
      }
      __syncwarp();
    };
    const int early = nsteps < C::STAGES ? nsteps : C::STAGES;
    for (int it = 0; it < early; it++) fetch_w(it, ks0 + it);  // weights do not depend on the quantisation kernel
    pdl_wait();
    int s = 0;
    uint32_t phase = 1;  // parity to wait for on bar_empty: the first round over the ring finds every stage free
    for (int it = 0; it < nsteps; it++) {
      if (it >= C::STAGES) {
        if (!tc_wait_warp(tc_smem_u32(&bar_empty[s]), phase)) {
          if (tc_elect()) atomicExch(p.t.err, 2u);
          break;
        }
        fetch_w(s, ks0 + it);
      }
      if (tc_elect()) {
        const uint32_t st = smem_base + (uint32_t)s * C::STAGE_BYTES, bar = tc_smem_u32(&bar_full[s]);
        tc_bulk_g2s(st + C::A_BYTES, p.xq + ((size_t)tm * p.ksteps + ks0 + it) * (C::B_BYTES + C::SX_BYTES), C::B_BYTES + C::SX_BYTES, bar);
      }
      __syncwarp();
      if (++s == C::STAGES) s = 0, phase ^= 1u;
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    // kind::i8: D = S32 (2), A = B = S8 (1), both K-major, N = TOK, M = 128
    constexpr uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TOK >> 3) << 17) | ((128u >> 4) << 24);
    constexpr bool HALF = I8Act64::serves(TOK, BS * 32);  // the B operand has a block's rows of 64 bytes
    const uint64_t desc0 = tc_smem_desc(smem_base), bdesc0 = HALF ? tc_smem_desc64(smem_base + C::A_BYTES) : tc_smem_desc(smem_base + C::A_BYTES);
    int s = 0, g = 0;  // g: groups handed out
    uint32_t phase = 0;
    bool dead = false;
    for (int left = nsteps; !dead && left > 0; left -= C::SG, g++) {
      const int grp = g % C::NGRP;
      if (g >= C::NGRP) {  // a recycled group: the epilogue must have read it
        if (!tc_wait_warp(tc_smem_u32(&d_free[grp]), (uint32_t)((g / C::NGRP - 1) & 1))) {
          if (tc_elect()) atomicExch(p.t.err, 3u);
          dead = true;
          break;
        }
        tc_fence_after();
      }
      const uint32_t d = tmem + grp * (C::GROUP * TOK);
#pragma unroll
      for (int t = 0; t < C::SG; t++) {
        if (t >= left || dead) continue;
        if (!tc_wait_warp(tc_smem_u32(&bar_full[s]), phase)) {
          if (tc_elect()) atomicExch(p.t.err, 4u);
          dead = true;
          continue;
        }
        tc_fence_after();
        if (tc_elect()) {
          const uint64_t at = (uint64_t)(s * (C::STAGE_BYTES >> 4));  // descriptors count 16-byte units
#pragma unroll
          for (int j = 0; j < 4; j++)
            i8_mma(d + (4 * t + j) / BS * TOK, desc0 + at + (uint64_t)(2 * j), bdesc0 + at + (uint64_t)(HALF ? (j >> 1) * TOK * 4 + 2 * (j & 1) : 2 * j), idesc,
                   (4 * t + j) % BS ? 1u : 0u);
        }
        __syncwarp();
        if (++s == C::STAGES) s = 0, phase ^= 1u;
      }
      // the epilogue also frees the stages that the group read, once it has used their scales
      if (!dead && tc_elect()) tc_commit(tc_smem_u32(&d_full[grp]));
      __syncwarp();
    }
  } else {
    // ------------------------------------------------------------ epilogue: thread = feature row of the tile
    const int sub = warp & 3;
    const uint32_t lane_base = ((uint32_t)(sub * 32)) << 16;
    const int row = sub * 32 + lane;
    const int cpart = (warp - 2) >> 2;  // this warp's tokens: [cpart * TW, +TW) of the tile
    pdl_wait();
    // The conversion instruction runs at a quarter of the rate of an addition. Sums of at most 256 products stay below 2^22: added to
    // the bits of 1.5 * 2^23 they are that float's low bits, exact either way.
    auto to_float = [](uint32_t d) { return BS <= 8 ? __uint_as_float(d + 0x4B400000u) - 12582912.0f : (float)(int)d; };
    int s = 0, g = 0;
    uint32_t phase = 0;
    bool dead = false;  // a warp that gave up still meets the others at their barriers
    const int n = tile * 128 + row;
    float acc[TW];  // this thread's tokens of its feature row
#pragma unroll
    for (int i = 0; i < TW; i++) acc[i] = 0.0f;
    int blk = BS == 2 ? 2 * ks0 : ks0 / C::ALIGN;
    for (int left = nsteps; left > 0 && !dead; left -= C::SG, g++, blk += C::GS) {
      const int grp = g % C::NGRP;
      const int steps = left < C::SG ? left : C::SG, cnt = BS == 2 ? 2 * steps : steps / C::ALIGN;
      uint32_t at[C::SG];  // the steps' stages: their scales were copied there
      const int s_first = s;
      bool ok = true;
#pragma unroll
      for (int t = 0; t < C::SG; t++) {
        at[t] = smem_base + (uint32_t)s * C::STAGE_BYTES + C::A_BYTES + C::B_BYTES;
        if (t >= steps) continue;
        ok = ok && tc_wait(tc_smem_u32(&bar_full[s]), phase);
        if (++s == C::STAGES) s = 0, phase ^= 1u;
      }
      if (!__all_sync(0xffffffffu, ok && tc_wait(tc_smem_u32(&d_full[grp]), (uint32_t)((g / C::NGRP) & 1)))) {
        if (lane == 0) atomicExch(p.t.err, 6u);
        dead = true;
        break;
      }
      tc_fence_after();
      constexpr int BATCH = C::EPI_SPLIT <= 2 ? C::GS : 1;  // blocks per round trip to tensor memory
#pragma unroll
      for (int q0 = 0; q0 < C::GS; q0 += BATCH) {
#pragma unroll
        for (int c0 = 0; c0 < TW; c0 += 16) {
          uint32_t d[BATCH][16];
#pragma unroll
          for (int q = 0; q < BATCH; q++)
            if (q0 + q < cnt) tc_ld_x16(tmem + lane_base + (grp * C::GROUP + q0 + q) * TOK + cpart * TW + c0, d[q]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int q = 0; q < BATCH; q++) {
            if (q0 + q >= cnt || blk + q0 + q >= p.nblk) continue;  // (a block of pure k padding has no scales)
            const uint32_t sc = at[((q0 + q + 1) * BS - 1) / 4];  // the block's last step
            const int r = BS == 2 ? (q0 + q) & 1 : 0;
            const float sw = i8_ld_shared(sc + C::SX_BYTES + r * 512 + row * 4);
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
              const float4 sx = i8_ld_shared4(sc + (r * TOK + cpart * TW + c0 + i) * 4);
              acc[c0 + i] += to_float(d[q][i]) * sx.x * sw;
              acc[c0 + i + 1] += to_float(d[q][i + 1]) * sx.y * sw;
              acc[c0 + i + 2] += to_float(d[q][i + 2]) * sx.z * sw;
              acc[c0 + i + 3] += to_float(d[q][i + 3]) * sx.w * sw;
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        tc_mbar_arrive(tc_smem_u32(&d_free[grp]));
#pragma unroll
        for (int t = 0; t < C::SG; t++)
          if (t < steps) tc_mbar_arrive(tc_smem_u32(&bar_empty[s_first + t < C::STAGES ? s_first + t : s_first + t - C::STAGES]));
      }
    }
    if (csize > 1) {
      asm volatile("bar.sync 1, %0;" ::"n"(C::THREADS - 64) : "memory");  // nobody still reads scales from the stages
      const uint32_t sp = smem_base + (uint32_t)((row * TOK + cpart * TW) * 4);
#pragma unroll
      for (int c0 = 0; c0 < TW; c0 += 4) tc_st_shared_f4(sp + c0 * 4, make_float4(acc[c0], acc[c0 + 1], acc[c0 + 2], acc[c0 + 3]));
    } else if (!dead) {
#pragma unroll
      for (int c0 = 0; c0 < TW; c0 += 16) {
        float v[16], v2[16];
#pragma unroll
        for (int i = 0; i < 16; i++) { v[i] = acc[c0 + i]; v2[i] = 0.0f; }
        const int tok0 = tm * TOK + cpart * TW + c0;
        if (n < p.t.N && tok0 < p.t.M) tc_finish16<false>(p.t, tok0, n, v, v2);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (csize > 1) {
    // every member's partial tile is in its own shared memory; 16-token chunks go round the members, each adds the
    // parts in rank order over distributed shared memory and finishes its chunks. Nobody leaves before all have read.
    tc_cluster_sync();
    if (warp >= 2 && warp < 6) {
      const int row = (warp & 3) * 32 + lane;
      const int n = tile * 128 + row;
#pragma unroll 1
      for (int c0 = crank * 16; c0 < TOK; c0 += 16 * csize) {
        float v[16], v2[16];
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = v2[i] = 0.0f;
        const uint32_t sp = smem_base + (uint32_t)((row * TOK + c0) * 4);
        tc_cluster_sum<4, 2>(sp, csize, v);
        if (n < p.t.N && tm * TOK + c0 < p.t.M) tc_finish16<false>(p.t, tm * TOK + c0, n, v, v2);
      }
    }
    tc_cluster_sync();
  }
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)C::TMEM_COLS) : "memory");
  }
}

// ---------------------------------------------------------------- host side
struct I8Plan {
  int tokp, ksteps, tiles, cluster, TM;  // tiles = feature tiles x token tiles
  int64_t Kp, Np, Mp;
  size_t off_xq, xq_bytes, total;
};

static I8Plan i8_plan(int64_t M, int64_t N, int64_t K, int64_t B) {
  I8Plan pl;
  pl.tokp = M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128;
  pl.TM = (int)((M + pl.tokp - 1) / pl.tokp);
  pl.Mp = (int64_t)pl.TM * pl.tokp;
  pl.Kp = (K + 127) / 128 * 128;
  pl.Np = (N + 127) / 128 * 128;
  pl.ksteps = (int)(pl.Kp / 128);
  pl.tiles = (int)(pl.Np / 128) * pl.TM;
  const int sms = sm_count();
  const int groups = (int)(B > 128 ? pl.ksteps / (B / 128) : pl.ksteps);  // units a cluster can cut K into
  int c = pl.tiles > 0 ? sms / pl.tiles : 1;
  if (c > 8) c = 8;
  if (c > groups) c = groups;
  pl.cluster = c < 1 ? 1 : c;
  size_t o = kTcCounterBytes;
  auto bump = [&](size_t bytes) { size_t r = o; o += (bytes + 1023) & ~(size_t)1023; return r; };
  pl.xq_bytes = (size_t)pl.TM * pl.ksteps * I8Act(pl.tokp, pl.ksteps, (int)B).bytes;
  pl.off_xq = bump(pl.xq_bytes);
  pl.total = o;
  return pl;
}

template <int TOK, int BS>
static int i8_launch(const CUtensorMap& w, I8Params p, int tiles, cudaStream_t st) {
  using C = I8Cfg<TOK, BS>;
  static bool opted[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16 || !opted[dev]) {
    TPX_CUDA_OK(cudaFuncSetAttribute(qlinear_i8_kernel<TOK, BS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM));
    if (dev >= 0 && dev < 16) opted[dev] = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(C::THREADS);
  cfg.dynamicSmemBytes = C::SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  // the largest cluster size, from the planned one down, of which one cluster per tile can be resident at once
  static int fits[16][9] = {};
  int c = p.t.cluster;
  for (; c >= 2; c--) {
    int& f = fits[(dev >= 0 && dev < 16) ? dev : 0][c];
    if (f == 0) {
      attr[1].val.clusterDim.x = (unsigned)c;
      cfg.gridDim = dim3((unsigned)(tiles * c));
      cfg.numAttrs = 2;
      int n = 0;
      cudaError_t e = cudaOccupancyMaxActiveClusters(&n, qlinear_i8_kernel<TOK, BS>, &cfg);
      if (e != cudaSuccess) { n = 0; (void)cudaGetLastError(); }
      f = 1 + n;
    }
    if (f - 1 >= tiles) break;
  }
  if (c < 2) c = 1;
  p.t.cluster = c;
  attr[1].val.clusterDim.x = (unsigned)c;
  cfg.gridDim = dim3((unsigned)(tiles * c));
  cfg.numAttrs = c > 1 ? 2 : 1;
  count_launch();
  TPX_CUDA_OK(cudaLaunchKernelEx(&cfg, qlinear_i8_kernel<TOK, BS>, w, p));
  return TPX_OK;
}

template <int BS>
static int i8_launch_tok(int tokp, const CUtensorMap& w, const I8Params& p, int tiles, cudaStream_t st) {
  switch (tokp) {
    case 16: return i8_launch<16, BS>(w, p, tiles, st);
    case 32: return i8_launch<32, BS>(w, p, tiles, st);
    case 64: return i8_launch<64, BS>(w, p, tiles, st);
    default: return i8_launch<128, BS>(w, p, tiles, st);
  }
}

static int make_map_u8(CUtensorMap* m, const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_rows) {
  typedef CUresult (*Fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                         const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static Fn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &ptr, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<Fn>(ptr);
  }
  TPX_REQUIRE(fn, TPX_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t gdim[2] = {row_bytes, rows};
  cuuint64_t gstr[1] = {row_bytes};
  cuuint32_t box[2] = {128, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  TPX_REQUIRE(r == CUDA_SUCCESS, TPX_ERR_CUDA, "cuTensorMapEncodeTiled failed with %d (rows=%llu row_bytes=%llu box_rows=%u)", (int)r,
              (unsigned long long)rows, (unsigned long long)row_bytes, box_rows);
  return TPX_OK;
}

}  // namespace tpx

using namespace tpx;

extern "C" int tpx_tc_packed_bytes_qint8(int64_t N, int64_t K, int64_t block_size, size_t* wq_bytes, size_t* sw_bytes) {
  TPX_REQUIRE(N > 0 && K > 0 && N % 16 == 0 && block_size % 64 == 0 && K % block_size == 0, TPX_ERR_ARG,
              "tc_packed_bytes_qint8: needs N %% 16 == 0 and a block size that is a multiple of 64 dividing K");
  const int64_t Np = (N + 127) / 128 * 128, Kp = (K + 127) / 128 * 128;
  if (wq_bytes) *wq_bytes = (size_t)Np * Kp;
  if (sw_bytes) *sw_bytes = (size_t)(K / block_size) * Np * sizeof(float);
  return TPX_OK;
}

extern "C" int tpx_repack_qint8_tc(const int8_t* q, const float* scales, int64_t N, int64_t K, int64_t block_size, int8_t* wq, float* swT,
                                   void* stream) {
  TPX_REQUIRE(q && scales && wq && swT, TPX_ERR_ARG, "repack_qint8_tc: null pointer");
  TPX_REQUIRE(N % 16 == 0 && block_size % 64 == 0 && K % block_size == 0, TPX_ERR_ARG,
              "repack_qint8_tc: needs N %% 16 == 0 and a block size that is a multiple of 64 dividing K");
  const int64_t Np = (N + 127) / 128 * 128, Kp = (K + 127) / 128 * 128;
  const int64_t total = Np * (Kp / 4) > (K / block_size) * Np ? Np * (Kp / 4) : (K / block_size) * Np;
  repack_qint8_tc_kernel<<<(unsigned)((total + 255) / 256), 256, 0, (cudaStream_t)stream>>>(q, scales, N, K, block_size, Np, Kp, wq, swT);
  TPX_LAUNCH_OK();
  return TPX_OK;
}

extern "C" size_t tpx_qlinear_qint8_tc_scratch_bytes(int64_t M, int64_t N, int64_t K, int64_t block_size) {
  if (M <= 0 || N <= 0 || K <= 0 || block_size <= 0) return 0;
  return i8_plan(M, N, K, block_size).total;
}

namespace tpx {
// The activations of a call as its GEMM reads them.
template <class LAYOUT>
static int i8_quantize(const uint16_t* x, const void* gamma, int gamma_is_f32, float eps, int M, int Mp, int64_t K, const LAYOUT& L, uint8_t* xq,
                       cudaStream_t st) {
  if (gamma) {
    TPX_CUDA_OK(launch_pdl(quantize_act_i8_row_kernel<4, LAYOUT>, dim3((unsigned)Mp), dim3(kQaThreads), 0, st, x, gamma, gamma_is_f32, eps, M, (int)K, L, xq));
  } else {
    TPX_CUDA_OK(launch_pdl(quantize_act_i8_row_kernel<1, LAYOUT>, dim3((unsigned)Mp, (unsigned)((K / 8 + kQaThreads - 1) / kQaThreads)), dim3(kQaThreads), 0,
                           st, x, gamma, gamma_is_f32, eps, M, (int)K, L, xq));
  }
  return TPX_OK;
}
}  // namespace tpx

// One linear, or with wq2 the pair act(x wq^T) * (x wq2^T): in one kernel for few tokens, else as two linears, the second multiplying by
// what the first left in y.
static int i8_linear(const int8_t* wq, const float* swT, const int8_t* wq2, const float* swT2, const uint16_t* x, const void* gamma, int gamma_is_f32,
                     float eps, int64_t M, int64_t N, int64_t K, int64_t block_size, int reuse_act, const uint16_t* bias, int act,
                     const uint16_t* mul_in, const uint16_t* res, float res_scale, uint16_t* y, void* scratch, size_t scratch_bytes, void* stream) {
  TPX_REQUIRE(M >= 0 && N > 0 && K > 0, TPX_ERR_ARG, "qlinear_qint8_tc: bad shape");
  if (M == 0) return TPX_OK;
  TPX_REQUIRE(M <= (1 << 20), TPX_ERR_UNSUPPORTED, "qlinear_qint8_tc: at most 2^20 tokens per call (M=%ld)", (long)M);
  TPX_REQUIRE(wq && swT && x && y, TPX_ERR_ARG, "qlinear_qint8_tc: null pointer");
  TPX_REQUIRE(block_size == 64 || block_size == 128 || block_size == 256 || block_size == 512, TPX_ERR_UNSUPPORTED,
              "qlinear_qint8_tc: block size %ld not supported (64, 128, 256, 512)", (long)block_size);
  TPX_REQUIRE(N % 16 == 0 && K % block_size == 0, TPX_ERR_ARG, "qlinear_qint8_tc: needs N %% 16 == 0 and K %% block_size == 0");
  TPX_REQUIRE(act >= TPX_ACT_NONE && act <= TPX_ACT_RELU, TPX_ERR_ARG, "qlinear_qint8_tc: unknown activation %d", act);
  TPX_REQUIRE((((uintptr_t)wq | (uintptr_t)wq2 | (uintptr_t)x | (uintptr_t)swT | (uintptr_t)swT2) & 15) == 0 && ((uintptr_t)scratch & 255) == 0,
              TPX_ERR_ARG, "qlinear_qint8_tc: misaligned pointer");
  I8Plan pl = i8_plan(M, N, K, block_size);
  TPX_REQUIRE(pl.Kp % block_size == 0, TPX_ERR_UNSUPPORTED, "qlinear_qint8_tc: K rounded up to 128 must stay a multiple of the block size");
  TPX_REQUIRE(scratch && scratch_bytes >= pl.total, TPX_ERR_SCRATCH, "qlinear_qint8_tc: scratch of %zu bytes needed, %zu given", pl.total,
              scratch_bytes);
  TPX_REQUIRE(!gamma || (K <= 8192 && block_size <= 256 && ((uintptr_t)gamma & 15) == 0), TPX_ERR_UNSUPPORTED,
              "qlinear_qint8_tc: the fused RMSNorm takes rows of up to 8192 values, blocks of up to 256 and a 16-byte aligned gamma");
  if (wq2 && !i8_rows_serves(M, N, K, block_size, true)) {
    int rc = i8_linear(wq, swT, nullptr, nullptr, x, gamma, gamma_is_f32, eps, M, N, K, block_size, reuse_act, bias, act, nullptr, nullptr, 1.0f, y,
                       scratch, scratch_bytes, stream);
    if (rc) return rc;
    return i8_linear(wq2, swT2, nullptr, nullptr, x, gamma, gamma_is_f32, eps, M, N, K, block_size, 1, nullptr, TPX_ACT_NONE, y, res, res_scale, y,
                     scratch, scratch_bytes, stream);
  }
  cudaStream_t st = (cudaStream_t)stream;
  unsigned char* sc = reinterpret_cast<unsigned char*>(scratch);
  uint8_t* xq = sc + pl.off_xq;
  TcParams t = {};
  t.bias = bias; t.mul_in = mul_in; t.res = res; t.res_scale = res_scale; t.y = y; t.act = act;
  t.M = (int)M; t.N = (int)N; t.K = (int)K; t.cluster = pl.cluster;
  t.err = reinterpret_cast<unsigned*>(sc + kTcCounterBytes - 4);
  const bool rows = i8_rows_serves(M, N, K, block_size, wq2 != nullptr);
  I8RowsParams r = {};
  // The order of the quantised activations depends on M, K and block_size alone, so that a call that reuses them may be of another N, and another kernel's.
  const I8Act L(pl.tokp, pl.ksteps, (int)block_size);
  if (!reuse_act && rows && i8_rows_quantizes(x, y, M, N, K)) {
    r.x = x; r.gamma = gamma; r.gamma_f32 = gamma_is_f32; r.eps = eps;
  } else if (!reuse_act && block_size <= 256) {
    if (!rows && pl.Kp != K) TPX_CUDA_OK(cudaMemsetAsync(xq, 0, pl.xq_bytes, st));  // the k padding reads as zero, as the weight's
    int rc = I8Act64::serves(pl.tokp, (int)block_size)
                 ? i8_quantize(x, gamma, gamma_is_f32, eps, (int)M, rows ? (int)M : pl.tokp, K, I8Act64{(uint32_t)pl.tokp}, xq, st)
                 : i8_quantize(x, gamma, gamma_is_f32, eps, (int)M, (int)pl.Mp, K, L, xq, st);
    if (rc) return rc;
  } else if (!reuse_act) {
    const long long warps = (long long)pl.Mp * (K / 512);
    TPX_CUDA_OK(launch_pdl(quantize_act_i8_block512_kernel, dim3((unsigned)((warps + kQbWarps - 1) / kQbWarps)), dim3(kQbWarps * 32), 0, st, x, (int)M, (int)K,
                           (int)pl.Mp, L, xq));
  }
  if (rows) {
    r.t = t;
    r.w[0] = wq; r.w[1] = wq2; r.swT[0] = swT; r.swT[1] = swT2; r.xq = xq;
    r.nkb = (int)(K / 64); r.Kp = (int)pl.Kp; r.Np = (int)pl.Np; r.tiles = (int)(N / 16);
    return i8_rows_launch(r, wq2 != nullptr, st);
  }
  CUtensorMap mw;
  int rc = make_map_u8(&mw, wq, (uint64_t)pl.Np, (uint64_t)pl.Kp, 128);
  if (rc) return rc;
  I8Params p = {};
  p.t = t;
  p.swT = swT; p.xq = xq; p.ksteps = pl.ksteps; p.Np = (int)pl.Np; p.nblk = (int)(K / block_size);
  p.tilesN = (int)(pl.Np / 128);
  switch (block_size) {
    case 64: return i8_launch_tok<2>(pl.tokp, mw, p, pl.tiles, st);
    case 128: return i8_launch_tok<4>(pl.tokp, mw, p, pl.tiles, st);
    case 256: return i8_launch_tok<8>(pl.tokp, mw, p, pl.tiles, st);
    default: return i8_launch_tok<16>(pl.tokp, mw, p, pl.tiles, st);
  }
}

extern "C" int tpx_qlinear_qint8_tc(const int8_t* wq, const float* swT, const uint16_t* x, const void* gamma, int gamma_is_f32, float eps,
                                    int64_t M, int64_t N, int64_t K, int64_t block_size, int reuse_act, const uint16_t* bias, int act, const uint16_t* mul_in,
                                    const uint16_t* res, float res_scale, uint16_t* y, void* scratch, size_t scratch_bytes, void* stream) {
  return i8_linear(wq, swT, nullptr, nullptr, x, gamma, gamma_is_f32, eps, M, N, K, block_size, reuse_act, bias, act, mul_in, res, res_scale, y,
                   scratch, scratch_bytes, stream);
}

extern "C" int tpx_qlinear_qint8_pair_tc(const int8_t* wq, const float* swT, const int8_t* wq2, const float* swT2, const uint16_t* x, const void* gamma,
                                         int gamma_is_f32, float eps, int64_t M, int64_t N, int64_t K, int64_t block_size, int act, uint16_t* y,
                                         void* scratch, size_t scratch_bytes, void* stream) {
  TPX_REQUIRE(M == 0 || (wq2 && swT2), TPX_ERR_ARG, "qlinear_qint8_pair_tc: null pointer");
  return i8_linear(wq, swT, wq2, swT2, x, gamma, gamma_is_f32, eps, M, N, K, block_size, 0, nullptr, act, nullptr, nullptr, 1.0f, y, scratch,
                   scratch_bytes, stream);
}


// ---------------------------------------------------------------- int8 weight -> bf16 matrix (many tokens)
// With many tokens the per-K-block drain of the int8 kernel (one pass over the accumulator per 64 to 512 k) costs more
// than the MMAs it serves (253 TOP/s at block 64), while the bf16 tensor-core kernel runs the same shapes at 1000-1170
// TFLOP/s: for more than 128 tokens the host unpacks the weight to bf16 (w = q * s, rounded once) into a transient
// buffer and runs tpx_linear_bf16_tc on it, i.e. weight-only arithmetic with bf16 activations (the reference's QINT8_EMU
// mode, src/csrc/qtypes.cpp:27, :928-930). One thread per 16 consecutive k of one output row.
namespace tpx {
__global__ void unpack_qint8_bf16_kernel(const int8_t* __restrict__ wq, const float* __restrict__ swT, long long N, long long K, long long Kp,
                                         long long Np, int block, uint16_t* __restrict__ out) {
  pdl_trigger();
  pdl_wait();
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long per_row = K / 16;
  if (idx >= N * per_row) return;
  const long long n = idx / per_row, k = (idx % per_row) * 16;
  const uint4 q = *reinterpret_cast<const uint4*>(wq + n * Kp + k);
  const float s = swT[(k / block) * Np + n];  // block sizes are multiples of 16: one scale for the sixteen values
  const uint32_t w[4] = {q.x, q.y, q.z, q.w};
  uint32_t o[8];
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const int a = (int)(int8_t)((w[j >> 1] >> (16 * (j & 1))) & 0xff), b = (int)(int8_t)((w[j >> 1] >> (16 * (j & 1) + 8)) & 0xff);
    o[j] = (uint32_t)f32_to_bf16_bits((float)a * s) | ((uint32_t)f32_to_bf16_bits((float)b * s) << 16);
  }
  uint4* dst = reinterpret_cast<uint4*>(out + n * K + k);
  dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
  dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
}
}  // namespace tpx

extern "C" int tpx_unpack_qint8_tc_bf16(const int8_t* wq, const float* swT, int64_t N, int64_t K, int64_t block_size, uint16_t* w_bf16,
                                        void* stream) {
  TPX_REQUIRE(wq && swT && w_bf16, TPX_ERR_ARG, "unpack_qint8_tc_bf16: null pointer");
  TPX_REQUIRE(N > 0 && K > 0 && K % 16 == 0 && block_size >= 16 && block_size % 16 == 0 && K % block_size == 0, TPX_ERR_ARG,
              "unpack_qint8_tc_bf16: bad shape (N=%ld K=%ld block=%ld)", (long)N, (long)K, (long)block_size);
  TPX_REQUIRE((((uintptr_t)wq | (uintptr_t)w_bf16) & 15) == 0, TPX_ERR_ARG, "unpack_qint8_tc_bf16: misaligned pointer");
  const long long Kp = (K + 127) / 128 * 128, Np = (N + 127) / 128 * 128;
  const long long total = N * (K / 16);
  TPX_CUDA_OK(tpx::launch_pdl(tpx::unpack_qint8_bf16_kernel, dim3((unsigned)((total + 255) / 256)), dim3(256), 0, (cudaStream_t)stream, wq, swT,
                              (long long)N, (long long)K, Kp, Np, (int)block_size, w_bf16));
  return TPX_OK;
}

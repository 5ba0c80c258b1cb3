// MXFP4 linear (and gate/up pair) of few tokens, optionally behind an RMSNorm: the weight through registers once, mma.sync beside the stream.
//
// The codes become fp16 pairs in registers (one instruction per two; every E2M1 value is an fp16 value), activations fp16 values too: a
// token's 128 values of a k step are multiplied by the power of two that brings the largest below 2^15. All 8 bits of a bf16 value fit in
// fp16 from there down to 2^-17, so that what is rounded is 2^-39 of the largest, less than fp32 sums lose. mma.sync in fp32 per block of 32 values, then
// times weight scale * activation factor (fp32, any scale byte).
//
// A CTA has T tiles of 16 features and all of K, its groups of warps take the k steps of 128 in turn (RowsSplit). The packed weight of the
// tensor-core kernels serves as it is: 16 rows of a k step are 1 KB in one piece. A warp copies its own pieces by cp.async into a ring of its own, the
// first before the wait for the previous kernel, 16-byte units swizzled by row so that the reads (a word per lane: 8 codes of its row and block)
// meet no bank twice.
//
// Bound by the instructions per weight byte (about 64 ALU ones per KB of codes, 32 of them the unpacking) and by what a launch in a chain costs at both ends: the
// tcgen05 kernels take activations as two E4M3 terms that a kernel in front has to make, and hold their weights unpacked, twice the shared memory
// per byte on the way. Chains of calls on one B200, tcgen05 / here: 1 token 4096 x 4096 8.4 / 4.7 us, 11008 x 4096 11.7 / 7.3, 4096 x 14336 13.1 / 10.1, pair of
// 14336 x 4096 behind a norm 17.6 / 15.9, of 11008 x 4096 20.3 / 12.7; 8 tokens 8.6 / 5.2, 12.0 / 8.6, 13.3 / 9.8, 17.7 / 16.3, 21.6 / 12.8.
#include "tpx_qlinear_mx_rows.cuh"
#include "tpx_rows.cuh"

namespace tpx {

// Slots of a warp's ring where a k step has no more tiles (whole k steps of them: 50 to 120 KB per SM). More of them hold the next kernel's weights, but the activations, asked for
// when the kernel before ends, queue behind them: a generation with 1 prompt on the Llama-3 shape took 24.4 ms with nine slots and 20.4 with five.
constexpr int kMrSlots = 5;
constexpr int kMrTiles16 = 5;  // tiles per CTA up to which more than 8 tokens are served
constexpr int kMrSlot = 1088;  // 16 features x 128 codes, then 16 words of 4 scale bytes

// Who turns bf16 activations into fp16 ones. kMrStage: every CTA all of them, first, into its shared memory. kMrNorm: that behind an RMSNorm. kMrReady:
// a kernel in front, mx_rows_prep_kernel.
enum { kMrStage, kMrNorm, kMrReady };

// MG: groups of 8 tokens; two of them need the registers of twelve warps
template <int T, int MG, int MODE>
struct MrCfg : RowsSplit<T, MG, MG == 2 ? 12 : 16, 8> {
  using S0 = RowsSplit<T, MG, MG == 2 ? 12 : 16, 8>;
  // D: k steps in the ring
  static constexpr int STAGED = MODE == kMrStage || MODE == kMrNorm, D = S0::N >= kMrSlots ? 1 : kMrSlots / S0::N;
  static constexpr int S = D * S0::N;
  static constexpr size_t RING = (size_t)S0::W * S * kMrSlot, SMEM = RING > S0::PARTS ? RING : S0::PARTS;
  static constexpr size_t ROOM = STAGED ? 32768 * 2 + 32768 / 128 * 4 : 0;  // staged activations and their factors
  static_assert(SMEM + ROOM <= 225 * 1024, "shared memory");
};

struct MxRowsParams {
  TcParams t;          // sfa, epilogue fields, M, N, K, cluster
  const uint8_t* wq;   // [tiles of 128][KS](pair: [2])[128][64]
  const uint16_t* x;   // [M][K]
  const uint8_t* xr;   // kMrReady: fp16 values [k step][block][Mp][32], then their factors [k step][Mp], Mp = 8 MG
  const void* gamma;   // RMSNorm of x, or null
  float eps;
  int gamma_f32, KS, steps, tiles;  // KS: k steps of the packed weight; steps: those that K reaches; tiles: N / 16
};

__device__ __forceinline__ void mr_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, float c0, float c1,
                                       float c2, float c3) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}
// eight codes -> four fp16 pairs, low nibble first
__device__ __forceinline__ void mr_unpack(uint32_t w, uint32_t (&h)[4]) {
  asm("{ .reg .b8 b0, b1, b2, b3; mov.b32 {b0, b1, b2, b3}, %4;\n"
      "  cvt.rn.f16x2.e2m1x2 %0, b0; cvt.rn.f16x2.e2m1x2 %1, b1; cvt.rn.f16x2.e2m1x2 %2, b2; cvt.rn.f16x2.e2m1x2 %3, b3; }"
      : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3])
      : "r"(w));
}
__device__ __forceinline__ uint32_t mr_lds(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ float2 mr_bf16x2(uint32_t v) { return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u)); }
__device__ __forceinline__ uint32_t mr_pack_bf16(float lo, float hi) {
  uint32_t v;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(v) : "f"(hi), "f"(lo));
  return v;
}
__device__ __forceinline__ uint32_t mr_pack_f16(float lo, float hi) {
  uint32_t v;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(v) : "f"(hi), "f"(lo));
  return v;
}

// exponent field of the power of two that brings `top` (the largest magnitude, bf16 bits) to 2^14 ... 2^15
__device__ __forceinline__ uint32_t mr_scale(uint32_t top) { return min(268u - (top >> 7), 253u); }
__device__ __forceinline__ float mr_unscale(uint32_t f) { return __uint_as_float((254u - f) << 23); }
// the larger magnitude of each half; the sign bit is of no use
__device__ __forceinline__ uint32_t mr_max(uint32_t a, uint32_t b) {
  uint32_t v;
  asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(v) : "r"(a), "r"(b));
  return v;
}
__device__ __forceinline__ uint32_t mr_top(uint32_t v) {
  v &= 0x7fff7fffu;
  return max(v >> 16, v & 0xffffu);
}
// bf16 pair -> fp16 pair times 2^(f - 127)
__device__ __forceinline__ uint32_t mr_to_f16(uint32_t v, uint32_t f) {
  uint32_t s;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(s) : "r"(v), "r"(f * 0x00800080u));
  const float2 w = mr_bf16x2(s);
  return mr_pack_f16(w.x, w.y);
}
// two scale bytes -> fp32 factors
__device__ __forceinline__ float2 mr_factors(uint16_t v) {
  uint32_t r;
  asm("cvt.rn.bf16x2.ue8m0x2 %0, %1;" : "=r"(r) : "h"(v));
  return mr_bf16x2(r);
}

// largest magnitude among the 128 values of sixteen lanes
__device__ __forceinline__ uint32_t mr_top16(uint4 v) {
  uint32_t top = mr_max(mr_max(v.x, v.y), mr_max(v.z, v.w));
#pragma unroll
  for (int o = 1; o < 16; o <<= 1) top = mr_max(top, __shfl_xor_sync(0xffffffffu, top, o));
  return mr_top(top);
}
__device__ __forceinline__ float mr_square(uint4 v) {
  const float2 a = mr_bf16x2(v.x), b = mr_bf16x2(v.y), c = mr_bf16x2(v.z), d = mr_bf16x2(v.w);
  return a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y + c.x * c.x + c.y * c.y + d.x * d.x + d.y * d.y;
}
__device__ __forceinline__ void mr_gamma(const void* gamma, int f32, int q, float (&gm)[8]) {  // weights of piece q
  if (f32) {
    const float4* s = reinterpret_cast<const float4*>(gamma) + q * 2;
    const float4 a = s[0], c = s[1];
    gm[0] = a.x; gm[1] = a.y; gm[2] = a.z; gm[3] = a.w; gm[4] = c.x; gm[5] = c.y; gm[6] = c.z; gm[7] = c.w;
  } else {
    const uint4 v = reinterpret_cast<const uint4*>(gamma)[q];
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const float2 f = mr_bf16x2(w[e]);
      gm[2 * e] = f.x;
      gm[2 * e + 1] = f.y;
    }
  }
}
__device__ __forceinline__ uint4 mr_normed(uint4 v, float inv, const float (&gm)[8]) {
  auto two = [&](uint32_t w, int e) {
    const float2 f = mr_bf16x2(w);
    return mr_pack_bf16(f.x * inv * gm[e], f.y * inv * gm[e + 1]);
  };
  return make_uint4(two(v.x, 0), two(v.y, 2), two(v.z, 4), two(v.w, 6));
}

// T: tiles of 16 features per CTA (of a pair: gate and up tiles in turn)
template <int T, int MG, bool DUAL, int MODE>
__global__ void __launch_bounds__(MrCfg<T, MG, MODE>::W * 32, 1) qlinear_mx_rows_kernel(MxRowsParams p) {
  using C = MrCfg<T, MG, MODE>;
  static_assert(MG == 1 || MODE == kMrReady, "more than 8 tokens");
  constexpr int KG = C::KG, N = C::N, D = C::D, S = C::S, TF = DUAL ? T / 2 : T, NW = DUAL ? 2 : 1;  // TF: feature tiles
  extern __shared__ __align__(16) unsigned char mr_smem[];
  __shared__ float norm_part[8][16], norm_inv[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int csize = p.t.cluster, crank = csize > 1 ? (int)tc_cluster_rank() : 0;
  // the last CTA starts early enough to have all its tiles, and stores those that are its own
  const int tile_own = (int)blockIdx.x / csize * TF, tile0 = min(tile_own, p.tiles - TF);
  const int first = warp / KG * N;  // this warp's first tile
  // its k steps: those that fall to its group when all groups of the cluster take turns
  const int groups = KG * csize, turn = crank * KG + warp % KG;
  const int cnt = p.steps > turn ? (p.steps - turn + groups - 1) / groups : 0;
  const uint32_t smem = tc_smem_u32(mr_smem), ring = smem + warp * (S * kMrSlot);
  // 16-byte unit `lane` of a piece is (row lane / 4, block lane % 4); units of a row are exchanged by (row / 2) % 4
  const uint32_t own = ring + ((lane & ~3) + ((lane & 3) ^ ((lane >> 3) & 3))) * 16;
  const uint32_t swz = (g >> 1) & 3, rd = ring + g * 64 + t * 4;
  // addresses: bases that are the same in the whole CTA, 32-bit offsets of this warp's feature tiles, and of its k step
  const uint8_t* const wbase = p.wq + (size_t)(tile0 >> 3) * p.KS * NW * 8192;
  const uint8_t* const sbase = p.t.sfa + (size_t)(tile0 >> 3) * p.KS * NW * 512;
  uint32_t woff[N], soff[N];
#pragma unroll
  for (int j = 0; j < N; j++) {
    const int f = tile0 + (DUAL ? (first + j) >> 1 : first + j), tile = ((f >> 3) - (tile0 >> 3)) * p.KS * NW + (DUAL ? (first + j) & 1 : 0);
    woff[j] = tile * 8192 + (f & 7) * 1024 + lane * 16;
    soff[j] = tile * 512 + (f & 1) * 256 + ((f & 7) >> 1) * 4 + lane * 16;
  }
  const uint32_t kstep = groups * NW;  // in pieces of 128 rows
  uint32_t k0 = turn * NW;
  pdl_trigger();

  // slot q of the ring, k step `ord` of this warp's, `td` steps behind the one that k0 points at
  auto issue = [&](int q, int td, int ord) {
    const int j = q % N;
    if (ord < cnt && (j < C::SURE || first + j < T)) {
      const uint32_t to = q % S * kMrSlot, k = k0 + td * kstep;
      const uint8_t* src = wbase + (woff[j] + k * 8192);
      rows_copy16(own + to, src);
      rows_copy16(own + to + 512, src + 512);
      if (lane < 16)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(ring + to + 1024 + lane * 4), "l"(sbase + (soff[j] + k * 512)) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int q = 0; q < S - 1; q++) issue(q, q / N, q / N);

  // kMrStage, kMrNorm: shared memory behind the ring, fp16 values [k step][block][token][32], then their factors [k step][token]
  const int M = p.t.M;
  const uint32_t xs = smem + (uint32_t)C::SMEM, fs = xs + p.steps * M * 256;
  // kMrReady: values and factors of block b of a k step
  uint32_t xh[MG][4][4];
  float2 sx[MG];  // factors of tokens 2t, 2t + 1
  constexpr int Mp = MG * 8;
  const uint8_t* const xf = p.xr + (size_t)p.steps * Mp * 256;
  auto ready = [&](int td, int b) {
    const uint32_t step = k0 / NW + td * groups;
#pragma unroll
    for (int m = 0; m < MG; m++) {
      const uint4 v = rows_ldg16(p.xr + (((step * 4 + b) * Mp + m * 8 + g) * 64 + t * 16));
      xh[m][b][0] = v.x, xh[m][b][1] = v.y, xh[m][b][2] = v.z, xh[m][b][3] = v.w;
    }
  };
  auto factors = [&](int td) {
    const uint32_t step = k0 / NW + td * groups;
#pragma unroll
    for (int m = 0; m < MG; m++) sx[m] = rows_ldg8(xf + ((step * Mp + m * 8 + 2 * t) * 4));
  };
  if constexpr (MODE == kMrReady) {
    pdl_wait();
    if (cnt > 0) {
#pragma unroll
      for (int b = 0; b < 4; b++) ready(0, b);
      factors(0);
    }
  } else {
    const int pieces = p.steps * 16;  // of 8 values, per token; sixteen threads have a k step
    auto at = [&](int q, int m) { return xs + (uint32_t)(((q >> 2) * M + m) * 64 + (q & 3) * 16); };
    auto load = [&](int q, int m) { return q * 8 < p.t.K ? rows_ldg16(p.x + (size_t)m * p.t.K + q * 8) : make_uint4(0, 0, 0, 0); };
    auto store = [&](uint32_t a, uint4 v) { asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory"); };
    auto convert = [&](int q, int m, uint4 v) {
      const uint32_t f = mr_scale(mr_top16(v));
      if (q >= pieces) return;
      store(at(q, m), make_uint4(mr_to_f16(v.x, f), mr_to_f16(v.y, f), mr_to_f16(v.z, f), mr_to_f16(v.w, f)));
      if ((q & 15) == 0) asm volatile("st.shared.f32 [%0], %1;" ::"r"(fs + (uint32_t)((q >> 4) * M + m) * 4), "f"(mr_unscale(f)) : "memory");
    };
    float gm[8], ss[8];
    if (MODE == kMrNorm)
      for (int q = threadIdx.x; q * 8 < p.t.K; q += C::W * 32) rows_prefetch_gamma(p.gamma, p.gamma_f32, q);
    pdl_wait();
#pragma unroll
    for (int m = 0; m < 8; m++) ss[m] = 0.0f;
    for (int q0 = 0; q0 < pieces; q0 += C::W * 32) {
      const int q = q0 + threadIdx.x;
      uint4 v[8];
#pragma unroll
      for (int m = 0; m < 8; m++)
        if (m < M) v[m] = load(q, m);
      if (MODE == kMrNorm && q0 == 0 && q * 8 < p.t.K) mr_gamma(p.gamma, p.gamma_f32, q, gm);
#pragma unroll
      for (int m = 0; m < 8; m++)
        if (m < M) {
          if (MODE == kMrStage) convert(q, m, v[m]);
          else if (q < pieces) store(at(q, m), v[m]), ss[m] += mr_square(v[m]);
        }
    }
    if constexpr (MODE == kMrNorm) {
#pragma unroll
      for (int m = 0; m < 8; m++)
        if (m < M) {
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) ss[m] += __shfl_xor_sync(0xffffffffu, ss[m], o);
          if (lane == 0) norm_part[m][warp] = ss[m];
        }
      __syncthreads();
      if (warp < M) {
        float tot = norm_part[warp][lane & 15];
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
        if (lane == 0) norm_inv[warp] = rsqrtf(tot / (float)p.t.K + p.eps);
      }
      __syncthreads();
      for (int q0 = 0; q0 < pieces; q0 += C::W * 32) {
        const int q = q0 + threadIdx.x;
        if (q0 > 0 && q * 8 < p.t.K) mr_gamma(p.gamma, p.gamma_f32, q, gm);
#pragma unroll
        for (int m = 0; m < 8; m++)
          if (m < M) {
            uint4 v = q < pieces ? rows_lds16(at(q, m)) : make_uint4(0, 0, 0, 0);
            if (q * 8 < p.t.K) v = mr_normed(v, norm_inv[m], gm);
            convert(q, m, v);
          }
      }
    }
    __syncthreads();
  }
  float2 acc[N][MG][2];  // [row g, row g + 8] of tokens 2t, 2t + 1
#pragma unroll
  for (int j = 0; j < N; j++)
#pragma unroll
    for (int m = 0; m < MG; m++) acc[j][m][0] = acc[j][m][1] = make_float2(0.0f, 0.0f);
  for (int i = 0; i < cnt; i += D) {
#pragma unroll
    for (int d = 0; d < D; d++) {
      if (i + d >= cnt) break;
      if constexpr (MODE != kMrReady) {  // columns behind the last token repeat it and are not stored
        const uint32_t step = k0 / NW + d * groups, xa = xs + (step * 4 * M + min(g, M - 1)) * 64 + t * 16, fa = fs + step * M * 4;
#pragma unroll
        for (int b = 0; b < 4; b++) {
          const uint4 v = rows_lds16(xa + b * M * 64);
          xh[0][b][0] = v.x, xh[0][b][1] = v.y, xh[0][b][2] = v.z, xh[0][b][3] = v.w;
        }
        sx[0] = make_float2(rows_lds4(fa + min(2 * t, M - 1) * 4), rows_lds4(fa + min(2 * t + 1, M - 1) * 4));
      }
#pragma unroll
      for (int j = 0; j < N; j++) {
        const int q = d * N + j;
        asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
        __syncwarp();  // other lanes copied parts of the slot; and all are done with the slot before, which is filled again
        uint32_t wa[4], wb[4];
#pragma unroll
        for (int b = 0; b < 4; b++) {
          wa[b] = mr_lds(rd + q * kMrSlot + ((b ^ swz) << 4));
          wb[b] = mr_lds(rd + q * kMrSlot + 512 + ((b ^ swz) << 4));
        }
        const uint32_t sa = mr_lds(ring + q * kMrSlot + 1024 + g * 4), sb = mr_lds(ring + q * kMrSlot + 1056 + g * 4);
        issue(q + S - 1, (q + S - 1) / N, i + (q + S - 1) / N);
        if (j >= C::SURE && MODE != kMrReady && first + j >= T) continue;  // (kMrReady: the last tile also fetches; its sums are not stored)
        float ga[4], gb[4];
        {
          const float2 a = mr_factors((uint16_t)sa), b = mr_factors((uint16_t)(sa >> 16)), c = mr_factors((uint16_t)sb), e = mr_factors((uint16_t)(sb >> 16));
          ga[0] = a.x, ga[1] = a.y, ga[2] = b.x, ga[3] = b.y, gb[0] = c.x, gb[1] = c.y, gb[2] = e.x, gb[3] = e.y;
        }
        const bool next = MODE == kMrReady && j == N - 1 && i + d + 1 < cnt;
        float2 fx[MG];
#pragma unroll
        for (int m = 0; m < MG; m++) fx[m] = sx[m];
        if (next) factors(d + 1);
#pragma unroll
        for (int b = 0; b < 4; b++) {
          uint32_t ha[4], hb[4];
          mr_unpack(wa[b], ha);
          mr_unpack(wb[b], hb);
          float e[MG][4];
#pragma unroll
          for (int m = 0; m < MG; m++) {
            const uint32_t(&x)[4] = xh[m][b];
            float h[4];
            mr_mma(h, ha[0], hb[0], ha[1], hb[1], x[0], x[1], 0.0f, 0.0f, 0.0f, 0.0f);
            mr_mma(e[m], ha[2], hb[2], ha[3], hb[3], x[2], x[3], h[0], h[1], h[2], h[3]);
          }
          if (next) ready(d + 1, b);  // this block's registers take the next step's values
#pragma unroll
          for (int m = 0; m < MG; m++) {
            acc[j][m][0] = __ffma2_rn(make_float2(e[m][0], e[m][1]), __fmul2_rn(fx[m], make_float2(ga[b], ga[b])), acc[j][m][0]);
            acc[j][m][1] = __ffma2_rn(make_float2(e[m][2], e[m][3]), __fmul2_rn(fx[m], make_float2(gb[b], gb[b])), acc[j][m][1]);
          }
        }
      }
    }
    k0 += D * kstep;
  }
  rows_finish<C, DUAL>(acc, mr_smem, p.t, tile0, tile_own, csize, crank);
}

// Activations for kMrReady, optionally behind an RMSNorm: sixteen threads have the 128 values of a (token, k step). With the norm a CTA has a row.
constexpr int kMpThreads = 256, kMpVecs = 4;
template <bool NORM>
__global__ void __launch_bounds__(kMpThreads) mx_rows_prep_kernel(MxRowsParams p, int Mp, uint8_t* out) {
  __shared__ float part[kMpThreads / 32];
  constexpr int V = NORM ? kMpVecs : 1;
  const int m = blockIdx.x, q0 = blockIdx.y * kMpThreads + threadIdx.x, pieces = p.steps * 16;
  pdl_trigger();
  if (NORM)
    for (int q = q0; q * 8 < p.t.K; q += kMpThreads) rows_prefetch_gamma(p.gamma, p.gamma_f32, q);
  pdl_wait();
  uint4 x[V];
#pragma unroll
  for (int v = 0; v < V; v++) {
    const int q = q0 + v * kMpThreads;
    x[v] = q * 8 < p.t.K ? rows_ldg16(p.x + (size_t)m * p.t.K + q * 8) : make_uint4(0, 0, 0, 0);
  }
  float gm[V][8];
  if (NORM)
#pragma unroll
    for (int v = 0; v < V; v++) {
      const int q = q0 + v * kMpThreads;
      if (q * 8 < p.t.K) mr_gamma(p.gamma, p.gamma_f32, q, gm[v]);
    }
  float inv = 1.0f;
  if (NORM) {
    float ss = 0.0f;
#pragma unroll
    for (int v = 0; v < V; v++) ss += mr_square(x[v]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
    __syncthreads();
    ss = 0.0f;
#pragma unroll
    for (int w = 0; w < kMpThreads / 32; w++) ss += part[w];
    inv = rsqrtf(ss / (float)p.t.K + p.eps);
  }
#pragma unroll
  for (int v = 0; v < V; v++) {
    const int q = q0 + v * kMpThreads;
    if (NORM && q * 8 < p.t.K) x[v] = mr_normed(x[v], inv, gm[v]);
    const uint32_t f = mr_scale(mr_top16(x[v]));
    if (q >= pieces) continue;
    const uint32_t step = q >> 4, b = (q >> 2) & 3;
    *reinterpret_cast<uint4*>(out + ((step * 4 + b) * Mp + m) * 64 + (q & 3) * 16) =
        make_uint4(mr_to_f16(x[v].x, f), mr_to_f16(x[v].y, f), mr_to_f16(x[v].z, f), mr_to_f16(x[v].w, f));
    if ((q & 15) == 0) *reinterpret_cast<float*>(out + (size_t)p.steps * Mp * 256 + (step * Mp + m) * 4) = mr_unscale(f);
  }
}

static size_t mr_stage_bytes(const MxRowsParams& p) { return (size_t)p.steps * p.t.M * (256 + 4); }

template <int T, int MG, bool DUAL, int MODE>
static int mr_launch_mode(const MxRowsParams& p, cudaStream_t st) {
  using C = MrCfg<T, MG, MODE>;
  const size_t smem = C::SMEM + (C::STAGED ? mr_stage_bytes(p) : 0);
  static bool opted[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16 || !opted[dev]) {
    TPX_CUDA_OK(cudaFuncSetAttribute(qlinear_mx_rows_kernel<T, MG, DUAL, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(C::SMEM + C::ROOM)));
    if (dev >= 0 && dev < 16) opted[dev] = true;
  }
  constexpr int TF = DUAL ? T / 2 : T;
  return rows_launch(qlinear_mx_rows_kernel<T, MG, DUAL, MODE>, (p.tiles + TF - 1) / TF, p.t.cluster, C::W * 32, smem, st, p);
}

template <int T, bool DUAL>
static int mr_launch(MxRowsParams p, uint8_t* scratch, cudaStream_t st) {
  // By every CTA while that costs about what the launch in front does, which a caller of single linears pays for as well: one weight up to 20480 values, a pair of more than
  // eight tiles 8 tokens of 4096, behind a norm 2 tokens of 4096. Recorded chains, us, a kernel in front / by every CTA: 4096 x 4096 at 1, 2, 4 and 5 tokens 4.7 / 4.4, 4.5 / 4.7,
  // 4.6 / 5.0 and 4.6 / 5.2, 6144 x 4096 5.6 / 5.1, 5.6 / 5.3, 5.7 / 5.7 and 5.7 / 5.9, 2048 x 2048 3.2 / 2.4, 3.3 / 2.6, 3.3 / 3.0 and 3.1 / 3.1, 4096 x 14336 at 1 token
  // 9.6 / 10.5; the pair of 14336 x 4096 at 1, 4 and 8 tokens 14.4 / 13.7, 14.7 / 14.5 and 15.3 / 15.9, behind a norm at 1 and 2 tokens 15.7 / 15.0 and 15.8 / 15.6. Launched one by
  // one, the launches count for more: an MLP of 8 tokens 29.5 / 27.5 us, a generation of 40 tokens on the Llama-3 shape 21.3 / 20.8 ms with limits after the recorded chains
  // (12288 values, 4096 with two tiles per CTA, 20480 of a pair). Activations in the host's memory are read once, and those that the result replaces before it is written.
  const long long values = (long long)p.steps * 128 * p.t.M;
  if (p.t.M <= (p.gamma ? 2 : 8) && values <= (p.gamma ? 8192 : T > 8 ? 32768 : 20480) &&
      rows_shared_x(p.x, (size_t)p.t.M * p.t.K * 2, p.t.y, (size_t)p.t.M * p.t.N * 2))
    return p.gamma ? mr_launch_mode<T, 1, DUAL, kMrNorm>(p, st) : mr_launch_mode<T, 1, DUAL, kMrStage>(p, st);
  const int Mp = p.t.M > 8 ? 16 : 8;
  p.xr = scratch;
  if (p.gamma)
    TPX_CUDA_OK(launch_pdl(mx_rows_prep_kernel<true>, dim3((unsigned)p.t.M), dim3(kMpThreads), 0, st, p, Mp, scratch));
  else
    TPX_CUDA_OK(launch_pdl(mx_rows_prep_kernel<false>, dim3((unsigned)p.t.M, (unsigned)((p.steps * 16 + kMpThreads - 1) / kMpThreads)), dim3(kMpThreads), 0, st, p,
                           Mp, scratch));
  if constexpr (T <= kMrTiles16)
    if (p.t.M > 8) return mr_launch_mode<T, 2, DUAL, kMrReady>(p, st);
  return mr_launch_mode<T, 1, DUAL, kMrReady>(p, st);
}

template <bool DUAL>
static int mr_launch_t(const MxRowsParams& p, int tf, uint8_t* scratch, cudaStream_t st) {
  constexpr int Z = DUAL ? 2 : 1;
  switch (tf) {
    case 1: return mr_launch<1 * Z, DUAL>(p, scratch, st);
    case 2: return mr_launch<2 * Z, DUAL>(p, scratch, st);
    case 3: return mr_launch<3 * Z, DUAL>(p, scratch, st);
    case 4: return mr_launch<4 * Z, DUAL>(p, scratch, st);
    case 5: return mr_launch<5 * Z, DUAL>(p, scratch, st);
    case 6: return mr_launch<6 * Z, DUAL>(p, scratch, st);
    default: return mr_launch<7 * Z, DUAL>(p, scratch, st);
  }
}

// Up to 8 tokens (the columns of an MMA) wherever one round of CTAs has all tiles (28672 x 8192 pair, two rounds, the second with 108 of 148 CTAs: 57 us,
// tcgen05 52). 9 to 16 tokens while a CTA has few tiles and steps: the MMAs and sums of the second group of tokens are what bounds the kernel there, at 16
// tokens, us, here / tcgen05: 4096 x 4096 6.7 / 8.7, its pair 9.8 / 11.3, 6144 x 4096 8.3 / 9.6, 11008 x 4096 11.5 / 12.6; not 4096 x 14336 14.6 / 13.7, 14336 x 4096
// 13.4 / 11.2, pairs of 6144 x 4096 13.2 / 13.0, 8192 x 2048 10.7 / 10.3.
bool mx_rows_serves(int64_t M, int64_t N, int64_t K, bool pair) {
  const int64_t tiles = (N + 15) / 16, T = rows_tiles(tiles) * (pair ? 2 : 1), steps = (K + 127) / 128;
  return M <= 16 && tiles <= 7LL * sm_count() && (M <= 8 || (T <= kMrTiles16 && T * steps <= 160));
}

size_t mx_rows_scratch_bytes(int64_t M, int64_t K) { return M > 16 ? 0 : (size_t)((K + 127) / 128) * (M > 8 ? 16 : 8) * 260; }

int mx_rows_run(const uint8_t* wq, const uint8_t* sfa, bool pair, const uint16_t* x, int64_t M, int64_t N, int64_t K, int KS, TcParams b, void* scratch,
                cudaStream_t st, const TcNorm* norm) {
  MxRowsParams p = {};
  p.t = b;
  p.t.sfa = sfa;
  p.t.M = (int)M; p.t.N = (int)N; p.t.K = (int)K;
  p.wq = wq; p.x = x; p.KS = KS; p.steps = (int)((K + 127) / 128); p.tiles = (int)(N / 16);
  if (norm && norm->gamma) p.gamma = norm->gamma, p.gamma_f32 = norm->gamma_f32, p.eps = norm->eps;
  const int sms = sm_count(), tf = rows_tiles(p.tiles);
  int c = tf == 1 ? sms / p.tiles : 1;  // few tiles: a cluster cuts k, as far as each warp keeps a step
  while (c > 1 && p.steps < 16 * c) c--;
  p.t.cluster = c >= 8 ? 8 : c >= 4 ? 4 : c >= 2 ? 2 : 1;
  return pair ? mr_launch_t<true>(p, tf, (uint8_t*)scratch, st) : mr_launch_t<false>(p, tf, (uint8_t*)scratch, st);
}

}  // namespace tpx

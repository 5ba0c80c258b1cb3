// Generalized delta rule (tpx_delta.cu) for prompts, heads of 64 channels, bf16 projections: sixteen tokens at a time as matrix products.
//
// With G the decay accumulated since the chunk's start, s = S / G, and per token the rows (64 channels)
//   u = G_(t-1) k,  K = k / G_t,  A = a k / G_t,  R = G_t r,  c = 1 / (sum k^2 + 1e-6),
// the token loop q = c u^T s, s <- s - A q + K v^T, o = R^T s is, over a chunk (rows: tokens; lower triangles, strict for N and M),
//   (I + N) q = c u s0 + M v,   N = c tril(u A^T),  M = c tril(u K^T)
//   o = R s0 + G1 v - G2 q,     G1 = tril(R K^T),  G2 = tril(R A^T)
//   s <- s0 + K^T v - A^T q
// and with W and Y solving (I + N) [W, Y] = [c u, M]:
//   q = W s0 + Y v,   o = (R - G2 W) s0 + (G1 - G2 Y) v.
// Only s0 ties a chunk to the one before: two groups of eight warps, a chunk each, prepare the next chunks' W, R - G2 W, Y, G1 - G2 Y, K, A while four warps apply
// the present one's, each to 16 value channels, whose state they hold as mma accumulators (transposed, so that an accumulator is the next product's left operand
// as it lies).
//
// The matrix products hold that form only for numbers: a token's infinity or NaN would reach the tokens before it through the zeros of the triangles, and the split
// below loses both. A chunk with one, or with a value so large that a product of two overflows, goes token by token (dc_token_loop), and so does one that finds
// such a state, for the value channels of that warp.
//
// State and sums are 32-bit. mma.sync in TF32 with both operands as a rounded value and the rounded remainder, which hold 23 of 24 bits, three products each (two
// where the operand is v, whose bf16 values are TF32 values; that of the two remainders, below 2^-22, is left out); an MMA's own sums are cut off, not rounded.
// Decays and rates take the library's exponential and division, without which the state was 1.25e-7 off 64 bits. As it is, here / token loop: keys of all
// directions 1.0e-7 / 1.05e-7, with slow decays 1.4e-7 / 2.35e-7 and less beside it the slower, with the fastest 1.04e-7 / 0.87e-7 (512 tokens); keys of four
// directions 1.2e-7 / 1.1e-7, of one 1.4e-7 / 1.1e-7 to 2.9e-7 / 1.6e-7. o's rounding to bf16, 1.66e-3, hides any of it.
// Bound by the instructions of the preparation (11000 of a chunk's 14700; splits, fragment loads, the triangular solve): issue slots 56 % busy, tensor pipe 31 %, the
// applying warps alone would take half the time. One sequence of 4096 tokens, 64 heads: 926 us, the token loop 1380; 2 of 512, 16 heads 126 / 177. One CTA per SM: with more
// heads than SMs the token loop is as fast (16 of 256, 64 heads 381 us, here 410).
#include "tpx_delta.cuh"

namespace tpx {

constexpr int kDcTok = 16, kDcMain = 4, kDcPrep = 8, kDcThreads = 32 * (kDcMain + 2 * kDcPrep);
constexpr int kDcMeet = 32 * (kDcMain + kDcPrep);  // threads that hand a buffer over
// floats: row strides are chosen so that the fragment loads meet no bank twice
constexpr int kDcY = 72, kDcH = 24, kDcK = 68, kDcN = 20;
struct __align__(16) DcBuf {  // what the four warps need of a chunk; h: rounded to TF32, l: the remainder
  float yh[32 * kDcY], yl[32 * kDcY];  // rows 0-15 W, 16-31 R - G2 W
  float hh[32 * kDcH], hl[32 * kDcH];  // rows 0-15 Y, 16-31 G1 - G2 Y
  float kh[kDcTok * kDcK], kl[kDcTok * kDcK], ah[kDcTok * kDcK], al[kDcTok * kDcK];
  float v[kDcTok * kDcK], gate[kDcTok * 64], g[64];
  float u[kDcTok * 64], r[kDcTok * 64], c[kDcTok];  // for the token loop, with K = kh + kl and A = ah + al
  int loop;  // the chunk is not for matrix products; yh to hl are not set
};
struct __align__(16) DcPrep {  // of the eight warps that prepare every other chunk
  float w[kDcTok * kDcY], u[kDcTok * kDcY], k[kDcTok * kDcY], a[kDcTok * kDcY], r[kDcTok * kDcY];
  float n[kDcTok * kDcN], m[kDcTok * kDcN], g1[kDcTok * kDcN], g2[kDcTok * kDcN];
  float v[kDcTok * 64], gate[kDcTok * 64], g[64], c[kDcTok];
  __align__(16) uint16_t raw[5 * kDcTok * 64];
  __align__(16) float wraw[kDcTok * 64];
};
struct DcSmem {
  DcBuf buf[2];
  DcPrep prep[2];
  float o[2][kDcTok * kDcK];
};
static_assert(offsetof(DcSmem, buf[1]) % 16 == 0 && offsetof(DcSmem, prep) % 16 == 0 && offsetof(DcSmem, prep[1]) % 16 == 0 && offsetof(DcBuf, u) % 16 == 0 &&
                  offsetof(DcPrep, raw) % 16 == 0 && sizeof(DcSmem) <= 227 * 1024,
              "vectors of 16 bytes");

__device__ __forceinline__ float dc_hi(float x) { return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u); }
__device__ __forceinline__ void dc_split(float x, float& h, float& l) {
  h = dc_hi(x);
  l = dc_hi(x - h);
}
__device__ __forceinline__ void dc_mma(float (&d)[4], const float (&a)[4], float b0, float b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])), "r"(__float_as_uint(a[3])), "r"(__float_as_uint(b0)),
        "r"(__float_as_uint(b1)));
}
// The larger magnitude, a NaN before all; the sign is of no use. Below the bounds a chunk's products are all finite, and so is the split.
constexpr float kDcBig = 1125899906842624.0f, kDcBigState = 1.2676506002282294e30f;  // 2^50, 2^100
__device__ __forceinline__ void dc_larger(float& m, float x) { asm("max.NaN.xorsign.abs.f32 %0, %0, %1;" : "+f"(m) : "f"(x)); }
__device__ __forceinline__ void dc_mma0(float (&d)[4], const float (&a)[4], float b0, float b1) {  // the product alone
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(__float_as_uint(a[0])), "r"(__float_as_uint(a[1])), "r"(__float_as_uint(a[2])), "r"(__float_as_uint(a[3])), "r"(__float_as_uint(b0)),
        "r"(__float_as_uint(b1)), "f"(0.0f));
}
__device__ __forceinline__ void dc_add(float (&d)[4], const float (&x)[4]) {
#pragma unroll
  for (int i = 0; i < 4; i++) d[i] += x[i];
}
__device__ __forceinline__ void dc_bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void dc_bar_arrive(int id, int n) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ bool dc_bar_any(int id, int n, bool mine) {
  int any;
  asm volatile("{ .reg .pred p, q; setp.ne.s32 p, %3, 0; bar.red.or.pred q, %1, %2, p; selp.s32 %0, 1, 0, q; }"
               : "=r"(any)
               : "r"(id), "r"(n), "r"((int)mine)
               : "memory");
  return any != 0;
}
// barriers: 1 and 7 the preparing warps, 2 the applying ones, 3 and 4 a buffer is ready, 5 and 6 it is free

// A chunk token by token, in the order and with the formulas of delta_fast_kernel: value channels e0 ... + 15, the warp's state as it lies in s; o to sh.o.
__device__ __forceinline__ void dc_token_loop(float (&s)[8][4], const DcBuf& B, float* o, int e0) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll 1
  for (int tok = 0; tok < kDcTok; tok++) {
    float2 k[8], a[8];
    float x[6] = {0, 0, 0, 0, 0, 0};  // u . s of both value channels, R . s, then r . k and r . a k
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int at = 8 * j + 2 * t;
      const float2 u = *reinterpret_cast<const float2*>(B.u + tok * 64 + at), r = *reinterpret_cast<const float2*>(B.r + tok * 64 + at);
      const float2 kh = *reinterpret_cast<const float2*>(B.kh + tok * kDcK + at), kl = *reinterpret_cast<const float2*>(B.kl + tok * kDcK + at);
      const float2 ah = *reinterpret_cast<const float2*>(B.ah + tok * kDcK + at), al = *reinterpret_cast<const float2*>(B.al + tok * kDcK + at);
      k[j] = make_float2(kh.x + kl.x, kh.y + kl.y);
      a[j] = make_float2(ah.x + al.x, ah.y + al.y);
#pragma unroll
      for (int e = 0; e < 2; e++) {
        x[e] = fmaf(u.y, s[j][2 * e + 1], fmaf(u.x, s[j][2 * e], x[e]));
        x[2 + e] = fmaf(r.y, s[j][2 * e + 1], fmaf(r.x, s[j][2 * e], x[2 + e]));
      }
      x[4] = fmaf(r.y, k[j].y, fmaf(r.x, k[j].x, x[4]));
      x[5] = fmaf(r.y, a[j].y, fmaf(r.x, a[j].x, x[5]));
    }
#pragma unroll
    for (int i = 0; i < 6; i++) {
      x[i] += __shfl_xor_sync(0xffffffffu, x[i], 1);
      x[i] += __shfl_xor_sync(0xffffffffu, x[i], 2);
    }
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const float q = -B.c[tok] * x[e], v = B.v[tok * kDcK + e0 + g + 8 * e];
      // times zero: as there, where all but one of a column's lanes add the last two terms so
      if (t == 0) o[tok * kDcK + e0 + g + 8 * e] = fmaf(x[4], v, fmaf(x[5], q, x[2 + e])) + fmaf(0.0f, v, 0.0f * q);
#pragma unroll
      for (int j = 0; j < 8; j++) {
        s[j][2 * e] = fmaf(a[j].x, q, fmaf(k[j].x, v, s[j][2 * e]));
        s[j][2 * e + 1] = fmaf(a[j].y, q, fmaf(k[j].y, v, s[j][2 * e + 1]));
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const float2 g2 = *reinterpret_cast<const float2*>(B.g + 8 * j + 2 * t);
#pragma unroll
    for (int i = 0; i < 4; i++) s[j][i] *= (i & 1) ? g2.y : g2.x;
  }
}

__global__ void __launch_bounds__(kDcThreads, 1) delta_chunk_kernel(DeltaFastParams p) {
  extern __shared__ __align__(16) unsigned char dc_smem[];
  DcSmem& sh = *reinterpret_cast<DcSmem*>(dc_smem);
  const int head = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int hd = p.H * 64;
  pdl_trigger();
  pdl_wait();
  const int past = p.dev_len ? *p.dev_len : p.past;
  const int first = p.start ? max(0, min(p.S, p.start[b] - past)) : 0;
  const int chunks = (p.S - first + kDcTok - 1) / kDcTok;
  float* st = p.state + (long long)(b * p.H + head) * 4096;
  if (warp < kDcMain) {
    // ------------------------------------------------------------ the chunk applied to value channels 16 warp ... + 15
    asm volatile("setmaxnreg.inc.sync.aligned.u32 184;");
    const int e0 = warp * 16;
    float s[8][4];  // state, transposed: rows e0 + g, + 8, key channels 8 j + 2 t, + 1
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
      for (int i = 0; i < 4; i++) s[j][i] = st[(8 * j + 2 * t + (i & 1)) * 64 + e0 + g + (i >> 1) * 8];
    for (int c = 0; c < chunks; c++) {
      DcBuf& B = sh.buf[c & 1];
      dc_bar_sync(3 + (c & 1), kDcMeet);
      float* o = sh.o[c & 1];
      float most = 0.0f;
#pragma unroll
      for (int j = 0; j < 8; j++)
#pragma unroll
        for (int i = 0; i < 4; i++) dc_larger(most, s[j][i]);
      if (B.loop || __any_sync(0xffffffffu, !(fabsf(most) < kDcBigState))) {
        dc_token_loop(s, B, o, e0);
      } else {
        // [q of tokens 0-7, 8-15, o of tokens 0-7, 8-15], transposed; small: the products with remainders, summed for themselves, and the others in
        // two sums: an MMA's addition is cut off, not rounded. Products that go to the same sum are four apart: an MMA waits for its accumulator. (Every product
        // added outside: 6 % slower, no nearer to 64 bits but for keys of one direction.)
        float x[4][4], y[4][4], small[4][4];
#pragma unroll
        for (int n = 0; n < 4; n++)
#pragma unroll
          for (int i = 0; i < 4; i++) x[n][i] = y[n][i] = small[n][i] = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; j++) {
          float h[4], l[4];  // as the left operand: slots t and t + 4 of k are channels 2 t and 2 t + 1
          dc_split(s[j][0], h[0], l[0]);
          dc_split(s[j][2], h[1], l[1]);
          dc_split(s[j][1], h[2], l[2]);
          dc_split(s[j][3], h[3], l[3]);
          float2 yh[4], yl[4];
#pragma unroll
          for (int n = 0; n < 4; n++) {
            yh[n] = *reinterpret_cast<const float2*>(B.yh + (8 * n + g) * kDcY + 8 * j + 2 * t);
            yl[n] = *reinterpret_cast<const float2*>(B.yl + (8 * n + g) * kDcY + 8 * j + 2 * t);
          }
#pragma unroll
          for (int n = 0; n < 4; n++) dc_mma(small[n], l, yh[n].x, yh[n].y);
#pragma unroll
          for (int n = 0; n < 4; n++) dc_mma((j & 1) ? y[n] : x[n], h, yh[n].x, yh[n].y);
#pragma unroll
          for (int n = 0; n < 4; n++) dc_mma(small[n], h, yl[n].x, yl[n].y);
        }
        float v[2][4];
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
          for (int e = 0; e < 4; e++) v[i][e] = B.v[(8 * i + 2 * t + (e >> 1)) * kDcK + e0 + g + (e & 1) * 8];
#pragma unroll
        for (int i = 0; i < 2; i++) {
          float2 hh[4], hl[4];
#pragma unroll
          for (int n = 0; n < 4; n++) {
            hh[n] = *reinterpret_cast<const float2*>(B.hh + (8 * n + g) * kDcH + 8 * i + 2 * t);
            hl[n] = *reinterpret_cast<const float2*>(B.hl + (8 * n + g) * kDcH + 8 * i + 2 * t);
          }
#pragma unroll
          for (int n = 0; n < 4; n++) dc_mma(small[n], v[i], hl[n].x, hl[n].y);
#pragma unroll
          for (int n = 0; n < 4; n++) dc_mma(x[n], v[i], hh[n].x, hh[n].y);
        }
#pragma unroll
        for (int n = 0; n < 4; n++)
#pragma unroll
          for (int i = 0; i < 4; i++) x[n][i] += y[n][i] + small[n][i];
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
          for (int i = 0; i < 4; i++) o[(8 * n + 2 * t + (i & 1)) * kDcK + e0 + g + (i >> 1) * 8] = x[2 + n][i];
        float zh[2][4], zl[2][4];
#pragma unroll
        for (int i = 0; i < 2; i++) {
          dc_split(-x[i][0], zh[i][0], zl[i][0]);
          dc_split(-x[i][2], zh[i][1], zl[i][1]);
          dc_split(-x[i][1], zh[i][2], zl[i][2]);
          dc_split(-x[i][3], zh[i][3], zl[i][3]);
        }
#pragma unroll
        for (int j0 = 0; j0 < 8; j0 += 4) {  // what the chunk adds, four groups of channels at a time; the state is added outside
          float d[4][4], dv[4][4], dz[4][4];
#pragma unroll
          for (int j = 0; j < 4; j++)
#pragma unroll
            for (int e = 0; e < 4; e++) d[j][e] = dv[j][e] = dz[j][e] = 0.0f;
#pragma unroll
          for (int i = 0; i < 2; i++) {
            float kh[4][2], kl[4][2], ah[4][2], al[4][2];
#pragma unroll
            for (int j = 0; j < 4; j++)
#pragma unroll
              for (int e = 0; e < 2; e++) {
                const int at = (8 * i + 2 * t + e) * kDcK + 8 * (j0 + j) + g;
                kh[j][e] = B.kh[at]; kl[j][e] = B.kl[at]; ah[j][e] = B.ah[at]; al[j][e] = B.al[at];
              }
#pragma unroll
            for (int j = 0; j < 4; j++) dc_mma(d[j], v[i], kl[j][0], kl[j][1]);
#pragma unroll
            for (int j = 0; j < 4; j++) dc_mma(d[j], zl[i], ah[j][0], ah[j][1]);
#pragma unroll
            for (int j = 0; j < 4; j++) dc_mma(d[j], zh[i], al[j][0], al[j][1]);
#pragma unroll
            for (int j = 0; j < 4; j++) dc_mma(dv[j], v[i], kh[j][0], kh[j][1]);
#pragma unroll
            for (int j = 0; j < 4; j++) dc_mma(dz[j], zh[i], ah[j][0], ah[j][1]);
          }
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const float2 gg = *reinterpret_cast<const float2*>(B.g + 8 * (j0 + j) + 2 * t);
            float(&z)[4] = s[j0 + j];
#pragma unroll
            for (int e = 0; e < 4; e++) z[e] = (z[e] + (dv[j][e] + (dz[j][e] + d[j][e]))) * ((e & 1) ? gg.y : gg.x);
          }
        }
      }
      dc_bar_sync(2, 32 * kDcMain);  // o is whole; the buffer of the chunk after next is written behind the next one's barrier
      const int t0 = first + c * kDcTok;
#pragma unroll
      for (int i = 0; i < kDcTok / kDcMain; i++) {
        const int tok = warp * (kDcTok / kDcMain) + i;
        const float2 y = *reinterpret_cast<const float2*>(o + tok * kDcK + 2 * lane), gt = *reinterpret_cast<const float2*>(B.gate + tok * 64 + 2 * lane);
        const float inv = rsqrtf(hy_warp_sum(y.x * y.x + y.y * y.y) * (1.0f / 64) + p.eps);
        if (t0 + tok < p.S)
          *reinterpret_cast<__nv_bfloat162*>(p.out + ((long long)b * p.S + t0 + tok) * p.ldo + head * 64 + 2 * lane) =
              __floats2bfloat162_rn(y.x * inv * gt.x, y.y * inv * gt.y);
      }
      if (c + 2 < chunks) dc_bar_arrive(5 + (c & 1), kDcMeet);
    }
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
      for (int i = 0; i < 4; i++) st[(8 * j + 2 * t + (i & 1)) * 64 + e0 + g + (i >> 1) * 8] = s[j][i];
    return;
  }
  // -------------------------------------------------------------- the next chunk prepared
  asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
  const int grp = (warp - kDcMain) / kDcPrep, pt = tid - 32 * (kDcMain + grp * kDcPrep), pw = pt >> 5, bar = 1 + 6 * grp;
  DcPrep& sm = sh.prep[grp];
  DcBuf& B = sh.buf[grp];
  const uint16_t* proj = p.proj + (long long)b * p.S * p.ldp + head * 64;
  const float* wraw = p.wraw + (long long)b * p.S * hd + head * 64;
  auto fetch = [&](int c) {
    const int t0 = first + c * kDcTok, n = min(kDcTok, p.S - t0);
    for (int i = pt; i < n * 40; i += 32 * kDcPrep) {
      const int q = i & 7, a = (i >> 3) % 5, tok = i / 40;
      dl_cp16(sm.raw + (a * kDcTok + tok) * 64 + q * 8, proj + (long long)(t0 + tok) * p.ldp + a * hd + q * 8);
    }
    for (int i = pt; i < n * 16; i += 32 * kDcPrep) dl_cp16(sm.wraw + i * 4, wraw + (long long)(t0 + i / 16) * hd + i % 16 * 4);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (grp < chunks) fetch(grp);
  float2 bias, nw;
  bias = make_float2(p.a_bias[head * 64 + 2 * lane], p.a_bias[head * 64 + 2 * lane + 1]);
  nw = make_float2(p.norm_w[head * 64 + 2 * lane], p.norm_w[head * 64 + 2 * lane + 1]);
  for (int c = grp; c < chunks; c += 2) {
    const int n = min(kDcTok, p.S - first - c * kDcTok);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    dc_bar_sync(bar, 32 * kDcPrep);
    // decays, rates, c, values and gates: a warp per token, two channels per lane; tokens behind the last leave the state as it is
    const uint16_t* raw = sm.raw;
    float most = 0.0f;  // of this thread's values of the chunk
#pragma unroll
    for (int q = 0; q < kDcTok / kDcPrep; q++) {
      const int tok = pw + q * kDcPrep;
      float2 w = make_float2(1, 1), k = make_float2(0, 0), a = k, r = k, v = k, gt = k;
      if (tok < n) {
        auto two = [&](int row) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(raw + (row * kDcTok + tok) * 64 + 2 * lane)); };
        const float2 ws = *reinterpret_cast<const float2*>(sm.wraw + tok * 64 + 2 * lane), as = two(3), gs = two(4);
        r = two(0); k = two(1); v = two(2);
        a = make_float2(hy_sigmoid(as.x + bias.x) * k.x, hy_sigmoid(as.y + bias.y) * k.y);
        w = make_float2(expf(-0.60653065971263342f * hy_sigmoid(ws.x)), expf(-0.60653065971263342f * hy_sigmoid(ws.y)));
        gt = make_float2(nw.x * dl_sigmoid(gs.x), nw.y * dl_sigmoid(gs.y));
      }
      dc_larger(most, v.x);
      dc_larger(most, v.y);
      const float k2 = hy_warp_sum(k.x * k.x + k.y * k.y);
      if (lane == 0) sm.c[tok] = 1.0f / (k2 + 1e-6f);
      *reinterpret_cast<float2*>(sm.w + tok * kDcY + 2 * lane) = w;
      *reinterpret_cast<float2*>(sm.k + tok * kDcY + 2 * lane) = k;
      *reinterpret_cast<float2*>(sm.a + tok * kDcY + 2 * lane) = a;
      *reinterpret_cast<float2*>(sm.r + tok * kDcY + 2 * lane) = r;
      *reinterpret_cast<float2*>(sm.v + tok * 64 + 2 * lane) = v;
      *reinterpret_cast<float2*>(sm.gate + tok * 64 + 2 * lane) = gt;
    }
    dc_bar_sync(bar, 32 * kDcPrep);
    if (c + 2 < chunks) fetch(c + 2);  // this chunk's rows have been read
    // accumulated decays: four tokens of a channel per thread, the decays in front of them multiplied again
    {
      const int ch = pt & 63, q0 = (pt >> 6) * 4;
      float G = 1.0f;
      float before[12];
#pragma unroll
      for (int i = 0; i < 12; i++) before[i] = i < q0 ? sm.w[i * kDcY + ch] : 1.0f;
#pragma unroll
      for (int i = 0; i < 12; i++) G *= before[i];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int at = (q0 + i) * kDcY + ch;
        const float k = sm.k[at], a = sm.a[at];
        sm.u[at] = G * k;
        G *= sm.w[at];
        const float gi = 1.0f / G, ki = k * gi, ai = a * gi, r = sm.r[at] * G;
        sm.k[at] = ki;
        sm.a[at] = ai;
        sm.r[at] = r;
        dc_larger(most, ki);  // G k is no larger
        dc_larger(most, ai);
        dc_larger(most, r);
      }
      if (q0 == 12) sm.g[ch] = G;
    }
    const bool loop = dc_bar_any(bar, 32 * kDcPrep, !(fabsf(most) < kDcBig));
    // [u; R] [K; A]^T: a tile of 16 x 8 per warp. The main products are added outside, rounded: keys of one direction have sums of terms of one sign, and cut
    // off they put the state 2.2e-7 off 64 bits, so 1.45e-7 (1030 tokens; the token loop 1.1e-7). 1 x 4096 tokens, 64 heads take 926 us instead of 916.
    if (!loop) {
      const float* left = (pw & 1) ? sm.r : sm.u;
      const float* right = ((pw >> 1) & 2) ? sm.a : sm.k;
      const int col0 = ((pw >> 1) & 1) * 8;
      float x[4] = {0, 0, 0, 0}, x1[4] = {0, 0, 0, 0}, x2[4] = {0, 0, 0, 0};
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const float2 l0 = *reinterpret_cast<const float2*>(left + g * kDcY + 8 * j + 2 * t), l1 = *reinterpret_cast<const float2*>(left + (g + 8) * kDcY + 8 * j + 2 * t);
        const float2 rr = *reinterpret_cast<const float2*>(right + (col0 + g) * kDcY + 8 * j + 2 * t);
        float h[4], l[4], bh[2], bl[2];
        dc_split(l0.x, h[0], l[0]);
        dc_split(l1.x, h[1], l[1]);
        dc_split(l0.y, h[2], l[2]);
        dc_split(l1.y, h[3], l[3]);
        dc_split(rr.x, bh[0], bl[0]);
        dc_split(rr.y, bh[1], bl[1]);
        dc_mma(x1, l, bh[0], bh[1]);
        dc_mma(x2, h, bl[0], bl[1]);
        float one[4];
        dc_mma0(one, h, bh[0], bh[1]);
        dc_add(x, one);
      }
      float* to = (pw & 1) ? (((pw >> 1) & 2) ? sm.g2 : sm.g1) : (((pw >> 1) & 2) ? sm.n : sm.m);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int row = g + (i >> 1) * 8, col = col0 + 2 * t + (i & 1);
        const bool in = (pw & 1) ? col <= row : col < row;
        to[row * kDcN + col] = in ? (x[i] + (x1[i] + x2[i])) * ((pw & 1) ? 1.0f : sm.c[row]) : 0.0f;
      }
    }
    if (!loop) dc_bar_sync(bar, 32 * kDcPrep);
    // W (in place of w) and Y (of M): a column per thread
    if (!loop && pt < 80) {
      const bool isy = pt >= 64;
      const int col = isy ? pt - 64 : pt;
      float y[kDcTok];
#pragma unroll
      for (int i = 0; i < kDcTok; i++) y[i] = isy ? sm.m[i * kDcN + col] : sm.c[i] * sm.u[i * kDcY + col];
#pragma unroll
      for (int i = 1; i < kDcTok; i++) {
        float nr[kDcTok];
#pragma unroll
        for (int z = 0; z < (i + 3) / 4; z++) *reinterpret_cast<float4*>(nr + 4 * z) = *reinterpret_cast<const float4*>(sm.n + i * kDcN + 4 * z);
        float a1 = 0.0f;
#pragma unroll
        for (int z = 0; z < i; z++) {
          if (z & 1) a1 = fmaf(-nr[z], y[z], a1);
          else y[i] = fmaf(-nr[z], y[z], y[i]);
        }
        y[i] += a1;
      }
#pragma unroll
      for (int i = 0; i < kDcTok; i++) {
        if (isy) sm.m[i * kDcN + col] = y[i];
        else sm.w[i * kDcY + col] = y[i];
      }
    }
    dc_bar_sync(bar, 32 * kDcPrep);
    if (c >= 2) dc_bar_sync(5 + grp, kDcMeet);  // only from here on is the buffer touched
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int tok = q * 4 + (pt >> 6), ch = pt & 63;
      const float k = sm.k[tok * kDcY + ch], a = sm.a[tok * kDcY + ch];
      float kh, kl, ah, al;
      dc_split(k, kh, kl);
      dc_split(a, ah, al);
      B.kh[tok * kDcK + ch] = loop ? k : kh;
      B.kl[tok * kDcK + ch] = loop ? 0.0f : kl;
      B.ah[tok * kDcK + ch] = loop ? a : ah;
      B.al[tok * kDcK + ch] = loop ? 0.0f : al;
      B.u[tok * 64 + ch] = sm.u[tok * kDcY + ch];
      B.r[tok * 64 + ch] = sm.r[tok * kDcY + ch];
      dc_split(sm.w[tok * kDcY + ch], B.yh[tok * kDcY + ch], B.yl[tok * kDcY + ch]);
      B.v[tok * kDcK + ch] = sm.v[tok * 64 + ch];
      B.gate[tok * 64 + ch] = sm.gate[tok * 64 + ch];
    }
    dc_split(sm.m[(pt >> 4) * kDcN + (pt & 15)], B.hh[(pt >> 4) * kDcH + (pt & 15)], B.hl[(pt >> 4) * kDcH + (pt & 15)]);
    if (pt < 64) B.g[pt] = sm.g[pt];
    if (pt < kDcTok) B.c[pt] = sm.c[pt];
    if (pt == 0) B.loop = loop;
    // what o takes: [R, G1] - G2 [W, Y], eight columns per warp (warps 0 and 1: and eight of the second)
#pragma unroll
    for (int part = 0; part < 2; part++) {
      if (loop || (part == 1 && pw >= 2)) break;
      const float *left = sm.g2, *right = part ? sm.m : sm.w, *base = part ? sm.g1 : sm.r;
      const int ld = part ? kDcN : kDcY, col0 = 8 * pw;
      float x[4] = {0, 0, 0, 0}, x1[4] = {0, 0, 0, 0}, x2[4] = {0, 0, 0, 0};
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const float2 l0 = *reinterpret_cast<const float2*>(left + g * kDcN + 8 * j + 2 * t), l1 = *reinterpret_cast<const float2*>(left + (g + 8) * kDcN + 8 * j + 2 * t);
        float h[4], l[4], bh[2], bl[2];
        dc_split(l0.x, h[0], l[0]);
        dc_split(l1.x, h[1], l[1]);
        dc_split(l0.y, h[2], l[2]);
        dc_split(l1.y, h[3], l[3]);
        dc_split(right[(8 * j + 2 * t) * ld + col0 + g], bh[0], bl[0]);
        dc_split(right[(8 * j + 2 * t + 1) * ld + col0 + g], bh[1], bl[1]);
        dc_mma(x1, l, bh[0], bh[1]);
        dc_mma(x2, h, bl[0], bl[1]);
        dc_mma(x, h, bh[0], bh[1]);
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int row = g + (i >> 1) * 8, col = col0 + 2 * t + (i & 1);
        const float y = base[row * ld + col] - (x[i] + (x1[i] + x2[i]));
        if (part) dc_split(y, B.hh[(kDcTok + row) * kDcH + col], B.hl[(kDcTok + row) * kDcH + col]);
        else dc_split(y, B.yh[(kDcTok + row) * kDcY + col], B.yl[(kDcTok + row) * kDcY + col]);
      }
    }
    dc_bar_arrive(3 + grp, kDcMeet);
  }
}

// Padding rows of `out` are the caller's (zero, or unread), as in the token loop.
int delta_chunk(const DeltaFastParams& p, int64_t B, cudaStream_t st) {
  static bool opted[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16 || !opted[dev]) {
    TPX_CUDA_OK(cudaFuncSetAttribute(delta_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(DcSmem)));
    if (dev >= 0 && dev < 16) opted[dev] = true;
  }
  TPX_CUDA_OK(launch_pdl(delta_chunk_kernel, dim3((unsigned)p.H, (unsigned)B), dim3(kDcThreads), sizeof(DcSmem), st, p));
  return TPX_OK;
}

}  // namespace tpx

// int8 linear (and gate/up pair) of few tokens: the weight streams through registers once, mma.sync beside it.
//
// Arithmetic of qlinear_i8_kernel (tpx_qlinear_i8.cu): int8 x int8 -> int32 per block of 64 k values, times s_x * s_w, added in fp32.
//
// Every weight byte is read once, which is 0.73 of a call of 11008 x 4096 at one token, 0.55 at 16 and 0.44 at 32 (7.3 us of HBM); the rest is a launch's start and end
// in the chain, the wait for the activations and, above 16 tokens, the instructions per weight byte (43 % of issue slots at 32). A CTA has T tiles of 16 features
// and all of K; its groups of warps take the 64-wide k blocks in turn, two neighbours (128 bytes of a row) at a time. A warp's weights come by
// cp.async into a ring of its own, each lane copying exactly the 16-byte pieces that it feeds to its MMAs: no barrier of the CTA in the loop,
// 100 to 200 KB per SM on the way, the first of them before the wait for the previous kernel. k is permuted inside a block (a lane's MMA slots
// are 16 consecutive values), which both operands share, so the plain row-major weight needs no repacking. Quantised activations come straight
// from L2 to registers, a block ahead; one or two tokens every CTA quantises for itself. The tcgen05 form has a chain per 256 k values (copies, MMAs, drain of int32 accumulators from tensor memory)
// on whole tiles of 128 features; here the drain is three packed fp32 operations per two sums in the registers where the MMA left them.
// With the quantisation of x, recorded chains of calls on one B200, tcgen05 form / here: 11008 x 4096 1 token 15.6 / 10.0 us, 16: 15.8 / 13.2, 32: 18.1 / 16.7; 4096 x 4096
// 9.8 / 5.4 at 1, 12.2 / 8.5 at 32; the pair 2 x 11008 x 4096 at 1 token 30.7 / 16.8 (one kernel instead of two).
#include "tpx_qlinear_i8_rows.cuh"
#include "tpx_rows.cuh"

namespace tpx {

constexpr int kIrSlot = 1088;  // 16 features x 64 values and the 16 scales
// A warp's ring holds D k blocks of its tiles: every address in the loop over D blocks is a constant offset. Sixteen warps hide the latencies (with eight, 11008 x 4096 took 18.4 us at
// 16 tokens, with sixteen 14.1); above 16 tokens the sums and the activations of the next block need the registers of twelve (18.2 / 17.2 us).
template <int T, int MG>
struct IrCfg : RowsSplit<T, MG, MG == 4 ? 12 : 16, MG == 4 ? 3 : 4> {
  using S0 = RowsSplit<T, MG, MG == 4 ? 12 : 16, MG == 4 ? 3 : 4>;
  static constexpr int D = S0::N == 1 ? 8 : S0::N == 2 ? 4 : 2, S = D * S0::N;
  static constexpr size_t RING = (size_t)S0::W * S * kIrSlot, SMEM = RING > S0::PARTS ? RING : S0::PARTS;
  static_assert(SMEM <= 225 * 1024, "shared memory");
};

__device__ __forceinline__ void ir_mma(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1,
                                       int c0, int c1, int c2, int c3) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c0), "r"(c1), "r"(c2), "r"(c3));
}
constexpr int kIrStaged = 65536;  // quantised values, at most, of one or two tokens in shared memory behind the ring

// Quantises the rows of x as quantize_act_i8_row_kernel does, behind the same norm, into shared memory: values [k block][token][64] at xs, scales [k block][token] at fs.
// Every CTA does all of them for itself; the first leaves them in p.xq too, for a call that reuses them.
template <int THREADS>
__device__ __forceinline__ void ir_quantize(const I8RowsParams& p, uint32_t xs, uint32_t fs) {
  __shared__ float part[2][THREADS / 32];
  const int M = p.t.M, nv = p.nkb * 8, tid = threadIdx.x;  // nv: pieces of 8 values per token
  float gm[2][8];
  if (p.gamma) {
#pragma unroll
    for (int r = 0; r < 2; r++)
      if (r * THREADS + tid < nv) rows_prefetch_gamma(p.gamma, p.gamma_f32, r * THREADS + tid);
  }
  pdl_wait();
  for (int q0 = 0; q0 < nv; q0 += 2 * THREADS) {  // with the norm (at most 8192 values) once
    uint4 v[2][2];
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
      for (int m = 0; m < 2; m++) {
        const int q = q0 + r * THREADS + tid;
        v[r][m] = q < nv && m < M ? rows_ldg16(p.x + (size_t)m * nv * 8 + q * 8) : make_uint4(0, 0, 0, 0);
      }
    float inv[2] = {};
    if (p.gamma) {
#pragma unroll
      for (int r = 0; r < 2; r++)
        if (r * THREADS + tid < nv) i8_gamma(p.gamma, p.gamma_f32, r * THREADS + tid, gm[r]);
#pragma unroll
      for (int m = 0; m < 2; m++) {
        float ss = 0.0f;
#pragma unroll
        for (int r = 0; r < 2; r++) {
          float f[8];
          i8_unpack_bf16(v[r][m], f);
#pragma unroll
          for (int j = 0; j < 8; j += 2) ss += f[j] * f[j] + f[j + 1] * f[j + 1];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if ((tid & 31) == 0) part[m][tid >> 5] = ss;
      }
      __syncthreads();
#pragma unroll
      for (int m = 0; m < 2; m++) {
        float tot = 0.0f;
#pragma unroll
        for (int w = 0; w < THREADS / 32; w++) tot += part[m][w];
        inv[m] = rsqrtf(tot / (float)(nv * 8) + p.eps);
      }
    }
#pragma unroll
    for (int r = 0; r < 2; r++)
#pragma unroll
      for (int m = 0; m < 2; m++) {
        const int q = q0 + r * THREADS + tid;
        if (m >= M || q0 + r * THREADS >= nv) continue;
        float f[8];
        i8_unpack_bf16(v[r][m], f);
        if (p.gamma && q < nv) {
#pragma unroll
          for (int j = 0; j < 8; j++) f[j] = bf16_bits_to_f32(f32_to_bf16_bits(f[j] * inv[m] * gm[r][j]));
        }
        uint2 o;
        const float scale = i8_quantize8(f, 8, o);
        if (q >= nv) continue;
        const int blk = q >> 3;
        asm volatile("st.shared.v2.u32 [%0], {%1,%2};" ::"r"(xs + (uint32_t)((blk * M + m) * 64 + (q & 7) * 8)), "r"(o.x), "r"(o.y) : "memory");
        if ((q & 7) == 0) asm volatile("st.shared.f32 [%0], %1;" ::"r"(fs + (uint32_t)(blk * M + m) * 4), "f"(scale) : "memory");
        if (blockIdx.x == 0) {
          const I8Act64 L = {16};
          *reinterpret_cast<uint2*>(L.value(p.xq, m, q * 8)) = o;
          if ((q & 7) == 0) *L.scale(p.xq, m, blk) = scale;
        }
      }
  }
  __syncthreads();
}

// T: tiles of 16 features per CTA (of a pair: gate and up tiles in turn), MG: groups of 8 tokens, QUANT: the kernel quantises the activations itself
template <int T, int MG, bool DUAL, bool QUANT>
__global__ void __launch_bounds__(IrCfg<T, MG>::W * 32, 1) qlinear_i8_rows_kernel(I8RowsParams p) {
  using C = IrCfg<T, MG>;
  constexpr int KG = C::KG, N = C::N, D = C::D, S = C::S, TF = DUAL ? T / 2 : T;  // TF: feature tiles
  extern __shared__ __align__(16) unsigned char ir_smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int csize = p.t.cluster, crank = csize > 1 ? (int)tc_cluster_rank() : 0;
  // the last CTA starts early enough to have all its tiles, and stores those that are its own
  const int tile_own = (int)blockIdx.x / csize * TF, tile0 = min(tile_own, p.tiles - TF);
  const int first = warp / KG * N;  // this warp's first tile
  // its k blocks: of the pairs of neighbours, those that fall to its group when all groups of the cluster take turns
  const int pairs = p.nkb >> 1, groups = KG * csize, turn = crank * KG + warp % KG;
  const int cnt = 2 * (pairs > turn ? (pairs - turn + groups - 1) / groups : 0) + ((p.nkb & 1) && pairs % groups == turn ? 1 : 0);
  const uint32_t ring = tc_smem_u32(ir_smem_raw) + warp * (S * kIrSlot), own = ring + lane * 16;
  // addresses: a base that is the same in the whole CTA, and 32-bit offsets behind it
  const int f0 = DUAL ? first >> 1 : first, odd = DUAL ? first & 1 : 0;  // odd: the first tile is one of the second weight
  const uint32_t row16 = 16 * p.Kp, row8 = 8 * p.Kp, wstep = groups * 128, sstep = groups * 8 * p.Np;
  const int8_t* const wb0 = p.w[0] + (size_t)tile0 * row16;
  const int8_t* const wb1 = DUAL ? p.w[1] + (size_t)tile0 * row16 : nullptr;
  const char* const sb0 = reinterpret_cast<const char*>(p.swT[0] + tile0 * 16);
  const char* const sb1 = DUAL ? reinterpret_cast<const char*>(p.swT[1] + tile0 * 16) : nullptr;
  uint32_t w0 = f0 * row16 + g * p.Kp + t * 16 + turn * 128, s0 = turn * 8 * p.Np + f0 * 64 + lane * 16;
  constexpr uint32_t TOK = MG == 4 ? 32 : 16;
  const uint32_t xrow = p.t.M * 64, xpair = QUANT ? 2 * xrow : I8Act64::bytes(TOK), xstep = groups * xpair;  // QUANT: rows in shared memory, a block's after another's
  uint32_t x0 = turn * xpair;
  const int last = p.t.M - 1;  // QUANT: columns behind the last token repeat it and are not stored
  const uint32_t xl = QUANT ? min(g, last) * 64 + t * 16 : g * 64 + (t ^ (g >> 1)) * 16;
  const uint32_t xs = tc_smem_u32(ir_smem_raw) + (uint32_t)C::SMEM, fs = xs + p.nkb * xrow;
  pdl_trigger();

  // slot q of the ring, k block `ord` of this warp's, `td` blocks behind the one that w0 and s0 point at
  auto issue = [&](int q, int td, int ord) {
    const int j = q % N;
    if (ord < cnt && (j < C::SURE || first + j < T)) {
      const uint32_t to = own + q % S * kIrSlot;
      const int f = DUAL ? (j + odd) >> 1 : j;
      const bool second = DUAL && ((j + odd) & 1);
      const int8_t* wb = second ? wb1 : wb0;
      const uint32_t w = w0 + (td >> 1) * wstep + (td & 1) * 64 + f * row16;
      rows_copy16(to, wb + w);
      rows_copy16(to + 512, wb + (w + row8));
      if (lane < 4) rows_copy16(to + 1024, (second ? sb1 : sb0) + (s0 + (td >> 1) * sstep + (td & 1) * 4 * p.Np + f * 64));
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int q = 0; q < S - 1; q++) issue(q, q / N, q / N);
  if constexpr (QUANT) ir_quantize<C::W * 32>(p, xs, fs);
  else pdl_wait();

  uint4 xv[2][MG];
  float2 sv[2][MG];
  auto fetch = [&](int z, int td) {
    const uint32_t x = x0 + (td >> 1) * xstep;
    if constexpr (QUANT) {
      const uint32_t xb = x + (td & 1) * xrow;
      xv[z][0] = rows_lds16(xs + xb + xl);
      sv[z][0] = make_float2(rows_lds4(fs + xb / 16 + min(2 * t, last) * 4), rows_lds4(fs + xb / 16 + min(2 * t + 1, last) * 4));
    } else {
#pragma unroll
      for (int m = 0; m < MG; m++) {
        xv[z][m] = rows_ldg16(p.xq + (x + xl + (td & 1) * (TOK * 64) + m * 512));
        sv[z][m] = rows_ldg8(p.xq + (x + TOK * 128 + (td & 1) * (TOK * 4) + t * 8 + m * 32));
      }
    }
  };
  if (cnt > 0) fetch(0, 0);
  float2 acc[N][MG][2];  // [row g, row g + 8] of tokens 2t, 2t + 1
#pragma unroll
  for (int j = 0; j < N; j++)
#pragma unroll
    for (int m = 0; m < MG; m++) acc[j][m][0] = acc[j][m][1] = make_float2(0.0f, 0.0f);
  for (int i = 0; i < cnt; i += D) {
#pragma unroll
    for (int d = 0; d < D; d++) {
      if (i + d >= cnt) break;
      const int z = d & 1;
      if (i + d + 1 < cnt) fetch(z ^ 1, d + 1);
#pragma unroll
      for (int j = 0; j < N; j++) {
        constexpr int kZero = 0x4B400000;
        const int q = d * N + j;
        asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
        __syncwarp();  // the scales were copied by other lanes; and all are done with the slot before, which is filled again
        const uint4 a = rows_lds16(own + q * kIrSlot), b = rows_lds16(own + q * kIrSlot + 512);
        const float sw0 = rows_lds4(ring + q * kIrSlot + 1024 + g * 4), sw1 = rows_lds4(ring + q * kIrSlot + 1056 + g * 4);
        issue(q + S - 1, (q + S - 1) / N, i + (q + S - 1) / N);
        if (j >= C::SURE && first + j >= T) continue;
#pragma unroll
        for (int m = 0; m < MG; m++) {
          // Sums of 64 products stay below 2^22: added to the bits of 1.5 * 2^23 they are that float's low bits (the conversion
          // instruction runs at a quarter of the rate of an addition).
          const float2 zero = make_float2(-12582912.0f, -12582912.0f);
          const uint4 x = xv[z][m];
          int e[4], h[4];
          ir_mma(h, a.x, b.x, a.y, b.y, x.x, x.y, kZero, kZero, kZero, kZero);
          ir_mma(e, a.z, b.z, a.w, b.w, x.z, x.w, h[0], h[1], h[2], h[3]);
          acc[j][m][0] = __ffma2_rn(__fadd2_rn(make_float2(__int_as_float(e[0]), __int_as_float(e[1])), zero),
                                    __fmul2_rn(sv[z][m], make_float2(sw0, sw0)), acc[j][m][0]);
          acc[j][m][1] = __ffma2_rn(__fadd2_rn(make_float2(__int_as_float(e[2]), __int_as_float(e[3])), zero),
                                    __fmul2_rn(sv[z][m], make_float2(sw1, sw1)), acc[j][m][1]);
        }
      }
    }
    w0 += D / 2 * wstep;
    s0 += D / 2 * sstep;
    x0 += D / 2 * xstep;
  }
  rows_finish<C, DUAL>(acc, ir_smem_raw, p.t, tile0, tile_own, csize, crank);
}

template <int T, int MG, bool DUAL, bool QUANT>
static int ir_launch_as(const I8RowsParams& p, cudaStream_t st) {
  constexpr size_t base = IrCfg<T, MG>::SMEM, most = base + (QUANT ? kIrStaged / 64 * 68 : 0);
  static_assert(most <= 225 * 1024, "shared memory");
  static bool opted[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16 || !opted[dev]) {
    TPX_CUDA_OK(cudaFuncSetAttribute(qlinear_i8_rows_kernel<T, MG, DUAL, QUANT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
    if (dev >= 0 && dev < 16) opted[dev] = true;
  }
  constexpr int TF = DUAL ? T / 2 : T;
  return rows_launch(qlinear_i8_rows_kernel<T, MG, DUAL, QUANT>, (p.tiles + TF - 1) / TF, p.t.cluster, IrCfg<T, MG>::W * 32,
                     base + (QUANT ? (size_t)p.nkb * p.t.M * 68 : 0), st, p);
}
template <int T, int MG, bool DUAL>
static int ir_launch(const I8RowsParams& p, cudaStream_t st) {
  if constexpr (MG == 1) {
    if (p.x) return ir_launch_as<T, 1, DUAL, true>(p, st);
  }
  return ir_launch_as<T, MG, DUAL, false>(p, st);
}

template <int MG>
static int ir_launch_t(const I8RowsParams& p, bool pair, int tf, cudaStream_t st) {
  if constexpr (MG <= 2) {
    if (pair) switch (tf) {
      case 1: return ir_launch<2, MG, true>(p, st);
      case 2: return ir_launch<4, MG, true>(p, st);
      case 3: return ir_launch<6, MG, true>(p, st);
      case 4: return ir_launch<8, MG, true>(p, st);
      case 5: return ir_launch<10, MG, true>(p, st);
      case 6: return ir_launch<12, MG, true>(p, st);
      default: return ir_launch<14, MG, true>(p, st);
    }
  }
  switch (tf) {
    case 1: return ir_launch<1, MG, false>(p, st);
    case 2: return ir_launch<2, MG, false>(p, st);
    case 3: return ir_launch<3, MG, false>(p, st);
    case 4: return ir_launch<4, MG, false>(p, st);
    case 5: return ir_launch<5, MG, false>(p, st);
    case 6: return ir_launch<6, MG, false>(p, st);
    default:
      if constexpr (MG < 4) return ir_launch<7, MG, false>(p, st);
      else return TPX_ERR_UNSUPPORTED;  // not a case of i8_rows_serves
  }
}

// Blocks of 64, up to 32 tokens; a pair up to 16 (its two sums do not fit in registers above), where two tcgen05 linears never win. One weight: where the tcgen05 kernel's
// tiles of 128 features fill its one wave of CTAs, it takes the same time for the largest N as for the smallest and for 16 tokens as for one, this kernel more with each. Chains, us,
// tcgen05 / here:
// up to 8 tokens only that wave's last part, which is two rounds here: 4 tokens of 18944 x 3584 15.9 / 17.5, of 17408 x 2048 11.0 / 11.3; 1 token 15.9 / 14.7 and 11.2 / 10.5, of 17408 x 256
//   4.5 / 6.1; with two waves again 27392 x 4096 31.4 / 23.5, 37888 x 4096 34.3 / 32.0 (8 tokens);
// 9 to 16 tokens: up to five tiles per CTA from 256 values on (11008 x 256 4.2 / 4.0, 9408 x 128 4.1 / 5.6), more tiles from 4096 on (14080 x 2048 9.9 / 10.7, 14336 x 2048 10.1 / 10.6,
//   14336 x 4096 16.2 / 15.6, 15360 x 4096 16.6 / 16.2, 16384 x 4096 17.0 / 18.4; 12 tokens);
// 17 to 32 tokens, fewer groups of warps: four tiles from 256 values on (9408 x 128 4.5 / 6.1, x 256 6.5 / 5.8), five from 1536 (11008 x 1024 7.4 / 8.2, x 1536 9.3 / 9.2), six from 3072
//   (14080 x 2048 11.6 / 12.0, x 3072 14.9 / 14.8, 12288 x 4096 18.1 / 17.2), seven nowhere (14336 x 4096 19.7 / 21.0); more rounds where waves are badly filled (25600 x 5120, 200 tiles:
//   42.0 / 36.6; 32000 x 4096, 250: 36.5 / 36.6; 37888 x 4096, 296: 38.6 / 45.4).
bool i8_rows_serves(int64_t M, int64_t N, int64_t K, int64_t block, bool pair) {
  if (block != 64 || M > 32) return false;
  if (pair) return M <= 16;
  const int64_t sms = sm_count(), tiles = N / 16, big = (N + 127) / 128, waves = (big + sms - 1) / sms;
  const int T = rows_tiles(tiles);
  const bool rounds = tiles > 7 * sms;
  if (M <= 8) return !rounds || waves > 1 || (M <= 2 && K >= 1024);
  if (M <= 16) return rounds ? waves > 1 : T <= 5 ? K >= 256 : K >= 4096 && 2 * tiles <= 13 * sms;
  if (rounds) return T < 7 && 10 * big < 7 * waves * sms && K >= 1536;
  return T <= 4 ? K >= 256 : T == 5 ? K >= 1536 : T == 6 && K >= 3072;
}

// One and two tokens: in every CTA. Recorded chains of calls, us, a kernel in front / in here. 1 token: 4096 x 4096 5.3 / 5.4, 6144 x 4096 8.1 / 7.1, 11008 x 4096
// 11.5 / 10.1, 4096 x 11008 11.4 / 10.8, the pair of 11008 x 4096 18.2 / 16.8; behind a norm 7.4 / 6.8, 10.3 / 8.0, 13.8 / 11.2, the pair 21.0 / 18.0. 2 tokens: 6144 x 4096 8.2 / 7.5,
// 11008 x 4096 11.3 / 10.5, the pair 18.3 / 17.3, behind a norm 7.6 / 7.3, 10.3 / 8.6, 13.6 / 11.7, 20.9 / 18.5; only with two tiles per CTA and no norm is the kernel in front
// ahead, 4096 x 4096 5.4 / 5.9, 4096 x 11008 11.5 / 12.0, by less than a launch costs a caller of single linears: a generation of two sequences, 8 layers of 4096 x 11008,
// takes 26.8 ms either way.
bool i8_rows_quantizes(const void* x, const void* y, int64_t M, int64_t N, int64_t K) {
  return M <= 2 && M * K <= kIrStaged && rows_shared_x(x, (size_t)M * K * 2, y, (size_t)M * N * 2);
}

int i8_rows_launch(I8RowsParams p, bool pair, cudaStream_t st) {
  const int sms = sm_count(), tf = rows_tiles(p.tiles);
  // few tiles: a cluster cuts k, as far as each warp keeps a pair of blocks
  int c = tf == 1 ? sms / p.tiles : 1;
  while (c > 1 && p.nkb < 32 * c) c--;
  p.t.cluster = c >= 8 ? 8 : c >= 4 ? 4 : c >= 2 ? 2 : 1;
  return p.t.M <= 8 ? ir_launch_t<1>(p, pair, tf, st) : p.t.M <= 16 ? ir_launch_t<2>(p, pair, tf, st) : ir_launch_t<4>(p, pair, tf, st);
}

}  // namespace tpx

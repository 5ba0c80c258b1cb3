// int8 linear (and gate/up pair) of few tokens: the weight streams through registers once, mma.sync beside it.
//
// Arithmetic of qlinear_i8_kernel (tpx_qlinear_i8.cu): int8 x int8 -> int32 per block of 64 k values, times s_x * s_w, added in fp32.
//
// Bound by HBM up to 16 tokens (every weight byte is used once), above by the instructions per weight byte. A CTA has T tiles of 16 features
// and all of K; its groups of warps take the 64-wide k blocks in turn, two neighbours (128 bytes of a row) at a time. A warp's weights come by
// cp.async into a ring of its own, each lane copying exactly the 16-byte pieces that it feeds to its MMAs: no barrier of the CTA in the loop,
// 100 to 200 KB per SM on the way, the first of them before the wait for the previous kernel. k is permuted inside a block (a lane's MMA slots
// are 16 consecutive values), which both operands share, so the plain row-major weight needs no repacking. Activations come straight
// from L2 to registers, a block ahead. The tcgen05 form has a chain per 256 k values (copies, MMAs, drain of int32 accumulators from tensor memory)
// on whole tiles of 128 features; here the drain is three packed fp32 operations per two sums in the registers where the MMA left them.
// With the quantisation of x, a chain of calls on one B200, tcgen05 form / here: 11008 x 4096 (7.4 us of HBM) 1 token 16.4 / 12.0 us, 16: 16.4 / 14.1,
// 32: 18.8 / 17.2; 4096 x 4096 10.2 / 5.7 at 1, 12.6 / 9.0 at 32; the pair 2 x 11008 x 4096 at 1 token 31.8 / 20.3 (one kernel instead of two).
#include "tpx_qlinear_i8_rows.cuh"

namespace tpx {

constexpr int kIrSlot = 1088;  // 16 features x 64 values and the 16 scales
// W warps: KG groups that take the k blocks in turn, each of H warps with N of the T tiles. A warp's ring holds D k blocks of its tiles:
// every address in the loop over D blocks is a constant offset. Sixteen warps hide the latencies (with eight, 11008 x 4096 took 18.4 us at
// 16 tokens, now 14.1); above 16 tokens the sums and the activations of the next block need the registers of twelve (18.2 / 17.2 us).
template <int T, int MG>
struct IrCfg {
  static constexpr int MOST = MG == 4 ? 3 : 6;  // tiles whose sums a warp has registers for
  static constexpr int W = MG == 4 ? 12 : 16, H = T <= MOST ? 1 : T <= 2 * MOST ? 2 : 4;
  static constexpr int KG = W / H, N0 = (T + H - 1) / H, N = T > 7 ? (N0 + 1) / 2 * 2 : N0;  // whole pairs of gate and up tiles
  static constexpr int D = N == 1 ? 8 : N == 2 ? 4 : 2, S = D * N;
  static constexpr bool AHEAD = !(MG == 2 && N == 6);  // activations a k block ahead, in registers of their own
  static constexpr int RP = 16 * T + 4;  // a token's row of sums: 4 banks past a multiple of 16, so that lanes' stores do not meet
  static constexpr size_t RING = (size_t)W * S * kIrSlot, PARTS = (size_t)(KG == 16 ? 8 : KG) * MG * 8 * RP * 4;
  static constexpr size_t SMEM = RING > PARTS ? RING : PARTS;
  static_assert(SMEM <= 225 * 1024, "shared memory");
};

__device__ __forceinline__ void ir_mma(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1,
                                       int c0, int c1, int c2, int c3) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c0), "r"(c1), "r"(c2), "r"(c3));
}
__device__ __forceinline__ void ir_copy16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ uint4 ir_lds16(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
// What the kernel before this one wrote: not __ldg, which may be moved in front of the wait for that kernel.
__device__ __forceinline__ uint4 ir_ldg16(const void* a) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(a) : "memory");
  return v;
}
__device__ __forceinline__ float2 ir_ldg8(const void* a) {
  float2 v;
  asm volatile("ld.global.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(a) : "memory");
  return v;
}
__device__ __forceinline__ float ir_lds4(uint32_t a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

// a float of the shared memory of member c of the cluster, at the address that it has here
__device__ __forceinline__ float ir_ld_member(uint32_t a, int c) {
  float v;
  asm volatile("{ .reg .b32 r; mapa.shared::cluster.u32 r, %1, %2; ld.shared::cluster.f32 %0, [r]; }" : "=f"(v) : "r"(a), "r"(c) : "memory");
  return v;
}

// T: tiles of 16 features per CTA (of a pair: gate and up tiles in turn), MG: groups of 8 tokens
template <int T, int MG, bool DUAL>
__global__ void __launch_bounds__(IrCfg<T, MG>::W * 32, 1) qlinear_i8_rows_kernel(I8RowsParams p) {
  using C = IrCfg<T, MG>;
  constexpr int KG = C::KG, N = C::N, D = C::D, S = C::S, RP = C::RP, TF = DUAL ? T / 2 : T;  // TF: feature tiles
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
  const int f0 = DUAL ? first >> 1 : first;
  const uint32_t row16 = 16 * p.Kp, row8 = 8 * p.Kp, wstep = groups * 128, sstep = groups * 8 * p.Np;
  const int8_t* const wb0 = p.w[0] + (size_t)tile0 * row16;
  const int8_t* const wb1 = DUAL ? p.w[1] + (size_t)tile0 * row16 : nullptr;
  const char* const sb0 = reinterpret_cast<const char*>(p.swT[0] + tile0 * 16);
  const char* const sb1 = DUAL ? reinterpret_cast<const char*>(p.swT[1] + tile0 * 16) : nullptr;
  uint32_t w0 = f0 * row16 + g * p.Kp + t * 16 + turn * 128, s0 = turn * 8 * p.Np + f0 * 64 + lane * 16;
  const uint32_t xrow = p.Mp * 64, xstep = groups * 2 * xrow;
  const uint8_t* const sxb = p.xq + (size_t)p.nkb * xrow;  // a scale is 4 bytes where its 64 values are 64
  uint32_t x0 = turn * 2 * xrow;
  const uint32_t xl = g * 64 + t * 16;
  pdl_trigger();

  // slot q of the ring, k block `ord` of this warp's, `td` blocks behind the one that w0 and s0 point at
  auto issue = [&](int q, int td, int ord) {
    const int j = q % N;
    if (ord < cnt && (T % N == 0 || first + j < T)) {
      const uint32_t to = own + q % S * kIrSlot;
      const int f = DUAL ? j >> 1 : j;
      const int8_t* wb = DUAL && (j & 1) ? wb1 : wb0;
      const uint32_t w = w0 + (td >> 1) * wstep + (td & 1) * 64 + f * row16;
      ir_copy16(to, wb + w);
      ir_copy16(to + 512, wb + (w + row8));
      if (lane < 4) ir_copy16(to + 1024, (DUAL && (j & 1) ? sb1 : sb0) + (s0 + (td >> 1) * sstep + (td & 1) * 4 * p.Np + f * 64));
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int q = 0; q < S - 1; q++) issue(q, q / N, q / N);
  pdl_wait();

  uint4 xv[2][MG];
  float2 sv[2][MG];
  auto fetch = [&](int z, int td) {
    const uint32_t x = x0 + (td >> 1) * xstep + (td & 1) * xrow;
#pragma unroll
    for (int m = 0; m < MG; m++) {
      xv[z][m] = ir_ldg16(p.xq + (x + xl + m * 512));
      sv[z][m] = ir_ldg8(sxb + (x / 16 + t * 8 + m * 32));
    }
  };
  if (C::AHEAD && cnt > 0) fetch(0, 0);
  float2 acc[N][MG][2];  // [row g, row g + 8] of tokens 2t, 2t + 1
#pragma unroll
  for (int j = 0; j < N; j++)
#pragma unroll
    for (int m = 0; m < MG; m++) acc[j][m][0] = acc[j][m][1] = make_float2(0.0f, 0.0f);
  for (int i = 0; i < cnt; i += D) {
#pragma unroll
    for (int d = 0; d < D; d++) {
      if (i + d >= cnt) break;
      const int z = C::AHEAD ? d & 1 : 0;
      if (!C::AHEAD) fetch(0, d);
      else if (i + d + 1 < cnt) fetch(z ^ 1, d + 1);
#pragma unroll
      for (int j = 0; j < N; j++) {
        constexpr int kZero = 0x4B400000;
        const int q = d * N + j;
        asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
        __syncwarp();  // the scales were copied by other lanes; and all are done with the slot before, which is filled again
        const uint4 a = ir_lds16(own + q * kIrSlot), b = ir_lds16(own + q * kIrSlot + 512);
        const float sw0 = ir_lds4(ring + q * kIrSlot + 1024 + g * 4), sw1 = ir_lds4(ring + q * kIrSlot + 1056 + g * 4);
        issue(q + S - 1, (q + S - 1) / N, i + (q + S - 1) / N);
        if (T % N != 0 && first + j >= T) continue;
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
  // the groups' sums, in their order
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  float* part_sums = reinterpret_cast<float*>(ir_smem_raw);
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
        if (T % N != 0 && first + j >= T) continue;
        float* o = part_sums + ((size_t)(warp % GS) * MG * 8 + m * 8 + 2 * t) * RP + (first + j) * 16 + g;
        o[0] = acc[j][m][0].x;
        o[RP] = acc[j][m][0].y;
        o[8] = acc[j][m][1].x;
        o[RP + 8] = acc[j][m][1].y;
      }
  __syncthreads();
  constexpr int R = 16 * TF;
  const int skip = (tile_own - tile0) * 16, outs = R * p.t.M;
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
    const size_t o = (size_t)tok * p.t.N + n;
    if (p.t.bias) v += bf16_bits_to_f32(p.t.bias[n]);
    if (p.t.act) v = apply_act(v, p.t.act);
    if (DUAL) v *= u;
    if (p.t.mul_in) v *= bf16_bits_to_f32(p.t.mul_in[o]);
    if (p.t.res) v += bf16_bits_to_f32(p.t.res[o]) * p.t.res_scale;
    p.t.y[o] = f32_to_bf16_bits(v);
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
      v += ir_ld_member(at, c);
      if (DUAL) u += ir_ld_member(at + 64, c);
    }
    finish(idx, v, u);
  }
  tc_cluster_sync();  // nobody leaves before all have read
}

template <int T, int MG, bool DUAL>
static int ir_launch(const I8RowsParams& p, cudaStream_t st) {
  constexpr size_t smem = IrCfg<T, MG>::SMEM;
  static bool opted[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16 || !opted[dev]) {
    TPX_CUDA_OK(cudaFuncSetAttribute(qlinear_i8_rows_kernel<T, MG, DUAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    if (dev >= 0 && dev < 16) opted[dev] = true;
  }
  constexpr int TF = DUAL ? T / 2 : T;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((p.tiles + TF - 1) / TF * p.t.cluster));
  cfg.blockDim = dim3(IrCfg<T, MG>::W * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = knobs().pdl;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)p.t.cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = p.t.cluster > 1 ? 2 : 1;
  count_launch();
  TPX_CUDA_OK(cudaLaunchKernelEx(&cfg, qlinear_i8_rows_kernel<T, MG, DUAL>, p));
  return TPX_OK;
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

// Feature tiles per CTA: one round of CTAs where that takes at most seven each, else the fewest rounds.
static int ir_tiles(int64_t tiles) {
  const int sms = sm_count();
  int64_t tf = (tiles + sms - 1) / sms;
  if (tf > 7) {
    const int64_t rounds = (tiles + 7 * sms - 1) / (7 * sms);
    tf = (tiles + rounds * sms - 1) / (rounds * sms);
  }
  return tf < 1 ? 1 : (int)tf;
}

// Blocks of 64, up to 32 tokens; a pair up to 16 (its two sums do not fit in registers above). Seven tiles per CTA leave too few warps per tile above 16
// tokens: 14336 x 4096 at 32 tokens 21.0 us here, 19.7 on the tcgen05 kernel; six tiles (12288 x 4096) 18.7 / 19.3, one (2048 x 8192) 10.1 / 14.0.
bool i8_rows_serves(int64_t M, int64_t N, int64_t block, bool pair) {
  return block == 64 && (M <= 16 || (M <= 32 && !pair && ir_tiles(N / 16) < 7));
}

int i8_rows_launch(I8RowsParams p, bool pair, cudaStream_t st) {
  const int sms = sm_count(), tf = ir_tiles(p.tiles);
  // few tiles: a cluster cuts k, as far as each warp keeps a pair of blocks
  int c = tf == 1 ? sms / p.tiles : 1;
  while (c > 1 && p.nkb < 32 * c) c--;
  p.t.cluster = c >= 8 ? 8 : c >= 4 ? 4 : c >= 2 ? 2 : 1;
  return p.t.M <= 8 ? ir_launch_t<1>(p, pair, tf, st) : p.t.M <= 16 ? ir_launch_t<2>(p, pair, tf, st) : ir_launch_t<4>(p, pair, tf, st);
}

}  // namespace tpx

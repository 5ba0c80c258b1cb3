// bf16 linear of few tokens: the weight streams through private rings of every warp, mma.sync beside it. Same results as linear_bf16_kernel
// (tpx_linear_bf16.cu) up to the order of its fp32 sums, all its epilogues.
//
// A large weight comes at 0.88 to 0.94 of HBM's rate at one token, 0.80 to 0.88 at 16; a small one (4096 x 4096 0.74, 2048 x 2048 0.43) is a launch's start and end in the chain and
// the wait for the first activations. A CTA has T tiles of 16 features (T: one round of CTAs) and all of K; its KG groups of warps take the 64-wide k blocks (a 128-byte line of a row) in
// turn, H warps of a group N tiles each. A lane copies (cp.async) exactly the 16-byte pieces that it feeds to its MMAs, k being permuted inside a block
// for both operands: no barrier in the loop, 25 instructions per 2 KB. Activations come straight from L2 to registers, a block ahead. The tcgen05 form streams a
// large weight as fast, but a decode step is a chain of small ones, and there it pays for tensor memory, tensor maps, tiles of 128 features cut between CTAs and put
// together over memory. Recorded chains of calls, us, tcgen05 / here (floor), 1 and 16 tokens: 2048 x 2048 8.2 / 3.0 and 8.2 / 3.8 (1.3), 4096 x 4096 13.2 / 6.9 and
// 13.4 / 8.1 (5.1), 4096 x 14336 25.6 / 19.2 and 25.5 / 21.1 (18.0), 14336 x 4096 25.2 / 20.4 and 25.4 / 22.5, 32000 x 4096 44.9 / 42.6 and 45.3 / 45.5 (40.1); 24 tokens
// 4096 x 4096 18.0 / 9.5.
#include "tpx_bf16_pair.cuh"
#include "tpx_rows.cuh"

namespace tpx {

constexpr int kBrWarps = 16, kBrSlot = 2048;  // 16 features x 64 values
constexpr int kBrSlots = 4;  // of a warp's ring, where a k block has no more tiles: 128 KB per SM (three or four: the same to 1 %)

template <int H, int N, int MG>
struct BrCfg {
  static constexpr int KG = kBrWarps / H, D = N >= kBrSlots ? 1 : (kBrSlots + N - 1) / N, S = D * N;  // D: k blocks in the ring
  static constexpr size_t RING = (size_t)kBrWarps * S * kBrSlot, PARTS = (size_t)KG * MG * 8 * (16 * H * N + 4) * 4;
  static constexpr size_t SMEM = RING > PARTS ? RING : PARTS;
  static_assert(SMEM <= 225 * 1024, "shared memory");
};

struct BrParams {
  BfParams b;  // epilogue, t.M, t.N, t.K, t.cluster
  const uint16_t *w, *x;
  long long ldw, ldx;
  int T, tiles;  // tiles per CTA; of the call
};

__device__ __forceinline__ void br_mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void br_copy16(uint32_t dst, const void* src, bool in) {  // zeros behind the end of k
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}

// One output (of gated units: both halves, at the even feature), as bf_finish16_ex, bf_finish16_glu and tc_finish16 do sixteen.
__device__ __forceinline__ void br_finish(const BfParams& p, int tok, int n, float v, float u) {
  const BfEx& e = p.ex;
  if (!e.on) {
    const TcParams& t = p.t;
    const size_t o = (size_t)tok * t.N + n;
    if (t.bias) v += bf16_bits_to_f32(t.bias[n]);
    if (t.act) v = apply_act(v, t.act);
    if (t.mul_in) v *= bf16_bits_to_f32(t.mul_in[o]);
    if (t.res) v += bf16_bits_to_f32(t.res[o]) * t.res_scale;
    t.y[o] = f32_to_bf16_bits(v);
    return;
  }
  if (e.bias) v += e.bias[n];
  if (e.x_out) {
    const float s = e.res[(long long)tok * e.ldr + n] + v + (e.add ? e.add[n] : 0.0f);
    e.x_out[(long long)tok * e.ldr + n] = s;
    e.h[(long long)tok * e.ldh + n] = f32_to_bf16_bits(fmaf(tanhf(e.nalpha * s), e.nw[n], e.nb[n]));
    return;
  }
  if (e.act && n >= e.act_from) {
    if (e.act == TPX_ACT_CLAMPED_GLU) {
      if (n & 1) return;
      if (e.bias) u += e.bias[n + 1];
      e.z[(long long)tok * e.ldz + (n - e.act_from) / 2] = f32_to_bf16_bits(hy_clamped_glu_fast(v, u, e.limit));
      return;
    }
    v = hy_act(v, e.act, e.ap ? e.ap[0] : 0.0f, e.ap ? e.ap[1] : 0.0f);
  }
  if (e.out_f32) reinterpret_cast<float*>(e.y)[(long long)tok * e.ldy + n] = v;
  else reinterpret_cast<uint16_t*>(e.y)[(long long)tok * e.ldy + n] = f32_to_bf16_bits(v);
}

template <int H, int N, int MG>
__global__ void __launch_bounds__(kBrWarps * 32, 1) linear_bf16_rows_kernel(const __grid_constant__ BrParams p) {
  using C = BrCfg<H, N, MG>;
  constexpr int KG = C::KG, D = C::D, S = C::S;
  extern __shared__ __align__(16) unsigned char br_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int csize = p.b.t.cluster, crank = csize > 1 ? (int)tc_cluster_rank() : 0;
  const int T = p.T, M = p.b.t.M, K = p.b.t.K, F = p.b.t.N;
  // the last CTA starts early enough to have all its tiles, and stores those that are its own
  const int tile_own = (int)blockIdx.x / csize * T, tile0 = min(tile_own, p.tiles - T);
  const int first = warp / KG * N, groups = KG * csize, turn = crank * KG + warp % KG;
  const int blocks = (K + 63) / 64, cnt = blocks > turn ? (blocks - turn + groups - 1) / groups : 0;
  const uint32_t own = tc_smem_u32(br_smem) + warp * (S * kBrSlot) + lane * 16;
  // rows g and g + 8 of this warp's tiles, offsets from the CTA's first row; rows behind the last feature repeat it
  const uint16_t* const wb = p.w + (long long)tile0 * 16 * p.ldw;
  uint32_t row[N][2];
#pragma unroll
  for (int j = 0; j < N; j++)
#pragma unroll
    for (int e = 0; e < 2; e++) row[j][e] = (uint32_t)(min((first + j) * 16 + g + e * 8, F - 1 - tile0 * 16) * p.ldw) + t * 8;
  pdl_trigger();

  // slot q of the ring, k block `ord` of this warp's
  auto issue = [&](int q, int ord) {
    const int j = q % N;
    if (ord < cnt && first + j < T) {
      const uint32_t to = own + q % S * kBrSlot;
      const int k = (ord * groups + turn) * 64;
      const bool in0 = k + t * 8 < K, in1 = k + 32 + t * 8 < K;
      const uint16_t *a = wb + (row[j][0] + k), *b = wb + (row[j][1] + k);
      br_copy16(to, in0 ? a : wb, in0);
      br_copy16(to + 512, in1 ? a + 32 : wb, in1);
      br_copy16(to + 1024, in0 ? b : wb, in0);
      br_copy16(to + 1536, in1 ? b + 32 : wb, in1);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int q = 0; q < S - 1; q++) issue(q, q / N);
  pdl_wait();

  constexpr bool AHEAD = MG <= 2;  // a block ahead in registers of their own; else asked for when the block's last tile is done
  uint4 xv[AHEAD ? 2 : 1][MG][2];
  auto fetch = [&](uint4 (&x)[MG][2], int ord) {
    const int k = (ord * groups + turn) * 64 + t * 8;
#pragma unroll
    for (int m = 0; m < MG; m++)
#pragma unroll
      for (int e = 0; e < 2; e++)
        x[m][e] = m * 8 + g < M && k + e * 32 < K ? rows_ldg16(p.x + (long long)(m * 8 + g) * p.ldx + k + e * 32) : make_uint4(0, 0, 0, 0);
  };
  if (cnt > 0) fetch(xv[0], 0);
  float acc[N][MG][4];
#pragma unroll
  for (int j = 0; j < N; j++)
#pragma unroll
    for (int m = 0; m < MG; m++)
#pragma unroll
      for (int e = 0; e < 4; e++) acc[j][m][e] = 0.0f;
  constexpr int U = D % 2 ? 2 * D : D;  // blocks per round of the loop: whole rings, and activations in turn in two places
  for (int i = 0; i < cnt; i += U) {
#pragma unroll
    for (int d = 0; d < U; d++) {
      if (i + d >= cnt) break;
      const uint4(&x)[MG][2] = xv[AHEAD ? d & 1 : 0];
      if (AHEAD && i + d + 1 < cnt) fetch(xv[(d & 1) ^ 1], i + d + 1);
#pragma unroll
      for (int j = 0; j < N; j++) {
        const int q = d * N + j;
        asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
        const uint32_t at = own + q % S * kBrSlot;
        const uint4 a0 = rows_lds16(at), a1 = rows_lds16(at + 512), b0 = rows_lds16(at + 1024), b1 = rows_lds16(at + 1536);
        issue(q + S - 1, i + (q + S - 1) / N);  // the slot before, which this lane alone reads
#pragma unroll
        for (int m = 0; m < MG; m++) {
          br_mma(acc[j][m], a0.x, b0.x, a0.y, b0.y, x[m][0].x, x[m][0].y);
          br_mma(acc[j][m], a0.z, b0.z, a0.w, b0.w, x[m][0].z, x[m][0].w);
        }
#pragma unroll
        for (int m = 0; m < MG; m++) {
          br_mma(acc[j][m], a1.x, b1.x, a1.y, b1.y, x[m][1].x, x[m][1].y);
          br_mma(acc[j][m], a1.z, b1.z, a1.w, b1.w, x[m][1].z, x[m][1].w);
        }
      }
      if (!AHEAD && i + d + 1 < cnt) fetch(xv[0], i + d + 1);
    }
  }
  // the groups' sums, in their order
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const int RP = 16 * T + 4, R = 16 * T;  // a token's row is 4 banks past a multiple of 16
  float* part = reinterpret_cast<float*>(br_smem);
#pragma unroll
  for (int j = 0; j < N; j++)
#pragma unroll
    for (int m = 0; m < MG; m++) {
      if (first + j >= T) continue;
      float* o = part + ((warp % KG) * MG * 8 + m * 8 + 2 * t) * RP + (first + j) * 16 + g;
      o[0] = acc[j][m][0];
      o[RP] = acc[j][m][1];
      o[8] = acc[j][m][2];
      o[RP + 8] = acc[j][m][3];
    }
  __syncthreads();
  const int skip = (tile_own - tile0) * 16, outs = R * M;
  const bool glu = p.b.ex.on && p.b.ex.act == TPX_ACT_CLAMPED_GLU;
  auto sum = [&](const float* s) {
    float v = 0.0f;
#pragma unroll
    for (int w = 0; w < KG; w++) v += s[w * MG * 8 * RP];
    return v;
  };
  if (csize == 1) {
    for (int idx = threadIdx.x; idx < outs; idx += kBrWarps * 32) {
      const int tok = idx / R, r = idx - tok * R, n = tile0 * 16 + r;
      const float* s = part + tok * RP + r;
      if (r >= skip && n < F) br_finish(p.b, tok, n, sum(s), glu && !(r & 1) ? sum(s + 1) : 0.0f);
    }
    return;
  }
  // each member sums over its own groups, then takes its turn at adding the members' sums over distributed shared memory
  for (int idx = threadIdx.x; idx < outs; idx += kBrWarps * 32) {
    float* s = part + idx / R * RP + idx % R;
    s[0] = sum(s);
  }
  tc_cluster_sync();
  for (int idx = crank * kBrWarps * 32 + threadIdx.x; idx < outs; idx += csize * kBrWarps * 32) {
    const int tok = idx / R, r = idx - tok * R, n = tile0 * 16 + r;
    const uint32_t at = tc_smem_u32(part + tok * RP + r);
    float v = 0.0f, u = 0.0f;
    for (int c = 0; c < csize; c++) {
      v += rows_ld_member(at, c);
      if (glu && !(r & 1)) u += rows_ld_member(at + 4, c);
    }
    if (r >= skip && n < F) br_finish(p.b, tok, n, v, u);
  }
  tc_cluster_sync();  // nobody leaves before all have read
}

template <int H, int N, int MG>
static int br_launch(const BrParams& p, cudaStream_t st) {
  using C = BrCfg<H, N, MG>;
  static bool opted[16] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 16 || !opted[dev]) {
    TPX_CUDA_OK(cudaFuncSetAttribute(linear_bf16_rows_kernel<H, N, MG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM));
    if (dev >= 0 && dev < 16) opted[dev] = true;
  }
  return rows_launch(linear_bf16_rows_kernel<H, N, MG>, (p.tiles + p.T - 1) / p.T, p.b.t.cluster, kBrWarps * 32, C::SMEM, st, p);
}

template <int MG>
static int br_launch_t(const BrParams& p, cudaStream_t st) {
  constexpr int MOST = MG == 4 ? 3 : 5;  // tiles whose sums a warp has registers for
  const int T = p.T, H = T <= MOST ? 1 : T <= 2 * MOST ? 2 : 4, N = (T + H - 1) / H;
  if (H == 1) {
    if (N == 1) return br_launch<1, 1, MG>(p, st);
    if (N == 2) return br_launch<1, 2, MG>(p, st);
    if (N == 3) return br_launch<1, 3, MG>(p, st);
    if constexpr (MOST > 3) return N == 4 ? br_launch<1, 4, MG>(p, st) : br_launch<1, 5, MG>(p, st);
  }
  if (H == 2) {
    if constexpr (MOST == 3) {
      if (N == 2) return br_launch<2, 2, MG>(p, st);
    }
    if (N == 3) return br_launch<2, 3, MG>(p, st);
    if constexpr (MOST > 3) return N == 4 ? br_launch<2, 4, MG>(p, st) : br_launch<2, 5, MG>(p, st);
  }
  if constexpr (MOST == 3) return br_launch<4, 2, MG>(p, st);  // up to eight tiles
  else return N == 3 ? br_launch<4, 3, MG>(p, st) : N == 4 ? br_launch<4, 4, MG>(p, st) : br_launch<4, 5, MG>(p, st);
}

// As many tiles per CTA as this kernel streams no slower than the tcgen05 one, which needs no more time for 16 tokens than for one. Chains, us, tcgen05 / here: 1 token 40960 x 4096
// (18 tiles) 55.9 / 54.1, the longest weights even (24192 x 11584, 11 tiles, 88.4 / 89.3; at 8 tokens 88.6 / 92.3); 16 tokens 20608 x 4096 (9) 32.0 / 30.4, 25600 x 5120 (11) 46.1 / 45.1, but 24192 x 8192 65.1 / 68.9; 32 tokens
// 16384 x 8192 (7) 54.1 / 52.5, but 16384 x 512 7.4 / 8.2, 11008 x 512 (5) 6.4 / 6.8 (x 1024 17.2 / 9.3), 8192 x 20480 (4) 62.5 / 65.4 (x 14336 47.7 / 43.9). Where the tcgen05
// kernel has a tile for every SM, so that none is cut, it is the faster one above 8 tokens: 18944 x 3584 at 8, 16 and 32 tokens 23.4 / 22.8, 23.3 / 24.6 and 25.1 / 28.2.
bool bf_rows_serves(int64_t M, int64_t N, int64_t K, int64_t ldw) {
  const int64_t sms = sm_count(), T = ((N + 15) / 16 + sms - 1) / sms;
  if (M > 32 || T > 20 || 336 * ldw + K >= (1ll << 31)) return false;
  if (M <= 8) return true;
  if ((N + 127) / 128 == sms) return false;
  if (M <= 16) return T <= 8 || (T <= 12 && K <= 6144);
  return T <= 3 || (T <= 8 && K <= 16384 && (T <= 4 || K >= 1024));
}

int bf_rows_run(const BfParams& b, const void* w, const void* x, int64_t M, int64_t N, int64_t K, int64_t ldw, int64_t ldx, cudaStream_t st) {
  BrParams p = {};
  p.b = b;
  p.b.t.M = (int)M; p.b.t.N = (int)N; p.b.t.K = (int)K;
  p.w = (const uint16_t*)w; p.x = (const uint16_t*)x; p.ldw = ldw; p.ldx = ldx;
  const int sms = sm_count();
  p.tiles = (int)((N + 15) / 16);
  p.T = (p.tiles + sms - 1) / sms;
  int c = p.T == 1 ? sms / p.tiles : 1;  // few tiles: a cluster cuts k, as far as each warp keeps a block
  while (c > 1 && (K + 63) / 64 < kBrWarps * c) c--;
  p.b.t.cluster = c >= 8 ? 8 : c >= 4 ? 4 : c >= 2 ? 2 : 1;
  return M <= 8 ? br_launch_t<1>(p, st) : M <= 16 ? br_launch_t<2>(p, st) : br_launch_t<4>(p, st);
}

}  // namespace tpx

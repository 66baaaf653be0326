// The three sums over the heads of a group in the backward of the SSD scan, as one kernel over tiles of one step (128 tokens) of
// one group (mamba2/ssd_ops.rs:201-234 and its autograd compute the same quantities op by op):
//   dG[t,s] = sum_h exp(S_h,t - S_h,s) [s <= t] <dY_h,t, x~_h,s>
//   dC[t,:] = dG B   + sum_h exp(S_h,t)            dY_h,t h_h      (h = state entering the step)
//   dB[s,:] = dG^T C + sum_h exp(S_h,end - S_h,s)  x~_h,s dh_h     (dh = adjoint of the state leaving it)
// Per head the tensor core forms dY x~^T, dY h^T and x~ dh^T from four tiles; the decays are applied where the products are added
// up in registers, so no copy of dY or x~ scaled by them exists and dG never leaves the SM.  With few tiles the heads of a group
// are split over CTAs; dC and dB are linear in dG, so every CTA finishes its own heads' share and the shares are added in a fixed
// order (heads_sum_kernel).
//
// warp 0 = TMA, 1 = MMA issuer, 2 = S of the heads, then dG (eight warps with 64 columns per thread; d_state above 64: four with 128), four of
// dC and four of dB (all of d_state).  Two or three operand stages, two accumulators of dG; dC and dB have two up to 64 states, the
// products of the next head running under the sums of this one, and one above, where the next head's dG product runs ahead instead.
// What bounds it: the operands' bytes, half of HBM's rate, and the latency of a head's chain (product, TMEM load, sum, hand-over).  Bf16, 8 x 4096
// tokens, 32 heads of 128 x 64: 197 us when d_state was taken in two passes over the heads (826 MB read) and dG's warps took nine instructions
// per element one by one; 235 in one pass (558 MB) with half as many dG warps: theirs was the longest chain; 150 now that exponents and sums go
// in pairs (12 to 15 % less with decays below 2^-126 as zeros, whose scaling doubles the operations of a pair; a test by 16 columns or by heads that skips it
// where no decay is that small cost more than it saved).  16 x 1024 of 64 x 64: 55 us; 16 x 8192 of 128 x 64: 512.
// (Three stages instead of two, a warp index from a shuffle and a look at the barrier before a wait brought 836 to 680 before.)
// At 24 heads of 64 x 64 on pairs, 4 x 512 tokens: 17 us + 4 us for the sum of the shares.
#include <cuda_bf16.h>
#include "tc_common.cuh"
#include "kernels.h"
#include "ssd_fused.h"

namespace pmb {

static __device__ unsigned int g_heads_status = 0;

pmb_status read_clear_device_status_heads(unsigned int* word) {
  unsigned int zero = 0;
  PMB_CUDA(cudaMemcpyFromSymbol(word, g_heads_status, sizeof(unsigned int)));
  if (*word) PMB_CUDA(cudaMemcpyToSymbol(g_heads_status, &zero, sizeof(unsigned int)));
  return PMB_OK;
}

namespace shd {

using namespace tcx;

constexpr int L = SCAN_STEP, T128 = L * 128, T64 = 64 * 128;

// NK = 64-wide blocks of d_state, all of them in one pass over the heads.
template <int NI, int ND, int NK>
struct Geo {
  // warps of dG, then four each of dC and dB; with two blocks their threads have 128 sums each, and there are half as many for dG
  static constexpr int GW = NK == 2 ? 4 : 8, W_G = 4, W_C = W_G + GW, NTHREADS = 32 * (W_C + 8);
  static constexpr int GC = L * 4 / GW, CC = 64 * NK;      // columns per thread
  static constexpr int CB = NK == 2 ? 1 : 2;               // accumulators of dC and dB (TMEM: two of 128 columns for dG, the rest is theirs)
  static constexpr int XT = NI * T128, HT = ND * NK * T64, BT = NI * NK * T128;
  static constexpr int STAGE = 2 * XT + 2 * HT;            // [dY | x~ | h | dh]; in the end [B | C]
  static constexpr int DG = ND * 2 * T128;                        // dG as an operand: two 64-column tiles (hi), then lo
  static constexpr bool OWN_DG = NI == 1 && NK == 1;       // otherwise dG goes over the stage that the last head has left
  static constexpr int RING = 4;                           // heads whose S is in shared memory
  static constexpr int STG = NI == 1 && ND == 1 ? 3 : 2;   // (what fits)
  static constexpr int TILES = STG * STAGE + (OWN_DG ? DG : 0);
  static_assert((OWN_DG || DG <= STAGE) && 2 * BT <= STAGE, "dG, and B and C, fit a stage");
  static constexpr int SMEM = TILES + 1024 /*alignment slack*/ + 256 /*barriers*/ + RING * L * 4;
};

struct Maps { CUtensorMap dy[2], xt[2], h[2], dh[2], b[2], c[2]; };

struct Params {
  int T, H, G, hpg, N, n, nsplit;
  const float* S;
  float *dc, *db; int64_t ld;                              // token rows, group g at column g * N
  uint16_t *dc16, *db16;                                   // the same as bf16 (instead)
  float* part;                                             // nsplit > 1: [tile][split][dC | dB][128][N]
  unsigned int* status;
};

template <int NI, int ND, int NK>
__global__ void __launch_bounds__(Geo<NI, ND, NK>::NTHREADS, 1) ssd_heads_kernel(const __grid_constant__ Maps maps, const Params p) {
  using GE = Geo<NI, ND, NK>;
  constexpr int W_G = GE::W_G, W_C = GE::W_C, CB = GE::CB;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);
  const uint32_t bars = base + GE::TILES;
  enum { FULL = 0 /*3*/, EMPTY = 3 /*3*/, MFULL = 6 /*2*/, MFREE = 8 /*2*/, CFULL = 10 /*2*/, CFREE = 12 /*2*/, SRDY = 14 /*4*/, SFREE = 18 /*4*/, DGRDY = 22, NBAR };
  static_assert(8 * NBAR + 8 <= 256, "barrier block");
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  uint8_t* bar_ptr = base_ptr + GE::TILES;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bar_ptr + 8 * NBAR);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  float* sS = reinterpret_cast<float*>(bar_ptr + 256);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  int id = (int)blockIdx.x;
  const int split = id % p.nsplit; id /= p.nsplit;
  const int tile = id;
  const int g = id % p.G; id /= p.G;
  const int i = id % p.n, bb = id / p.n;
  const int nh = (p.hpg - split + p.nsplit - 1) / p.nsplit;
  auto head = [&](int j) { return g * p.hpg + split + j * p.nsplit; };
  const int nitems = nh + 1;                                // the heads, then the product with dG
  if (threadIdx.x == 0) {
    for (int q = 0; q < 2; ++q) {
      mbar_init(bar(MFULL + q), 1); mbar_init(bar(MFREE + q), GE::GW);
      mbar_init(bar(CFULL + q), 1); mbar_init(bar(CFREE + q), 8);
    }
    for (int q = 0; q < GE::STG; ++q) { mbar_init(bar(FULL + q), 1); mbar_init(bar(EMPTY + q), 1); }
    for (int q = 0; q < 4; ++q) { mbar_init(bar(SRDY + q), 1); mbar_init(bar(SFREE + q), GE::GW + 8); }
    mbar_init(bar(DGRDY), GE::GW);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "n"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  pdl_launch();
  pdl_wait();
  const uint32_t tM = tmem, tC = tmem + 256, tB = tmem + 384;
  // the stage that dG goes over: the one the last head was in
  const uint32_t dg_s = GE::OWN_DG ? base + GE::STG * GE::STAGE : base + (uint32_t)((nh - 1) % GE::STG) * GE::STAGE;

  auto give_up = [&](unsigned int code) { atomicOr(p.status, code); *abort_flag = 1; };
  auto wait = [&](int b, uint32_t parity, unsigned int code) -> bool {
    if (mbar_wait(bar(b), parity & 1u, 1u)) return true;
    if (*abort_flag) return false;
    if (mbar_wait(bar(b), parity & 1u)) return true;
    give_up(code);
    return false;
  };
  auto all = [&](bool v) -> bool { return __all_sync(0xffffffffu, v); };

  if (warp < W_G) {
  if (NK == 2) regs_dec<40>();
  if (warp == 0) {
    if (lane == 0) {
      int issued = 0;
      for (int m = 0; m < nitems; ++m) {
        const int s = m % GE::STG, j = m;
        if (!wait(EMPTY + s, (uint32_t)(m / GE::STG) ^ 1u, 1u)) break;
        const uint32_t st = base + s * GE::STAGE;
        if (j < nh) {
          const int h = head(j);
          mbar_expect_tx(bar(FULL + s), GE::STAGE);
#pragma unroll
          for (int sp = 0; sp < NI; ++sp) {
            tma_load_4d(st + sp * T128, &maps.dy[sp], 0, i * L, h, bb, bar(FULL + s));
            tma_load_4d(st + GE::XT + sp * T128, &maps.xt[sp], 0, i * L, h, bb, bar(FULL + s));
          }
#pragma unroll
          for (int sp = 0; sp < ND; ++sp)
#pragma unroll
            for (int kt = 0; kt < NK; ++kt) {
              tma_load_4d(st + 2 * GE::XT + (sp * NK + kt) * T64, &maps.h[sp], 0, 64 * kt, h, bb * p.n + i, bar(FULL + s));
              tma_load_4d(st + 2 * GE::XT + GE::HT + (sp * NK + kt) * T64, &maps.dh[sp], 0, 64 * kt, h, bb * p.n + i, bar(FULL + s));
            }
        } else {
          mbar_expect_tx(bar(FULL + s), 2 * GE::BT);
#pragma unroll
          for (int sp = 0; sp < NI; ++sp)
#pragma unroll
            for (int kt = 0; kt < NK; ++kt) {
              tma_load_4d(st + (sp * NK + kt) * T128, &maps.b[sp], 64 * kt, i * L, g, bb, bar(FULL + s));
              tma_load_4d(st + GE::BT + (sp * NK + kt) * T128, &maps.c[sp], 64 * kt, i * L, g, bb, bar(FULL + s));
            }
        }
        issued = m + 1;
      }
      if (*abort_flag)
        for (int m = (issued > GE::STG ? issued - GE::STG : 0); m < issued; ++m) mbar_wait(bar(FULL + m % GE::STG), (uint32_t)((m / GE::STG) & 1));
    }
  } else if (warp == 1) {
    const uint32_t dhi = desc_hi(1024, 2);
    const uint32_t id_m = idesc_bf16(0, 0, L, L), id_h = idesc_bf16(0, 0, L, 64 * NK);      // both operands K-major
    const uint32_t id_c = idesc_bf16(0, 1, L, 64 * NK), id_b = idesc_bf16(1, 1, L, 64 * NK);     // dG B and dG^T C
    const uint32_t XS = T128 >> 4, HS = (NK * T64) >> 4, BS = (NK * T128) >> 4, DS = (2 * T128) >> 4;
    bool ok = true;
#pragma unroll 1
    for (int m = 0; m < nitems && ok; ++m) {
      const int s = m % CB, sg = m % GE::STG;
      const uint32_t st = base + sg * GE::STAGE;
      const uint32_t y0 = desc_lo(st, 16), x0 = desc_lo(st + GE::XT, 16);
      ok = all(wait(FULL + sg, (uint32_t)(m / GE::STG), 2u) && (m >= nh || m < 2 || wait(MFREE + (m & 1), (uint32_t)((m >> 1) - 1), 8u)));
      if (!ok) break;
      if (CB == 1 && m < nh) {                               // (the other products wait for dC and dB of the head before to be taken)
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (elect_one()) {
#pragma unroll
          for (int q = 0; q < 4; ++q) mma_split<NI, NI>(tM + (uint32_t)(128 * (m & 1)), y0 + 2 * q, XS, x0 + 2 * q, XS, dhi, id_m, q ? 1u : 0u);
          umma_commit(bar(MFULL + (m & 1)));
        }
        __syncwarp();
      }
      if (!(ok = all((m < CB || wait(CFREE + s, (uint32_t)(m / CB - 1), 4u)) && (m < nh || wait(DGRDY, 0u, 16u))))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (elect_one()) {
        const uint32_t dC = tC + (uint32_t)(64 * s), dB = tB + (uint32_t)(64 * s);
        if (m < nh) {
          const uint32_t h0 = desc_lo(st + 2 * GE::XT, 16), d0 = desc_lo(st + 2 * GE::XT + GE::HT, 16);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            if (CB == 2) mma_split<NI, NI>(tM + (uint32_t)(128 * (m & 1)), y0 + 2 * q, XS, x0 + 2 * q, XS, dhi, id_m, q ? 1u : 0u);
            mma_split<NI, ND>(dC, y0 + 2 * q, XS, h0 + 2 * q, HS, dhi, id_h, q ? 1u : 0u);
            mma_split<NI, ND>(dB, x0 + 2 * q, XS, d0 + 2 * q, HS, dhi, id_h, q ? 1u : 0u);
          }
          if (CB == 2) umma_commit(bar(MFULL + (m & 1)));
        } else {
          const uint32_t gk = desc_lo(dg_s, 16), gm = desc_lo(dg_s, T128), b0 = desc_lo(st, T128), c0 = desc_lo(st + GE::BT, T128);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const uint32_t o = (uint32_t)(q * 2048) >> 4;
            mma_split<ND, NI>(dC, gk + ((uint32_t)((q >> 2) * T128 + (q & 3) * 32) >> 4), DS, b0 + o, BS, dhi, id_c, q ? 1u : 0u);
            mma_split<ND, NI>(dB, gm + o, DS, c0 + o, BS, dhi, id_b, q ? 1u : 0u);
          }
        }
        umma_commit(bar(CFULL + s));
        umma_commit(bar(EMPTY + sg));
      }
      __syncwarp();
    }
  } else if (warp == 2) {
    // S of a head's 128 tokens (a = 0 past the end of the sequence)
    for (int m = 0; m < nh; ++m) {
      const int r = m % GE::RING;
      if (m >= GE::RING && !all(wait(SFREE + r, (uint32_t)(m / GE::RING - 1), 32u))) break;
      const float* Sg = p.S + ((int64_t)bb * p.H + head(m)) * p.T;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = i * L + lane + 32 * e;
        sS[r * L + lane + 32 * e] = Sg[t < p.T ? t : p.T - 1];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(SRDY + r));
    }
  }
  } else if (warp < W_C) {
    // ---------------- dG ----------------
    if (NK == 2) regs_inc<152>();
    constexpr int GC = GE::GC;
    const int quarter = warp & 3, grp = (warp - W_G) >> 2, row = quarter * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    F2 acc[GC / 2];
#pragma unroll
    for (int e = 0; e < GC / 2; ++e) acc[e] = 0;
    bool ok = true;
    for (int j = 0; j < nh && ok; ++j) {
      const float* S = sS + (j % GE::RING) * L;
      ok = all(wait(SRDY + (j % GE::RING), (uint32_t)(j / GE::RING), 64u) && wait(MFULL + (j & 1), (uint32_t)(j >> 1), 64u));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float S_row = S[row];
      const F2 Sr2 = pack2(S_row, S_row), neg = pack2(-1.0f, -1.0f), log2e = pack2(1.4426950408889634f, 1.4426950408889634f);
#pragma unroll
      for (int q = 0; q < GC / 16; ++q) {
        const int c0 = grp * GC + 16 * q;
        if (c0 > quarter * 32 + 31) continue;                // every one of these columns is past every row of this warp
        uint32_t v[16];
        tmem_ld16(tM + lane_addr + (uint32_t)(128 * (j & 1) + c0), v);
        F2 w[8];
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
          const ulonglong2 s4 = *reinterpret_cast<const ulonglong2*>(S + c0 + 2 * e);
          w[e] = ex2_two(mul2(fma2(s4.x, neg, Sr2), log2e)); w[e + 1] = ex2_two(mul2(fma2(s4.y, neg, Sr2), log2e));
        }
        if (c0 + 15 > quarter * 32) {                        // (the diagonal may cross)
#pragma unroll
          for (int e = 0; e < 8; ++e) { const float2 u = unpack2(w[e]); w[e] = pack2(c0 + 2 * e <= row ? u.x : 0.0f, c0 + 2 * e + 1 <= row ? u.y : 0.0f); }
        }
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[8 * q + e] = fma2(pack2(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1])), w[e], acc[8 * q + e]);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) { mbar_arrive(bar(MFREE + (j & 1))); mbar_arrive(bar(SFREE + (j % GE::RING))); }
    }
    // (over a stage: when all products of the last head are done)
    if (ok && !GE::OWN_DG && CB == 1) ok = all(wait(CFULL + (nh - 1) % CB, (uint32_t)((nh - 1) / CB), 64u));
    if (ok) {
#pragma unroll
      for (int c = 0; c < GC / 8; ++c) {
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 u = unpack2(acc[4 * c + e]);
          hi[e] = bf16_of_two(u.x, u.y);
          lo[e] = bf16_rest_of_two(u.x, u.y, hi[e]);
        }
        const int cg = grp * (GC / 8) + c;                     // eight columns of the row
        const uint32_t a = dg_s + (uint32_t)((cg >> 3) * T128 + row * 128 + (((cg & 7) ^ (row & 7)) << 4));
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(hi[0]), "r"(hi[1]), "r"(hi[2]), "r"(hi[3]) : "memory");
        if (ND == 2) asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a + 2 * T128), "r"(lo[0]), "r"(lo[1]), "r"(lo[2]), "r"(lo[3]) : "memory");
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(DGRDY));
    }
  } else {
    // ---------------- dC (first four warps) and dB ----------------
    if (NK == 2) regs_inc<152>();
    constexpr int CC = GE::CC;
    const int quarter = warp & 3, which = (warp - W_C) >> 2, row = quarter * 32 + lane;
    const uint32_t src = (which ? tB : tC) + ((uint32_t)(quarter * 32) << 16);
    F2 acc[CC / 2];
#pragma unroll
    for (int e = 0; e < CC / 2; ++e) acc[e] = 0;
    bool ok = true;
    for (int j = 0; j <= nh && ok; ++j) {
      const int s = j % CB;
      float f = 1.0f;
      if (j < nh) {
        ok = all(wait(SRDY + (j % GE::RING), (uint32_t)(j / GE::RING), 128u));
        if (!ok) break;
        const float* S = sS + (j % GE::RING) * L;
        f = __expf(which ? S[L - 1] - S[row] : S[row]);
      }
      ok = all(wait(CFULL + s, (uint32_t)(j / CB), 128u));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const F2 f2 = pack2(f, f);
#pragma unroll
      for (int q = 0; q < CC / 16; ++q) {
        uint32_t v[16];
        tmem_ld16(src + (uint32_t)(64 * s + 16 * q), v);
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 8; ++e) acc[8 * q + e] = fma2(pack2(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1])), f2, acc[8 * q + e]);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) { mbar_arrive(bar(CFREE + s)); if (j < nh) mbar_arrive(bar(SFREE + (j % GE::RING))); }
    }
    const int t = i * L + row;
    if (ok && p.nsplit > 1) {
      float* dst = p.part + ((((int64_t)tile * p.nsplit + split) * 2 + which) * L + row) * p.N;
#pragma unroll
      for (int e = 0; e < CC / 4; ++e) if (4 * e < p.N) store_quad(dst + 4 * e, Quad{acc[2 * e], acc[2 * e + 1]});
    } else if (ok && t < p.T) {
      const int64_t o = ((int64_t)bb * p.T + t) * p.ld + (int64_t)g * p.N;
      uint16_t* o16 = which ? p.db16 : p.dc16;
      if (o16) {
        auto two = [&](int e) { const float2 u = unpack2(acc[e]); return bf16_of_two(u.x, u.y); };
#pragma unroll
        for (int e = 0; e < CC / 8; ++e)
          if (8 * e < p.N) *reinterpret_cast<uint4*>(o16 + o + 8 * e) = make_uint4(two(4 * e), two(4 * e + 1), two(4 * e + 2), two(4 * e + 3));
      } else {
        float* dst = (which ? p.db : p.dc) + o;
#pragma unroll
        for (int e = 0; e < CC / 4; ++e) if (4 * e < p.N) store_quad(dst + 4 * e, Quad{acc[2 * e], acc[2 * e + 1]});
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
  }
}

// Adds the shares of the splits in a fixed order; four columns per thread.
__global__ void __launch_bounds__(256) heads_sum_kernel(const float* __restrict__ part, Params p, int64_t total) {
  pdl_launch();
  pdl_wait();
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= total) return;
  const int n4 = p.N / 4, c = (int)(q % n4); int64_t r = q / n4;
  const int row = (int)(r % L); r /= L;
  const int which = (int)(r & 1); r >>= 1;
  const int g = (int)(r % p.G); const int64_t bi = r / p.G;
  const int t = (int)(bi % p.n) * L + row;
  if (t >= p.T) return;
  const float4* src = reinterpret_cast<const float4*>(part) + ((r * p.nsplit * 2 + which) * L + row) * n4 + c;
  float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
  for (int k = 0; k < p.nsplit; ++k) {
    const float4 v = src[(int64_t)k * 2 * L * n4];
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  const int64_t o = ((bi / p.n) * p.T + t) * p.ld + (int64_t)g * p.N + 4 * c;
  uint16_t* o16 = which ? p.db16 : p.dc16;
  if (o16) *reinterpret_cast<uint2*>(o16 + o) = make_uint2(bf16_of_two(s.x, s.y), bf16_of_two(s.z, s.w));
  else *reinterpret_cast<float4*>((which ? p.db : p.dc) + o) = s;
}

static unsigned int* status_ptr() {
  static unsigned int* known[PMB_MAX_DEVICES] = {nullptr};
  return status_address(g_heads_status, known);
}

template <int NI, int ND, int NK>
static pmb_status launch(cudaStream_t st, const HeadsArgs& a, int nsplit) {
  using GE = Geo<NI, ND, NK>;
  static_assert(GE::SMEM <= 227 * 1024, "shared-memory plan");
  const int n = (int)cdiv(a.T, L);
  Maps ms{};
  for (int sp = 0; sp < 2; ++sp) {
    const bool lo = sp && NI == 2, lod = sp && ND == 2;
    const int64_t st_h = (int64_t)a.N * a.P, hp = (int64_t)a.H * a.P;
    PMB_TRY(sf::bf16_map4(&ms.dy[sp], lo ? a.dy.lo : a.dy.hi, a.P, a.T, a.H, a.B, hp, a.P, a.T * hp, 64, L));
    PMB_TRY(sf::bf16_map4(&ms.xt[sp], lo ? a.xt.lo : a.xt.hi, a.P, a.T, a.H, a.B, hp, a.P, a.T * hp, 64, L));
    PMB_TRY(sf::bf16_map4(&ms.h[sp], lod ? a.hp_lo : a.hp_hi, a.P, a.N, a.H, (int64_t)a.B * n, a.P, st_h, a.H * st_h, 64, 64));
    PMB_TRY(sf::bf16_map4(&ms.dh[sp], lod ? a.dh_lo : a.dh_hi, a.P, a.N, a.H, (int64_t)a.B * n, a.P, st_h, a.H * st_h, 64, 64));
    PMB_TRY(sf::bf16_map4(&ms.b[sp], lo ? a.b.lo : a.b.hi, a.N, a.T, a.G, a.B, a.b.pitch, a.N, (int64_t)a.T * a.b.pitch, 64, L));
    PMB_TRY(sf::bf16_map4(&ms.c[sp], lo ? a.c.lo : a.c.hi, a.N, a.T, a.G, a.B, a.c.pitch, a.N, (int64_t)a.T * a.c.pitch, 64, L));
  }
  Params p{};
  p.T = a.T; p.H = a.H; p.G = a.G; p.hpg = a.H / a.G; p.N = a.N; p.n = n; p.nsplit = nsplit;
  p.S = a.S; p.dc = a.dc; p.db = a.db; p.ld = a.ld; p.dc16 = a.dc16; p.db16 = a.db16; p.part = a.part; p.status = status_ptr();
  const int64_t tiles = (int64_t)a.B * n * a.G;
  PMB_SMEM_OPT_IN(GE::SMEM, ssd_heads_kernel<NI, ND, NK>);
  PMB_TRY(launch_pdl(st, ssd_heads_kernel<NI, ND, NK>, dim3((unsigned)((tiles * nsplit))), GE::NTHREADS, GE::SMEM, ms, p));
  if (nsplit > 1) {
    const int64_t total = tiles * 2 * L * (a.N / 4);
    PMB_TRY(launch_pdl(st, heads_sum_kernel, dim3((unsigned)cdiv(total, 256)), 256, 0, a.part, p, total));
  }
  return PMB_OK;
}

}  // namespace shd

// One CTA per SM: as many splits as fill the machine once, then the fewest with the same number of heads per CTA.
int ssd_heads_nsplit(int B, int T, int H, int G) {
  const int64_t tiles = (int64_t)B * cdiv(T, SCAN_STEP) * G;
  const int hpg = H / G;
  int want = tiles >= 148 ? 1 : (int)(148 / tiles);
  if (want > hpg) want = hpg;
  const int per = (int)cdiv(hpg, want);
  return (int)cdiv(hpg, per);
}
size_t ssd_heads_part_floats(int B, int T, int H, int N, int G) {
  const int ns = ssd_heads_nsplit(B, T, H, G);
  return ns > 1 ? (size_t)B * cdiv(T, SCAN_STEP) * G * ns * 2 * SCAN_STEP * N : 0;
}

pmb_status ssd_heads(cudaStream_t st, const HeadsArgs& a) {
  const bool pairs = a.b.lo != nullptr;
  if (!ssd_chain_bwd_shape(a.P, a.N, pairs) || a.H % a.G != 0) return fail(PMB_ERR_UNSUPPORTED, "ssd_heads: unsupported shape (P=%d N=%d)", a.P, a.N);
  if ((a.dy.lo != nullptr) != pairs || (a.xt.lo != nullptr) != pairs) return fail(PMB_ERR_ARG, "ssd_heads: operands must be all pairs or all plain bf16");
  const int nsplit = ssd_heads_nsplit(a.B, a.T, a.H, a.G);
  const int64_t tiles = (int64_t)a.B * cdiv(a.T, SCAN_STEP) * a.G;
  if (tiles * nsplit > 0x7fffffff) return fail(PMB_ERR_SHAPE, "ssd_heads: too many tiles");
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (!al16(a.dc) || !al16(a.db) || !al16(a.dc16) || !al16(a.db16) || !al16(a.part) || (a.ld & (a.dc16 ? 7 : 3))) return fail(PMB_ERR_SHAPE, "ssd_heads: dB and dC rows must be 16-byte aligned");
  const double tok = (double)a.B * a.T;
  ProfScope prof(st, "ssd_heads", tok * (a.H * ((double)SCAN_STEP * a.P + 4.0 * a.N * a.P) + 2.0 * a.G * SCAN_STEP * a.N), 0.0);
  if (pairs) return shd::launch<2, 2, 1>(st, a, nsplit);      // (d_state up to 64)
  if (a.N > 64) return a.hp_lo ? shd::launch<1, 2, 2>(st, a, nsplit) : shd::launch<1, 1, 2>(st, a, nsplit);
  return a.hp_lo ? shd::launch<1, 2, 1>(st, a, nsplit) : shd::launch<1, 1, 1>(st, a, nsplit);
}

}  // namespace pmb

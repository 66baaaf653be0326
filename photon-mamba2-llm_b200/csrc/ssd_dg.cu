// dG[t,s] = sum over the heads of a group of exp(S_h,t - S_h,s) <dY_h,t, x~_h,s>  [s <= t],  per (batch, chunk, group): the gradient w.r.t.
// C B^T of a chunked scan (mamba2/ssd_ops.rs:83-138 backwards), on plain bf16 operands or (hi, lo) pairs, chunks that are multiples of 128.
// One CTA owns a 128 x 128 tile on or below the diagonal and walks the heads: operands and S by TMA into a ring, the product into one of two
// TMEM buffers, and sixteen warps fold it, times that head's decay, into sums that stay in registers (heads in ascending order).
// warp 0 = TMA, warp 1 = MMAs (one elected lane), warps 2..17 = sums: a warp has 32 rows and 32 columns.
// Bound by the exponentials: 16 per clock and SM.  A warp may read one quarter of TMEM's lanes only, which is also one scheduler; with the
// tile's rows in order the quarters of a tile on the diagonal would have one to four blocks of it to compute.  So the rows are dealt to the lanes in
// groups of eight (lane 32 q + 8 i + r = row 32 i + 8 q + r, a rank-5 tensor map): every quarter has the same 10/16 of a diagonal tile.
// 16384 tokens of 24 heads, chunks of 256 (192 tiles on 148 SMs): 45 us, 95 as a contraction whose warps loaded each head's S between two barriers;
// 8192 tokens 25; pairs, 8192 tokens of 16 heads 24 (58).
#include <cuda_bf16.h>
#include <type_traits>
#include "tc_common.cuh"
#include "kernels.h"
#include "ssd_fused.h"

namespace pmb {
namespace sdg {

using namespace tcx;

constexpr int L = 128, NSUMW = 16, NTHREADS = 64 + 32 * NSUMW, T128 = L * 128;

template <int NS> struct Geo {
  static constexpr int STAGE = 2 * NS * T128 + 2 * L * 4;   // [dY | x~] (hi, then lo), S of the rows and of the columns
  static constexpr int PITCH = 2 * NS * T128 + 1024;        // (tiles start 1024-byte aligned)
  static constexpr int STAGES = NS == 1 ? 4 : 3;
  static constexpr int SMEM = STAGES * PITCH + 1024 + 256;
};

struct Maps { CUtensorMap a[2], b[2]; };
struct Params {
  int H, hpg, G, Q, nc, T, nsplit, noff;
  const float* S;
  float* part;                                              // nsplit > 1: (batch, chunk, group, split, Q, Q)
  uint16_t *dg_hi, *dg_lo;
  unsigned int* status;
};

template <int NS>
__global__ void __launch_bounds__(NTHREADS, 1) ssd_dg_kernel(const __grid_constant__ Maps maps, const Params p) {
  using GE = Geo<NS>;
  constexpr int STAGES = GE::STAGES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t ring = (raw + 1023u) & ~1023u, bars = ring + STAGES * GE::PITCH;
  uint8_t* ring_ptr = smem_raw + (ring - raw);
  enum { FULL = 0, EMPTY = STAGES, GFULL = 2 * STAGES, GFREE = GFULL + 2, NBAR = GFREE + 2 };
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(ring_ptr + STAGES * GE::PITCH + 8 * NBAR);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  // tiles below the diagonal come first, they are the longer ones
  int mt = (int)blockIdx.y - p.noff, nt = mt;
  if (mt < 0) { int k = (int)blockIdx.y; mt = 1; while (k >= mt) { k -= mt; ++mt; } nt = k; }
  const int split = (int)blockIdx.x % p.nsplit, bcg = (int)blockIdx.x / p.nsplit, g = bcg % p.G, bc = bcg / p.G, cc = bc % p.nc, bb = bc / p.nc;
  const int tok0 = bc * p.Q, m0 = mt * L, n0 = nt * L;
  const int nh = (p.hpg - split + p.nsplit - 1) / p.nsplit;
  auto head = [&](int j) { return g * p.hpg + split + j * p.nsplit; };
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(bar(FULL + s), 1); mbar_init(bar(EMPTY + s), 1 + NSUMW); }
    for (int i = 0; i < 2; ++i) { mbar_init(bar(GFULL + i), 1); mbar_init(bar(GFREE + i), NSUMW); }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "n"(2 * L) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  auto give_up = [&](unsigned int code) { atomicOr(p.status, code); *abort_flag = 1; };
  // bounded waits that also end as soon as another role of the CTA has given up
  auto wait = [&](int b, uint32_t parity, unsigned int code) -> bool {
    if (*abort_flag) return false;
    if (mbar_wait(bar(b), parity & 1u)) return true;
    give_up(code);
    return false;
  };

  if (warp == 0) {
    if (lane == 0) {
      int issued = 0;
      for (int j = 0; j < nh; ++j) {
        const int s = j % STAGES, h = head(j);
        if (!wait(EMPTY + s, (uint32_t)(j / STAGES) ^ 1u, 1u)) break;
        mbar_expect_tx(bar(FULL + s), GE::STAGE);
        const uint32_t dst = ring + s * GE::PITCH;
#pragma unroll
        for (int sp = 0; sp < NS; ++sp) {
          tma_load_5d(dst + 2 * sp * T128, &maps.a[sp], 0, 0, (tok0 + m0) / 32, 0, h, bar(FULL + s));
          tma_load_3d(dst + (2 * sp + 1) * T128, &maps.b[sp], 0, tok0 + n0, h, bar(FULL + s));
        }
        const float* Sp = p.S + ((int64_t)bb * p.H + h) * p.T + (int64_t)cc * p.Q;
        bulk_load(dst + 2 * NS * T128, Sp + m0, L * 4, bar(FULL + s));
        bulk_load(dst + 2 * NS * T128 + L * 4, Sp + n0, L * 4, bar(FULL + s));
        issued = j + 1;
      }
      if (*abort_flag)
        for (int j = (issued > STAGES ? issued - STAGES : 0); j < issued; ++j) mbar_wait(bar(FULL + j % STAGES), (uint32_t)((j / STAGES) & 1));
    }
  } else if (warp == 1) {
    auto wait_all = [&](int b, uint32_t parity, unsigned int code) -> bool { return __all_sync(0xffffffffu, wait(b, parity, code)); };
    const uint32_t dh = desc_hi(1024, 2), id = idesc_bf16(0, 0, L, L);
    for (int j = 0; j < nh; ++j) {
      const int s = j % STAGES, b = j & 1;
      if (!wait_all(FULL + s, (uint32_t)(j / STAGES), 2u) || (j >= 2 && !wait_all(GFREE + b, (uint32_t)(j >> 1) - 1u, 4u))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t a0 = desc_lo(ring + s * GE::PITCH, 16), b0 = desc_lo(ring + s * GE::PITCH + T128, 16);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          mma_split<NS, NS>(tmem + (uint32_t)(b * L), a0 + ((k * 32) >> 4), (2 * T128) >> 4, b0 + ((k * 32) >> 4), (2 * T128) >> 4, dh, id, k ? 1u : 0u);
        umma_commit(bar(GFULL + b));
        umma_commit(bar(EMPTY + s));
      }
      __syncwarp();
    }
  } else {
    const int q = warp & 3, c = (warp - 2) >> 2;            // the TMEM quarter this warp may read; its 32 columns
    const int er = lane >> 2, ec = (lane & 3) * 2;          // fragments: rows 32 i + 8 q + er of the tile, columns 32 c + 8 o + ec + {0, 1}
    const bool diag = mt == nt;
    F2 acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int o = 0; o < 4; ++o) acc[i][o] = 0ull;
    bool ok = true;
#pragma unroll 1
    for (int j = 0; j < nh; ++j) {
      const int s = j % STAGES, b = j & 1;
      ok = __all_sync(0xffffffffu, wait(FULL + s, (uint32_t)(j / STAGES), 16u) && wait(GFULL + b, (uint32_t)(j >> 1), 16u));
      if (!ok) break;
      const float* Sr = reinterpret_cast<const float*>(ring_ptr + s * GE::PITCH + 2 * NS * T128);
      float nSr[4];
      F2 sc[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) { nSr[i] = Sr[32 * i + 8 * q + er]; sc[i] = neg2(*reinterpret_cast<const F2*>(Sr + L + 32 * c + 8 * i + ec)); }
      uint32_t r[2][16];
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int rh = 0; rh < 2; ++rh) tmem_ld16x256_x4(tmem + ((uint32_t)(32 * q + 16 * rh) << 16) + (uint32_t)(b * L + 32 * c), r[rh]);
      tmem_wait_ld();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) { mbar_arrive(bar(GFREE + b)); mbar_arrive(bar(EMPTY + s)); }
      // rows 32 i + 8 q + er: all of them are past the columns (below), or the block crosses the diagonal
      auto fold = [&](int i, auto below) {
#pragma unroll
        for (int o = 0; o < 4; ++o) {
          const int x = 4 * o + 2 * (i & 1);
          float2 w = unpack2(ex2_two(mul2(add2(pack2(nSr[i], nSr[i]), sc[o]), pack2(1.4426950408889634f, 1.4426950408889634f))));
          if (!decltype(below)::value) { const int d = 8 * (q - o) + er - ec; w.x = d >= 0 ? w.x : 0.0f; w.y = d >= 1 ? w.y : 0.0f; }
          acc[i][o] = fma2(pack2(__uint_as_float(r[i >> 1][x]), __uint_as_float(r[i >> 1][x + 1])), pack2(w.x, w.y), acc[i][o]);
        }
      };
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (!diag || i > c) fold(i, std::true_type{});
        else if (i == c) fold(i, std::false_type{});
      }
    }
    if (ok && !__any_sync(0xffffffffu, *abort_flag != 0)) {
      const int64_t base = (int64_t)blockIdx.x * p.Q * p.Q;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int64_t row = base + (int64_t)(m0 + 32 * i + 8 * q + er) * p.Q + n0 + 32 * c + ec;
#pragma unroll
        for (int o = 0; o < 4; ++o) {
          const float2 v = unpack2(acc[i][o]);
          if (p.nsplit > 1) *reinterpret_cast<float2*>(p.part + row + 8 * o) = v;
          else {
            uint32_t hi, lo = 0u;
            split2(v.x, v.y, hi, lo, NS == 2);
            *reinterpret_cast<uint32_t*>(p.dg_hi + row + 8 * o) = hi;
            if (NS == 2) *reinterpret_cast<uint32_t*>(p.dg_lo + row + 8 * o) = lo;
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(2 * L) : "memory");
  }
}

template <int NS>
static pmb_status launch(cudaStream_t st, const SsdIn& in, const SsdWs& ws, int nsplit) {
  const int nc = in.T / in.Q, qt = in.Q / L, chunks = in.B * nc;
  const int64_t tok = (int64_t)in.B * in.T, hp = (int64_t)in.H * in.P;
  Maps ms{};
  for (int sp = 0; sp < 2; ++sp) {
    const bool lo = NS == 2 && sp;
    PMB_TRY(sf::bf16_map_rows8(&ms.a[sp], lo ? ws.dy_lo : ws.dy_hi, in.P, tok, in.H, hp, in.P));
    PMB_TRY(sf::bf16_map3(&ms.b[sp], lo ? ws.xt_lo : ws.xt_hi, in.P, tok, in.H, hp, in.P, 64, L));
  }
  Params p{};
  p.H = in.H; p.hpg = in.H / in.G; p.G = in.G; p.Q = in.Q; p.nc = nc; p.T = in.T; p.nsplit = nsplit; p.noff = qt * (qt - 1) / 2;
  p.S = ws.S; p.part = ws.splitk; p.dg_hi = ws.dg_hi; p.dg_lo = ws.dg_lo; p.status = ssd_fused_status();
  PMB_SMEM_OPT_IN(Geo<NS>::SMEM, ssd_dg_kernel<NS>);
  ssd_dg_kernel<NS><<<dim3((unsigned)(chunks * in.G * nsplit), (unsigned)(qt * (qt + 1) / 2)), NTHREADS, Geo<NS>::SMEM, st>>>(ms, p);
  PMB_LAUNCHED();
  return PMB_OK;
}

}  // namespace sdg

// As many splits of a group's heads as fit the machine in one wave of a CTA per SM, then the fewest that give the same number of heads per CTA
// (fewer partial tiles to write and add up).
int ssd_dg_nsplit(int B, int T, int H, int G, int Q) {
  const int hpg = H / G, qt = Q / sdg::L;
  const int64_t ctas = (int64_t)B * (T / Q) * G * (qt * (qt + 1) / 2);
  int want = (int)(148 / (ctas > 0 ? ctas : 1));
  if (want < 1) want = 1;
  if (want > hpg) want = hpg;
  const int per = (hpg + want - 1) / want;
  return (hpg + per - 1) / per;
}

pmb_status ssd_dg(cudaStream_t st, const SsdIn& in, const SsdWs& ws, int nsplit) {
  return in.plain16 || !ws.dy_lo ? sdg::launch<1>(st, in, ws, nsplit) : sdg::launch<2>(st, in, ws, nsplit);
}

}  // namespace pmb

// Gradient of the chunked scan w.r.t. its input, chunk by chunk on plain bf16 operands (bf16-storage blocks on whole chunks of 128 or 256
// tokens at d_state = d_head = 64; mamba2/ssd_ops.rs:83-138,201-234 backwards), with everything else that a row of it needs:
//   dx~[s,:] = sum_{t>=s} (C_t.B_s) exp(S_t-S_s) dY_t + exp(S_end-S_s) B_s dh,   dx = dx~ dt + D dY,
//   <dx~, x>, <dY, exp(S) C h>, <dY, x> of every row and the terms of dS (see ssd_dx_finish_kernel).
// One CTA owns 128 rows s of one (batch, chunk, head) and walks the 64-wide column blocks t that the causal mask leaves:
//   G = B C^T and dM = x~ dY^T (tensor core, TMEM), M = G exp(S_t - S_s) [t >= s] -> bf16 in shared memory, W = dM M [t > s] in registers
//   (its row and column sums, see ssd_fused.cu on why both come from the same registers), acc1 += M dY;  acc2 = B dh.
// warp 0 = TMA, warp 1 = MMAs (one elected lane), warps 2..9 = mask: a warp has 32 rows and one half of a block's columns; G and dM are given
// back as soon as all eight have them in registers, so that the next block's products run while this one is masked.
// Bound by the latency of one CTA's chain (load, products, mask, product, epilogue), so the plan is sized for two CTAs per SM: 102 KB of shared
// memory, 256 columns of TMEM (G 64, dM 64, two accumulators of 64), 96 registers.  Tiles of 32 x 32 above the diagonal are not computed.
// The epilogue takes the accumulators as 16 x 8 fragments: a quad of lanes reads and writes whole 32-byte sectors of x, dY, exp(S) C h and dx.
// 16384 tokens of 24 heads, chunks of 256: 206 us with one CTA per SM that wrote dx~ alone and 107 us for a pass over the rows behind it;
// 163 us and 12 now (500 MB: 77 us at the copy rate).
#include <cuda_bf16.h>
#include "tc_common.cuh"
#include "kernels.h"
#include "ssd_fused.h"

namespace pmb {
namespace sdx {

using namespace tcx;

constexpr int RB = 128, CW = 64, NMASKW = 8, NMASK = 32 * NMASKW, NTHREADS = 64 + NMASK;
constexpr int PW = 64, MAXQ = 256;
constexpr int T128 = RB * 128, T64 = CW * 128;
constexpr int STAGES = 2, STAGE = 2 * T64;                  // [C | dY] of a column block; slot use 0 carries the state tiles, [dh | h]
constexpr int TILES = 2 * T128 + STAGES * STAGE + 2 * T128; // [B | x~], ring, two masked tiles
constexpr int NSUM = 5;                                     // per row: sum of W over t, e, <dx~, x>, <dY, exp(S) C h>, <dY, x>
constexpr int SMEM = TILES + 1024 + 256 + (MAXQ + 4 * MAXQ + 2 * NSUM * RB) * 4;
constexpr int TMEM_COLS = 256;
static_assert(2 * (SMEM + 1024) <= 227 * 1024, "two CTAs per SM");

struct Maps { CUtensorMap b, x, c, cr, dy, st, hp; };       // cr: C in tiles of 128 rows
struct Params {
  int H, hpg, Q, nc, nb, T;
  const float* S;
  const float* dt;
  const float* x; int64_t ldx;
  const float* dy; int64_t lddy;
  const float* D;
  float* dx; int64_t lddx;
  float* rpart;                                             // (B*nc*H, nb, Q)
  float* sums;                                              // (B*nc*H, NSUM, Q)
  unsigned int* status;
};

__device__ __forceinline__ void tmem_ld32_nowait(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}

// On entry every lane holds v[0..31]: its row's values for 32 consecutive columns.  On exit lane l holds the sum of column l over the
// warp's 32 rows, in a fixed order.
__device__ __forceinline__ float warp_column_sums(float (&v)[32], int lane) {
#pragma unroll
  for (int w = 16; w >= 1; w >>= 1) {
    const bool upper = (lane & w) != 0;
#pragma unroll
    for (int k = 0; k < w; ++k) {
      const float keep = upper ? v[k + w] : v[k], send = upper ? v[k] : v[k + w];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, w);
    }
  }
  return v[0];
}

__global__ void __launch_bounds__(NTHREADS, 2) ssd_dx_kernel(const __grid_constant__ Maps maps, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);
  const uint32_t b_s = base, x_s = b_s + T128, ring_s = x_s + T128, mop_s = ring_s + STAGES * STAGE, bars = mop_s + 2 * T128;
  enum { R_FULL = 0, F_FULL, LD_FULL, LD_EMPTY = LD_FULL + STAGES, G_FULL = LD_EMPTY + STAGES, G_FREE, M_READY, M_FREE = M_READY + 2, ACC_FULL = M_FREE + 2, NBAR };
  static_assert(8 * NBAR + 8 <= 256, "barrier block");
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  uint8_t* bar_ptr = base_ptr + (bars - base);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bar_ptr + 8 * NBAR);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  float* sS = reinterpret_cast<float*>(bar_ptr + 256);
  float* colsum = sS + MAXQ;                                // [quarter][t]: sums of W over a warp's 32 rows
  float* xchg = colsum + 4 * MAXQ;                          // [column half][NSUM][row]

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int bch = (int)blockIdx.x, rb = (int)blockIdx.y;    // (b * nc + chunk) * H + head; the row blocks with the most column blocks come first
  const int h = bch % p.H, bc = bch / p.H, cc = bc % p.nc, bb = bc / p.nc, g = h / p.hpg;
  const int tok0 = bc * p.Q;                                // first token of the chunk (T = nc * Q)
  const int cb0 = 2 * rb, ncb = p.Q / CW - cb0;
  if (threadIdx.x == 0) {
    mbar_init(bar(R_FULL), 1); mbar_init(bar(F_FULL), 1);
    for (int s = 0; s < STAGES; ++s) { mbar_init(bar(LD_FULL + s), 1); mbar_init(bar(LD_EMPTY + s), 1); }
    mbar_init(bar(G_FULL), 1); mbar_init(bar(G_FREE), NMASKW);
    for (int i = 0; i < 2; ++i) { mbar_init(bar(M_READY + i), NMASKW); mbar_init(bar(M_FREE + i), 1); }
    mbar_init(bar(ACC_FULL), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "n"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const uint32_t tG = tmem, tDM = tmem + CW, tA1 = tmem + 2 * CW, tA2 = tA1 + PW;

  auto give_up = [&](unsigned int code) { atomicOr(p.status, code); *abort_flag = 1; };
  // bounded waits that also end as soon as another role of the CTA has given up
  auto wait = [&](int b, uint32_t parity, unsigned int code) -> bool {
    if (*abort_flag) return false;
    if (mbar_wait(bar(b), parity & 1u)) return true;
    give_up(code);
    return false;
  };
  auto wait_idle = [&](int b, uint32_t parity, unsigned int code) -> bool {
    if (*abort_flag) return false;
    if (mbar_wait_idle(bar(b), parity & 1u)) return true;
    give_up(code);
    return false;
  };

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      mbar_expect_tx(bar(R_FULL), 3 * T128);
      tma_load_3d(b_s, &maps.b, 0, tok0 + RB * rb, g, bar(R_FULL));
      tma_load_3d(x_s, &maps.x, 0, tok0 + RB * rb, h, bar(R_FULL));
      tma_load_3d(mop_s, &maps.cr, 0, tok0 + RB * rb, g, bar(R_FULL));      // (over the first masked tile, which waits for its product)
      int issued = 0;
      for (int it = 0; it <= ncb; ++it) {
        const int s = it % STAGES;
        if (!wait(LD_EMPTY + s, (uint32_t)(it / STAGES) ^ 1u, 1u)) break;
        const uint32_t dst = ring_s + s * STAGE;
        if (it == 0) {
          mbar_expect_tx(bar(LD_FULL + s), STAGE);
          tma_load_3d(dst, &maps.st, 0, bch * PW, 0, bar(LD_FULL + s));
          tma_load_3d(dst + T64, &maps.hp, 0, bch * PW, 0, bar(LD_FULL + s));
        } else {
          const int row0 = tok0 + CW * (cb0 + it - 1);
          mbar_expect_tx(bar(LD_FULL + s), STAGE);
          tma_load_3d(dst, &maps.c, 0, row0, g, bar(LD_FULL + s));
          tma_load_3d(dst + T64, &maps.dy, 0, row0, h, bar(LD_FULL + s));
        }
        issued = it + 1;
      }
      if (*abort_flag) {
        // give the copies already in flight a bounded chance to land before the CTA exits
        mbar_wait(bar(R_FULL), 0);
        for (int it = (issued > STAGES ? issued - STAGES : 0); it < issued; ++it) mbar_wait(bar(LD_FULL + it % STAGES), (uint32_t)((it / STAGES) & 1));
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (the whole warp waits, one elected lane issues) ----------------
    auto wait_all = [&](int b, uint32_t parity, unsigned int code) -> bool { return __all_sync(0xffffffffu, wait(b, parity, code)); };
    const uint32_t id_g = idesc_bf16(0, 0, RB, CW);         // G, dM: both operands K-major
    const uint32_t id_v = idesc_bf16(0, 1, RB, PW);         // M dY and B dh: B operand MN-major
    const uint32_t dh = desc_hi(1024, 2);
    const uint32_t b0 = desc_lo(b_s, 16), x0 = desc_lo(x_s, 16);
    bool ok = wait_all(R_FULL, 0u, 2u) && wait_all(LD_FULL + 0, 0u, 2u);
    if (ok) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t s0 = desc_lo(ring_s, T64), h0 = desc_lo(ring_s + T64, T64), c0 = desc_lo(mop_s, 16);
      if (elect_one()) {
        // C h, where the first product of a masked tile will land once the mask warps have read it
#pragma unroll
        for (int k = 0; k < 4; ++k) mma_f16_h(tA1, c0 + ((k * 32) >> 4), dh, h0 + ((k * 2048) >> 4), dh, id_v, k ? 1u : 0u);
        umma_commit(bar(F_FULL));
#pragma unroll
        for (int k = 0; k < 4; ++k) mma_f16_h(tA2, b0 + ((k * 32) >> 4), dh, s0 + ((k * 2048) >> 4), dh, id_v, k ? 1u : 0u);
        umma_commit(bar(LD_EMPTY + 0));
      }
      __syncwarp();
    }
    // G and dM of column block jj
    auto mma_g = [&](int jj) -> bool {
      const int it = jj + 1, s = it % STAGES;
      if (!wait_all(LD_FULL + s, (uint32_t)(it / STAGES), 2u)) return false;
      if (jj > 0 && !wait_all(G_FREE, (uint32_t)(jj - 1), 4u)) return false;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t c0 = desc_lo(ring_s + s * STAGE, 16), y0 = desc_lo(ring_s + s * STAGE + T64, 16);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 4; ++k) mma_f16_h(tG, b0 + ((k * 32) >> 4), dh, c0 + ((k * 32) >> 4), dh, id_g, k ? 1u : 0u);
        // dM[s,t] = <x~_s, dY_t>: the dY tile read as a K-major operand (the same bytes that M dY reads MN-major)
#pragma unroll
        for (int k = 0; k < 4; ++k) mma_f16_h(tDM, x0 + ((k * 32) >> 4), dh, y0 + ((k * 32) >> 4), dh, id_g, k ? 1u : 0u);
        umma_commit(bar(G_FULL));
      }
      __syncwarp();
      return true;
    };
    ok = ok && mma_g(0);
    for (int jj = 0; jj < ncb && ok; ++jj) {
      const int mb = jj & 1, s = (jj + 1) % STAGES;
      if (jj + 1 < ncb && !mma_g(jj + 1)) { ok = false; break; }
      if (!wait_all(M_READY + mb, (uint32_t)(jj >> 1), 8u)) { ok = false; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t m0 = desc_lo(mop_s + mb * T128, 16), v0 = desc_lo(ring_s + s * STAGE + T64, T64);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 4; ++k) mma_f16_h(tA1, m0 + ((k * 32) >> 4), dh, v0 + ((k * 2048) >> 4), dh, id_v, (jj | k) ? 1u : 0u);
        umma_commit(bar(LD_EMPTY + s));
        umma_commit(bar(M_FREE + mb));
      }
      __syncwarp();
    }
    if (elect_one()) umma_commit(bar(ACC_FULL));
    __syncwarp();
  } else {
    // ---------------- mask (TMEM -> registers -> shared-memory operand), then epilogue ----------------
    const int quarter = warp & 3;                           // the TMEM lane quarter this warp may read
    const int grp = (warp - 2) >> 2;                        // half of a block's (and of the output's) columns
    const int tid = (int)threadIdx.x - 64, r_local = quarter * 32 + lane, row0 = rb * RB + quarter * 32;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    // fragments: this thread's rows are er + {0, 8, 16, 24}, its columns cw + 8 o + {0, 1}
    const int er = quarter * 32 + (lane >> 2), cw = 32 * grp + (lane & 3) * 2;
    const int64_t tkr = (int64_t)tok0 + rb * RB + er;
    const int col = h * PW + cw;
    float2 dyf[4][4];                                       // dY of all four rows, on its way while the first operands are
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int o = 0; o < 4; ++o) dyf[e][o] = *reinterpret_cast<const float2*>(p.dy + (tkr + 8 * e) * p.lddy + col + 8 * o);
    {
      const float* Sp = p.S + ((int64_t)bb * p.H + h) * p.T + (int64_t)cc * p.Q;
      if (tid < p.Q) sS[tid] = Sp[tid];
      // the epilogue's rows of x on their way into L2, a line per thread
      asm volatile("prefetch.global.L2 [%0];" ::"l"(p.x + ((int64_t)tok0 + rb * RB + (tid >> 1)) * p.ldx + h * PW + 32 * (tid & 1)));
      asm volatile("bar.sync 3, %0;" ::"n"(NMASK) : "memory");
    }
    const float S_row = sS[rb * RB + r_local];
    bool ok = __all_sync(0xffffffffu, wait_idle(F_FULL, 0u, 64u));
    if (ok) {
      // f_t = <dY_t, exp(S_t) C_t h> of the same 128 tokens
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int rh = 0; rh < 2; ++rh) {
        uint32_t a[16];
        tmem_ld16x256_x4(tA1 + lane_addr + ((uint32_t)(16 * rh) << 16) + (uint32_t)(32 * grp), a);
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float fs = __expf(sS[rb * RB + er + 16 * rh + 8 * e]);
          float f = 0.0f;
#pragma unroll
          for (int o = 0; o < 4; ++o) {
            const float2 dy = dyf[2 * rh + e][o];
            f = fmaf(dy.x, fs * __uint_as_float(a[4 * o + 2 * e]), fmaf(dy.y, fs * __uint_as_float(a[4 * o + 2 * e + 1]), f));
          }
          f += __shfl_xor_sync(0xffffffffu, f, 1);
          f += __shfl_xor_sync(0xffffffffu, f, 2);
          if ((lane & 3) == 0) xchg[(grp * NSUM + 3) * RB + er + 16 * rh + 8 * e] = f;
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    float c_acc = 0.0f;                                     // sum over t > s of W[t,s] for this thread's row s, this half's columns
    // (nothing in this loop waits for another warp but through the bounded waits, so a warp that gave up just leaves it)
#pragma unroll 1
    for (int jj = 0; jj < ncb && ok; ++jj) {
      const int mb = jj & 1, c0 = (cb0 + jj) * CW + 32 * grp;
      ok = __all_sync(0xffffffffu, wait_idle(G_FULL, (uint32_t)jj, 16u));
      if (!ok) break;
      uint8_t* mrow = base_ptr + (mop_s - base) + mb * T128 + (r_local >> 3) * 1024 + (r_local & 7) * 128;
      if (c0 < row0) {                                      // every t of the tile is before every s
        if (lane == 0) mbar_arrive(bar(G_FREE));
        ok = __all_sync(0xffffffffu, jj < 2 || wait_idle(M_FREE + mb, (uint32_t)((jj >> 1) - 1), 32u));
        if (!ok) break;
#pragma unroll
        for (int q8 = 0; q8 < 4; ++q8) *reinterpret_cast<uint4*>(mrow + (((grp * 4 + q8) ^ (r_local & 7)) << 4)) = make_uint4(0u, 0u, 0u, 0u);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(M_READY + mb));
        colsum[quarter * MAXQ + c0 + lane] = 0.0f;
        continue;
      }
      uint32_t r[32], d[32];
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      tmem_ld32_nowait(tG + lane_addr + (uint32_t)(32 * grp), r);
      tmem_ld32_nowait(tDM + lane_addr + (uint32_t)(32 * grp), d);
      tmem_wait_ld();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(G_FREE));
      ok = __all_sync(0xffffffffu, jj < 2 || wait_idle(M_FREE + mb, (uint32_t)((jj >> 1) - 1), 32u));
      if (!ok) break;
      float wv[32];
      const bool diag = c0 == row0;
#pragma unroll
      for (int q8 = 0; q8 < 4; ++q8) {
        uint32_t hi[4], z;
#pragma unroll
        for (int e2 = 0; e2 < 4; ++e2) {
          const int e = q8 * 8 + 2 * e2;
          const float2 sc = *reinterpret_cast<const float2*>(sS + c0 + e);
          // row = s, column = t: exp(S_t - S_s) for t >= s; W for t > s (the diagonal does not depend on S)
          float m0 = __uint_as_float(r[e]) * __expf(sc.x - S_row), m1 = __uint_as_float(r[e + 1]) * __expf(sc.y - S_row);
          if (diag) { m0 = e >= lane ? m0 : 0.0f; m1 = e + 1 >= lane ? m1 : 0.0f; }
          wv[e] = __uint_as_float(d[e]) * m0; wv[e + 1] = __uint_as_float(d[e + 1]) * m1;
          if (diag) { wv[e] = e > lane ? wv[e] : 0.0f; wv[e + 1] = e + 1 > lane ? wv[e + 1] : 0.0f; }
          c_acc += wv[e] + wv[e + 1];
          split2(m0, m1, hi[e2], z, false);
        }
        *reinterpret_cast<uint4*>(mrow + (((grp * 4 + q8) ^ (r_local & 7)) << 4)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(M_READY + mb));
      colsum[quarter * MAXQ + c0 + lane] = warp_column_sums(wv, lane);
    }
    const float Dv = p.D ? p.D[h] : 0.0f;
    float2 xv[2][4], dyv[2][4];
    float dtv[2];
    auto fetch = [&](int rh) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int64_t tk = tkr + 16 * rh + 8 * e;
        dtv[e] = p.dt[tk * p.H + h];
#pragma unroll
        for (int o = 0; o < 4; ++o) {
          xv[e][o] = *reinterpret_cast<const float2*>(p.x + tk * p.ldx + col + 8 * o);
          dyv[e][o] = *reinterpret_cast<const float2*>(p.dy + tk * p.lddy + col + 8 * o);
        }
      }
    };
    fetch(0);
    const bool acc_ok = __all_sync(0xffffffffu, ok && wait_idle(ACC_FULL, 0u, 64u) && wait(R_FULL, 0u, 64u));
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const bool run = acc_ok && !__any_sync(0xffffffffu, *abort_flag != 0);
    xchg[(grp * NSUM + 0) * RB + r_local] = c_acc;
    if (run) {
      const float S_end = sS[p.Q - 1];
      const uint8_t* xt = base_ptr + (x_s - base);
#pragma unroll 1
      for (int rh = 0; rh < 2; ++rh) {
        float es[2] = {0.0f, 0.0f}, s1[2] = {0.0f, 0.0f}, s3[2] = {0.0f, 0.0f}, fac[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) fac[e] = __expf(S_end - sS[rb * RB + er + 16 * rh + 8 * e]);
#pragma unroll
        for (int c16 = 0; c16 < 2; ++c16) {
          uint32_t a1[8], a2[8];
          const uint32_t ta = lane_addr + ((uint32_t)(16 * rh) << 16) + (uint32_t)(32 * grp + 16 * c16);
          tmem_ld16x256_x2(tA1 + ta, a1);
          tmem_ld16x256_x2(tA2 + ta, a2);
          tmem_wait_ld();
#pragma unroll
          for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int r = 4 * q + 2 * e, o = 2 * c16 + q, rl = er + 16 * rh + 8 * e;
              const float b0 = __uint_as_float(a2[r]), b1 = __uint_as_float(a2[r + 1]);
              // x~ of these two columns, from the operand tile (128-byte rows, 16-byte pieces xor-swizzled by the row)
              const uint32_t xp = *reinterpret_cast<const uint32_t*>(xt + rl * 128 + (((4 * grp + o) ^ (rl & 7)) << 4) + (lane & 3) * 4);
              es[e] = fmaf(__uint_as_float(xp << 16), b0, fmaf(__uint_as_float(xp & 0xffff0000u), b1, es[e]));
              const float v0 = fmaf(fac[e], b0, __uint_as_float(a1[r])), v1 = fmaf(fac[e], b1, __uint_as_float(a1[r + 1]));
              const float2 xx = xv[e][o], dy = dyv[e][o];
              s1[e] = fmaf(v0, xx.x, fmaf(v1, xx.y, s1[e]));
              s3[e] = fmaf(dy.x, xx.x, fmaf(dy.y, xx.y, s3[e]));
              *reinterpret_cast<float2*>(p.dx + (tkr + 16 * rh + 8 * e) * p.lddx + col + 8 * o) = make_float2(fmaf(v0, dtv[e], Dv * dy.x), fmaf(v1, dtv[e], Dv * dy.y));
            }
        }
        if (rh == 0) fetch(1);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
#pragma unroll
          for (int o = 1; o <= 2; o <<= 1) {
            es[e] += __shfl_xor_sync(0xffffffffu, es[e], o); s1[e] += __shfl_xor_sync(0xffffffffu, s1[e], o);
            s3[e] += __shfl_xor_sync(0xffffffffu, s3[e], o);
          }
          const int which = lane & 3;
          if (which < 3) xchg[(grp * NSUM + (which == 2 ? 4 : 1 + which)) * RB + er + 16 * rh + 8 * e] = which == 0 ? es[e] * fac[e] : which == 1 ? s1[e] : s3[e];
        }
      }
    }
    // every warp comes here, whatever happened before
    asm volatile("bar.sync 3, %0;" ::"n"(NMASK) : "memory");
    if (run) {
      if (tid >= RB * rb && tid < p.Q) {
        const float* q = colsum + tid;
        p.rpart[((int64_t)bch * p.nb + rb) * p.Q + tid] = ((q[0] + q[MAXQ]) + q[2 * MAXQ]) + q[3 * MAXQ];
      }
      for (int i = tid; i < NSUM * RB; i += NMASK)
        p.sums[((int64_t)bch * NSUM + i / RB) * p.Q + rb * RB + i % RB] = xchg[i] + xchg[NSUM * RB + i];
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TMEM_COLS) : "memory");
  }
}

// The gradient w.r.t. the in-chunk cumulative sum S and what follows from it, one thread per token of a (batch, chunk, head):
//   dS_t = r_t - c_t + f_t - e_t,      dS_{Q-1} += sum_s e_s + exp(S_end) <dh, h_prev>
//   r_t = sum_{s<t} W[t,s], c_t = sum_{u>t} W[u,t], f_t = <dY_t, exp(S_t) C_t h_prev>, e_s = exp(S_end - S_s) <x~_s, B_s dh>
// da = reverse cumsum(dS);  ddt = <dx~, x> + A da, through the softplus into the dt columns of the in_proj gradient; per-chunk sums of dA, dD, d_dt_bias.
__global__ void __launch_bounds__(MAXQ) ssd_dx_finish_kernel(const float* __restrict__ rpart, const float* __restrict__ sums, const float* __restrict__ S,
                                                             const float* __restrict__ dt, const float* __restrict__ A, const float* __restrict__ dd,
                                                             float* __restrict__ part, SsdGrads::RawDt raw, int H, int T, int Q, int nc, int parts) {
  __shared__ float wsum[MAXQ / 32], red[32];
  const int w = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int h = w % H, bc = w / H, cc = bc % nc, bb = bc / nc, nb = Q / RB;
  const int t = Q - 1 - tid;                                // thread 0 owns the last token
  const int64_t tk = (int64_t)bc * Q + t;
  const float* own = sums + (int64_t)w * NSUM * Q + t;
  float rr = 0.0f;
  for (int rb = 0; rb <= t / RB; ++rb) rr += rpart[((int64_t)w * nb + rb) * Q + t];      // row blocks whose rows s can be < t
  const float cs = own[0], es = own[Q], s1 = own[2 * Q], s2 = own[3 * Q], s3 = own[4 * Q], dtv = dt[tk * H + h], Ah = A[h];
  float v = ((rr - cs) + s2) - es;
  const float esum = block_sum(es, red);
  if (tid == 0) v += esum + expf(S[((int64_t)bb * H + h) * T + (int64_t)cc * Q + Q - 1]) * dd[w];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) { const float u = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += u; }
  if (lane == 31) wsum[wid] = v;
  __syncthreads();
  float off = 0.0f;
  for (int j = 0; j < wid; ++j) off += wsum[j];
  v += off;
  const float gr = fmaf(Ah, v, s1) * (-expm1f(-dtv));       // d softplus(u) / du = sigmoid(u) = 1 - exp(-softplus(u))
  uint32_t hh, ll;
  split_bf16_pair(gr, hh, ll);
  raw.hi[tk * raw.ld + raw.col0 + h] = (uint16_t)hh;
  const float tA = block_sum(v * dtv, red), tD = block_sum(s3, red), tB = block_sum(gr, red);
  if (tid == 0) {
    part[(int64_t)bc * H + h] = tA;
    part[(int64_t)parts * H + (int64_t)bc * H + h] = tD;
    part[2 * (int64_t)parts * H + (int64_t)bc * H + h] = tB;
  }
}

}  // namespace sdx

size_t ssd_dx_sum_floats(int B, int T, int H) { return (size_t)sdx::NSUM * B * T * H; }

pmb_status ssd_dx(cudaStream_t st, const DxArgs& a) {
  if (a.P != 64 || a.N != 64 || (a.Q != 128 && a.Q != 256) || a.T % a.Q || a.H % a.G || (a.ldx | a.lddy | a.lddx) & 1 || (int64_t)a.B * a.T * a.H >= (1LL << 31) / 64)
    return fail(PMB_ERR_UNSUPPORTED, "ssd_dx: unsupported shape (P=%d N=%d Q=%d)", a.P, a.N, a.Q);
  const int nc = a.T / a.Q, chunks = a.B * nc;
  const int64_t tok = (int64_t)a.B * a.T, HP = (int64_t)a.H * sdx::PW;
  sdx::Maps ms{};
  PMB_TRY(sf::bf16_map3(&ms.b, a.b.hi, 64, tok, a.G, a.b.pitch, 64, 64, sdx::RB));
  PMB_TRY(sf::bf16_map3(&ms.c, a.c.hi, 64, tok, a.G, a.c.pitch, 64, 64, sdx::CW));
  PMB_TRY(sf::bf16_map3(&ms.cr, a.c.hi, 64, tok, a.G, a.c.pitch, 64, 64, sdx::RB));
  PMB_TRY(sf::bf16_map3(&ms.x, a.xt, 64, tok, a.H, HP, 64, 64, sdx::RB));
  PMB_TRY(sf::bf16_map3(&ms.dy, a.dy16, 64, tok, a.H, HP, 64, 64, sdx::CW));
  PMB_TRY(sf::bf16_map3(&ms.st, a.dh, 64, (int64_t)chunks * a.H * 64, 1, 64, 64 * 64, 64, sdx::CW));
  PMB_TRY(sf::bf16_map3(&ms.hp, a.hp, 64, (int64_t)chunks * a.H * 64, 1, 64, 64 * 64, 64, sdx::CW));
  sdx::Params p{};
  p.H = a.H; p.hpg = a.H / a.G; p.Q = a.Q; p.nc = nc; p.nb = a.Q / sdx::RB; p.T = a.T;
  p.S = a.S; p.dt = a.dt; p.x = a.x; p.ldx = a.ldx; p.dy = a.dy; p.lddy = a.lddy; p.D = a.D; p.dx = a.dx; p.lddx = a.lddx;
  p.rpart = a.rpart; p.sums = a.sums; p.status = ssd_fused_status();
  {
    ProfScope prof(st, "ssd_dx", 2.0 * tok * a.H * 64 * (3.0 * a.Q + 64), 0.0);
    PMB_SMEM_OPT_IN(sdx::SMEM, sdx::ssd_dx_kernel);
    static DeviceOnce once;                                  // two CTAs per SM need the largest shared-memory carve-out
    int dev = 0;
    PMB_CUDA(cudaGetDevice(&dev));
    if (once.pending(dev)) {
      PMB_CUDA(cudaFuncSetAttribute(sdx::ssd_dx_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared));
      once.mark(dev);
    }
    sdx::ssd_dx_kernel<<<dim3((unsigned)(chunks * a.H), (unsigned)p.nb), sdx::NTHREADS, sdx::SMEM, st>>>(ms, p);
    PMB_LAUNCHED();
  }
  ProfScope prof(st, "ssd_dx_finish", 0.0, 4.0 * tok * a.H * 8.0);
  sdx::ssd_dx_finish_kernel<<<(unsigned)(chunks * a.H), a.Q, 0, st>>>(a.rpart, a.sums, a.S, a.dt, a.A, a.dd, a.part, a.raw, a.H, a.T, a.Q, nc, chunks);
  PMB_LAUNCHED();
  return PMB_OK;
}

}  // namespace pmb

// Gradient of the chunked scan w.r.t. its input, chunk by chunk on plain bf16 operands (bf16-storage blocks on whole chunks of 128 or 256
// tokens at d_state = d_head = 64; mamba2/ssd_ops.rs:83-138,201-234 backwards), with everything else that a row of it needs:
//   dx~[s,:] = sum_{t>=s} (C_t.B_s) exp(S_t-S_s) dY_t + exp(S_end-S_s) B_s dh,   dx = dx~ dt + D dY,
//   <dx~, x>, <dY, exp(S) C h>, <dY, x> of every row and the terms of dS (see ssd_dx_finish_kernel).
// One CTA owns 128 rows s of one (batch, chunk, head) and walks the 64-wide column blocks t that the causal mask leaves:
//   G = B C^T and dM = x~ dY^T (tensor core, TMEM), M = G exp(S_t - S_s) [t >= s] -> bf16 in shared memory, W = dM M [t > s] in registers
//   (its row and column sums, see ssd_fused.cu on why both come from the same registers), acc1 += M dY;  acc2 = B dh.
// The last use of G's columns is C h of the same 128 tokens, for <dY, exp(S) C h>.
// warp 0 = TMA, warp 1 = MMAs (one elected lane), warps 2..9 = mask: a warp has 32 rows and one half of a block's columns, as 16 x 8
// fragments; G and dM are given back as soon as all eight have them in registers, so that the next block's products run while this one is masked.
// Bound by the latency of one CTA's chain (load, products, mask, product, epilogue), so the plan is sized for two CTAs per SM: 103 KB of shared
// memory, 256 columns of TMEM (G 64, dM 64, two accumulators of 64), 96 registers.  Tiles of 32 x 32 above the diagonal are not computed.
// 16384 tokens of 24 heads, chunks of 256: 206 us with one CTA per SM that wrote dx~ alone and 107 us for a pass over the rows behind it; with two
// CTAs and the rows' work in the epilogue 158 and 12; 124 us now (400 MB: 61 us at the copy rate), by what clocks inside a CTA showed: a row per
// thread cost 31 shuffles per 32 x 32 sums of columns (fragments: 7), fp32 operations in pairs shortened a block's mask of 3500 clocks, and the epilogue's rows pass through shared memory, so that loads and
// stores are whole lines (a quad of lanes per row took half of the L1's cycles).
#include <cuda_bf16.h>
#include <type_traits>
#include "tc_common.cuh"
#include "kernels.h"
#include "ssd_fused.h"

namespace pmb {
namespace sdx {

using namespace tcx;

constexpr int RB = 128, CW = 64, NMASKW = 8, NMASK = 32 * NMASKW, NTHREADS = 64 + NMASK;
constexpr int PW = 64, MAXQ = 256;
constexpr int T128 = RB * 128, T64 = CW * 128;
constexpr int STAGES = 3, STAGE = 2 * T64;                  // [C | dY] of a column block, then [dh | h] and the CTA's own rows of C
constexpr int TILES = 2 * T128 + STAGES * STAGE + T128;     // [B | x~], ring, masked tile
constexpr int NSUM = 5;                                     // per row: sum of W over t, e, <dx~, x>, <dY, exp(S) C h>, <dY, x>
static_assert(NSUM <= PW, "the sums take the place of dx~ (B,T,H,P)");
constexpr int SMEM = TILES + 1024 + 256 + (MAXQ + 4 * MAXQ + RB) * 4;
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

__global__ void __launch_bounds__(NTHREADS, 2) ssd_dx_kernel(const __grid_constant__ Maps maps, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);
  const uint32_t b_s = base, x_s = b_s + T128, ring_s = x_s + T128, mop_s = ring_s + STAGES * STAGE, bars = mop_s + T128;
  enum { R_FULL = 0, LD_FULL, LD_EMPTY = LD_FULL + STAGES, G_FULL = LD_EMPTY + STAGES, G_FREE, M_READY, M_FREE, ACC_FULL, NBAR };
  static_assert(8 * NBAR + 8 <= 256, "barrier block");
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  uint8_t* bar_ptr = base_ptr + (bars - base);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bar_ptr + 8 * NBAR);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  float* sS = reinterpret_cast<float*>(bar_ptr + 256);
  float* colsum = sS + MAXQ;                                // [quarter][t]: sums of W over a warp's 32 rows
  float* sdt = colsum + 4 * MAXQ;                           // dt of the CTA's rows
  float* xchg = reinterpret_cast<float*>(base_ptr + (b_s - base));     // over B, once all products are done: [column half][c, e][row], then [3][row]

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int bch = (int)blockIdx.x, rb = (int)blockIdx.y;    // (b * nc + chunk) * H + head; the row blocks with the most column blocks come first
  const int h = bch % p.H, bc = bch / p.H, cc = bc % p.nc, bb = bc / p.nc, g = h / p.hpg;
  const int tok0 = bc * p.Q;                                // first token of the chunk (T = nc * Q)
  const int cb0 = 2 * rb, ncb = p.Q / CW - cb0;
  if (threadIdx.x == 0) {
    mbar_init(bar(R_FULL), 1);
    for (int s = 0; s < STAGES; ++s) { mbar_init(bar(LD_FULL + s), 1); mbar_init(bar(LD_EMPTY + s), 1); }
    mbar_init(bar(G_FULL), 1); mbar_init(bar(G_FREE), NMASKW);
    mbar_init(bar(M_READY), NMASKW); mbar_init(bar(M_FREE), 1); mbar_init(bar(ACC_FULL), 1);
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
  const uint32_t tG = tmem /*last: C h*/, tDM = tmem + CW, tA1 = tmem + 2 * CW, tA2 = tA1 + PW;

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
      mbar_expect_tx(bar(R_FULL), 2 * T128);
      tma_load_3d(b_s, &maps.b, 0, tok0 + RB * rb, g, bar(R_FULL));
      tma_load_3d(x_s, &maps.x, 0, tok0 + RB * rb, h, bar(R_FULL));
      int issued = 0;
      for (int it = 0; it < ncb + 2; ++it) {
        const int s = it % STAGES;
        if (!wait(LD_EMPTY + s, (uint32_t)(it / STAGES) ^ 1u, 1u)) break;
        const uint32_t dst = ring_s + s * STAGE;
        mbar_expect_tx(bar(LD_FULL + s), STAGE);
        if (it < ncb) {
          tma_load_3d(dst, &maps.c, 0, tok0 + CW * (cb0 + it), g, bar(LD_FULL + s));
          tma_load_3d(dst + T64, &maps.dy, 0, tok0 + CW * (cb0 + it), h, bar(LD_FULL + s));
        } else if (it == ncb) {
          tma_load_3d(dst, &maps.st, 0, bch * PW, 0, bar(LD_FULL + s));
          tma_load_3d(dst + T64, &maps.hp, 0, bch * PW, 0, bar(LD_FULL + s));
        } else {
          tma_load_3d(dst, &maps.cr, 0, tok0 + RB * rb, g, bar(LD_FULL + s));
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
    bool ok = wait_all(R_FULL, 0u, 2u);
    // G and dM of column block jj
    auto mma_g = [&](int jj) -> bool {
      const int s = jj % STAGES;
      if (!wait_all(LD_FULL + s, (uint32_t)(jj / STAGES), 2u)) return false;
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
    // acc2 = B dh, and C h of the CTA's own rows over the last G
    auto mma_states = [&]() -> bool {
      const int sd = ncb % STAGES, sc = (ncb + 1) % STAGES;
      if (!wait_all(LD_FULL + sd, (uint32_t)(ncb / STAGES), 2u) || !wait_all(LD_FULL + sc, (uint32_t)((ncb + 1) / STAGES), 2u) || !wait_all(G_FREE, (uint32_t)(ncb - 1), 4u)) return false;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t d0 = desc_lo(ring_s + sd * STAGE, T64), h0 = desc_lo(ring_s + sd * STAGE + T64, T64), c0 = desc_lo(ring_s + sc * STAGE, 16);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 4; ++k) mma_f16_h(tA2, b0 + ((k * 32) >> 4), dh, d0 + ((k * 2048) >> 4), dh, id_v, k ? 1u : 0u);
#pragma unroll
        for (int k = 0; k < 4; ++k) mma_f16_h(tG, c0 + ((k * 32) >> 4), dh, h0 + ((k * 2048) >> 4), dh, id_v, k ? 1u : 0u);
      }
      __syncwarp();
      return true;
    };
    ok = ok && mma_g(0);
    for (int jj = 0; jj < ncb && ok; ++jj) {
      const int s = jj % STAGES;
      if (!(jj + 1 < ncb ? mma_g(jj + 1) : mma_states()) || !wait_all(M_READY, (uint32_t)jj, 8u)) { ok = false; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t m0 = desc_lo(mop_s, 16), v0 = desc_lo(ring_s + s * STAGE + T64, T64);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < 4; ++k) mma_f16_h(tA1, m0 + ((k * 32) >> 4), dh, v0 + ((k * 2048) >> 4), dh, id_v, (jj | k) ? 1u : 0u);
        umma_commit(bar(LD_EMPTY + s));
        umma_commit(bar(M_FREE));
      }
      __syncwarp();
    }
    if (elect_one()) umma_commit(bar(ACC_FULL));
    __syncwarp();
  } else {
    // ---------------- mask (TMEM -> registers -> shared-memory operand), then epilogue ----------------
    const int quarter = warp & 3;                           // the TMEM lane quarter this warp may read
    const int grp = (warp - 2) >> 2;                        // half of a block's columns
    const int tid = (int)threadIdx.x - 64, row0 = rb * RB + quarter * 32;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    // fragments: this thread's rows of the warp's 32 are er + {0, 8, 16, 24}, its columns of a half 8 o + ec + {0, 1}
    const int er = lane >> 2, ec = (lane & 3) * 2;
    {
      const float* Sp = p.S + ((int64_t)bb * p.H + h) * p.T + (int64_t)cc * p.Q;
      if (tid < p.Q) sS[tid] = Sp[tid];
      if (tid < RB) sdt[tid] = p.dt[((int64_t)tok0 + rb * RB + tid) * p.H + h];
      // the epilogue's rows on their way into L2: a thread has one line of each tensor
      const int64_t tk = (int64_t)tok0 + rb * RB + (tid >> 1);
      asm volatile("prefetch.global.L2 [%0];" ::"l"(p.x + tk * p.ldx + h * PW + 32 * (tid & 1)));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(p.dy + tk * p.lddy + h * PW + 32 * (tid & 1)));
      asm volatile("bar.sync 3, %0;" ::"n"(NMASK) : "memory");
    }
    float S_row[4];
    F2 c_acc[4];                                            // sum over t > s of W[t,s] for this thread's rows s, its even and its odd columns t
#pragma unroll
    for (int i = 0; i < 4; ++i) { S_row[i] = sS[row0 + er + 8 * i]; c_acc[i] = 0ull; }
    // stmatrix: the lane's row of eight and its 16-byte piece of a half (rows of 128 bytes, pieces xor-swizzled by the row)
    const uint32_t m_st = mop_s + (uint32_t)(quarter * 32 + (lane & 7)) * 128u + (uint32_t)(((grp * 4 + (lane >> 3)) ^ (lane & 7)) << 4);
    bool ok = true;
    // (nothing in this loop waits for another warp but through the bounded waits, so a warp that gave up just leaves it)
#pragma unroll 1
    for (int jj = 0; jj < ncb && ok; ++jj) {
      const int c0 = (cb0 + jj) * CW + 32 * grp;
      ok = __all_sync(0xffffffffu, wait_idle(G_FULL, (uint32_t)jj, 16u));
      if (!ok) break;
      if (c0 < row0) {                                      // every t of the tile is before every s
        if (lane == 0) mbar_arrive(bar(G_FREE));
        ok = __all_sync(0xffffffffu, jj < 1 || wait_idle(M_FREE, (uint32_t)(jj - 1), 32u));
        if (!ok) break;
#pragma unroll
        for (int i = 0; i < 4; ++i) st_matrix_x4(m_st + (uint32_t)(i * 1024), 0u, 0u, 0u, 0u);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(M_READY));
        colsum[quarter * MAXQ + c0 + lane] = 0.0f;
        continue;
      }
      uint32_t r[2][16], d[2][16];
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int rh = 0; rh < 2; ++rh) {
        tmem_ld16x256_x4(tG + lane_addr + ((uint32_t)(16 * rh) << 16) + (uint32_t)(32 * grp), r[rh]);
        tmem_ld16x256_x4(tDM + lane_addr + ((uint32_t)(16 * rh) << 16) + (uint32_t)(32 * grp), d[rh]);
      }
      tmem_wait_ld();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(G_FREE));
      F2 cs[4];
      uint32_t m[4][4];
      // row = s, column = t: exp(S_t - S_s) for t >= s; W for t > s (the diagonal does not depend on S)
      auto mask = [&](auto diag) {
#pragma unroll
        for (int o = 0; o < 4; ++o) {
          const F2 sc = *reinterpret_cast<const F2*>(sS + c0 + 8 * o + ec);
          cs[o] = 0ull;
#pragma unroll
          for (int i = 0; i < 4; ++i) {                     // rows er + 8 i
            const int x = 4 * o + 2 * (i & 1), past = 8 * (o - i) + ec - er;      // t - s of the first of the two
            const F2 w2 = ex2_two(mul2(add2(sc, pack2(-S_row[i], -S_row[i])), pack2(1.4426950408889634f, 1.4426950408889634f)));
            F2 mv = mul2(pack2(__uint_as_float(r[i >> 1][x]), __uint_as_float(r[i >> 1][x + 1])), w2);
            if (decltype(diag)::value) { const float2 v = unpack2(mv); mv = pack2(past >= 0 ? v.x : 0.0f, past >= -1 ? v.y : 0.0f); }
            F2 w = mul2(pack2(__uint_as_float(d[i >> 1][x]), __uint_as_float(d[i >> 1][x + 1])), mv);
            if (decltype(diag)::value) { const float2 v = unpack2(w); w = pack2(past > 0 ? v.x : 0.0f, past > -1 ? v.y : 0.0f); }
            c_acc[i] = add2(c_acc[i], w);
            cs[o] = add2(cs[o], w);
            const float2 v = unpack2(mv);
            uint32_t z;
            split2(v.x, v.y, m[i][o], z, false);
          }
        }
      };
      if (c0 == row0) mask(std::true_type{}); else mask(std::false_type{});
      ok = __all_sync(0xffffffffu, jj < 1 || wait_idle(M_FREE, (uint32_t)(jj - 1), 32u));
      if (!ok) break;
#pragma unroll
      for (int i = 0; i < 4; ++i) st_matrix_x4(m_st + (uint32_t)(i * 1024), m[i][0], m[i][1], m[i][2], m[i][3]);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(M_READY));
      // column sums over the warp's 32 rows: lanes with the same ec add up, halving the columns they keep
      float v[8];
#pragma unroll
      for (int o = 0; o < 4; ++o) { const float2 q = unpack2(cs[o]); v[2 * o] = q.x; v[2 * o + 1] = q.y; }
#pragma unroll
      for (int w = 4; w >= 1; w >>= 1) {
        const bool upper = (lane & (4 * w)) != 0;
#pragma unroll
        for (int k = 0; k < w; ++k) {
          const float keep = upper ? v[k + w] : v[k], send = upper ? v[k] : v[k + w];
          v[k] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * w);
        }
      }
      colsum[quarter * MAXQ + c0 + 8 * (lane >> 3) + ec + ((lane >> 2) & 1)] = v[0];
    }
    // Epilogue.  The accumulators pass through shared memory (the ring and the masked tiles are idle then), so that a half-warp has a whole
    // row of x, dY and dx: the warp's rows are grp * 16 + 2 i + (lane / 16), a lane has four columns.
    const int l16 = lane & 15;
    const int64_t tkr = (int64_t)tok0 + row0 + grp * 16 + (lane >> 4);
    const float Dv = p.D ? p.D[h] : 0.0f;
    float4 xv[8], dyv[8];
    auto fetch = [&](int i0) {
#pragma unroll
      for (int i = i0; i < i0 + 4; ++i) {
        xv[i] = reinterpret_cast<const float4*>(p.x + (tkr + 2 * i) * p.ldx + h * PW)[l16];
        dyv[i] = reinterpret_cast<const float4*>(p.dy + (tkr + 2 * i) * p.lddy + h * PW)[l16];
      }
    };
    fetch(0);
    const bool acc_ok = __all_sync(0xffffffffu, ok && wait_idle(ACC_FULL, 0u, 64u) && wait(R_FULL, 0u, 64u));
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const bool run = acc_ok && !__any_sync(0xffffffffu, *abort_flag != 0);
    uint8_t* const st_f = base_ptr + (ring_s - base);       // C h, rows of 256 bytes, 16-byte pieces xor-swizzled by twice the row
    uint8_t* const st_v = st_f + RB * 256;                  // dx~
    static_assert(2 * RB * 256 <= STAGES * STAGE + T128, "both fit over the ring and the masked tile");
    if (run) {
      const float S_end = sS[p.Q - 1];
      const uint8_t* xt = base_ptr + (x_s - base);
#pragma unroll
      for (int i = 0; i < 4; i += 2) {
        float es[2] = {0.0f, 0.0f};
        uint32_t a1[16], a2[16];
        const uint32_t ta = lane_addr + ((uint32_t)(8 * i) << 16) + (uint32_t)(32 * grp);
        tmem_ld16x256_x4(tA1 + ta, a1);
        tmem_ld16x256_x4(tA2 + ta, a2);
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int rl = quarter * 32 + er + 8 * (i + e);
          const float fac = __expf(S_end - S_row[i + e]);
#pragma unroll
          for (int o = 0; o < 4; ++o) {
            const float b0 = __uint_as_float(a2[4 * o + 2 * e]), b1 = __uint_as_float(a2[4 * o + 2 * e + 1]);
            // x~ of these two columns, from the operand tile
            const uint32_t xp = *reinterpret_cast<const uint32_t*>(xt + rl * 128 + (((4 * grp + o) ^ (rl & 7)) << 4) + ec * 2);
            es[e] = fmaf(__uint_as_float(xp << 16), b0, fmaf(__uint_as_float(xp & 0xffff0000u), b1, es[e]));
            *reinterpret_cast<float2*>(st_v + rl * 256 + (((8 * grp + 2 * o + (ec >> 2)) ^ ((rl & 7) << 1)) << 4) + (ec & 2) * 4) =
                make_float2(fmaf(fac, b0, __uint_as_float(a1[4 * o + 2 * e])), fmaf(fac, b1, __uint_as_float(a1[4 * o + 2 * e + 1])));
          }
          es[e] *= fac;
        }
        tmem_ld16x256_x4(tG + ta, a1);
        tmem_wait_ld();
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int rl = quarter * 32 + er + 8 * (i + e);
#pragma unroll
          for (int o = 0; o < 4; ++o)
            *reinterpret_cast<float2*>(st_f + rl * 256 + (((8 * grp + 2 * o + (ec >> 2)) ^ ((rl & 7) << 1)) << 4) + (ec & 2) * 4) =
                make_float2(__uint_as_float(a1[4 * o + 2 * e]), __uint_as_float(a1[4 * o + 2 * e + 1]));
          const float2 cc2 = unpack2(c_acc[i + e]);
          float c = cc2.x + cc2.y;
#pragma unroll
          for (int w = 1; w <= 2; w <<= 1) { es[e] += __shfl_xor_sync(0xffffffffu, es[e], w); c += __shfl_xor_sync(0xffffffffu, c, w); }
          if ((lane & 3) < 2) xchg[(grp * 2 + (lane & 3)) * RB + rl] = (lane & 3) == 0 ? c : es[e];
        }
      }
    }
    fetch(4);                                               // (the accumulators' registers are free now)
    // every warp comes here, whatever happened before; the two warps of a quarter exchange its rows
    if (quarter == 0) asm volatile("bar.sync 4, 64;" ::: "memory");
    else if (quarter == 1) asm volatile("bar.sync 5, 64;" ::: "memory");
    else if (quarter == 2) asm volatile("bar.sync 6, 64;" ::: "memory");
    else asm volatile("bar.sync 7, 64;" ::: "memory");
    if (run) {
#pragma unroll
      for (int i0 = 0; i0 < 8; i0 += 4) {
        float s[3][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int rr = grp * 16 + 2 * (i0 + i) + (lane >> 4), rl = quarter * 32 + rr;
          const int at = rl * 256 + ((l16 ^ ((rl & 7) << 1)) << 4);
          const float4 v = *reinterpret_cast<const float4*>(st_v + at), f = *reinterpret_cast<const float4*>(st_f + at);
          const float4 xx = xv[i0 + i], dy = dyv[i0 + i];
          const float dtv = sdt[rl];
          s[0][i] = fmaf(v.x, xx.x, fmaf(v.y, xx.y, fmaf(v.z, xx.z, v.w * xx.w)));
          s[1][i] = __expf(sS[rb * RB + rl]) * fmaf(dy.x, f.x, fmaf(dy.y, f.y, fmaf(dy.z, f.z, dy.w * f.w)));
          s[2][i] = fmaf(dy.x, xx.x, fmaf(dy.y, xx.y, fmaf(dy.z, xx.z, dy.w * xx.w)));
          reinterpret_cast<float4*>(p.dx + (tkr + 2 * (i0 + i)) * p.lddx + h * PW)[l16] =
              make_float4(fmaf(v.x, dtv, Dv * dy.x), fmaf(v.y, dtv, Dv * dy.y), fmaf(v.z, dtv, Dv * dy.z), fmaf(v.w, dtv, Dv * dy.w));
        }
        // four rows' sums over sixteen lanes: lanes l16 / 4 = i end up with row i
#pragma unroll
        for (int q = 0; q < 3; ++q) {
#pragma unroll
          for (int w = 2; w >= 1; w >>= 1) {
            const bool upper = (lane & (4 * w)) != 0;
#pragma unroll
            for (int k = 0; k < w; ++k) {
              const float keep = upper ? s[q][k + w] : s[q][k], send = upper ? s[q][k] : s[q][k + w];
              s[q][k] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * w);
            }
          }
          s[q][0] += __shfl_xor_sync(0xffffffffu, s[q][0], 2);
          s[q][0] += __shfl_xor_sync(0xffffffffu, s[q][0], 1);
        }
        const int q = lane & 3, rl = quarter * 32 + grp * 16 + 2 * (i0 + (l16 >> 2)) + (lane >> 4);
        if (q < 3) xchg[(4 + q) * RB + rl] = q == 0 ? s[0][0] : q == 1 ? s[1][0] : s[2][0];
      }
    }
    asm volatile("bar.sync 3, %0;" ::"n"(NMASK) : "memory");
    if (run) {
      if (tid >= RB * rb && tid < p.Q) {
        const float* q = colsum + tid;
        p.rpart[((int64_t)bch * p.nb + rb) * p.Q + tid] = ((q[0] + q[MAXQ]) + q[2 * MAXQ]) + q[3 * MAXQ];
      }
      for (int i = tid; i < NSUM * RB; i += NMASK)          // [c, e] of the two column halves, then the three sums of a whole row
        p.sums[((int64_t)bch * NSUM + i / RB) * p.Q + rb * RB + i % RB] = i < 2 * RB ? xchg[i] + xchg[2 * RB + i] : xchg[2 * RB + i];
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

pmb_status ssd_dx_check(const DxArgs& a) {
  if (a.P != 64 || a.N != 64 || (a.Q != 128 && a.Q != 256) || a.T % a.Q || a.H % a.G)
    return fail(PMB_ERR_UNSUPPORTED, "ssd_dx: unsupported shape (P=%d N=%d Q=%d)", a.P, a.N, a.Q);
  if ((int64_t)a.B * a.T >= (1LL << 31) || (int64_t)a.B * (a.T / a.Q) * a.H * a.N >= (1LL << 31))
    return fail(PMB_ERR_UNSUPPORTED, "ssd_dx: too many rows for 32-bit tile coordinates");
  auto off16 = [](const void* q, int64_t ld) { return (reinterpret_cast<uintptr_t>(q) & 15) != 0 || (ld & 3) != 0; };
  if (off16(a.x, a.ldx) || off16(a.dy, a.lddy) || off16(a.dx, a.lddx)) return fail(PMB_ERR_UNSUPPORTED, "ssd_dx: x, dy and dx rows must be 16-byte aligned");
  return PMB_OK;
}

pmb_status ssd_dx(cudaStream_t st, const DxArgs& a) {
  PMB_TRY(ssd_dx_check(a));
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

// Backward of the chunked SSD scan along a sequence as one kernel: the adjoint of ssd_chain.cu's forward except for the three
// sums over heads (dG, dC, dB), which ssd_heads.cu forms after it.  One CTA owns one (batch, head) and walks its steps of 128
// tokens from the last to the first with the state's adjoint dh in registers.
//
// Per step (rows s, columns t of the masked tile; S = inclusive cumulative sum of a in the step; h = state entering it, as the forward
// left it; dh = adjoint of the state leaving it):
//   GT = B C^T,  dMT = x~ dY^T   (128 x 128 each)                             tensor core
//   MT[s,t] = GT exp(S_t - S_s) [t >= s];  W[s,t] = dMT MT [t > s]            mask warps: MT back into TMEM, W summed along
//                                                                             rows and columns in fixed orders
//   dx~ = MT dY + exp(S_end - S_s) B dh                                       tensor core, mask warps' epilogue
//   f_t = exp(S_t) <dY_t, C_t h>,  e_s = exp(S_end - S_s) <x~_s, B_s dh>      tensor core, epilogue
//   dS_t = sum_s W[s,t] - sum_u W[t,u] + f_t - e_t, dS_last += sum_s e_s + exp(S_end) <dh, h>;  da = reverse cumulative sum
//   dh <- exp(S_end) dh + C^T (exp(S) dY)                                     tensor core, state warps' registers
// The row and column sums of W come from the same registers, so that the near-total cancellation in sum_t S_t dS_t (the gradient of
// A) is between identically rounded numbers; <dY, y> - <x~, dx~> from separately rounded products loses it.
//
// <dx~_s, x~_s>, which the gradient of dt needs, is the same sum over t >= s plus e_s: W's row sum with its diagonal.
//
// warp 0 = TMA loads (B, C, h, bf16 x and dY), 1 = products of the masked tile (GT, dMT, MT dY), 2 = per-token gradients (da / ddt and the
// per-head sums), 3 = products of the state (B dh, C h, U) and TMA stores of the operands x~ and dY that the sums over heads read, 4..11 = two
// mask groups of four warps, then the output of the same step, 12..19 = transform (x -> x~, dY -> dY and dY exp(S), into shared memory; bf16
// x and dY are operands as they are), 20..23 = state.
// What bounds it: instructions and their chains, 15000 warp instructions a step at d_state 128, issued in 44 % of the cycles.  On plain
// operands mask (4100 clocks), MT dY and output (2300) follow one another; on pairs, whose one buffer of x~ and dY has to be drained first, the
// transform (6500) comes on top.  Warps of their own for the output (28 of 72 registers) were no faster: 1317 us against 1271 for
// 16 x 8192 tokens, 32 heads of 128 x 64 (1412 with one MMA warp, sums by 16 shuffles per 16 columns and an exponential per element), nor x and dY
// prefetched into registers (50 us for 4 x 512 tokens, 24 heads of 64 x 64, on pairs) or read again by the output (49).
// Measured at 24 heads of 64 x 64 on pairs: 44 us for 4 x 512 tokens (the d(states) product, reverse pass, masked product and row
// kernel it replaces: 118 us), 30 us for 2 x 384, 50 us in segments for 2 x 1000 (1.7 ms of FMA contractions with ssd_heads.cu's share).
// On bf16 inputs, 16 x 8192 tokens of 32 heads of 128 x 64 take 1055 us where 148 SMs share 512 chains in equal stretches (ssd_chain_wrap), 1146 whole.
// Every mbarrier wait is bounded, as in the forward.
#include <cuda_bf16.h>
#include <type_traits>
#include "tc_common.cuh"
#include "kernels.h"
#include "ssd_fused.h"
#include "ssd_wrap.cuh"

namespace pmb {

static __device__ unsigned int g_chain_bwd_status = 0;

pmb_status read_clear_device_status_chain_bwd(unsigned int* word) {
  unsigned int zero = 0;
  PMB_CUDA(cudaMemcpyFromSymbol(word, g_chain_bwd_status, sizeof(unsigned int)));
  if (*word) PMB_CUDA(cudaMemcpyToSymbol(g_chain_bwd_status, &zero, sizeof(unsigned int)));
  return PMB_OK;
}

namespace scb {

using namespace tcx;

constexpr int L = SCAN_STEP, PW = 64, T128 = L * 128, T64 = 64 * 128;
constexpr int W_MASK = 4, W_XF = 12, W_ST = 20, NTHREADS = 32 * 24, XF_THREADS = 256;
// (shares of the block's 80 x 768 registers: 56, 2 x 88, 2 x 72 and 104 per thread of the six warpgroups)

template <int NI, int ND, int NK, bool IN16>
struct Geo {
  static constexpr int BT = NI * NK * T128;              // B (or C)
  static constexpr int HT = ND * NK * T64;               // h, dh: rows n of 128 bytes
  static constexpr int STAGE = 2 * BT + HT;              // [B | C | h]
  static constexpr int XT = NI * T128;                   // x~ (or dY)
  static constexpr int XBUF = 2 * XT + ND * T128;        // [x~ | dY | dY exp(S)]
  static constexpr int XB = ND == 1 ? 2 : 1;
  static constexpr int NSB = 4;                          // copies of S: see the transform warps
  static constexpr int AHEAD = IN16 ? 0 : 2;             // fp32: pieces of x and of dY that a transform thread has in flight (bf16: the tiles are copied as they are)
  static constexpr int TILES = STAGE + XB * XBUF + HT;
  static constexpr int ROWS = 11 * L;                    // per-row sums: [2 groups] of W, e, f; W[s,s]; [4 quarters] column sums of W
  static constexpr int SLOT = 3 * L;                     // a step's [S | dt | column factors]
  static constexpr int SMEM = TILES + 1024 /*alignment slack*/ + 512 /*barriers, small sums*/ + (NSB * SLOT + 2 * ROWS) * 4 + 2 * AHEAD * XF_THREADS * 16;
};

struct Maps { CUtensorMap b[2], c[2], h[2], dh[2], xt[2], dy[2]; };      // [0] = hi (or the plain bf16 tensor), [1] = lo; bf16: xt and dy are the inputs; dh goes out, 32 rows to a box

struct Params {
  int T, H, hpg, N, P, nsteps;
  const float* S;                                        // (B,H,T)
  const float* x; int64_t ldx;                           // fp32
  const float* dy; int64_t lddy;
  const float* dt; const float* A;                       // (B,T,H), (H); NULL: x~ = x and da is the result
  const float* D;
  float* dx; uint16_t* dx16; int64_t lddx;
  int store_ops;                                         // x~ and dY go out as bf16 operands (maps xt, dy)
  float* da;                                             // (B,T,H)
  uint16_t *raw_hi, *raw_lo; int64_t ld_raw; int raw_col;                  // dt mode: gradient before the softplus as a bf16 pair (raw_lo may be NULL)
  float* part; int64_t part_pitch;                       // dt mode: per (b, h) sums for dA, dD and d_dt_bias, `part_pitch` apart
  int first, nseg, per;                                  // first chain of this launch (grid: chains x segments); segments of a sequence, steps per segment
  int late;                                              // needs nothing from the kernel before, which lets this one in after its own wait: waits when it is done
  int rows, fill;                                        // rows of `part` per (b, h); of them a block writes its own, a chain in one piece all (zeros: no more than a warp has lanes)
  int state_only;                                        // first of two passes over segments: only seg_h and seg_d are formed
  float *seg_h, *seg_d;                                  // (B*H-whole,nseg-1,N,P), (B*H-whole,nseg-1): adjoint that a segment hands back when it receives none, decay over it (nobody receives the first one's)
  uint32_t* flags;                                       // equal stretches of all chains: seg_h (CHAIN_SMS,N,P) and flags are the hand-overs
  unsigned int* status;
};

__device__ __forceinline__ uint32_t ld_shared(uint32_t a) { uint32_t v; asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a)); return v; }
__device__ __forceinline__ float2 bf2(uint32_t v) { return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u)); }

// On entry v[2 o + c] is a lane's sum over its four rows of column 8 o + 2 (lane & 3) + c of 32; on exit the lane returns the sum over the
// warp's 32 rows of the column column_of(lane).  Fixed order.
__device__ __forceinline__ float warp_column_sums32(float (&v)[8], int lane) {
#pragma unroll
  for (int w = 4; w >= 1; w >>= 1) {
    const bool upper = (lane & (4 * w)) != 0;
#pragma unroll
    for (int k = 0; k < w; ++k) {
      const float keep = upper ? v[k + w] : v[k], send = upper ? v[k] : v[k + w];
      v[k] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * w);
    }
  }
  return v[0];
}
__device__ __forceinline__ int column_of(int lane) { return 8 * (lane >> 3) + 2 * (lane & 3) + ((lane >> 2) & 1); }

template <int NI, int ND, int NK, bool IN16, bool WRAP>
__global__ void __launch_bounds__(NTHREADS, 1) ssd_chain_bwd_kernel(const __grid_constant__ Maps maps, const __grid_constant__ ChainWrap wr, const Params p) {
  using GE = Geo<NI, ND, NK, IN16>;
  constexpr int XB = GE::XB, NSB = GE::NSB;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - raw);
  const uint32_t b_s = base, c_s = b_s + GE::BT, hin_s = c_s + GE::BT, xbuf_s = base + GE::STAGE, dh_s = xbuf_s + XB * GE::XBUF, bars = dh_s + GE::HT;
  enum { FULL = 0, EMPTY, XRDY /*2*/, XFREE = XRDY + 2 /*2*/, SRDY = XFREE + 2 /*4*/, GFULL = SRDY + 4, MRDY, ACCFULL, ACCFREE, UFULL, UFREE, HRDY, HFREE,
         RRDY /*2*/, RFREE = RRDY + 2 /*2*/, XIN = RFREE + 2 /*2*/, NBAR = XIN + 2 };
  static_assert(8 * NBAR + 16 + 80 + 64 <= 512 && NSB <= 4, "barrier block");
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  uint8_t* bar_ptr = base_ptr + (bars - base);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bar_ptr + 8 * NBAR);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  float* ddw = reinterpret_cast<float*>(bar_ptr + 8 * NBAR + 16);      // [2 steps][4 state warps] <dh, h>
  float* dDw = ddw + 8;                                                // [8 transform warps] <dY, x>
  float* sWend = dDw + 8;                                              // [4 transform warps] S of their last token
  float* sM = sWend + 4;                                               // IN16: [NSB][4] m of 32 tokens
  float* sS = reinterpret_cast<float*>(bar_ptr + 512);                 // [NSB] S, dt and column factor exp(S_t - m) of a step's tokens, m = the largest S of the token's 32 and of the one before them
  float* sRows = sS + NSB * GE::SLOT;                                     // [2 steps] per-row sums

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int state_only = WRAP ? 0 : p.state_only, seg = WRAP ? 0 : (int)blockIdx.y + state_only;
  int bh = p.first + (int)blockIdx.x, n = min(p.per, p.nsteps - seg * p.per), last = seg * p.per + n - 1;      // chain, steps of this CTA, the last one of them
  if (WRAP) {
    const ChainItem it = chain_item(wr, (int)blockIdx.x, p.nsteps);
    bh = __shfl_sync(0xffffffffu, it.chain, 0); n = __shfl_sync(0xffffffffu, it.count, 0); last = p.nsteps - 1 - __shfl_sync(0xffffffffu, it.from, 0);      // (uniform, as the warp index)
    if (n <= 0) return;
  }
  const int h = bh % p.H, bb = bh / p.H, g = h / p.hpg;
  const int64_t tokb = (int64_t)bb * p.T;
  if (threadIdx.x == 0) {
    mbar_init(bar(FULL), 1); mbar_init(bar(EMPTY), state_only ? 1 : 6);
    for (int i = 0; i < 2; ++i) { mbar_init(bar(XIN + i), 1); mbar_init(bar(XRDY + i), 8); mbar_init(bar(XFREE + i), state_only ? 1 : IN16 ? 10 : 11); mbar_init(bar(RRDY + i), 12); mbar_init(bar(RFREE + i), 1); }
    for (int i = 0; i < 4; ++i) mbar_init(bar(SRDY + i), 8);
    mbar_init(bar(GFULL), 1); mbar_init(bar(MRDY), 8); mbar_init(bar(ACCFULL), 2); mbar_init(bar(ACCFREE), 8);
    mbar_init(bar(UFULL), 1); mbar_init(bar(UFREE), 4); mbar_init(bar(HRDY), 4); mbar_init(bar(HFREE), 1);
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
  if (WRAP || !p.late) pdl_wait();
  pdl_launch();
  const uint32_t tG = tmem, tM = tmem + 128, tA1 = tmem + 256, tA2 = tmem + 320, tA3 = tmem + 384, tU = tmem + 448;

  auto give_up = [&](unsigned int code) { atomicOr(p.status, code); *abort_flag = 1; };
  // bounded waits that also end as soon as another role of the CTA has given up
  auto wait = [&](int b, uint32_t parity, unsigned int code) -> bool {
    if (mbar_wait(bar(b), parity & 1u, 1u)) return true;
    if (*abort_flag) return false;
    if (mbar_wait(bar(b), parity & 1u)) return true;
    give_up(code);
    return false;
  };
  auto all = [&](bool v) -> bool { return __all_sync(0xffffffffu, v); };

  // k = 0, 1, ... counts the steps as they are walked; step last - k of the sequence
  if (warp < W_MASK) {
    regs_dec<56>();
    if (warp == 0) {
      // ---------------- TMA producer: B, C and the entering state ----------------
      if (lane == 0) {
        int issued = 0;
        int xissued = 0;
        // bf16: the operand tiles x~ and dY are the inputs as they are (two buffers: room for a step's is there before that for its other tiles)
        auto xload = [&](int k) -> bool {
          const int xb = k % XB;
          if (!wait(XFREE + xb, (uint32_t)(k / XB) ^ 1u, 4096u)) return false;
          mbar_expect_tx(bar(XIN + xb), (state_only ? 1 : 2) * T128);
          if (!state_only) tma_load_4d(xbuf_s + xb * GE::XBUF, &maps.xt[0], 0, (last - k) * L, h, bb, bar(XIN + xb));
          tma_load_4d(xbuf_s + xb * GE::XBUF + GE::XT, &maps.dy[0], 0, (last - k) * L, h, bb, bar(XIN + xb));
          xissued = k + 1;
          return true;
        };
        for (int k = 0; k < n; ++k) {
          const int i = last - k;
          if (IN16 && XB == 2 && !xload(k)) break;
          if (!wait(EMPTY, (uint32_t)k ^ 1u, 1u)) break;
          mbar_expect_tx(bar(FULL), state_only ? GE::BT : GE::STAGE);
#pragma unroll
          for (int kt = 0; kt < NK; ++kt) {
#pragma unroll
            for (int sp = 0; sp < NI; ++sp) {
              tma_load_4d(c_s + (sp * NK + kt) * T128, &maps.c[sp], 64 * kt, i * L, g, bb, bar(FULL));
              if (!state_only) tma_load_4d(b_s + (sp * NK + kt) * T128, &maps.b[sp], 64 * kt, i * L, g, bb, bar(FULL));
            }
#pragma unroll
            for (int sp = 0; sp < ND; ++sp)
              if (!state_only) tma_load_4d(hin_s + (sp * NK + kt) * T64, &maps.h[sp], 0, 64 * kt, h, bb * p.nsteps + i, bar(FULL));
          }
          issued = k + 1;
          if (IN16 && XB == 1 && !xload(k)) break;
        }
        if (*abort_flag && issued > 0) mbar_wait(bar(FULL), (uint32_t)((issued - 1) & 1));
        if (IN16 && *abort_flag)
          for (int k = (xissued > XB ? xissued - XB : 0); k < xissued; ++k) mbar_wait(bar(XIN + k % XB), (uint32_t)((k / XB) & 1));
      }
    } else if (warp == 1 || warp == 3) {
      // ---------------- MMA issuers (the whole warp waits; one elected lane issues) ----------------
      const uint32_t dhi = desc_hi(1024, 2);
      const uint32_t id_g = idesc_bf16(0, 0, L, L);            // both operands K-major
      const uint32_t id_v = idesc_bf16(0, 1, L, PW);           // B operand MN-major
      const uint32_t id_u = idesc_bf16(1, 1, L, PW);           // both operands MN-major
      const uint32_t BS = (NK * T128) >> 4, HS = (NK * T64) >> 4, XS = T128 >> 4;      // from a hi tile to its lo tile
      bool ok = !(warp == 1 && state_only);
#pragma unroll 1
      for (int k = 0; k < n && ok; ++k) {
        const int xb = k % XB;
        const uint32_t xt_s = xbuf_s + xb * GE::XBUF, dy_s = xt_s + GE::XT, dys_s = dy_s + GE::XT;
        auto xready = [&]() -> bool { return all(wait(XRDY + xb, (uint32_t)(k / XB), 2u) && (!IN16 || wait(XIN + xb, (uint32_t)(k / XB), 2u))); };
        if (!(ok = all(wait(FULL, (uint32_t)k, 2u)))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (warp == 1) {
          // the masked tile's: GT and dMT (both accumulators were read by the mask warps before they reported the last tile; the products that
          // read the masked tile over GT were issued before this)
          if (elect_one()) {
            const uint32_t b0 = desc_lo(b_s, 16), c0 = desc_lo(c_s, 16);
#pragma unroll
            for (int kt = 0; kt < NK; ++kt)
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const uint32_t o = (uint32_t)(kt * T128 + q * 32) >> 4;
                mma_split<NI, NI>(tG, b0 + o, BS, c0 + o, BS, dhi, id_g, (kt | q) ? 1u : 0u);
              }
            umma_commit(bar(EMPTY));
          }
          __syncwarp();
          if (!(ok = xready())) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (elect_one()) {
            const uint32_t x0 = desc_lo(xt_s, 16), y0 = desc_lo(dy_s, 16);
#pragma unroll
            for (int q = 0; q < 4; ++q) mma_split<NI, NI>(tM, x0 + 2 * q, XS, y0 + 2 * q, XS, dhi, id_g, q ? 1u : 0u);
            umma_commit(bar(GFULL));
          }
          __syncwarp();
          // MT dY, the masked tile read from TMEM: per 32 columns [hi: 16 | lo: 16], 8 columns per k-step of 16
          if (!(ok = all((k == 0 || wait(ACCFREE, (uint32_t)(k - 1), 8u)) && wait(MRDY, (uint32_t)k, 16u)))) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          if (elect_one()) {
            const uint32_t y0 = desc_lo(dy_s, T128);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              const uint32_t ta = tG + (uint32_t)((q >> 1) * 32 + (q & 1) * 8), vb = y0 + ((uint32_t)(q * 2048) >> 4);
              mma_split_ts<ND, NI>(tA1, ta, 16u, vb, XS, dhi, id_v, q ? 1u : 0u);
            }
            umma_commit(bar(ACCFULL));
            umma_commit(bar(XFREE + xb));
          }
          __syncwarp();
        } else {
          // the state's: B dh and C h, and U
          auto carried = [&]() -> bool {
            if (!all(wait(HRDY, (uint32_t)k, 8u) && (k == 0 || wait(ACCFREE, (uint32_t)(k - 1), 8u)))) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) {
              const uint32_t b0 = desc_lo(b_s, 16), c0 = desc_lo(c_s, 16), d0 = desc_lo(dh_s, T64), h0 = desc_lo(hin_s, T64);
#pragma unroll
              for (int kt = 0; kt < NK; ++kt)
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                  const uint32_t oa = (uint32_t)(kt * T128 + q * 32) >> 4, ob = (uint32_t)(kt * T64 + q * 2048) >> 4;
                  mma_split<NI, ND>(tA2, b0 + oa, BS, d0 + ob, HS, dhi, id_v, (kt | q) ? 1u : 0u);
                  mma_split<NI, ND>(tA3, c0 + oa, BS, h0 + ob, HS, dhi, id_v, (kt | q) ? 1u : 0u);
                }
              umma_commit(bar(ACCFULL));
              umma_commit(bar(HFREE));
              if (XB == 2) umma_commit(bar(EMPTY));
            }
            __syncwarp();
            return true;
          };
          auto update = [&]() -> bool {
            if (!(xready() && all(k == 0 || wait(UFREE, (uint32_t)(k - 1), 4u)))) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // U = C^T (exp(S) dY): the step's contribution to the state's adjoint (with one 64-wide block of d_state the second half
            // of M reads the tile behind it and its rows of U are never looked at)
            if (elect_one()) {
              const uint32_t cm = desc_lo(c_s, T128), y0 = desc_lo(dys_s, T128);
#pragma unroll
              for (int q = 0; q < 8; ++q) mma_split<NI, ND>(tU, cm + ((uint32_t)(q * 2048) >> 4), BS, y0 + ((uint32_t)(q * 2048) >> 4), XS, dhi, id_u, q ? 1u : 0u);
              umma_commit(bar(UFULL)); umma_commit(bar(XFREE + xb));
              if (XB == 1 || state_only) umma_commit(bar(EMPTY));
            }
            __syncwarp();
            return true;
          };
          // (two buffers: exp(S) dY has been there for a while, and the state's chain does not wait for the draining; one: it is being formed)
          if (!(ok = state_only ? update() : XB == 2 ? update() && carried() : carried() && update())) break;
          if (!IN16 && !state_only && lane == 0) {
            // x~ and dY go out as the operands that the sums over heads read
            if (p.store_ops) {
#pragma unroll
              for (int sp = 0; sp < NI; ++sp) {
                tma_store_4d(&maps.xt[sp], xt_s + sp * T128, 0, (last - k) * L, h, bb);
                tma_store_4d(&maps.dy[sp], dy_s + sp * T128, 0, (last - k) * L, h, bb);
              }
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
              asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            }
            mbar_arrive(bar(XFREE + xb));
          }
          __syncwarp();
        }
      }
      if (!IN16 && warp == 3 && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    } else if (state_only) {
    } else if (warp == 2) {
      // ---------------- per-token gradients (lane = four consecutive tokens) ----------------
      const bool dtm = p.dt != nullptr;
      const float Ah = dtm ? p.A[h] : 1.0f;
      float accA = 0.0f, accB = 0.0f;
      for (int k = 0; k < n; ++k) {
        const int i = last - k;
        if (!all(wait(SRDY + (k % NSB), (uint32_t)(k / NSB), 1024u) && wait(RRDY + (k & 1), (uint32_t)(k >> 1), 1024u))) break;
        const float4* R = reinterpret_cast<const float4*>(sRows + (k & 1) * GE::ROWS) + lane;
        const float* S = sS + (k % NSB) * GE::SLOT;
        const float4 S4 = reinterpret_cast<const float4*>(S)[lane], dt4 = reinterpret_cast<const float4*>(S + L)[lane];
        const float send = S[L - 1];
        auto two = [&](int a) { const float4 u = R[a * 32], v = R[(a + 1) * 32]; return make_float4(u.x + v.x, u.y + v.y, u.z + v.z, u.w + v.w); };
        const float4 r4 = two(0), e4 = two(2), f4 = two(4), w4 = R[6 * 32], ca = two(7), cb = two(9);
        const float Sv[4] = {S4.x, S4.y, S4.z, S4.w}, dtv[4] = {dt4.x, dt4.y, dt4.z, dt4.w};
        float qv[4] = {r4.x + w4.x, r4.y + w4.y, r4.z + w4.z, r4.w + w4.w};      // <dx~_s, x~_s> = sum_{t >= s} W[s,t] + e_s
        float d[4] = {ca.x + cb.x - r4.x, ca.y + cb.y - r4.y, ca.z + cb.z - r4.z, ca.w + cb.w - r4.w};
        const float ev[4] = {e4.x, e4.y, e4.z, e4.w}, fv[4] = {f4.x, f4.y, f4.z, f4.w};
        float es = 0.0f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float e = __expf(send - Sv[j]) * ev[j];
          es += e;
          qv[j] += e;
          d[j] += __expf(Sv[j]) * fv[j] - e;
        }
        es = warp_sum(es);
        const float* dw = ddw + (k & 1) * 4;
        if (lane == 31) d[3] += es + __expf(send) * ((dw[0] + dw[1]) + (dw[2] + dw[3]));
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(RFREE + (k & 1)));
        // reverse cumulative sum over the step
        d[2] += d[3]; d[1] += d[2]; d[0] += d[1];
        float tail = d[0];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const float u = __shfl_down_sync(0xffffffffu, tail, o); if (lane + o < 32) tail += u; }
        tail -= d[0];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int t = i * L + 4 * lane + j;
          if (t >= p.T) continue;
          const float da = d[j] + tail;
          if (p.da) p.da[(tokb + t) * p.H + h] = da;
          if (dtm) {
            // gradient w.r.t. the pre-softplus dt: (<dx~, x> + A da) (1 - exp(-dt)), with <dx~, x> = <dx~, x~> / dt
            const float sg = -expm1f(-dtv[j]);
            const float gr = fmaf(Ah * da, sg, qv[j] * (dtv[j] > 0.0f ? sg / dtv[j] : 1.0f));
            uint32_t hh, ll;
            split_bf16_pair(gr, hh, ll);
            const int64_t o = (tokb + t) * p.ld_raw + p.raw_col + h;
            p.raw_hi[o] = (uint16_t)hh;
            if (p.raw_lo) p.raw_lo[o] = (uint16_t)ll;
            accA = fmaf(da, dtv[j], accA);
            accB += gr;
          }
        }
      }
      if (dtm) {
        accA = warp_sum(accA); accB = warp_sum(accB);
        // (row of `part`: segment by segment of a sequence; a chain in one piece fills its rows with zeros)
        if (lane < p.fill) {
          const int64_t o = ((int64_t)bb * p.rows + seg + lane) * p.H + h;
          p.part[o] = lane == 0 ? accA : 0.0f; p.part[2 * p.part_pitch + o] = lane == 0 ? accB : 0.0f;
        }
      }
    }
  } else if (warp < W_XF) {
    regs_inc<88>();
    const int quarter = warp & 3, grp = (warp - W_MASK) >> 2;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const bool dtm = p.dt != nullptr;
    const float dv = p.D ? p.D[h] : 0.0f;
    const int er = quarter * 32 + (lane >> 2), ec = (lane & 3) * 2, cw = 32 * grp;
    // ---------------- output of a step: half of the columns, in pieces of 16 rows x 16 columns, fragments of 16 x 8 (whole 32-byte
    // sectors per store) ----------------
    auto output = [&](int k) -> bool {
      float* R = sRows + (k & 1) * GE::ROWS;
      const float* S = sS + (k % NSB) * GE::SLOT;
      const int xb = k % XB, i = last - k;
      const uint32_t xt_s = xbuf_s + xb * GE::XBUF, dy_s = xt_s + GE::XT;
      auto fetch = [&](int rh, int c16, float2 (&xo)[2][2], float2 (&yo)[2][2]) {
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const uint32_t at = (uint32_t)((er + 16 * rh + 8 * e) * 128) + (uint32_t)(((4 * grp + 2 * c16 + q) ^ (lane >> 2)) << 4) + (uint32_t)((lane & 3) * 4);
            xo[q][e] = bf2(ld_shared(xt_s + at)); yo[q][e] = bf2(ld_shared(dy_s + at));
            if (NI == 2) {
              const float2 xl = bf2(ld_shared(xt_s + T128 + at)), yl = bf2(ld_shared(dy_s + T128 + at));
              xo[q][e].x += xl.x; xo[q][e].y += xl.y; yo[q][e].x += yl.x; yo[q][e].y += yl.y;
            }
          }
      };
      if (!all(wait((IN16 ? XIN : XRDY) + xb, (uint32_t)(k / XB), 64u) && wait(ACCFULL, (uint32_t)k, 64u))) return false;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float send = S[L - 1];
      float fx[2], dtr[2], es[2], fs[2];
#pragma unroll 1
      for (int rh = 0; rh < 2; ++rh) {                      // 16 rows, in two pieces
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int row = er + 16 * rh + 8 * e;
          fx[e] = __expf(send - S[row]);
          dtr[e] = dtm ? S[L + row] : 1.0f;
          es[e] = fs[e] = 0.0f;
        }
#pragma unroll
        for (int c16 = 0; c16 < 2; ++c16) {
          float2 xn[2][2], yn[2][2];                        // [8-column group][row, row + 8]
          fetch(rh, c16, xn, yn);
          uint32_t a1[8], a2[8], a3[8];
          const uint32_t ta = lane_addr + ((uint32_t)(16 * rh) << 16) + (uint32_t)(cw + 16 * c16);
          tmem_ld16x256_x2(tA1 + ta, a1);
          tmem_ld16x256_x2(tA2 + ta, a2);
          tmem_ld16x256_x2(tA3 + ta, a3);
          tmem_wait_ld();
          float2 o[2][2];
#pragma unroll
          for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int r = 4 * q + 2 * e;
              const float2 yv = yn[q][e], xv = xn[q][e];
              const float u0 = __uint_as_float(a2[r]), u1 = __uint_as_float(a2[r + 1]);
              const float d0 = fmaf(fx[e], u0, __uint_as_float(a1[r])), d1 = fmaf(fx[e], u1, __uint_as_float(a1[r + 1]));
              es[e] = fmaf(u0, xv.x, fmaf(u1, xv.y, es[e]));
              fs[e] = fmaf(__uint_as_float(a3[r]), yv.x, fmaf(__uint_as_float(a3[r + 1]), yv.y, fs[e]));
              o[q][e] = make_float2(fmaf(d0, dtr[e], dv * yv.x), fmaf(d1, dtr[e], dv * yv.y));
            }
          if (rh == 1 && c16 == 1) {
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) { mbar_arrive(bar(ACCFREE)); mbar_arrive(bar(XFREE + xb)); }
          }
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int t = i * L + er + 16 * rh + 8 * e;
            if (!IN16) {
              if (t < p.T) {
                float* dr = p.dx + (tokb + t) * p.lddx + h * p.P + cw + 16 * c16 + ec;
#pragma unroll
                for (int q = 0; q < 2; ++q) if (cw + 16 * c16 + 8 * q < p.P) *reinterpret_cast<float2*>(dr + 8 * q) = o[q][e];
              }
            } else {
              // neighbouring lanes swap halves, so that a lane writes four columns and a quad one whole sector
              uint32_t v0, v1, z;
              split2(o[0][e].x, o[0][e].y, v0, z, false); split2(o[1][e].x, o[1][e].y, v1, z, false);
              const bool odd = lane & 1;
              const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? v0 : v1, 1);
              const uint2 wv = odd ? make_uint2(got, v1) : make_uint2(v0, got);
              if (t < p.T && cw + 16 * c16 + (odd ? 8 : 0) < p.P)
                *reinterpret_cast<uint2*>(p.dx16 + (tokb + t) * p.lddx + h * p.P + cw + 16 * c16 + ec + (odd ? 6 : 0)) = wv;
            }
          }
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
#pragma unroll
          for (int w = 1; w < 4; w <<= 1) {                 // the quad of lanes that shares a row
            es[e] += __shfl_xor_sync(0xffffffffu, es[e], w);
            fs[e] += __shfl_xor_sync(0xffffffffu, fs[e], w);
          }
          const int row = er + 16 * rh + 8 * e;
          if ((lane & 3) == 0) { R[(2 + grp) * L + row] = es[e]; R[(4 + grp) * L + row] = fs[e]; }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(RRDY + (k & 1)));
      return true;
    };
    // ---------------- mask groups: blocks of 32 columns, group g those of index g and g + 2 ----------------
    // Fragments of 16 rows x 8 columns: a lane holds rows fr + {0, 8, 16, 24} of the warp's 32 and two adjacent columns of every eight, so
    // a column's sum over the warp takes four additions in the lane and three exchanges of a halving number of columns.
    const int fr = lane >> 2, fc = 2 * (lane & 3);
    bool ok = !state_only;
#pragma unroll 1
    for (int k = 0; k < n && ok; ++k) {
      float* R = sRows + (k & 1) * GE::ROWS;
      const float* S = sS + (k % NSB) * GE::SLOT;
      ok = all((k < 2 || wait(RFREE + (k & 1), (uint32_t)((k >> 1) - 1), 32u)) && wait(SRDY + (k % NSB), (uint32_t)(k / NSB), 32u) &&
               wait(GFULL, (uint32_t)k, 32u));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      float Sr[4], rs[4] = {0.0f, 0.0f, 0.0f, 0.0f};        // rows fr + 8 e
#pragma unroll
      for (int e = 0; e < 4; ++e) Sr[e] = S[quarter * 32 + fr + 8 * e];
#pragma unroll 1
      for (int cb = grp; cb < 4; cb += 2) {
        const uint32_t tb = lane_addr + (uint32_t)(32 * cb);
        float cs[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) cs[e] = 0.0f;
        if (cb < quarter) {                                 // every column is before every row of this warp
          uint32_t z[16];
#pragma unroll
          for (int e = 0; e < 16; ++e) z[e] = 0u;
          tmem_st16(tG + tb, z);
          if (ND == 2) tmem_st16(tG + tb + 16u, z);
        } else {
          // past the diagonal (every column past every row): exp(S_t - S_s) = exp(S_t - m) exp(m - S_s), m as below where the factors are formed
          auto block = [&](auto diagonal) {
            constexpr bool DIAG = decltype(diagonal)::value;
            float rf[4];
            if (!DIAG) {
              const float m = IN16 ? sM[(k % NSB) * 4 + cb] : S[32 * cb - 1];
#pragma unroll
              for (int e = 0; e < 4; ++e) rf[e] = __expf(m - Sr[e]);
            }
            const float* Sc = S + (DIAG ? 0 : 2 * L) + 32 * cb + fc;      // S, or the columns' factors
#pragma unroll
            for (int rh = 0; rh < 2; ++rh) {
              const uint32_t at = tb + ((uint32_t)(16 * rh) << 16);
              uint32_t gr[16], dr[16], mh[8], ml[8];
              tmem_ld16x256_x4(tG + at, gr);
              tmem_ld16x256_x4(tM + at, dr);
              tmem_wait_ld();
#pragma unroll
              for (int o = 0; o < 4; ++o) {
                const float2 sv = *reinterpret_cast<const float2*>(Sc + 8 * o);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                  const int r = 4 * o + 2 * e;
                  float m0, m1, w0, w1;
                  if (!DIAG) {
                    m0 = __uint_as_float(gr[r]) * (rf[2 * rh + e] * sv.x); m1 = __uint_as_float(gr[r + 1]) * (rf[2 * rh + e] * sv.y);
                    w0 = m0 * __uint_as_float(dr[r]); w1 = m1 * __uint_as_float(dr[r + 1]);
                  } else {
                    const int d = 8 * o + fc - (fr + 8 * e + 16 * rh);    // column - row
                    m0 = __uint_as_float(gr[r]) * __expf(sv.x - Sr[2 * rh + e]); m1 = __uint_as_float(gr[r + 1]) * __expf(sv.y - Sr[2 * rh + e]);
                    m0 = d >= 0 ? m0 : 0.0f; m1 = d >= -1 ? m1 : 0.0f;
                    w0 = d >= 0 ? m0 * __uint_as_float(dr[r]) : 0.0f; w1 = d >= -1 ? m1 * __uint_as_float(dr[r + 1]) : 0.0f;
                    if (o == 2 * rh + e && (d == 0 || d == -1)) {          // (the diagonal lies in the fragments on it)
                      R[6 * L + quarter * 32 + fr + 8 * o] = d == 0 ? w0 : w1;
                      if (d == 0) w0 = 0.0f; else w1 = 0.0f;
                    }
                  }
                  rs[2 * rh + e] += w0 + w1;
                  cs[2 * o] += w0; cs[2 * o + 1] += w1;
                  ml[2 * o + e] = 0u;
                  split2(m0, m1, mh[2 * o + e], ml[2 * o + e], ND == 2);
                }
              }
              tmem_st16x128_x4(tG + at, mh);
              if (ND == 2) tmem_st16x128_x4(tG + at + 16u, ml);
            }
          };
          if (cb == quarter) block(std::true_type{}); else block(std::false_type{});
        }
        R[(7 + quarter) * L + 32 * cb + column_of(lane)] = cb < quarter ? 0.0f : warp_column_sums32(cs, lane);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        rs[e] += __shfl_xor_sync(0xffffffffu, rs[e], 1);
        rs[e] += __shfl_xor_sync(0xffffffffu, rs[e], 2);
        if ((lane & 3) == e) R[grp * L + quarter * 32 + fr + 8 * e] = rs[e];
      }
      tmem_wait_st();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(MRDY));
      ok = output(k);
    }
  } else if (warp < W_ST) {
    // ---------------- transform: x -> x~, dY -> dY and dY exp(S) ----------------
    regs_dec<72>();
    const int wx = warp - W_XF, tid = threadIdx.x - 32 * W_XF;
    const bool dtm = p.dt != nullptr;
    constexpr int LPR = IN16 ? 8 : 16;                      // lanes per row, 16 bytes each
    constexpr int RPI = 8 * (32 / LPR), NIT = L / RPI;    // rows per pass of the role, passes
    constexpr int EPL = IN16 ? 8 : 4;                       // elements per lane
    constexpr int AHEAD = GE::AHEAD;
    const int j = lane % LPR, r0 = wx * (32 / LPR) + lane / LPR;
    const bool jcol = EPL * j < p.P;
    const uint32_t place = (uint32_t)(r0 * 128) + (IN16 ? (uint32_t)((j ^ (r0 & 7)) << 4) : (uint32_t)((((j >> 1) ^ (r0 & 7)) << 4) + (j & 1) * 8));
    // every thread copies the pieces that it will read itself, AHEAD passes before it reads them (cp.async into slots of its own; no
    // barrier; rows past the end and columns past d_head arrive as zeros)
    const uint32_t ring = smem_u32(sRows + 2 * GE::ROWS) + (uint32_t)tid * 16u;
    constexpr uint32_t SLOT = 2 * XF_THREADS * 16;          // [x | dY]
    const char* xsrc = reinterpret_cast<const char*>(p.x) + (int64_t)(h * p.P + (jcol ? EPL * j : 0)) * 4;
    const char* ysrc = reinterpret_cast<const char*>(p.dy) + (int64_t)(h * p.P + (jcol ? EPL * j : 0)) * 4;
    int rrow = last * L + r0, rit = 0;                      // row and pass of the next piece to request; rows are walked up inside a step
    auto request = [&](uint32_t slot) {
      if (rrow >= (last - n + 1) * L) {
        const bool in = rrow < p.T && jcol;
        const int64_t tk = tokb + (rrow < p.T ? rrow : p.T - 1);      // (the address stays inside the tensor)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ring + slot), "l"(xsrc + tk * (p.ldx * 4)), "r"(in ? 16 : 0) : "memory");
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ring + slot + XF_THREADS * 16), "l"(ysrc + tk * (p.lddy * 4)), "r"(in ? 16 : 0) : "memory");
        rrow += RPI;
        if (++rit == NIT) { rit = 0; rrow -= 2 * L; }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const float* Sg = p.S + ((int64_t)bb * p.H + h) * p.T;
    float s_next = 0.0f, d_next = 1.0f;
    auto fetch_s = [&](int k) {                             // S and dt of this thread's token of the step
      if (tid >= L || k >= n) return;
      const int t = (last - k) * L + tid;
      s_next = Sg[t < p.T ? t : p.T - 1];                   // (a = 0 past the end)
      if (dtm) d_next = t < p.T ? p.dt[(tokb + t) * p.H + h] : 0.0f;
    };
    if (!IN16) {
#pragma unroll 1
      for (int q = 0; q < AHEAD; ++q) request((uint32_t)q * SLOT);
    }
    fetch_s(0);
    uint32_t slot = 0;
    float dD = 0.0f;
    bool ok = true;
    for (int k = 0; k < n; ++k) {
      const int xb = k % XB;
      float* S = sS + (k % NSB) * GE::SLOT;
      if (IN16 && ok) ok = all(wait(XIN + xb, (uint32_t)(k / XB), 128u));
      // fp32: S is formed ahead of the wait for the one buffer of x, whose transform is what every step waits for.  (Whoever reads the copy's old
      // entry, of step k - 4, has finished: the buffer of step k - 2 has been waited for, by fp32 in the step before, by bf16's loads here.
      // It is free when that step has been masked, for which the masks wait for the row sums of step k - 4, and when its product U
      // is done, which waits for the state warps' end of step k - 3.)
      const float sv = s_next;
      if (ok && tid < L) { S[tid] = sv; S[L + tid] = d_next; }
      if (lane == 31 && tid < L) sWend[wx] = sv;
      const float most = IN16 && tid < L ? warp_max(sv) : sv;       // (on its way while the warps meet)
      asm volatile("bar.sync 4, %0;" ::"n"(256) : "memory");        // (a warp that gave up keeps reaching the named barriers)
      if (ok && tid < L) {
        // m = the largest S of the 32 columns and of the token before them, that token's where a <= 0: as in the forward, no factor
        // exp(S_t - m) is above 1, and exp(m - S_s) overflows only where an exponential of the row does
        float m = sWend[wx > 0 ? wx - 1 : 0];
        if (IN16) m = fmaxf(m, most);
        S[2 * L + tid] = __expf(sv - m);
        if (IN16 && lane == 0) sM[(k % NSB) * 4 + wx] = m;
      }
      asm volatile("bar.sync 4, %0;" ::"n"(256) : "memory");
      if (!ok) continue;
      if (lane == 0) mbar_arrive(bar(SRDY + (k % NSB)));
      fetch_s(k + 1);
      if (!IN16 && k >= XB && !(ok = all(wait(XFREE + xb, (uint32_t)(k / XB - 1), 128u)))) continue;
      uint32_t dst = xbuf_s + xb * GE::XBUF + place;
#pragma unroll (IN16 ? 4 : 2)
      for (int it = 0; it < NIT; ++it, dst += RPI * 128) {
        uint4 xq = make_uint4(0u, 0u, 0u, 0u), yq;
        if (IN16) {
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(yq.x), "=r"(yq.y), "=r"(yq.z), "=r"(yq.w) : "r"(dst + GE::XT));
        } else {
          asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD > 0 ? AHEAD - 1 : 0) : "memory");
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(xq.x), "=r"(xq.y), "=r"(xq.z), "=r"(xq.w) : "r"(ring + slot) : "memory");
          asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(yq.x), "=r"(yq.y), "=r"(yq.z), "=r"(yq.w) : "r"(ring + slot + XF_THREADS * 16) : "memory");
        }
        const int row = it * RPI + r0;
        const float f = __expf(S[row]);
        if (IN16) {
          const uint32_t y4[4] = {yq.x, yq.y, yq.z, yq.w};
          uint32_t s4[4], k4[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) { const float2 v = bf2(y4[e]); split2(v.x * f, v.y * f, s4[e], k4[e], ND == 2); }
          st_shared_v4(dst + 2 * GE::XT, s4[0], s4[1], s4[2], s4[3]);
          if (ND == 2) st_shared_v4(dst + 2 * GE::XT + T128, k4[0], k4[1], k4[2], k4[3]);
        } else {
          const float dt = S[L + row];
          const float xv[4] = {__uint_as_float(xq.x), __uint_as_float(xq.y), __uint_as_float(xq.z), __uint_as_float(xq.w)};
          const float yv[4] = {__uint_as_float(yq.x), __uint_as_float(yq.y), __uint_as_float(yq.z), __uint_as_float(yq.w)};
          uint32_t h0, h1, l0 = 0u, l1 = 0u;
          split2(xv[0] * dt, xv[1] * dt, h0, l0, ND == 2); split2(xv[2] * dt, xv[3] * dt, h1, l1, ND == 2);
          st_shared_v2(dst, h0, h1);
          if (ND == 2) st_shared_v2(dst + T128, l0, l1);
          split2(yv[0], yv[1], h0, l0, ND == 2); split2(yv[2], yv[3], h1, l1, ND == 2);
          st_shared_v2(dst + GE::XT, h0, h1);
          if (ND == 2) st_shared_v2(dst + GE::XT + T128, l0, l1);
          split2(yv[0] * f, yv[1] * f, h0, l0, ND == 2); split2(yv[2] * f, yv[3] * f, h1, l1, ND == 2);
          st_shared_v2(dst + 2 * GE::XT, h0, h1);
          if (ND == 2) st_shared_v2(dst + 2 * GE::XT + T128, l0, l1);
#pragma unroll
          for (int e = 0; e < 4; ++e) dD = fmaf(xv[e], yv[e], dD);
        }
        if (!IN16) {
          request(slot);                                    // (this pass has consumed the slot)
          slot = slot + SLOT == AHEAD * SLOT ? 0u : slot + SLOT;
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(XRDY + xb));
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    dD = warp_sum(dD);
    if (lane == 0) dDw[wx] = dD;
  } else {
    // ---------------- state: dh in registers (thread = row n of the state) ----------------
    regs_inc<104>();
    const int quarter = warp & 3, nr = quarter * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const bool active = nr < p.N;                           // rows past d_state hold zeros
    const bool tile = quarter * 32 < 64 * NK;               // this warp's rows exist in the operand tile
    const bool kept = !state_only && quarter * 32 < p.N;      // (N <= 64 NK; rows from N on are outside the map)
    const int64_t NP = (int64_t)p.N * p.P;
    float hv[PW];
#pragma unroll
    for (int q = 0; q < PW; ++q) hv[q] = 0.0f;
    if (!WRAP && !state_only && active)
      for (int j = p.nseg - 1; j > seg; --j) {              // what the segments after this one hand back
        const int64_t row = (int64_t)(bh - p.first) * (p.nseg - 1) + j - 1;
        const float* F = p.seg_h + row * NP + (int64_t)nr * p.P;
        const float dj = p.seg_d[row];
#pragma unroll
        for (int q = 0; q < PW / 4; ++q) {
          if (4 * q >= p.P) continue;
          const float4 v = *reinterpret_cast<const float4*>(F + 4 * q);
          hv[4 * q] = fmaf(dj, hv[4 * q], v.x); hv[4 * q + 1] = fmaf(dj, hv[4 * q + 1], v.y);
          hv[4 * q + 2] = fmaf(dj, hv[4 * q + 2], v.z); hv[4 * q + 3] = fmaf(dj, hv[4 * q + 3], v.w);
          if (q % 4 == 3) asm volatile("" ::: "memory");      // (no more than four loads in flight: registers)
        }
      }
    bool ok = true;
    if (WRAP && last + 1 < p.nsteps) {            // the rest of a chain: dh comes from the CTA that walked its end
      const int from = wr.e[blockIdx.x % CHAIN_SMS].sm;
      ok = chain_take(p.flags + from, abort_flag);
      if (!ok) give_up(8192u);
      if (ok && active) {
        const float4* F = reinterpret_cast<const float4*>(p.seg_h + (int64_t)from * NP + (int64_t)nr * p.P);
#pragma unroll
        for (int q = 0; q < PW / 4; ++q) {
          if (4 * q >= p.P) continue;
          const float4 v = __ldcg(F + q);
          hv[4 * q] = v.x; hv[4 * q + 1] = v.y; hv[4 * q + 2] = v.z; hv[4 * q + 3] = v.w;
          if (q % 4 == 3) asm volatile("" ::: "memory");
        }
      }
    }
    float stot = 0.0f;
    for (int k = 0; k < n && ok; ++k) {
      const int i = last - k;
      if (!state_only) {
        if (k > 0) ok = all(wait(HFREE, (uint32_t)(k - 1), 256u));
        if (!ok) break;
        if (kept && k > 0) {                                  // (the stores of the adjoint before have read its rows)
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          __syncwarp();
        }
        if (tile) {
#pragma unroll
          for (int c = 0; c < 8; ++c) {                       // eight 16-byte chunks of the row
            uint32_t hi[4], lo[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int e = 0; e < 4; ++e) split2(hv[8 * c + 2 * e], hv[8 * c + 2 * e + 1], hi[e], lo[e], ND == 2);
            const uint32_t a = dh_s + (uint32_t)(nr * 128 + ((c ^ (nr & 7)) << 4));
            st_shared_v4(a, hi[0], hi[1], hi[2], hi[3]);
            if (ND == 2) st_shared_v4(a + NK * T64, lo[0], lo[1], lo[2], lo[3]);
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(HRDY));
        // dh goes out as it lies in the operand tile, a warp's 32 rows by themselves (stored by the threads that hold its rows, an instruction
        // touched 32 lines; backward of the scan at 9 x 1400 tokens, 32 heads of 64 x 64, kept as pairs, 216 -> 204 us, 16 x 1024 of 128 x 64
        // 225 -> 220, four layers of 2 x 384 on pairs 935 -> 927 in all)
        if (kept && lane == 0) {
          tma_store_4d(&maps.dh[0], dh_s + (uint32_t)quarter * (32 * 128), 0, quarter * 32, h, bb * p.nsteps + i);
          if (ND == 2) tma_store_4d(&maps.dh[1], dh_s + NK * T64 + (uint32_t)quarter * (32 * 128), 0, quarter * 32, h, bb * p.nsteps + i);
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
        // <dh, h>
        ok = all(wait(FULL, (uint32_t)k, 512u) && (k < 2 || wait(RFREE + (k & 1), (uint32_t)((k >> 1) - 1), 512u)));
        if (!ok) break;
        float dot = 0.0f;
        if (active) {
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const uint32_t a = hin_s + (uint32_t)(nr * 128 + ((c ^ (nr & 7)) << 4));
            uint32_t v[4];
#pragma unroll
            for (int sp = 0; sp < ND; ++sp) {
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(a + sp * NK * T64) : "memory");
#pragma unroll
              for (int e = 0; e < 4; ++e) { const float2 u = bf2(v[e]); dot = fmaf(u.x, hv[8 * c + 2 * e], fmaf(u.y, hv[8 * c + 2 * e + 1], dot)); }
            }
          }
        }
        dot = warp_sum(dot);
        if (lane == 0) {
          ddw[(k & 1) * 4 + quarter] = dot;
          mbar_arrive(bar(RRDY + (k & 1)));
          mbar_arrive(bar(EMPTY));
        }
      }
      ok = all(wait(SRDY + (k % NSB), (uint32_t)(k / NSB), 512u) && wait(UFULL, (uint32_t)k, 512u));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float send = sS[(k % NSB) * GE::SLOT + L - 1], dec = __expf(send);
      stot += send;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t u[16];
        tmem_ld16(tU + lane_addr + (uint32_t)(16 * q), u);
        tmem_wait_ld();
        if (active) {
#pragma unroll
          for (int e = 0; e < 16; ++e) hv[16 * q + e] = fmaf(dec, hv[16 * q + e], __uint_as_float(u[e]));
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(UFREE));
    }
    if (kept && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    const bool handed = WRAP && last + 1 > n;     // the end of a chain whose rest another CTA walks
    if (ok && (state_only || handed)) {
      const int64_t row = handed ? wr.e[blockIdx.x % CHAIN_SMS].sm + 1 : (int64_t)blockIdx.x * gridDim.y + blockIdx.y;
      if (nr == 0 && !handed) p.seg_d[row] = __expf(stot);
      float* dst = p.seg_h + row * NP + (int64_t)nr * p.P;
      if (active) {
#pragma unroll
        for (int q = 0; q < PW / 4; ++q)
          if (4 * q < p.P) *reinterpret_cast<float4*>(dst + 4 * q) = make_float4(hv[4 * q], hv[4 * q + 1], hv[4 * q + 2], hv[4 * q + 3]);
      }
      if (handed) chain_hand_over(p.flags + row);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if ((int)threadIdx.x < p.fill && p.part && !state_only) {
    float t = 0.0f;                                         // fixed order
    for (int q = 0; q < 8; ++q) t += dDw[q];
    p.part[p.part_pitch + ((int64_t)bb * p.rows + seg + threadIdx.x) * p.H + h] = threadIdx.x == 0 ? t : 0.0f;
  }
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
  }
  if (!WRAP && p.late) pdl_wait();                                  // (a kernel completes after those before it)
}

// ---- host side -------------------------------------------------------------------------------------------
static unsigned int* status_ptr() {
  static unsigned int* known[PMB_MAX_DEVICES] = {nullptr};
  return status_address(g_chain_bwd_status, known);
}

template <int NI, int ND, int NK, bool IN16>
static pmb_status launch(cudaStream_t st, const ChainBwdArgs& a) {
  using GE = Geo<NI, ND, NK, IN16>;
  static_assert(GE::SMEM <= 227 * 1024, "shared-memory plan");
  static_assert(IN16 ? NI == 1 : NI == ND, "fp32 tensors take pairs throughout");
  const int n = (int)cdiv(a.T, L);
  Maps ms{};
  for (int sp = 0; sp < 2; ++sp) {
    const bool lo = sp && NI == 2, lod = sp && ND == 2;
    const int64_t st_h = (int64_t)a.N * a.P, hp = (int64_t)a.H * a.P;
    PMB_TRY(sf::bf16_map4(&ms.b[sp], lo ? a.b.lo : a.b.hi, a.N, a.T, a.G, a.B, a.b.pitch, a.N, (int64_t)a.T * a.b.pitch, 64, L));
    PMB_TRY(sf::bf16_map4(&ms.c[sp], lo ? a.c.lo : a.c.hi, a.N, a.T, a.G, a.B, a.c.pitch, a.N, (int64_t)a.T * a.c.pitch, 64, L));
    PMB_TRY(sf::bf16_map4(&ms.h[sp], lod ? a.hp_lo : a.hp_hi, a.P, a.N, a.H, (int64_t)a.B * n, a.P, st_h, a.H * st_h, 64, 64));
    PMB_TRY(sf::bf16_map4(&ms.dh[sp], lod ? a.dh_lo : a.dh_hi, a.P, a.N, a.H, (int64_t)a.B * n, a.P, st_h, a.H * st_h, 64, 32));
    if (IN16 && !sp) {
      PMB_TRY(sf::bf16_map4(&ms.xt[0], a.x16, a.P, a.T, a.H, a.B, a.ldx, a.P, a.T * a.ldx, 64, L));
      PMB_TRY(sf::bf16_map4(&ms.dy[0], a.dy16, a.P, a.T, a.H, a.B, a.lddy, a.P, a.T * a.lddy, 64, L));
    }
    if (!IN16 && a.xt_hi) {
      PMB_TRY(sf::bf16_map4(&ms.xt[sp], lo ? a.xt_lo : a.xt_hi, a.P, a.T, a.H, a.B, hp, a.P, a.T * hp, 64, L));
      PMB_TRY(sf::bf16_map4(&ms.dy[sp], lo ? a.dyo_lo : a.dyo_hi, a.P, a.T, a.H, a.B, hp, a.P, a.T * hp, 64, L));
    }
  }
  Params p{};
  p.T = a.T; p.H = a.H; p.hpg = a.H / a.G; p.N = a.N; p.P = a.P; p.nsteps = n;
  p.S = a.S; p.x = a.x; p.ldx = a.ldx; p.dy = a.dy; p.lddy = a.lddy; p.dt = a.dt; p.A = a.A; p.D = a.D;
  p.dx = a.dx; p.dx16 = a.dx16; p.lddx = a.lddx; p.store_ops = a.xt_hi != nullptr; p.da = a.da;
  p.raw_hi = a.raw_hi; p.raw_lo = a.raw_lo; p.ld_raw = a.ld_raw; p.raw_col = a.raw_col; p.part = a.part; p.status = status_ptr();
  const int chains = a.B * a.H;
  ChainWrap wr{};
  if constexpr (IN16) {
    if (a.seg && !a.part && ssd_chain_wrap(chains, n, 1, 0.0, &wr)) {
      p.seg_h = a.seg; p.flags = ssd_chain_flags(a.seg, a.P, a.N);
      PMB_CUDA(cudaMemsetAsync(p.flags, 0, CHAIN_FLAG_BYTES, st));
      PMB_SMEM_OPT_IN(GE::SMEM, ssd_chain_bwd_kernel<NI, ND, NK, IN16, true>);
      return launch_pdl(st, ssd_chain_bwd_kernel<NI, ND, NK, IN16, true>, dim3((unsigned)(wr.rounds * CHAIN_SMS)), NTHREADS, GE::SMEM, ms, wr, p);
    }
  }
  const ChainPlan plan = a.seg ? ssd_chain_plan(a.B, a.T, a.H) : ChainPlan{chains, 1, n};
  const unsigned cut = (unsigned)((chains - plan.whole) * plan.nseg);      // blocks of segments
  if (cut) { p.seg_h = a.seg; p.seg_d = a.seg + (size_t)cut * a.N * a.P; }
  p.rows = plan.nseg; p.fill = 1; p.part_pitch = (int64_t)chains * plan.nseg;
  PMB_SMEM_OPT_IN(GE::SMEM, ssd_chain_bwd_kernel<NI, ND, NK, IN16, false>);
  auto run = [&](int count, int segments) { return launch_pdl(st, ssd_chain_bwd_kernel<NI, ND, NK, IN16, false>, dim3((unsigned)count, (unsigned)segments), NTHREADS, GE::SMEM, ms, wr, p); };
  // the segments' adjoints, the segments, and beside both the chains in one piece
  if (cut) {
    p.first = plan.whole; p.nseg = plan.nseg; p.per = plan.per;
    p.state_only = 1;
    PMB_TRY(run(chains - plan.whole, plan.nseg - 1));
    p.state_only = 0;
    PMB_TRY(run(chains - plan.whole, plan.nseg));
  }
  if (plan.whole) {
    p.first = 0; p.nseg = 1; p.per = n; p.late = cut > 0; p.fill = plan.nseg;
    PMB_TRY(run(plan.whole, 1));
  }
  return PMB_OK;
}

}  // namespace scb

pmb_status ssd_chain_bwd(cudaStream_t st, const ChainBwdArgs& a) {
  const bool pairs = a.b.lo != nullptr, in16 = a.x16 != nullptr;
  if (!ssd_chain_bwd_shape(a.P, a.N, pairs) || a.H % a.G != 0 || (int64_t)a.B * a.H > 0x7fffffff)
    return fail(PMB_ERR_UNSUPPORTED, "ssd_chain_bwd: unsupported shape (P=%d N=%d)", a.P, a.N);
  if (in16 == pairs || (in16 && (!a.dy16 || !a.dx16 || a.dt)) || (!in16 && (!a.x || !a.dy || !a.dx)) || (a.dt && (!a.A || !a.raw_hi || !a.part)))
    return fail(PMB_ERR_ARG, "ssd_chain_bwd: operands must be all pairs of fp32 values or all plain bf16");
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (!al16(a.x) || !al16(a.x16) || !al16(a.dy) || !al16(a.dy16) || !al16(a.dx) || !al16(a.dx16) || (a.ldx & (in16 ? 7 : 3)) || (a.lddy & (in16 ? 7 : 3)) || (a.lddx & 3))
    return fail(PMB_ERR_SHAPE, "ssd_chain_bwd: x, dy and dx rows must be 16-byte aligned");
  const double tok = (double)a.B * a.T;
  ProfScope prof(st, "ssd_chain_bwd", tok * a.H * ((double)SCAN_STEP * (a.N + 2.0 * a.P) + 6.0 * a.N * a.P), 0.0);
  if (pairs) return scb::launch<2, 2, 1, false>(st, a);
  if (a.hp_lo) return a.N > 64 ? scb::launch<1, 2, 2, true>(st, a) : scb::launch<1, 2, 1, true>(st, a);
  return a.N > 64 ? scb::launch<1, 1, 2, true>(st, a) : scb::launch<1, 1, 1, true>(st, a);
}

}  // namespace pmb

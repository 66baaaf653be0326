// Forward of the chunked SSD scan as one kernel (mamba2/ssd_ops.rs:167-284 computes the same chain op by op): one CTA
// owns one (batch, head) and walks its sequence in steps of 128 tokens with the state in registers, so that neither
// C B^T, nor the decay mask, nor the chunk states pass through HBM and a call is one launch.
//
// Per step (t, s = tokens of the step, S = inclusive cumulative sum of a inside it, h = state entering it):
//   x~[s,:] = x[s,:] dt[s],  xs[s,:] = x~[s,:] exp(S_end - S_s)             transform warps -> shared memory (bf16 operands)
//   G = C B^T   (128 x 128)                                                 tensor core, TMEM
//   M[t,s] = G[t,s] exp(S_t - S_s) [s <= t]                                 mask warps, TMEM -> registers -> TMEM over G
//   y[t,:] = M x~ + exp(S_t) C_t h + D x[t,:]                               tensor core, output warps
//   h <- exp(S_end) h + B^T xs                                              tensor core, state warps' registers
// S, xs and h can also be kept per chunk of two steps (plain bf16 operands): the second step's rows then see the first
// one's columns through a masked tile of their own and h as it entered the chunk.
// Operands are plain bf16 or (hi, lo) bf16 pairs: NI = 1 / 2 for x~, B and C, ND = 1 / 2 for what is formed here (M, xs, h).  fp32
// tensors take pairs throughout; bf16 tensors have inputs that are exact as they are, with (ND = 2) or without pairs of the rest.  Sequences of
// any length: rows past the end arrive as zeros (TMA fills them per batch) and carry a = 0.  d_state up to 128 and d_head
// up to 64, in multiples of 8: the 64-wide tiles are zero-filled beyond them.
//
// warp 0 = TMA loads (B, C, bf16 x), 1 = products of the masked tile (G one item ahead, M x~), 2 = products of the state (C h, U), 3 = TMA
// stores, 4..11 = two mask groups of four warps, then twelve warps of output and transform (eight and four; on fp32 pairs, whose
// transform rounds every element twice, four and eight), 24..27 = state.
// What bounds it: no pipe and no memory level.  A step takes 7000 warp instructions at d_state 128 on plain operands, issued in 45 % of the
// cycles; every role is a chain of TMEM loads, shared memory and arithmetic with two warps of it on a scheduler.  What shaped the roles are
// clocks read inside a step of 16 x 8192 tokens, 32 heads of 128 x 64, bf16 (927 us when masking and output were one role and one warp issued
// all products, 584 now):
//  - the products are issued by two warps: with one, its waits and the issue took 5000 of a step's 5200 clocks.  The warp index comes from a
//    shuffle, so that the roles' branches and the descriptors are uniform to the compiler (742 -> 711 us, this kernel alone);
//  - B and C are given back before the masked product waits for the mask, so that the next tiles (2200 clocks) land while it is masked;
//  - bf16 x is the operand x~ as it is and comes by TMA: copied by the transform warps, their few pieces in flight took 4200 clocks a step;
//  - a and dt are requested two chunks ahead (a head's tokens are a line apart), and below the diagonal the masked tile takes one
//    exponential per row and block of 32 columns instead of one per element (not where M is rounded for a stream of bf16 values, see FACT);
//  - the masked tile's exponents and products go in pairs, and a block whose smallest decay is a normal number takes exponentials without the scaling
//    that smaller ones need (16 x 8192 633 us with the scaling everywhere, 602 with it where needed; a bf16 block of 8 x 2048 tokens 317 and 315);
//  - the states that a backward reads leave by TMA from the operand tile, where they lie: stored by the threads that hold their rows, 32 lines to an
//    instruction, they took half of the state's 4900 clocks of a step's 5700 (16 x 8192 710 -> 622 us, 9 x 1400 of 64 x 64 118 -> 102,
//    16 x 512 of 128 x 64 61.5 -> 56.5);
//  - the kernel's 63 KB are about what the instruction cache holds for seven roles: an early return and a few selects by block, 72 KB, cost 8 %;
//  - the segment is the grid's y and not a remainder that stays in a register: on pairs its spills cost 10 % (24.6 -> 22.2 us at 4 x 512).
// Measured at 24 heads of 64 x 64: 23 us for 4 x 512 tokens on pairs, with what a backward reads or without; 8 x 2048 on
// plain operands in chunks of 256, 96 us, and 109 with all that a chunk-by-chunk backward reads (136 where every CTA walks whole chains, see
// ssd_chain_wrap); 30 us (two launches over segments) for 1 x 1337 on pairs.  Every mbarrier wait is bounded; on expiry the CTA raises the status
// word, every role stops issuing work, copies in flight are waited for (bounded) and TMEM is freed on the way out.
#include <cuda_bf16.h>
#include <algorithm>
#include <mutex>
#include <type_traits>
#include <unordered_map>
#include "tc_common.cuh"
#include "kernels.h"
#include "ssd_fused.h"
#include "ssd_wrap.cuh"

namespace pmb {

static __device__ unsigned int g_chain_status = 0;

pmb_status read_clear_device_status_chain(unsigned int* word) {
  unsigned int zero = 0;
  PMB_CUDA(cudaMemcpyFromSymbol(word, g_chain_status, sizeof(unsigned int)));
  if (*word) PMB_CUDA(cudaMemcpyToSymbol(g_chain_status, &zero, sizeof(unsigned int)));
  return PMB_OK;
}

namespace sc {

using namespace tcx;

constexpr int L = SCAN_STEP;            // tokens per step (= the MMA's M)
constexpr int PW = 64;                  // width of the head tile
constexpr int T128 = L * 128;           // bytes of a 128-row x 64-element bf16 tile (128-byte rows)
constexpr int T64 = 64 * 128;
// Seven warpgroups: 0 loads, stores and MMAs, 1 and 2 mask, then three of output and transform warps, 6 state.  setmaxnreg shares the
// block's 72 x 896 registers out by what a role keeps live.  Per thread: 40, 2 x 64 or 72, then 96 + 2 x 64 or 2 x 72 + 72, and 104.
constexpr int W_MASK = 4, W_OUT = 12, W_ST = 24, NWARPS = 28, NTHREADS = 32 * NWARPS;

// NB = 128-token blocks per chunk: S, the decay of xs and the state are relative to chunks of NB blocks.
template <int NI, int ND, int NK, int NB, bool XIN16>
struct Geo {
  // fp32 pairs spend most on the transform (two roundings of every element, twice), the others on the output
  static constexpr int OUTW = NI == 2 ? 4 : 8, XFW = 12 - OUTW, XF_THREADS = 32 * XFW;
  static constexpr int BT = NI * NK * T128;              // B (or C) of a step
  static constexpr int STAGE = 2 * BT;                   // [B | C]
  static constexpr int XT = NI * T128;                   // x~
  static constexpr int XBUF = XT + ND * T128;                    // [x~ | xs]
  static constexpr int HB = ND * NK * T64;               // state operand, rows n of 128 bytes
  static constexpr bool BIG = NI * NK == 4;              // pairs at d_state 128: one stage of B | C is all that fits
  static constexpr int STG = BIG ? 1 : 2;
  static constexpr int XB = ND == 1 ? 2 : 1;
  // copies of S: a chunk's S is read until its last tile has been masked and its output scaled, which the transform warps know of the
  // step XB + 2 (two blocks to a chunk: the chunk three) before the one they begin (see there)
  static constexpr int NSB = NB == 1 ? XB + 2 : 3;
  static_assert(NB == 1 || (STG == 2 && XB == 2), "both blocks of a chunk are resident");
  static constexpr int TILES = STG * STAGE + XB * XBUF + HB;
  // fp32 x: 16-byte pieces that every transform thread has in flight (bf16 x is copied into the operand tile as it is)
  static constexpr int AHEAD = BIG || XIN16 ? 0 : ND == 2 ? 3 : 16;
  // (BIG: no room for column factors and half of the alignment slack; shared memory starts 1024-byte aligned where nothing static
  // precedes it, and the kernel checks)
  // The masked tile by factors of blocks instead of an exponential per element.  Not for storage blocks on plain operands, whose M is rounded to
  // bf16 in a stream of bf16 values: a flipped rounding grows through the layers behind it, so that the gradients of 24 layers would move
  // by as much as bf16 storage itself puts them off fp64 (2e-2).  That is a choice, for results that repeat.
  static constexpr bool FACT = NB == 1 && !BIG && (ND == 2 || XIN16);
  static constexpr int BARS = XIN16 ? 320 : 256;         // bytes of barriers and small sums
  static constexpr int SLOT = (BIG ? 1 : 2) * L, SLACK = BIG ? 512 : 1024;    // floats per copy of S: [S | column factors]
  static constexpr int SMEM = TILES + SLACK + BARS + NSB * SLOT * 4 + (BIG ? 4 : 8) * NB * L /*row factors*/ + AHEAD * XF_THREADS * 16;
};

struct Maps { CUtensorMap b[2], c[2], x, xt, xs, h[2]; };      // [0] = hi (or the plain bf16 tensor), [1] = lo; x = bf16 x; h = the states kept, 32 rows to a box

struct Params {
  int T, H, hpg, N, P, nsteps;
  const float* x; int64_t ldx;                           // fp32
  const float* dt_raw; int64_t ld_raw; const float* dt_bias; const float* a_log;   // raw mode: dt and A are formed here
  const float* dt; const float* A; const float* a;                                 // (dt, A) or a alone
  const float* D;
  const float* init;                                     // (B,H,N,P) or NULL
  float* y; uint16_t* y16; int64_t ldy;
  float* dt_out; float* A_out; float* S_out;             // optional from here on: what a backward reads
  int keep_h;                                            // the states entering the chunks go out, (B,chunks,H,N,P)
  float* last;                                           // (B,H,N,P)
  // plain operands, for a backward that works chunk by chunk: state entering each chunk in fp32, and (store_ops) x~ and xs as the
  // kernel formed them.  bf16 x: store_ops leaves a copy of it.
  float* hprev;
  int store_ops;
  int first, nseg, per;                                  // first chain of this launch (grid: chains x segments); segments of a sequence, steps per segment
  int late;                                              // needs nothing from the kernel before, which lets this one in after its own wait: waits when it is done
  int state_only;                                        // first of two passes over segments: only seg_h and seg_d are formed
  float *seg_h, *seg_d;                                  // (B*H-whole,nseg-1,N,P), (B*H-whole,nseg-1): state that a segment leaves when it starts from none, decay over it (nobody reads the last one's)
  uint32_t* flags;                                       // equal stretches of all chains: seg_h (CHAIN_SMS,N,P) and flags are the hand-overs
  unsigned int* status;
};

template <int NI, int ND, int NK, int NB, bool XIN16, bool WRAP>
__global__ void __launch_bounds__(NTHREADS, 1) ssd_chain_fwd_kernel(const __grid_constant__ Maps maps, const __grid_constant__ ChainWrap wr, const Params p) {
  using GE = Geo<NI, ND, NK, NB, XIN16>;
  constexpr bool FACT = GE::FACT;
  constexpr int STG = GE::STG, XB = GE::XB, NSB = GE::NSB, OUTW = GE::OUTW, XFW = GE::XFW, XF_THREADS = GE::XF_THREADS, W_XF = W_OUT + OUTW;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  if (base - raw > (uint32_t)GE::SLACK) { if (threadIdx.x == 0) atomicOr(p.status, 4096u); return; }
  uint8_t* base_ptr = smem_raw + (base - raw);
  const uint32_t ring_s = base, xbuf_s = ring_s + STG * GE::STAGE, h_s = xbuf_s + XB * GE::XBUF, bars = h_s + GE::HB;
  enum { FULL = 0, EMPTY = 2, XRDY = 4, XFREE = 6, SRDY = 8 /*4*/, GFULL = 12, MRDY = 14, UFULL = 16, UFREE, HRDY, HFREE, ACCFULL, ACCFREE, XIN = 22 /*2*/, NBAR = 24 };
  static_assert(8 * NBAR + 8 + 48 + (XIN16 ? 64 : 0) <= GE::BARS && NSB <= 4, "barrier block");
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  uint8_t* bar_ptr = base_ptr + (bars - base);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bar_ptr + 8 * NBAR);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  float* wsum = reinterpret_cast<float*>(bar_ptr + 8 * NBAR + 8);
  float* sEnd = wsum + 8;                                   // S_end of the last four chunks
  float* sM = sEnd + 4;                                     // XIN16: [NSB][4] smallest S of 32 tokens
  float* sS = reinterpret_cast<float*>(bar_ptr + GE::BARS); // [NSB][S | FACT: exp(m - S), m = smallest S of the token's 32]
  float2* sfac = reinterpret_cast<float2*>(sS + NSB * GE::SLOT);    // (dt, exp(S_end - S)) of the step's rows
  float* sdt = sS + NSB * GE::SLOT;                                 // BIG: dt alone, the last kilobyte is not there

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int state_only = WRAP ? 0 : p.state_only;
  int bh = p.first + (int)blockIdx.x, i0 = (int)blockIdx.y * p.per, n = min(p.per, p.nsteps - i0);      // chain, first step and steps of this CTA
  if (WRAP) {
    const ChainItem it = chain_item(wr, (int)blockIdx.x, p.nsteps / NB);
    bh = __shfl_sync(0xffffffffu, it.chain, 0); i0 = __shfl_sync(0xffffffffu, NB * it.from, 0); n = __shfl_sync(0xffffffffu, NB * it.count, 0);      // (uniform to the compiler, as the warp index)
    if (n <= 0) return;
  }
  const int seg = WRAP ? 0 : (int)blockIdx.y;
  const int h = bh % p.H, bb = bh / p.H, g = h / p.hpg;
  const int toff = i0 * L;                                 // first token
  const int64_t tokb = (int64_t)bb * p.T;
  if (threadIdx.x == 0) {
    const int mmas = state_only ? 1 : 2;                  // warps that issue products
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(FULL + i), 1); mbar_init(bar(EMPTY + i), mmas);
      mbar_init(bar(XIN + i), 1); mbar_init(bar(XRDY + i), XFW); mbar_init(bar(XFREE + i), mmas + (p.store_ops ? 1 : 0));
      mbar_init(bar(GFULL + i), 1); mbar_init(bar(MRDY + i), 8);
    }
    for (int i = 0; i < 4; ++i) mbar_init(bar(SRDY + i), XFW);
    mbar_init(bar(UFULL), 1); mbar_init(bar(UFREE), 4); mbar_init(bar(HRDY), 4); mbar_init(bar(HFREE), 1);
    mbar_init(bar(ACCFULL), 2); mbar_init(bar(ACCFREE), OUTW);
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
  const uint32_t tG = tmem, tA1 = tmem + 256, tA2 = tmem + 320, tU = tmem + 384;

  auto give_up = [&](unsigned int code) { atomicOr(p.status, code); *abort_flag = 1; };
  // bounded waits that also end as soon as another role of the CTA has given up
  auto wait = [&](int b, uint32_t parity, unsigned int code) -> bool {
    if (mbar_wait(bar(b), parity & 1u, 1u)) return true;
    if (*abort_flag) return false;
    if (mbar_wait(bar(b), parity & 1u)) return true;
    give_up(code);
    return false;
  };

  if (warp < W_MASK) {
  regs_dec<40>();
  if (warp == 0) {
    // ---------------- TMA producer: B and C tiles of each step ----------------
    if (lane == 0) {
      int issued = 0, xissued = 0;
      for (int i = 0; i < n; ++i) {
        const int s = i % STG;
        if (!wait(EMPTY + s, (uint32_t)(i / STG) ^ 1u, 1u)) break;
        mbar_expect_tx(bar(FULL + s), state_only ? GE::BT : GE::STAGE);
        const uint32_t dst = ring_s + s * GE::STAGE;
#pragma unroll
        for (int sp = 0; sp < NI; ++sp)
#pragma unroll
          for (int kt = 0; kt < NK; ++kt) {
            tma_load_4d(dst + (sp * NK + kt) * T128, &maps.b[sp], 64 * kt, toff + i * L, g, bb, bar(FULL + s));
            if (!state_only) tma_load_4d(dst + GE::BT + (sp * NK + kt) * T128, &maps.c[sp], 64 * kt, toff + i * L, g, bb, bar(FULL + s));
          }
        issued = i + 1;
        if (XIN16) {                                         // bf16 x is the operand tile x~ as it is
          const int xb = i % XB;
          if (!wait(XFREE + xb, (uint32_t)(i / XB) ^ 1u, 2048u)) break;
          mbar_expect_tx(bar(XIN + xb), T128);
          tma_load_4d(xbuf_s + xb * GE::XBUF, &maps.x, 0, toff + i * L, h, bb, bar(XIN + xb));
          xissued = i + 1;
        }
      }
      if (*abort_flag) {
        for (int i = (issued > STG ? issued - STG : 0); i < issued; ++i) mbar_wait(bar(FULL + i % STG), (uint32_t)((i / STG) & 1));
        for (int i = (xissued > XB ? xissued - XB : 0); i < xissued; ++i) mbar_wait(bar(XIN + i % XB), (uint32_t)((i / XB) & 1));
      }
    }
  } else if ((XIN16 || ND == 1) && warp == 3 && p.store_ops) {
    // ---------------- x~ and xs go out as they lie in shared memory ----------------
    if (lane == 0) {
      for (int i = 0; i < n; ++i) {
        const int xb = i % XB;
        if (!wait((XIN16 ? XIN : XRDY) + xb, (uint32_t)(i / XB), 1024u)) break;
        tma_store_4d(&maps.xt, xbuf_s + xb * GE::XBUF, 0, toff + i * L, h, bb);
        if (!XIN16) tma_store_4d(&maps.xs, xbuf_s + xb * GE::XBUF + GE::XT, 0, toff + i * L, h, bb);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        mbar_arrive(bar(XFREE + xb));
      }
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
  } else if (warp == 1) {
    // ---------------- products of the masked tile: G and M x~ (the whole warp waits; one elected lane issues) ----------------
    const uint32_t dh = desc_hi(1024, 2);
    const uint32_t id_g = idesc_bf16(0, 0, L, L);            // G: both operands K-major
    const uint32_t id_v = idesc_bf16(0, 1, L, PW);           // x x~: B operand MN-major
    auto all = [&](bool v) -> bool { return __all_sync(0xffffffffu, v); };
    // G of the item (block k, earlier or same block kb of its chunk) into buffer m & 1
    auto mma_g = [&](int m, int k, int kb) -> bool {
      if (!all(wait(FULL + k % STG, (uint32_t)(k / STG), 2u))) return false;      // (block kb <= k has landed before)
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t b0 = desc_lo(ring_s + (kb % STG) * GE::STAGE, 16), c0 = desc_lo(ring_s + (k % STG) * GE::STAGE + GE::BT, 16);
      // (the buffer's previous content, the masked tile of item m - 2, is read by products issued before this one)
      if (elect_one()) {
#pragma unroll
        for (int kt = 0; kt < NK; ++kt)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint32_t o = (uint32_t)(kt * T128 + q * 32) >> 4;
            mma_split<NI, NI>(tG + (uint32_t)((m & 1) * L), c0 + o, (NK * T128) >> 4, b0 + o, (NK * T128) >> 4, dh, id_g, (kt | q) ? 1u : 0u);
          }
        umma_commit(bar(GFULL + (m & 1)));
        if (NB == 1 || k % NB > 0) umma_commit(bar(EMPTY + kb % STG));      // (that block's B and C have been in their last G)
      }
      __syncwarp();
      return true;
    };
    bool ok = !state_only && mma_g(0, 0, 0);
    int m = 0;                                               // item: (block, column block), the diagonal one last
#pragma unroll 1
    for (int k = 0; k < n && ok; ++k) {
      const int xb = k % XB, rb = k % NB;
#pragma unroll 1
      for (int cb = 0; cb <= rb; ++cb, ++m) {
        if (STG == 2) {                                      // one item ahead
          if (cb < rb) ok = mma_g(m + 1, k, k - rb + cb + 1);
          else if (k + 1 < n) ok = mma_g(m + 1, k + 1, k + 1 - (k + 1) % NB);
          if (!ok) break;
        }
        // acc1 += M x~, the masked tile read from TMEM: per 32 columns [hi: 16 | lo: 16], 8 columns per k-step of 16
        if (!(ok = all((cb < rb || wait((XIN16 ? XIN : XRDY) + xb, (uint32_t)(k / XB), 4u)) && (cb > 0 || k == 0 || wait(ACCFREE, (uint32_t)(k - 1), 8u)) &&
                       wait(MRDY + (m & 1), (uint32_t)(m >> 1), 16u)))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t xt0 = desc_lo(xbuf_s + ((k - rb + cb) % XB) * GE::XBUF, T128);
        if (elect_one()) {
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const uint32_t ta = tG + (uint32_t)((m & 1) * L + (q >> 1) * 32 + (q & 1) * 8), vb = xt0 + ((uint32_t)(q * 2048) >> 4);
            const uint32_t acc = (q | cb) ? 1u : 0u;
            mma_split_ts<ND, NI>(tA1, ta, 16u, vb, T128 >> 4, dh, id_v, acc);
          }
          if (cb == rb) umma_commit(bar(ACCFULL));
          if (cb < rb || rb == NB - 1) umma_commit(bar(XFREE + (k - rb + cb) % XB));      // (that block of the chunk is done with)
        }
        __syncwarp();
        if (STG == 1 && k + 1 < n) ok = mma_g(m + 1, k + 1, k + 1);
      }
    }
  } else if (warp == 2) {
    // ---------------- products of the state: C h and U (a warp of their own: the waits and the issue of one warp took 5000 of a
    // step's 5200 clocks) ----------------
    const uint32_t dh = desc_hi(1024, 2);
    const uint32_t id_v = idesc_bf16(0, 1, L, PW);           // x h: B operand MN-major
    const uint32_t id_u = idesc_bf16(1, 1, L, PW);           // B^T xs: both operands MN-major
    auto all = [&](bool v) -> bool { return __all_sync(0xffffffffu, v); };
    bool ok = true;
#pragma unroll 1
    for (int k = 0; k < n && ok; ++k) {
      const int s = k % STG, xb = k % XB, rb = k % NB, c = k / NB;
      // acc2 = C h
      auto carried = [&]() -> bool {
        if (!all(wait(FULL + s, (uint32_t)(k / STG), 4u) && wait(HRDY, (uint32_t)c, 8u) && (k == 0 || wait(ACCFREE, (uint32_t)(k - 1), 8u)))) return false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (elect_one()) {
          const uint32_t c0 = desc_lo(ring_s + s * GE::STAGE + GE::BT, 16), h0 = desc_lo(h_s, T64);
#pragma unroll
          for (int kt = 0; kt < NK; ++kt)
#pragma unroll
            for (int q = 0; q < 4; ++q)
              mma_split<NI, ND>(tA2, c0 + ((uint32_t)(kt * T128 + q * 32) >> 4), (NK * T128) >> 4, h0 + ((uint32_t)(kt * T64 + q * 2048) >> 4), (NK * T64) >> 4, dh, id_v,
                                (kt | q) ? 1u : 0u);
          umma_commit(bar(ACCFULL));
          if (XB == 2) umma_commit(bar(EMPTY + s));
          if (rb == NB - 1 || k + 1 == n) umma_commit(bar(HFREE));
        }
        __syncwarp();
        return true;
      };
      // U (+)= B^T xs: the chunk's contribution to the state
      auto update = [&]() -> bool {
        if (!all(wait(FULL + s, (uint32_t)(k / STG), 4u) && wait(XRDY + xb, (uint32_t)(k / XB), 4u) && (rb > 0 || c == 0 || wait(UFREE, (uint32_t)(c - 1), 4u)))) return false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (elect_one()) {
          // (M = 128 over one or two 64-wide blocks of d_state; with one block the second reads the tile behind it and
          // its rows of U are never looked at)
          const uint32_t b0 = desc_lo(ring_s + s * GE::STAGE, T128), xs0 = desc_lo(xbuf_s + xb * GE::XBUF + GE::XT, T128);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const uint32_t o = (uint32_t)(q * 2048) >> 4;
            mma_split<NI, ND>(tU, b0 + o, (NK * T128) >> 4, xs0 + o, T128 >> 4, dh, id_u, (q | rb) ? 1u : 0u);
          }
          if (rb == NB - 1 || k + 1 == n) umma_commit(bar(UFULL));
          umma_commit(bar(XFREE + xb));
          if (XB == 1 || state_only) umma_commit(bar(EMPTY + s));
        }
        __syncwarp();
        return true;
      };
      // (two buffers of x: xs has been there for a while, and the state's chain does not wait for C h; one: xs is being formed)
      ok = state_only ? update() : XB == 2 ? update() && carried() : carried() && update();
    }
  }
  } else if (warp < W_OUT) {
    // ---------------- mask groups: blocks of 32 columns, group g those of index g and g + 2 ----------------
    if (NI == 2) regs_dec<64>();
    const int quarter = warp & 3, grp = (warp - W_MASK) >> 2, r_local = quarter * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    bool ok = !state_only;
    int k = 0, rb = 0, kc = 0;                              // this item: block k = block rb of its chunk, column block kc
#pragma unroll 1
    for (int m = 0; k < n && ok; ++m) {
      const int c = k / NB;
      const float* S = sS + (c % NSB) * GE::SLOT;
      ok = __all_sync(0xffffffffu, wait(SRDY + (c % NSB), (uint32_t)(c / NSB), 32u) && wait(GFULL + (m & 1), (uint32_t)(m >> 1), 32u));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int diag = NB == 1 || kc == rb ? quarter : 4;   // the block of 32 columns that the diagonal crosses (none: all are before every row)
      const float S_row = S[rb * L + r_local];
      S += kc * L;                                          // of the columns
#pragma unroll 1
      for (int cb = grp; cb < 4; cb += 2) {
        const uint32_t tg = tG + lane_addr + (uint32_t)((m & 1) * L + 32 * cb);
        uint32_t mh[16], ml[16];
        if (cb > diag) {                                 // every column is past every row of this warp
#pragma unroll
          for (int e = 0; e < 16; ++e) { mh[e] = 0u; ml[e] = 0u; }
        } else {
          uint32_t r[32];
          tmem_ld32(tg, r);
          const F2 Sr2 = pack2(S_row, S_row), neg = pack2(-1.0f, -1.0f), log2e = pack2(1.4426950408889634f, 1.4426950408889634f);
          if (FACT && cb < diag) {
            // every column is before every row: exp(S_t - S_s) = exp(S_t - m) exp(m - S_s), m as below where the factors are formed
            const float rf = __expf(S_row - (XIN16 ? sM[(c % NSB) * 4 + cb] : S[32 * cb + 31]));
            const F2 rf2 = pack2(rf, rf);
#pragma unroll
            for (int e4 = 0; e4 < 8; ++e4) {
              const ulonglong2 cf = *reinterpret_cast<const ulonglong2*>(S + L + 32 * cb + 4 * e4);
              const float2 m0 = unpack2(mul2(pack2(__uint_as_float(r[4 * e4]), __uint_as_float(r[4 * e4 + 1])), mul2(rf2, cf.x)));
              const float2 m1 = unpack2(mul2(pack2(__uint_as_float(r[4 * e4 + 2]), __uint_as_float(r[4 * e4 + 3])), mul2(rf2, cf.y)));
              ml[2 * e4] = ml[2 * e4 + 1] = 0u;
              split2(m0.x, m0.y, mh[2 * e4], ml[2 * e4], ND == 2);
              split2(m1.x, m1.y, mh[2 * e4 + 1], ml[2 * e4 + 1], ND == 2);
            }
          } else {
            auto block = [&](auto normal) {
#pragma unroll
              for (int e4 = 0; e4 < 8; ++e4) {
                const ulonglong2 sv = *reinterpret_cast<const ulonglong2*>(S + 32 * cb + 4 * e4);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                  const int e2 = 2 * e4 + u;
                  const F2 x = mul2(fma2(u ? sv.y : sv.x, neg, Sr2), log2e);
                  float2 m = unpack2(mul2(pack2(__uint_as_float(r[2 * e2]), __uint_as_float(r[2 * e2 + 1])), decltype(normal)::value ? ex2_two_normal(x) : ex2_two(x)));
                  if (FACT || cb == diag) { m.x = 2 * e2 <= lane ? m.x : 0.0f; m.y = 2 * e2 + 1 <= lane ? m.y : 0.0f; }
                  ml[e2] = 0u;
                  split2(m.x, m.y, mh[e2], ml[e2], ND == 2);
                }
              }
            };
            // exp(S_t - S_s) of a block is a normal number (2^-125.5 and up) where that of the highest S_s is, for all rows
            if (__any_sync(0xffffffffu, S_row - warp_max(S[32 * cb + lane]) < -87.0f)) block(std::false_type{}); else block(std::true_type{});
          }
        }
        tmem_st16(tg, mh);
        if (ND == 2) tmem_st16(tg + 16u, ml);
      }
      tmem_wait_st();
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(MRDY + (m & 1)));
      if (kc == rb) { ++k; rb = rb + 1 == NB ? 0 : rb + 1; kc = 0; } else ++kc;
    }
  } else if (warp < W_XF) {
    // ---------------- output: drains the accumulators of a step while the next one is masked ----------------
    constexpr int NG = 8 / OUTW;                            // halves of the output columns that a warp takes
    if (NG == 2) regs_inc<96>();
    const int quarter = warp & 3, grp = NG == 1 ? (warp - W_OUT) >> 2 : 0;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const float dv = p.D ? p.D[h] : 0.0f;
    // fragments of 16 rows x 8 columns (a quad of lanes holds 8 columns of a row: whole 32-byte sectors per store): this thread's
    // output rows are er + {0, 8, 16, 24}
    const int er = quarter * 32 + (lane >> 2), cw = 32 * grp, col = h * p.P + cw + (lane & 3) * 2;
    bool ok = !state_only;
#pragma unroll 1
    for (int k = 0; k < n && ok; ++k) {
      const int c = k / NB;
      const float* S = sS + (c % NSB) * GE::SLOT + (k % NB) * L;
      const int t0 = toff + k * L + er;
      float2 o[2][4 * NG][2];                               // [16-row half][8-column group][row, row + 8]
      auto fetch_x = [&](int rh, int q, int e) -> float2 {  // the skip term's x
        const int t = t0 + 16 * rh + 8 * e;
        return p.D && t < p.T && cw + 8 * q < p.P ? *reinterpret_cast<const float2*>(p.x + (tokb + t) * p.ldx + col + 8 * q) : make_float2(0.0f, 0.0f);
      };
      if (!XIN16 && NG == 1) {                              // (requested ahead of the accumulators)
#pragma unroll
        for (int rh = 0; rh < 2; ++rh)
#pragma unroll
          for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int q = 0; q < 4; ++q) o[rh][q][e] = fetch_x(rh, q, e);
      }
      ok = __all_sync(0xffffffffu, wait(SRDY + (c % NSB), (uint32_t)(c / NSB), 64u));
      if (!ok) break;
      float f[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) f[e] = __expf(S[er + 8 * e]);
      ok = __all_sync(0xffffffffu, wait(ACCFULL, (uint32_t)k, 64u));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int rh = 0; rh < 2; ++rh)
#pragma unroll
        for (int c16 = 0; c16 < 2 * NG; ++c16) {
          uint32_t a1[8], a2[8];
          const uint32_t ta = lane_addr + ((uint32_t)(16 * rh) << 16) + (uint32_t)(cw + 16 * c16);
          tmem_ld16x256_x2(tA1 + ta, a1);
          tmem_ld16x256_x2(tA2 + ta, a2);
          tmem_wait_ld();
#pragma unroll
          for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int r = 4 * q + 2 * e;
              float2& v = o[rh][2 * c16 + q][e];
              const float u0 = fmaf(f[2 * rh + e], __uint_as_float(a2[r]), __uint_as_float(a1[r])), u1 = fmaf(f[2 * rh + e], __uint_as_float(a2[r + 1]), __uint_as_float(a1[r + 1]));
              v = XIN16 || NG == 2 ? make_float2(u0, u1) : make_float2(fmaf(dv, v.x, u0), fmaf(dv, v.y, u1));
            }
        }
      // handed back before anything waits for memory
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(ACCFREE));
#pragma unroll
      for (int rh = 0; rh < 2; ++rh)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int t = t0 + 16 * rh + 8 * e;
          if (!XIN16) {
            if (NG == 2) {
              float2 x[4 * NG];
#pragma unroll
              for (int q = 0; q < 4 * NG; ++q) x[q] = fetch_x(rh, q, e);
#pragma unroll
              for (int q = 0; q < 4 * NG; ++q) o[rh][q][e] = make_float2(fmaf(dv, x[q].x, o[rh][q][e].x), fmaf(dv, x[q].y, o[rh][q][e].y));
            }
            if (t < p.T) {
              float* yr = p.y + (tokb + t) * p.ldy + col;
#pragma unroll
              for (int q = 0; q < 4 * NG; ++q) if (cw + 8 * q < p.P) *reinterpret_cast<float2*>(yr + 8 * q) = o[rh][q][e];
            }
          } else {
            // neighbouring lanes swap halves, so that a lane writes four columns and a quad one whole sector
#pragma unroll
            for (int q = 0; q < 4 * NG; q += 2) {
              uint32_t v0, v1, z;
              split2(o[rh][q][e].x, o[rh][q][e].y, v0, z, false); split2(o[rh][q + 1][e].x, o[rh][q + 1][e].y, v1, z, false);
              const bool odd = lane & 1;
              const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? v0 : v1, 1);
              const uint2 w = odd ? make_uint2(got, v1) : make_uint2(v0, got);
              // even lanes: the lane's columns and the next two of the first eight; odd lanes: the two before and its own of the second
              if (t < p.T && cw + 8 * (q + (odd ? 1 : 0)) < p.P)
                *reinterpret_cast<uint2*>(p.y16 + (tokb + t) * p.ldy + col + 8 * q + (odd ? 6 : 0)) = w;
            }
          }
        }
    }
  } else if (warp < W_ST) {
    // ---------------- transform: S of the step, x -> x~ and xs ----------------
    if (XFW == 8) regs_dec<64>();
    const int wx = warp - W_XF, tid = threadIdx.x - 32 * W_XF;
    const float Ah = p.dt_raw ? -expf(p.a_log[h]) : (p.dt ? p.A[h] : 1.0f);
    const float bias = p.dt_raw ? p.dt_bias[h] : 0.0f;
    if (p.dt_raw && p.A_out && bb == 0 && tid == 0) p.A_out[h] = Ah;
    constexpr int LPR = XIN16 ? 8 : 16;                     // lanes per row, 16 bytes each
    constexpr int RPI = XFW * (32 / LPR), NIT = L / RPI;    // rows per pass of the role, passes
    constexpr int EPL = XIN16 ? 8 : 4;                      // elements per lane
    const int j = lane % LPR, r0 = wx * (32 / LPR) + lane / LPR;
    const bool jcol = EPL * j < p.P;
    // this lane's place in a row of an operand tile (rows of 128 bytes, 16-byte pieces xor-swizzled by the row)
    const uint32_t place = (uint32_t)(r0 * 128) + (XIN16 ? (uint32_t)((j ^ (r0 & 7)) << 4) : (uint32_t)((((j >> 1) ^ (r0 & 7)) << 4) + (j & 1) * 8));
    // x: every thread copies the pieces that it will read itself, AHEAD passes before it reads them, into a ring of its own
    // (cp.async; no barrier; rows past the end arrive as zeros)
    constexpr int RING = GE::AHEAD > 0 ? GE::AHEAD : 1;
    // Pieces that a thread takes, and requests, together: one by one, a piece's wait, shared memory and roundings were a chain of their own, and on plain
    // operands this role is the busiest (6700 of a step's 6900 clocks).  Block forward of 24 heads, chunks of 256, 8 x 2048 tokens 317 -> 314 us,
    // 8 x 4096 580 -> 574.  S formed a chunk ahead by warp 3 alone, which takes it out of this role, lost: 16 x 8192 of bf16 x 2342 -> 2448
    constexpr int UB = RING % 4 == 0 ? 4 : 1;
    static_assert(RING == 1 || UB == 1 || RING == NIT, "a ring of a step's pieces");
    const uint32_t xring = smem_u32(sfac + NB * L) + (uint32_t)tid * 16u;
    const char* src = reinterpret_cast<const char*>(p.x + (tokb + toff + r0) * p.ldx + h * p.P + (jcol ? EPL * j : 0));
    const int64_t sstep = (int64_t)RPI * p.ldx * 4;
    int frow = toff + r0;                                          // row of the next piece to request
    auto request = [&](uint32_t slot) {
      const bool in = frow < p.T && jcol;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(xring + slot), "l"(src), "r"(in ? 16 : 0) : "memory");
      frow += RPI;
      if (frow < p.T) src += sstep;                         // (the address stays inside the tensor)
    };
    constexpr int TPT = NB * L > XF_THREADS ? NB * L / XF_THREADS : 1;      // tokens of a chunk per thread
    float av[TPT], an[TPT];                                 // requested two chunks ahead: the tokens of a head are a line apart
    auto fetch_a = [&](int c, float (&av)[TPT]) {           // of this thread's tokens of chunk c
#pragma unroll
      for (int u = 0; u < TPT; ++u) {
        const int t = toff + c * NB * L + u * XF_THREADS + tid;
        const int64_t tk = tokb + t;
        av[u] = 0.0f;
        if (tid < NB * L && t < p.T) av[u] = p.dt_raw ? p.dt_raw[tk * p.ld_raw + h] : p.dt ? p.dt[tk * p.H + h] : p.a[tk * p.H + h];
      }
    };
    if (GE::AHEAD > 0) {
      if (frow >= p.T) src = reinterpret_cast<const char*>(p.x);
#pragma unroll 1
      for (int q = 0; q < RING; ++q) {
        request((uint32_t)q * (XF_THREADS * 16));
        if (q % UB == UB - 1) asm volatile("cp.async.commit_group;" ::: "memory");
      }
    }
    fetch_a(0, av);
    fetch_a(1, an);
    uint32_t slot = 0;
    bool ok = true;
    for (int i = 0; i < n; ++i) {
      const int c = i / NB, rb = i % NB;
      float* S = sS + (c % NSB) * GE::SLOT;
      if (rb == 0) {
        // S of the chunk.  A warp that gave up keeps reaching the named barriers: it skips the work, not the barrier.
        float dtv[TPT], v[TPT], least[TPT];
#pragma unroll
        for (int u = 0; u < TPT; ++u) {
          const bool in = toff + c * NB * L + u * XF_THREADS + tid < p.T;
          dtv[u] = 1.0f; v[u] = av[u];
          if (p.dt_raw) { dtv[u] = in ? softplus_acc(av[u] + bias) : 0.0f; v[u] = Ah * dtv[u]; }
          else if (p.dt) { dtv[u] = av[u]; v[u] = Ah * av[u]; }
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) { const float w = __shfl_up_sync(0xffffffffu, v[u], o); if (lane >= o) v[u] += w; }
          if (lane == 31 && tid < NB * L) wsum[u * XFW + wx] = v[u];
          if (FACT && XIN16) least[u] = warp_min(v[u]);     // (on its way while the warps meet)
        }
        asm volatile("bar.sync 4, %0;" ::"n"(XF_THREADS) : "memory");
        if (tid < NB * L) {
          float off[TPT], send = 0.0f;                      // fixed order
#pragma unroll
          for (int q = 0; q < 4 * NB; ++q) { if (q % XFW == wx) off[q / XFW] = send; send += wsum[q]; }
          // (nobody reads the buffer's old content any more: in the step before this one the thread has waited for the products of step
          // i - 1 - XB, which follow the masking of that step and the draining of the one before, and with it of everything earlier)
#pragma unroll
          for (int u = 0; u < TPT; ++u) {
            const int q = u * XF_THREADS + tid, t = toff + c * NB * L + q;
            v[u] += off[u];
            if (q == NB * L - 1) v[u] = send;
            S[q] = v[u];
            if (FACT) {
              // m = the smallest S of the 32 columns, their last where a <= 0.  Where a is positive for a while (bf16 x comes with any a)
              // S can rise and fall by more than fp32's exponent inside a step: no factor exp(m - S_s) is above 1, and exp(S_t - m)
              // overflows only where an exponential of the row does.
              const float m = XIN16 ? least[u] + off[u] : __shfl_sync(0xffffffffu, v[u], 31);
              S[L + q] = __expf(m - v[u]);
              if (XIN16 && lane == 0) sM[(c % NSB) * 4 + q / 32] = m;
            }
            if (GE::BIG) sdt[q] = dtv[u]; else sfac[q] = make_float2(dtv[u], __expf(send - v[u]));
            if (q == NB * L - 1) sEnd[c & 3] = send;
            if (t < p.T) {
              if (p.S_out && !state_only) p.S_out[((int64_t)bb * p.H + h) * p.T + t] = v[u];
              if (p.dt_out && !state_only) p.dt_out[(tokb + t) * p.H + h] = dtv[u];
            }
          }
        }
        asm volatile("bar.sync 4, %0;" ::"n"(XF_THREADS) : "memory");
        if (lane == 0) mbar_arrive(bar(SRDY + (c % NSB)));
#pragma unroll
        for (int u = 0; u < TPT; ++u) av[u] = an[u];
        if (i + 2 * NB < n) fetch_a(c + 2, an);
      }
      if (ok && XIN16) ok = __all_sync(0xffffffffu, wait(XIN + (i % XB), (uint32_t)(i / XB), 128u));
      else if (ok && i >= XB) ok = __all_sync(0xffffffffu, wait(XFREE + (i % XB), (uint32_t)(i / XB - 1), 128u));
      if (ok) {
        uint32_t dst = xbuf_s + (i % XB) * GE::XBUF + place;
#pragma unroll (XIN16 ? 4 : UB == 1 ? 2 : 1)
        for (int it = 0; it < NIT; it += UB, dst += UB * RPI * 128) {
          uint4 xq[UB];
          if (GE::AHEAD > 0) asm volatile("cp.async.wait_group %0;" ::"n"(RING / UB - 1) : "memory");
#pragma unroll
          for (int u = 0; u < UB; ++u) {
            xq[u] = make_uint4(0u, 0u, 0u, 0u);
            if (XIN16) {
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(xq[u].x), "=r"(xq[u].y), "=r"(xq[u].z), "=r"(xq[u].w) : "r"(dst));
            } else if (GE::AHEAD > 0) {
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(xq[u].x), "=r"(xq[u].y), "=r"(xq[u].z), "=r"(xq[u].w) : "r"(xring + slot + (uint32_t)(u * XF_THREADS * 16)) : "memory");
            } else {
              if (frow < p.T && jcol) xq[u] = *reinterpret_cast<const uint4*>(src);
              frow += RPI; src += sstep;
            }
          }
#pragma unroll
          for (int u = 0; u < UB; ++u) {
            const uint32_t du = dst + (uint32_t)(u * RPI * 128);
            const int rc = rb * L + (it + u) * RPI + r0;      // row of the chunk
            const float2 f = GE::BIG ? make_float2(sdt[rc], __expf(sEnd[c & 3] - S[rc])) : sfac[rc];
            if (XIN16) {
              const uint32_t in4[4] = {xq[u].x, xq[u].y, xq[u].z, xq[u].w};
              uint32_t s4[4], k4[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) split2(__uint_as_float(in4[e] << 16) * f.y, __uint_as_float(in4[e] & 0xffff0000u) * f.y, s4[e], k4[e], ND == 2);
              st_shared_v4(du + GE::XT, s4[0], s4[1], s4[2], s4[3]);
              if (ND == 2) st_shared_v4(du + GE::XT + T128, k4[0], k4[1], k4[2], k4[3]);
            } else {
              const float x0 = __uint_as_float(xq[u].x), x1 = __uint_as_float(xq[u].y), x2 = __uint_as_float(xq[u].z), x3 = __uint_as_float(xq[u].w);
              const float f0 = x0 * f.x, f1 = x1 * f.x, f2 = x2 * f.x, f3 = x3 * f.x;
              uint32_t h0, h1, l0 = 0u, l1 = 0u, g0, g1, k0 = 0u, k1 = 0u;
              split2(f0, f1, h0, l0, ND == 2); split2(f2, f3, h1, l1, ND == 2);
              if (ND == 2) { split2(f0 * f.y, f1 * f.y, g0, k0, true); split2(f2 * f.y, f3 * f.y, g1, k1, true); }
              else {                                          // (x (dt exp): rounded as the chunk-by-chunk kernels round it)
                const float fx = f.x * f.y;
                split2(x0 * fx, x1 * fx, g0, k0, false); split2(x2 * fx, x3 * fx, g1, k1, false);
              }
              st_shared_v2(du, h0, h1);
              st_shared_v2(du + GE::XT, g0, g1);
              if (ND == 2) { st_shared_v2(du + T128, l0, l1); st_shared_v2(du + GE::XT + T128, k0, k1); }
            }
          }
          if (GE::AHEAD > 0) {                              // (this pass has consumed the slots)
#pragma unroll
            for (int u = 0; u < UB; ++u) request(slot + (uint32_t)(u * XF_THREADS * 16));
            asm volatile("cp.async.commit_group;" ::: "memory");
            slot = slot + UB * XF_THREADS * 16 == RING * XF_THREADS * 16 ? 0u : slot + UB * XF_THREADS * 16;
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(XRDY + (i % XB)));
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    // ---------------- state: h in registers (thread = row n of the state) ----------------
    regs_inc<104>();
    const int quarter = warp & 3, nr = quarter * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const bool active = nr < p.N;                           // rows past d_state hold zeros
    const bool tile = quarter * 32 < 64 * NK;               // this warp's rows exist in the operand tile
    const bool kept = p.keep_h && !state_only && quarter * 32 < p.N;      // (N <= 64 NK; rows from N on are outside the map)
    const int64_t NP = (int64_t)p.N * p.P;
    float hv[PW];
    bool ok = true;
    const float* enters = p.init && !state_only ? p.init + ((int64_t)bb * p.H + h) * NP : nullptr;
    if (WRAP && i0 > 0) {                                   // the rest of a chain: the state comes from the CTA that walked its beginning
      const int from = wr.e[blockIdx.x % CHAIN_SMS].sm;
      ok = chain_take(p.flags + from, abort_flag);
      if (!ok) give_up(8192u);
      enters = p.seg_h + (int64_t)from * NP;
    }
#pragma unroll
    for (int q = 0; q < PW / 4; ++q) {
      float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (enters && active && 4 * q < p.P) v = __ldcg(reinterpret_cast<const float4*>(enters + (int64_t)nr * p.P + 4 * q));
      hv[4 * q] = v.x; hv[4 * q + 1] = v.y; hv[4 * q + 2] = v.z; hv[4 * q + 3] = v.w;
    }
    if (!WRAP && !state_only && active)
      for (int j = 0; j < seg; ++j) {                       // what the segments before this one leave
        const int64_t row = (int64_t)(bh - p.first) * (p.nseg - 1) + j;
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
    float stot = 0.0f;
    const int nch = (n + NB - 1) / NB, ncht = (p.nsteps + NB - 1) / NB;
    for (int i = 0; i < nch && ok; ++i) {                   // chunk after chunk
      if (i > 0 && !state_only) ok = __all_sync(0xffffffffu, wait(HFREE, (uint32_t)(i - 1), 256u));
      if (!ok) break;
      const int64_t so = (((int64_t)bb * ncht + i0 / NB + i) * p.H + h) * NP + (int64_t)nr * p.P;
      if (kept && i > 0) {                                  // (the stores of the state before have read its rows)
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncwarp();
      }
      if (tile && !state_only) {
#pragma unroll
        for (int c = 0; c < 8; ++c) {                       // eight 16-byte chunks of the row
          uint32_t hi[4], lo[4] = {0u, 0u, 0u, 0u};
#pragma unroll
          for (int e = 0; e < 4; ++e) split2(hv[8 * c + 2 * e], hv[8 * c + 2 * e + 1], hi[e], lo[e], ND == 2);
          const uint32_t a = h_s + (uint32_t)(nr * 128 + ((c ^ (nr & 7)) << 4));
          st_shared_v4(a, hi[0], hi[1], hi[2], hi[3]);
          if (ND == 2) st_shared_v4(a + NK * T64, lo[0], lo[1], lo[2], lo[3]);
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(HRDY));
      // What a backward keeps goes out as it lies in the operand tile, a warp's 32 rows by themselves, under the products that read it (a thread
      // that stored its own row would touch 32 lines with every instruction)
      if (kept && lane == 0) {
        tma_store_4d(&maps.h[0], h_s + (uint32_t)quarter * (32 * 128), 0, quarter * 32, h, bb * ncht + i0 / NB + i);
        if (ND == 2) tma_store_4d(&maps.h[1], h_s + NK * T64 + (uint32_t)quarter * (32 * 128), 0, quarter * 32, h, bb * ncht + i0 / NB + i);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
      if (ND == 1 && p.hprev && active) {
#pragma unroll
        for (int q = 0; q < PW / 4; ++q)
          if (4 * q < p.P) *reinterpret_cast<float4*>(p.hprev + so + 4 * q) = make_float4(hv[4 * q], hv[4 * q + 1], hv[4 * q + 2], hv[4 * q + 3]);
      }
      ok = __all_sync(0xffffffffu, wait(SRDY + (i % NSB), (uint32_t)(i / NSB), 512u) && wait(UFULL, (uint32_t)i, 512u));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const float dec = __expf(sEnd[i & 3]);
      stot += sEnd[i & 3];
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
    const int64_t row = (int64_t)blockIdx.x * gridDim.y + blockIdx.y;
    if (ok && state_only && nr == 0) p.seg_d[row] = __expf(stot);
    const bool handed = WRAP && i0 + n < p.nsteps;      // the beginning of a chain whose rest another CTA walks
    const int to = handed ? wr.e[blockIdx.x % CHAIN_SMS].sm + 1 : 0;
    float* const leave = state_only ? p.seg_h + row * NP : handed ? p.seg_h + to * NP : p.last && (WRAP || seg + 1 == p.nseg) ? p.last + (int64_t)bh * NP : nullptr;
    if (ok && leave && active) {
      float* dst = leave + (int64_t)nr * p.P;
#pragma unroll
      for (int q = 0; q < PW / 4; ++q)
        if (4 * q < p.P) *reinterpret_cast<float4*>(dst + 4 * q) = make_float4(hv[4 * q], hv[4 * q + 1], hv[4 * q + 2], hv[4 * q + 3]);
    }
    if (ok && handed) chain_hand_over(p.flags + to);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
  }
  if (!WRAP && p.late) pdl_wait();                                  // (a kernel completes after those before it)
}

// ---- host side -------------------------------------------------------------------------------------------
static unsigned int* status_ptr() {
  static unsigned int* known[PMB_MAX_DEVICES] = {nullptr};
  return status_address(g_chain_status, known);
}

template <int NI, int ND, int NK, int NB, bool XIN16>
static pmb_status launch(cudaStream_t st, const ChainArgs& a) {
  using GE = Geo<NI, ND, NK, NB, XIN16>;
  static_assert(GE::SMEM <= 227 * 1024, "shared-memory plan");
  static_assert(XIN16 ? NI == 1 : NI == ND, "fp32 tensors take pairs throughout or not at all");
  Maps ms{};
  for (int sp = 0; sp < 2; ++sp) {
    const bool lo = sp && NI == 2;
    PMB_TRY(sf::bf16_map4(&ms.b[sp], lo ? a.b.lo : a.b.hi, a.N, a.T, a.G, a.B, a.b.pitch, a.N, (int64_t)a.T * a.b.pitch, 64, L));
    PMB_TRY(sf::bf16_map4(&ms.c[sp], lo ? a.c.lo : a.c.hi, a.N, a.T, a.G, a.B, a.c.pitch, a.N, (int64_t)a.T * a.c.pitch, 64, L));
  }
  Params p{};
  p.T = a.T; p.H = a.H; p.hpg = a.H / a.G; p.N = a.N; p.P = a.P; p.nsteps = (int)cdiv(a.T, L);
  p.x = a.x; p.ldx = a.ldx;
  p.dt_raw = a.dt_raw; p.ld_raw = a.ld_raw; p.dt_bias = a.dt_bias; p.a_log = a.a_log; p.dt = a.dt; p.A = a.A; p.a = a.a; p.D = a.D;
  p.init = a.init; p.y = a.y; p.y16 = a.y16; p.ldy = a.ldy; p.dt_out = a.dt_out; p.A_out = a.A_out; p.S_out = a.S_out;
  p.hprev = a.hprev;
  uint16_t* const keep = XIN16 ? a.x_keep : a.xt;
  if (XIN16) PMB_TRY(sf::bf16_map4(&ms.x, a.x16, a.P, a.T, a.H, a.B, a.ldx, a.P, a.T * a.ldx, 64, L));
  if (keep) {
    const int64_t hp = (int64_t)a.H * a.P;
    PMB_TRY(sf::bf16_map4(&ms.xt, keep, a.P, a.T, a.H, a.B, hp, a.P, a.T * hp, 64, L));
    if (!XIN16) PMB_TRY(sf::bf16_map4(&ms.xs, a.xs, a.P, a.T, a.H, a.B, hp, a.P, a.T * hp, 64, L));
  }
  p.keep_h = a.hp_hi != nullptr; p.last = a.last; p.status = status_ptr();
  for (int sp = 0; sp < ND && a.hp_hi; ++sp) {
    const int64_t st_h = (int64_t)a.N * a.P, chunks = cdiv(p.nsteps, NB);
    PMB_TRY(sf::bf16_map4(&ms.h[sp], sp ? a.hp_lo : a.hp_hi, a.P, a.N, a.H, a.B * chunks, a.P, st_h, a.H * st_h, 64, 32));
  }
  const int chains = a.B * a.H;
  ChainWrap wr{};
  if constexpr (NI == 1 && !XIN16) {
    if (a.seg && p.nsteps % NB == 0 && ssd_chain_wrap(chains, p.nsteps / NB, NB, 1.0 / 7.0, &wr)) {
      p.seg_h = a.seg; p.flags = ssd_chain_flags(a.seg, a.P, a.N); p.store_ops = keep != nullptr;
      if (!a.flags_clear) PMB_CUDA(cudaMemsetAsync(p.flags, 0, CHAIN_FLAG_BYTES, st));
      PMB_SMEM_OPT_IN(GE::SMEM, ssd_chain_fwd_kernel<NI, ND, NK, NB, XIN16, true>);
      return launch_pdl(st, ssd_chain_fwd_kernel<NI, ND, NK, NB, XIN16, true>, dim3((unsigned)(wr.rounds * CHAIN_SMS)), NTHREADS, GE::SMEM, ms, wr, p);
    }
  }
  // (storage blocks on plain operands keep the sums of one chain, see FACT)
  const ChainPlan plan = (NI == 2 || XIN16) && a.seg ? ssd_chain_plan(a.B, a.T, a.H) : ChainPlan{chains, 1, p.nsteps};
  const unsigned cut = (unsigned)((chains - plan.whole) * plan.nseg);      // blocks of segments
  if (cut) { p.seg_h = a.seg; p.seg_d = a.seg + (size_t)cut * a.N * a.P; }
  PMB_SMEM_OPT_IN(GE::SMEM, ssd_chain_fwd_kernel<NI, ND, NK, NB, XIN16, false>);
  auto run = [&](int count, int segments) { return launch_pdl(st, ssd_chain_fwd_kernel<NI, ND, NK, NB, XIN16, false>, dim3((unsigned)count, (unsigned)segments), NTHREADS, GE::SMEM, ms, wr, p); };
  // the segments' states, the segments, and beside both the chains in one piece
  if (cut) {
    p.first = plan.whole; p.nseg = plan.nseg; p.per = plan.per;
    p.state_only = 1;
    PMB_TRY(run(chains - plan.whole, plan.nseg - 1));
    p.state_only = 0;
  }
  p.store_ops = keep != nullptr;
  if (cut) PMB_TRY(run(chains - plan.whole, plan.nseg));
  if (plan.whole) {
    p.first = 0; p.nseg = 1; p.per = p.nsteps; p.late = cut > 0;
    PMB_TRY(run(plan.whole, 1));
  }
  return PMB_OK;
}

}  // namespace sc

// Few sequences leave most SMs without a chain to walk: sequences are then cut into segments that are walked at the same time, after
// a first pass that only forms the state each segment leaves (about a quarter of a step's time).  Two steps per segment at least;
// under four steps the second launch costs what the cut saves.  Measured at
// 8 heads of 64 x 64, 1 x 2048 tokens: a block's forward 137 us uncut, 90 us in eight segments; training step of four layers 1588 and 934 us.
// With more chains than SMs the same goes for those of the last round: the others need nothing from the first pass and start beside it.  From
// three segments on, forward and backward of the bf16 scan: 160 chains of 64 x 64, 1000 tokens 220 -> 188 us, 192 of 64 x 128, 2048 tokens
// 352 -> 330; an fp32 prefill of 5 x 1200 tokens, 32 heads, 364 -> 352.  With two, 208 chains of 64 x 64 took 67 us forward instead of 59 and
// 113 backward instead of 118, 512 of 64 x 128 241 and 513 instead of 211 and 514: the first pass takes what the last round gives.
ChainPlan ssd_chain_plan(int B, int T, int H) {
  const int64_t chains = (int64_t)B * H;
  const int n = (int)cdiv(T, SCAN_STEP), rest = (int)(chains % 148 ? chains % 148 : 148);
  const int most = chains > 148 && rest < 5 ? 32 : 148 / rest, nseg = most < n / 2 ? most : n / 2;      // (32: ChainBwdArgs.part)
  if (n < 4 || nseg < (chains > 148 ? 3 : 2)) return ChainPlan{(int)chains, 1, n};
  const int per = (int)cdiv(n, nseg);
  return ChainPlan{(int)(chains - rest), (int)cdiv(n, per), per};
}
size_t ssd_chain_seg_floats(int B, int T, int H, int P, int N) {
  const ChainPlan plan = ssd_chain_plan(B, T, H);
  const size_t cut = plan.nseg > 1 ? ((size_t)B * H - plan.whole) * plan.nseg * ((size_t)N * P + 1) : 0;
  const size_t wrap = (int64_t)B * H > CHAIN_SMS ? (size_t)CHAIN_SMS * N * P + CHAIN_FLAG_BYTES / sizeof(float) : 0;
  return cut > wrap ? cut : wrap;
}

// Chains that fill the SMs a number of times and a bit (192 or 512 of them on 148) leave most SMs idle in the last round.  All their steps laid end to
// end are cut into 148 equal stretches instead: a chain that lies across a cut begins on one SM and ends on the next, which gets the state in
// fp32 through memory and so computes the same bits.  An SM walks the beginning of the chain that its stretch ends in FIRST, then its whole
// chains, then the rest of the chain that its stretch begins in: that one was begun when the launch did, on another SM, and has its state there
// before this SM comes to it, because a stretch is at least as long as a chain (McNaughton, Management Science 6(1), 1959).  The items are
// blocks of one launch in the order of their starts, which blocks are placed in; a block waits only for one of the first CHAIN_SMS.
// An item costs the kernel's filling and draining, two to three steps, which the blocks of a grid that is not cut pay less often.  Same bits, us:
// the forward of a bf16 block in chunks of 256, 24 heads of 64 x 64, 8 x 1024 tokens 191 -> 184, 8 x 2048 345 -> 320, 7 x 2048 342 -> 304, 32 heads
// 10 x 1024 296 -> 280, but 8 x 2048 412 -> 421 (an eighth of the steps saved); the scan's backward on bf16 inputs, 32 heads of 128 x 64, 16 x 8192
// 1927 -> 1750, 5 x 2048 207 -> 194, 8 x 4096 523 -> 485 (an eighth), 30 x 640 of 64 x 64 308 -> 301 (a 17th).  The forward on bf16 inputs, whose
// steps are shorter, lost as often as it gained (16 x 8192 724 -> 744, 7 x 1024 58 -> 68, 8 x 2048 of 64 x 64 92 -> 92): it stays uncut.
// Chains on pairs keep the segments of ssd_chain_plan, whose sums are others.  The forward of an fp32 block of 24 heads, segments / stretches: 8 x 384
// tokens 120 / 121, 8 x 512 149 / 157, 9 x 768 231 / 233, 8 x 1024 270 / 266, 7 x 2048 443 / 439, 8 x 2048 502 / 485; 32 heads, 10 x 512 256 / 258,
// 10 x 1024 487 / 466, 5 x 2048 484 / 462: from some 1000 tokens on stretches would give 1 to 5 %.
bool ssd_chain_wrap(int64_t chains, int units, int steps_per_unit, double least_share, ChainWrap* w) {
  const int64_t total = chains * units, uncut = cdiv(chains, CHAIN_SMS) * units, saved = uncut - cdiv(total, CHAIN_SMS);
  if (chains <= CHAIN_SMS || chains > 0xffff || units < 2 || units > 0xffff) return false;
  if (saved * steps_per_unit < 2 || (double)saved < least_share * (double)uncut) return false;
  auto cut = [&](int j) { return j * total / CHAIN_SMS; };
  auto wholes = [&](int j) { return (int)(cut(j + 1) / units - cdiv(cut(j), units)); };      // one of two numbers
  int order[CHAIN_SMS], given[CHAIN_SMS] = {}, place = 0;
  w->wholes = wholes(0);
  for (int j = 0; j < CHAIN_SMS; ++j) { order[j] = j; w->wholes = std::min(w->wholes, wholes(j)); }
  std::stable_sort(order, order + CHAIN_SMS, [&](int a, int b) { return cut(a + 1) % units < cut(b + 1) % units; });
  // Chains are numbered in the order of their starts, so that those under way at a time are neighbours and find B and C of their sequence in L2
  // (numbered along the stretches, 16 x 8192 tokens of 32 heads of 128 x 64 took 797 us forward instead of 694 uncut)
  for (int s = 0; s < CHAIN_SMS; ++s) {
    ChainWrap::Entry& e = w->e[s];
    const int j = order[s];
    e.sm = (uint16_t)j; e.head_units = (uint16_t)(cut(j + 1) % units); e.tail_from = (uint16_t)(cut(j) % units); e.head = e.extra = e.tail = 0;
    if (e.head_units) given[j + 1] = e.head = (uint16_t)place++;
  }
  w->first_whole = place;
  place += w->wholes * CHAIN_SMS;
  w->rounds = 0;
  for (int s = 0; s < CHAIN_SMS; ++s) {
    ChainWrap::Entry& e = w->e[s];
    if (wholes(e.sm) > w->wholes) e.extra = (uint16_t)place++;
    if (e.tail_from) e.tail = (uint16_t)given[e.sm];
    w->rounds = std::max(w->rounds, 1 + w->wholes + (e.extra > 0) + (e.tail_from > 0));
  }
  return true;
}

pmb_status ssd_chain_fwd(cudaStream_t st, const ChainArgs& a) {
  const bool pairs = a.b.lo != nullptr;
  if (!ssd_chain_shape(a.P, a.N) || a.H % a.G != 0 || (int64_t)a.B * a.H > 0x7fffffff) return fail(PMB_ERR_UNSUPPORTED, "ssd_chain: unsupported shape (P=%d N=%d)", a.P, a.N);
  if ((a.c.lo != nullptr) != pairs || (a.x16 && pairs) || (!a.x && !a.x16)) return fail(PMB_ERR_ARG, "ssd_chain: operands must be all pairs or all plain bf16");
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  if (!al16(a.x) || !al16(a.x16) || !al16(a.y) || !al16(a.y16) || !al16(a.init) || (a.ldx & (a.x16 ? 7 : 3)) || (a.ldy & 3))
    return fail(PMB_ERR_SHAPE, "ssd_chain: x, y and state rows must be 16-byte aligned");
  if (!pairs && !a.x16 && a.N > 64) return fail(PMB_ERR_UNSUPPORTED, "ssd_chain: fp32 x with plain bf16 B and C takes d_state up to 64");
  if ((a.hprev || a.xt) && (pairs || a.x16 || (a.xt != nullptr) != (a.xs != nullptr))) return fail(PMB_ERR_ARG, "ssd_chain: the chunk outputs go with fp32 x on plain operands");
  const double tok = (double)a.B * a.T;
  // G and the masked product over the causal half of a step, the state update and the carried-state product
  ProfScope prof(st, "ssd_chain_fwd", tok * a.H * ((double)SCAN_STEP * (a.N + a.P) + 4.0 * a.N * a.P), 0.0);
  const bool wide = a.N > 64;
  if (a.blocks == 2) {
    if (pairs || wide || a.x16 || a.T % (2 * SCAN_STEP)) return fail(PMB_ERR_UNSUPPORTED, "ssd_chain: chunks of two steps need plain bf16 operands, d_state <= 64 and whole chunks");
    return sc::launch<1, 1, 1, 2, false>(st, a);
  }
  if (a.x16 && a.exact) return wide ? sc::launch<1, 2, 2, 1, true>(st, a) : sc::launch<1, 2, 1, 1, true>(st, a);
  if (a.x16) return wide ? sc::launch<1, 1, 2, 1, true>(st, a) : sc::launch<1, 1, 1, 1, true>(st, a);
  if (!pairs) return sc::launch<1, 1, 1, 1, false>(st, a);
  return wide ? sc::launch<2, 2, 2, 1, false>(st, a) : sc::launch<2, 2, 1, 1, false>(st, a);
}

}  // namespace pmb

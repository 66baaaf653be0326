// Fused intra-chunk kernels of the chunked SSD scan (tcgen05 / TMEM); see ssd_fused.cu.  Internal to the library.
#pragma once
#include <cuda.h>
#include "kernels.h"

namespace pmb {

// A matrix operand stored as bf16: `hi` alone (lo == NULL: one MMA per product, the bf16-storage mode) or the
// (hi, lo) pair of an fp32 matrix (three MMAs per product).  `pitch` = elements between consecutive rows (tokens).
struct Op16 { const uint16_t* hi; const uint16_t* lo; int64_t pitch; };

struct FusedArgs {
  int B, T, H, P, N, G, Q;
  const float* S;          // (B,H,T) inclusive cumulative sums of a within each chunk
  Op16 c, b;               // (B*T, G*N) token rows; group g occupies columns [g*N, (g+1)*N)
  Op16 v;                  // mode 0: x~ = x*dt (B*T, H*P);  mode 1: dY (B*T, H*P)
  Op16 state;              // mode 0: h_prev (B*nc*H*N, P);  mode 1: dh (B*nc*H*N, P)   (rows of P, contiguous)
  float* out; int64_t ldo; // mode 0: y;  mode 1: dx~   (token rows, head h at column h*P)
  const float* x; int64_t ldx; const float* D;   // mode 0: skip term D[h] * x (D == NULL: none)
  float* off_out;          // mode 0, optional: (B,T,H,P) the carried-state part of y, exp(S_t) C_t h_prev
  // mode 1 only: x~ (the rows of the CTA, for dM = dY x~^T) and the sums of W[t,s] = dM[t,s] G[t,s] exp(S_t - S_s), s < t
  Op16 xt;                 // (B*T, H*P)
  float* csum;             // (B,T,H)  c_s = sum_{t>s} W[t,s]
  float* esum;             // (B,T,H)  e_s = exp(S_end - S_s) <x~_s, B_s dh>
  float* rpart;            // (B*nc*H, Q/128, Q)  r_t = sum_{s<t} W[t,s], one partial per row block of s (valid for t >= 128*block)
};

// ---- forward of the whole scan as one kernel (ssd_chain.cu), in steps of SCAN_STEP tokens
constexpr int SCAN_STEP = 128;
struct ChainArgs {
  int B, T, H, P, N, G;
  bool exact = false;                          // x16: what is formed from the inputs (M, xs, the states) is kept as pairs, so that nothing is rounded to bf16 but y
  int blocks = 1;                              // steps per chunk (what S, xs and the states are relative to): 1 or 2
  Op16 b, c;                                   // (B,T,G,N), pitch = elements between tokens, group stride N
  const float* x; const uint16_t* x16; int64_t ldx;      // one of the two: fp32 (scaled by dt here) or bf16 (taken as x~)
  const float* dt_raw; int64_t ld_raw; const float* dt_bias; const float* a_log;   // either these four (dt and A formed here),
  const float* dt; const float* A;             // or dt and A,
  const float* a;                              // or a (x~ = x)
  const float* D;                              // skip weights or NULL (fp32 x only)
  const float* init;                           // (B,H,N,P) or NULL
  float* y; uint16_t* y16; int64_t ldy;        // one of the two
  float *dt_out, *A_out, *S_out;               // optional: what the backward reads
  uint16_t* x_keep;                            // copy of x16, (B,T,H,P)
  uint16_t *hp_hi, *hp_lo;                     // state entering each step, (B,steps,H,N,P)
  float* last;                                 // (B,H,N,P)
  float *hprev;                                // plain operands with fp32 x: (B,chunks,H,N,P) state entering each chunk
  uint16_t *xt, *xs;                           // ... and the operands x~ and xs, (B,T,H,P)
  float* seg = nullptr;                        // ssd_chain_seg_floats() floats: lets chains be walked in pieces
  bool flags_clear = false;                    // ssd_chain_flags() of it are zero already
};
// The first `whole` chains (b, h) are walked in one piece, each of the others in `nseg` segments of `per` steps (the last may have fewer).
struct ChainPlan { int whole, nseg, per; };
ChainPlan ssd_chain_plan(int B, int T, int H);
size_t ssd_chain_seg_floats(int B, int T, int H, int P, int N);
// More chains than SMs on plain operands: every SM takes an equal stretch of all chains' steps laid end to end (ssd_chain.cu says how a chain
// that two SMs share is handed over).  One entry per SM, sorted by when it comes to its second item: in units of steps, the chains that its
// stretch begins and ends in and the places there, and the SM's place in the unsorted order, which numbers the hand-overs.
constexpr int CHAIN_SMS = 148;
struct ChainWrap {
  struct Entry {
    uint16_t head, head_units;                 // the chain that the stretch ends in and how much of it (0: none), walked first
    uint16_t extra;                            // a last whole chain beyond `wholes` (0: none)
    uint16_t tail, tail_from;                  // the chain that the stretch begins in and where (0: none), walked last
    uint16_t sm;                               // place in the order of the stretches, which numbers the hand-overs: sm + 1 is given, sm taken
  } e[CHAIN_SMS];
  int wholes, first_whole;                     // whole chains that every SM has, between the other two: first_whole + i CHAIN_SMS + the entry's place
  int rounds;                                  // blocks: rounds x CHAIN_SMS
};
// false: the chains are better walked whole.  `units` of steps to a chain; least_share: of the steps one after the other, what has to be saved
bool ssd_chain_wrap(int64_t chains, int units, int steps_per_unit, double least_share, ChainWrap* w);
// counters of the hand-overs, in the buffer `seg` of the two kernels below: zero when a launch begins
constexpr size_t CHAIN_FLAG_BYTES = (CHAIN_SMS + 12) * sizeof(uint32_t);
static_assert(CHAIN_FLAG_BYTES == CONV_CLEAR_WORDS * sizeof(uint32_t), "the conv kernel clears them");
inline uint32_t* ssd_chain_flags(float* seg, int P, int N) { return reinterpret_cast<uint32_t*>(seg + (size_t)CHAIN_SMS * N * P); }
inline bool ssd_chain_shape(int P, int N) { return P > 0 && P <= 64 && P % 8 == 0 && N > 0 && N <= 128 && N % 8 == 0; }
bool ssd_chain_enabled();      // false when PMB_SSD_FUSED=0 or PMB_SSD_ENGINE=simt
// bf16-storage blocks: shapes whose scan reads its operands rounded to bf16 (whole chunks of 128 or 256 tokens at d_state =
// d_head = 64); every other shape keeps (hi, lo) pairs of the fp32 values there
bool ssd_plain16_shape(int P, int N, int Q);
pmb_status ssd_chain_fwd(cudaStream_t st, const ChainArgs& a);
pmb_status read_clear_device_status_chain(unsigned int* word);

// ---- its backward (ssd_chain_bwd.cu): everything but the sums over heads.  fp32 tensors with (hi, lo) pairs of B, C and the states, or
// bf16 tensors with plain bf16 operands (x is then x~ and `da` the result).
struct ChainBwdArgs {
  int B, T, H, P, N, G;
  Op16 b, c;                                   // as in ChainArgs
  const uint16_t *hp_hi, *hp_lo;               // (B,steps,H,N,P) as the forward left it
  const float* S;                              // (B,H,T) relative to steps
  const float* x; const uint16_t* x16; int64_t ldx;
  const float* dy; const uint16_t* dy16; int64_t lddy;
  const float* dt; const float* A; const float* D;       // dt mode (fp32): (B,T,H), (H), skip weights or NULL
  float* dx; uint16_t* dx16; int64_t lddx;
  uint16_t *xt_hi, *xt_lo, *dyo_hi, *dyo_lo;   // optional (B,T,H,P): x~ and dY as operand pairs
  uint16_t *dh_hi, *dh_lo;                     // (B,steps,H,N,P) adjoint of the state leaving each step
  float* da;                                   // (B,T,H) or NULL
  uint16_t *raw_hi, *raw_lo; int64_t ld_raw; int raw_col;   // dt mode: gradient before the softplus, at [token * ld_raw + raw_col + h]
  float* part;                                 // dt mode: 3 x (B * segments,H): sums for dA, dD, d_dt_bias
  float* seg;                                  // as in ChainArgs, or NULL: no segments
};
inline bool ssd_chain_bwd_shape(int P, int N, bool pairs) { return P > 0 && P <= 64 && P % 8 == 0 && N > 0 && N <= (pairs ? 64 : 128) && N % 8 == 0; }
// the per-head sums over `rows` rows of each of part's three sections; d_a_log = A dA
pmb_status ssd_head_finish(cudaStream_t st, const float* part, int rows, int H, const float* A, float* dA, float* dD, float* d_dt_bias, float* d_a_log);
pmb_status ssd_chain_bwd(cudaStream_t st, const ChainBwdArgs& a);
pmb_status read_clear_device_status_chain_bwd(unsigned int* word);

// ---- the sums over heads next to it (ssd_heads.cu): dB and dC from the operands that the two passes leave
struct HeadsArgs {
  int B, T, H, P, N, G;
  Op16 b, c, dy, xt;                           // b, c as in ChainArgs; dy and xt (B,T,H,P)
  const uint16_t *hp_hi, *hp_lo, *dh_hi, *dh_lo;       // (B,steps,H,N,P)
  const float* S;                              // (B,H,T)
  float *dc, *db; uint16_t *dc16, *db16; int64_t ld;   // fp32 or bf16 token rows, group g at column g * N
  float* part;                                 // ssd_heads_part_floats() floats
};
int ssd_heads_nsplit(int B, int T, int H, int G);
size_t ssd_heads_part_floats(int B, int T, int H, int N, int G);
pmb_status ssd_heads(cudaStream_t st, const HeadsArgs& a);
pmb_status read_clear_device_status_heads(unsigned int* word);

// Shapes the fused kernels and the other contractions below take: block_len a multiple of 128 (at most 1024), d_state = d_head = 64.
bool ssd_fused_supported(int P, int N, int Q);

// mode 0: Y[t,:]   = sum_{s<=t} (C_t.B_s) exp(S_t-S_s) x~_s + exp(S_t) C_t h_prev + D x_t          per (b, chunk, head)
// mode 1: dx~[s,:] = sum_{t>=s} (C_t.B_s) exp(S_t-S_s) dY_t  + exp(S_end-S_s) B_s dh               per (b, chunk, head)
//         plus csum, esum, rpart (see FusedArgs)
pmb_status ssd_fused(cudaStream_t st, int mode, const FusedArgs& a);

// ---- the backward on plain bf16 operands (ssd_dx.cu): chunks of 128 or 256 tokens at d_state = d_head = 64
struct DxArgs {
  int B, T, H, P, N, G, Q;
  const float* S; const float* dt; const float* A; const float* D;      // D = NULL: no skip term
  Op16 b, c;               // as in FusedArgs
  const uint16_t *xt, *dy16, *hp, *dh;   // x~ and dY (B,T,H,P); state entering each chunk and adjoint of the one leaving it (B,T/Q,H,N,P)
  const float* x; int64_t ldx; const float* dy; int64_t lddy;
  float* dx; int64_t lddx; // dx~ dt + D dY
  const float* dd;         // (B*T/Q,H) <dh, h_prev>
  float *rpart, *sums;     // scratch: (B*T/Q*H, Q/128, Q) and, within the room of dx~ (B,T,H,P), five sums per row
  float* part;             // 3 x (B*T/Q,H): sums for dA, dD, d_dt_bias
  SsdGrads::RawDt raw;     // gradient before the softplus (hi alone)
};
pmb_status ssd_dx_check(const DxArgs& a);      // what ssd_dx takes; touches no memory
pmb_status ssd_dx(cudaStream_t st, const DxArgs& a);

unsigned int* ssd_fused_status();
pmb_status read_clear_device_status_fused(unsigned int* word);
pmb_status read_clear_device_status_pairs(unsigned int* word);

// ---- the other contractions of the scan on the same bf16 pairs (ssd_pairs.cu; shapes of ssd_fused_supported(pairs)):
// states / dstates (per head), dG (summed over the heads of a group, decay mask folded in registers), dC / dB.
pmb_status ssd_pairs_state(cudaStream_t st, const SsdIn& in, const SsdWs& ws, int mode);      // 0: chunk states, 1: d(states)
// dG (ssd_dg.cu)
int ssd_dg_nsplit(int B, int T, int H, int G, int Q);
pmb_status ssd_dg(cudaStream_t st, const SsdIn& in, const SsdWs& ws, int nsplit);       // -> ws.dg_hi/lo (nsplit == 1) or ws.splitk partials
int ssd_pairs_dbc_nsplit(int B, int T, int H, int N, int G, int Q);
// mode 0: dC, 1: dB; `part` = where the head-split partial tiles go (nsplit * B * nc * G * Q * N floats)
pmb_status ssd_pairs_dbc(cudaStream_t st, const SsdIn& in, const SsdWs& ws, int mode, float* out, int64_t ld, int nsplit, float* part);

namespace sf {
// cached rank-3 bf16 tensor map: dims (d0 contiguous, d1 rows with pitch s0 elements, d2 with pitch s1), box (b0, b1, 1)
pmb_status bf16_map3(CUtensorMap* out, const uint16_t* base, int64_t d0, int64_t d1, int64_t d2, int64_t s0, int64_t s1, int b0, int b1);
// cached rank-4 bf16 tensor map of a token-major operand: dims (d0 contiguous, T tokens with pitch s0, d2 heads / groups
// with pitch s1, B sequences with pitch s2), box (b0, b1, 1, 1).  A box that reaches past the end of a sequence (or past
// d0) is filled with zeros there, never with the next sequence's rows.
// cached map of 128 token rows (tokens a multiple of 32, 64 columns from 0) that a copy deals to a tile in groups of eight: tile row
// 32 q + 8 i + r = token row 32 i + 8 q + r; coordinates (0, 0, first row / 32, 0, head)
pmb_status bf16_map_rows8(CUtensorMap* out, const uint16_t* base, int64_t d0, int64_t tokens, int64_t H, int64_t pitch, int64_t head);
pmb_status bf16_map4(CUtensorMap* out, const uint16_t* base, int64_t d0, int64_t T, int64_t d2, int64_t B, int64_t s0, int64_t s1, int64_t s2, int b0, int b1);
}

}  // namespace pmb

// Chunked SSD scan (forward and fused-recompute backward) as a set of batched tile contractions.
//
// Per (batch b, chunk c, head h), with S = inclusive cumsum of a inside the chunk, L[t,s] = exp(S_t - S_s) (s <= t),
// x~ = x * dt:
//   forward   CB = C B^T                                   (per group)
//             states = sum_q exp(S_end - S_q) B_q (x) x~_q  -> exclusive scan over chunks -> h_prev
//             Y = (CB o L) x~ + diag(exp S) C h_prev (+ D x)
//   backward  dh_prev = sum_t exp(S_t) C_t (x) dY_t + exp(S_end) dh   (reverse scan over chunks)
//             dx~ = (CB o L)^T dY + exp(S_end - S_s) B_s dh
//             dG = sum_heads L o (dY x~^T);  dC = dG B + sum_h exp(S_t) dY_t h_prev^T;
//             dB = dG^T C + sum_h exp(S_end - S_s) x~_s dh^T
//             dS_t = <dY_t, Y_t> - <x~_t, dx~_t>, dS_{Q-1} += <dh, h_next>;  da = reverse cumsum(dS)   (Y without the skip term)
// The reference computes the same quantities with ~40 primitive ops and autograd
// (crates/pm-core/src/mamba2/ssd_ops.rs:167-284); nothing of size (Q,Q) per head is stored here.
//
// This file holds the SIMT (fp32 FMA) engine: one 64x64-tile kernel template, specialised by small functor
// structs that say how to read operand elements and where results go.
#include <cstdlib>
#include <cuda_bf16.h>
#include "common.cuh"
#include "kernels.h"
#include "bgemm.cuh"
#include "ssd_tc.h"
#include "ssd_fused.h"

namespace pmb {

struct SsdP {
  int B, T, H, P, N, G, Q, nc, hpg;
  const float* x; int64_t ldx;
  const float* dt; const float* A; const float* a;
  const float* b; const float* c; int64_t ldbc;
  const float* D;
  float* S; float* hprev; float* hlast; float* CB; float* dh; float* dG; float* dxt;
  const float* y; int64_t ldy; bool skip_in_y; const float* yp;      // yp: y without the skip term, for the rows that want it
  const float* dy; int64_t lddy;
  float* yout; int64_t ldyo; float* yplain;
  float* db; float* dc; int64_t lddbc;

  __device__ __forceinline__ int64_t tok(int bb, int cc, int q) const { return (int64_t)bb * T + (int64_t)cc * Q + q; }
  __device__ __forceinline__ float Sv(int bb, int h, int cc, int q) const { return S[((int64_t)bb * H + h) * T + (int64_t)cc * Q + q]; }
  __device__ __forceinline__ float dtv(int64_t tk, int h) const { return dt ? dt[tk * H + h] : 1.0f; }
};

// ---- F1: CB[t,s] = sum_n C[t,n] B[s,n], per (b,c,g) --------------------------------------------
struct OpCB {
  static constexpr bool SEG_SCALE = false;
  SsdP p; int Mdim, Ndim;
  int bb, cc, g; const float* cp; const float* bp; float* out;
  __device__ bool init(int batch, int m0, int n0) {
    if (n0 > m0 + BM - 1) return false;  // strictly above the diagonal: never read
    g = batch % p.G; int bc = batch / p.G; cc = bc % p.nc; bb = bc / p.nc;
    cp = p.c + p.tok(bb, cc, 0) * p.ldbc + g * p.N;
    bp = p.b + p.tok(bb, cc, 0) * p.ldbc + g * p.N;
    out = p.CB + (int64_t)batch * p.Q * p.Q;
    return true;
  }
  __device__ int nseg() const { return 1; }
  __device__ void krange(int, int, int, int& k0, int& k1) const { k0 = 0; k1 = p.N; }
  __device__ bool a_kcontig(int) const { return true; }
  __device__ bool b_kcontig(int) const { return true; }
  __device__ float a(int, int m, int k) const { return cp[(int64_t)m * p.ldbc + k]; }
  __device__ float b(int, int k, int n) const { return bp[(int64_t)n * p.ldbc + k]; }
  __device__ float seg_scale(int, int, int) const { return 1.0f; }
  __device__ bool seg_active(int) const { return true; }
  __device__ void store(int m, int n, float v) const { out[(int64_t)m * p.Q + n] = v; }
};

// Common context for per-(b,c,h) ops.
struct HeadCtx {
  int bb, cc, h, g; int64_t t0;  // first token of the chunk
  __device__ void set(const SsdP& p, int batch) {
    h = batch % p.H; int bc = batch / p.H; cc = bc % p.nc; bb = bc / p.nc; g = h / p.hpg;
    t0 = p.tok(bb, cc, 0);
  }
};

// ---- F2: states[n,p] = sum_q B[q,n] exp(S_end - S_q) x~[q,p], per (b,c,h) -----------------------
struct OpState {
  static constexpr bool SEG_SCALE = false;
  SsdP p; int Mdim, Ndim;
  HeadCtx cx; float send; const float* sp; float* out;
  __device__ bool init(int batch, int, int) {
    cx.set(p, batch);
    sp = p.S + ((int64_t)cx.bb * p.H + cx.h) * p.T + (int64_t)cx.cc * p.Q;
    send = sp[p.Q - 1];
    out = p.hprev + (int64_t)batch * p.N * p.P;
    return true;
  }
  __device__ int nseg() const { return 1; }
  __device__ void krange(int, int, int, int& k0, int& k1) const { k0 = 0; k1 = p.Q; }
  __device__ bool a_kcontig(int) const { return false; }
  __device__ bool b_kcontig(int) const { return false; }
  __device__ float a(int, int m, int k) const {
    int64_t tk = cx.t0 + k;
    return p.b[tk * p.ldbc + cx.g * p.N + m] * expf(send - sp[k]) * p.dtv(tk, cx.h);
  }
  __device__ float b(int, int k, int n) const { return p.x[(cx.t0 + k) * p.ldx + cx.h * p.P + n]; }
  __device__ float seg_scale(int, int, int) const { return 1.0f; }
  __device__ bool seg_active(int) const { return true; }
  __device__ void store(int m, int n, float v) const { out[(int64_t)m * p.P + n] = v; }
};

// ---- F4: Y[t,p] = sum_{s<=t} CB[t,s] L[t,s] x~[s,p] + exp(S_t) sum_n C[t,n] h_prev[n,p] (+ D x) --
struct OpScan {
  static constexpr bool SEG_SCALE = false;
  SsdP p; int Mdim, Ndim;
  HeadCtx cx; const float* sp; const float* cb; const float* hp;
  __device__ bool init(int batch, int, int) {
    cx.set(p, batch);
    sp = p.S + ((int64_t)cx.bb * p.H + cx.h) * p.T + (int64_t)cx.cc * p.Q;
    cb = p.CB + (((int64_t)cx.bb * p.nc + cx.cc) * p.G + cx.g) * p.Q * p.Q;
    hp = p.hprev + (int64_t)batch * p.N * p.P;
    return true;
  }
  __device__ int nseg() const { return 2; }
  __device__ void krange(int seg, int m0, int, int& k0, int& k1) const {
    k0 = 0; k1 = seg == 0 ? min(p.Q, m0 + BM) : p.N;
  }
  __device__ bool a_kcontig(int) const { return true; }
  __device__ bool b_kcontig(int) const { return false; }
  __device__ float a(int seg, int m, int k) const {
    if (seg == 0) {
      if (k > m) return 0.0f;
      return cb[(int64_t)m * p.Q + k] * expf(sp[m] - sp[k]) * p.dtv(cx.t0 + k, cx.h);
    }
    return p.c[(cx.t0 + m) * p.ldbc + cx.g * p.N + k] * expf(sp[m]);
  }
  __device__ float b(int seg, int k, int n) const {
    if (seg == 0) return p.x[(cx.t0 + k) * p.ldx + cx.h * p.P + n];
    return hp[(int64_t)k * p.P + n];
  }
  __device__ float seg_scale(int, int, int) const { return 1.0f; }
  __device__ bool seg_active(int) const { return true; }
  __device__ void store(int m, int n, float v) const {
    if (p.yplain) p.yplain[((cx.t0 + m) * p.H + cx.h) * p.P + n] = v;
    if (p.D) v = fmaf(p.D[cx.h], p.x[(cx.t0 + m) * p.ldx + cx.h * p.P + n], v);
    p.yout[(cx.t0 + m) * p.ldyo + cx.h * p.P + n] = v;
  }
};

// ---- B1: contrib[n,p] = sum_t C[t,n] exp(S_t) dY[t,p], per (b,c,h) ------------------------------
struct OpDstate {
  static constexpr bool SEG_SCALE = false;
  SsdP p; int Mdim, Ndim;
  HeadCtx cx; const float* sp; float* out;
  __device__ bool init(int batch, int, int) {
    cx.set(p, batch);
    sp = p.S + ((int64_t)cx.bb * p.H + cx.h) * p.T + (int64_t)cx.cc * p.Q;
    out = p.dh + (int64_t)batch * p.N * p.P;
    return true;
  }
  __device__ int nseg() const { return 1; }
  __device__ void krange(int, int, int, int& k0, int& k1) const { k0 = 0; k1 = p.Q; }
  __device__ bool a_kcontig(int) const { return false; }
  __device__ bool b_kcontig(int) const { return false; }
  __device__ float a(int, int m, int k) const { return p.c[(cx.t0 + k) * p.ldbc + cx.g * p.N + m] * expf(sp[k]); }
  __device__ float b(int, int k, int n) const { return p.dy[(cx.t0 + k) * p.lddy + cx.h * p.P + n]; }
  __device__ float seg_scale(int, int, int) const { return 1.0f; }
  __device__ bool seg_active(int) const { return true; }
  __device__ void store(int m, int n, float v) const { out[(int64_t)m * p.P + n] = v; }
};

// ---- B3: dx~[s,p] = sum_{t>=s} CB[t,s] L[t,s] dY[t,p] + exp(S_end - S_s) sum_n B[s,n] dh[n,p] ----
struct OpDx {
  static constexpr bool SEG_SCALE = false;
  SsdP p; int Mdim, Ndim;
  HeadCtx cx; const float* sp; const float* cb; const float* dhp; float send;
  __device__ bool init(int batch, int, int) {
    cx.set(p, batch);
    sp = p.S + ((int64_t)cx.bb * p.H + cx.h) * p.T + (int64_t)cx.cc * p.Q;
    send = sp[p.Q - 1];
    cb = p.CB + (((int64_t)cx.bb * p.nc + cx.cc) * p.G + cx.g) * p.Q * p.Q;
    dhp = p.dh + (int64_t)batch * p.N * p.P;
    return true;
  }
  __device__ int nseg() const { return 2; }
  __device__ void krange(int seg, int m0, int, int& k0, int& k1) const {
    if (seg == 0) { k0 = m0; k1 = p.Q; } else { k0 = 0; k1 = p.N; }
  }
  __device__ bool a_kcontig(int seg) const { return seg != 0; }
  __device__ bool b_kcontig(int) const { return false; }
  __device__ float a(int seg, int m, int k) const {
    if (seg == 0) {
      if (k < m) return 0.0f;
      return cb[(int64_t)k * p.Q + m] * expf(sp[k] - sp[m]);
    }
    return p.b[(cx.t0 + m) * p.ldbc + cx.g * p.N + k] * expf(send - sp[m]);
  }
  __device__ float b(int seg, int k, int n) const {
    if (seg == 0) return p.dy[(cx.t0 + k) * p.lddy + cx.h * p.P + n];
    return dhp[(int64_t)k * p.P + n];
  }
  __device__ float seg_scale(int, int, int) const { return 1.0f; }
  __device__ bool seg_active(int) const { return true; }
  __device__ void store(int m, int n, float v) const { p.dxt[(cx.t0 + m) * (int64_t)(p.H * p.P) + cx.h * p.P + n] = v; }
};

// ---- B5: dG[t,s] = sum_{h in group} L_h[t,s] sum_p dY_h[t,p] x~_h[s,p], per (b,c,g) --------------
struct OpDG {
  static constexpr bool SEG_SCALE = true;
  SsdP p; int Mdim, Ndim;
  int nsplit; float* part;      // split-K over heads: partial tiles go to `part`, summed by splitk_reduce_kernel
  int bb, cc, g, split; int64_t t0; float* out;
  __device__ bool init(int batch, int m0, int n0) {
    if (n0 > m0 + BM - 1) return false;
    split = batch % nsplit; batch /= nsplit;
    g = batch % p.G; int bc = batch / p.G; cc = bc % p.nc; bb = bc / p.nc;
    t0 = p.tok(bb, cc, 0);
    out = nsplit > 1 ? part + (int64_t)blockIdx.z * p.Q * p.Q : p.dG + (int64_t)batch * p.Q * p.Q;
    return true;
  }
  __device__ bool seg_active(int seg) const { return seg % nsplit == split; }
  __device__ int nseg() const { return p.hpg; }
  __device__ void krange(int, int, int, int& k0, int& k1) const { k0 = 0; k1 = p.P; }
  __device__ bool a_kcontig(int) const { return true; }
  __device__ bool b_kcontig(int) const { return true; }
  __device__ float a(int seg, int m, int k) const { return p.dy[(t0 + m) * p.lddy + (g * p.hpg + seg) * p.P + k]; }
  __device__ float b(int seg, int k, int n) const {
    int h = g * p.hpg + seg;
    return p.x[(t0 + n) * p.ldx + h * p.P + k] * p.dtv(t0 + n, h);
  }
  __device__ float seg_scale(int seg, int m, int n) const {
    if (n > m) return 0.0f;
    int h = g * p.hpg + seg;
    const float* sp = p.S + ((int64_t)bb * p.H + h) * p.T + (int64_t)cc * p.Q;
    return expf(sp[m] - sp[n]);
  }
  __device__ void store(int m, int n, float v) const { out[(int64_t)m * p.Q + n] = v; }
};

// ---- B6a: dC[t,n] = sum_{s<=t} dG[t,s] B[s,n] + sum_h exp(S_h,t) sum_p dY_h[t,p] h_prev_h[n,p] ----
struct OpDC {
  static constexpr bool SEG_SCALE = false;
  SsdP p; int Mdim, Ndim;
  int nsplit; float* part;
  int bb, cc, g, split; int64_t t0; const float* dg; float* pout;
  __device__ bool init(int batch, int, int) {
    split = batch % nsplit; batch /= nsplit;
    g = batch % p.G; int bc = batch / p.G; cc = bc % p.nc; bb = bc / p.nc;
    t0 = p.tok(bb, cc, 0);
    dg = p.dG + (int64_t)batch * p.Q * p.Q;
    pout = part + (int64_t)blockIdx.z * Mdim * Ndim;
    return true;
  }
  __device__ bool seg_active(int seg) const { return seg == 0 ? split == 0 : (seg - 1) % nsplit == split; }
  __device__ int nseg() const { return 1 + p.hpg; }
  __device__ void krange(int seg, int m0, int, int& k0, int& k1) const {
    k0 = 0; k1 = seg == 0 ? min(p.Q, m0 + BM) : p.P;
  }
  __device__ bool a_kcontig(int) const { return true; }
  __device__ bool b_kcontig(int seg) const { return seg != 0; }
  __device__ float a(int seg, int m, int k) const {
    if (seg == 0) return dg[(int64_t)m * p.Q + k];
    int h = g * p.hpg + seg - 1;
    return p.dy[(t0 + m) * p.lddy + h * p.P + k] * expf(p.Sv(bb, h, cc, m));
  }
  __device__ float b(int seg, int k, int n) const {
    if (seg == 0) return p.b[(t0 + k) * p.ldbc + g * p.N + n];
    int h = g * p.hpg + seg - 1;
    return p.hprev[((((int64_t)bb * p.nc + cc) * p.H + h) * p.N + n) * p.P + k];
  }
  __device__ float seg_scale(int, int, int) const { return 1.0f; }
  __device__ void store(int m, int n, float v) const {
    if (nsplit > 1) pout[(int64_t)m * Ndim + n] = v; else p.dc[(t0 + m) * p.lddbc + g * p.N + n] = v;
  }
};

// ---- B6b: dB[s,n] = sum_{t>=s} dG[t,s] C[t,n] + sum_h exp(S_end - S_s) sum_p x~_h[s,p] dh_h[n,p] --
struct OpDB {
  static constexpr bool SEG_SCALE = false;
  SsdP p; int Mdim, Ndim;
  int nsplit; float* part;
  int bb, cc, g, split; int64_t t0; const float* dg; float* pout;
  __device__ bool init(int batch, int, int) {
    split = batch % nsplit; batch /= nsplit;
    g = batch % p.G; int bc = batch / p.G; cc = bc % p.nc; bb = bc / p.nc;
    t0 = p.tok(bb, cc, 0);
    dg = p.dG + (int64_t)batch * p.Q * p.Q;
    pout = part + (int64_t)blockIdx.z * Mdim * Ndim;
    return true;
  }
  __device__ bool seg_active(int seg) const { return seg == 0 ? split == 0 : (seg - 1) % nsplit == split; }
  __device__ int nseg() const { return 1 + p.hpg; }
  __device__ void krange(int seg, int m0, int, int& k0, int& k1) const {
    if (seg == 0) { k0 = m0; k1 = p.Q; } else { k0 = 0; k1 = p.P; }
  }
  __device__ bool a_kcontig(int seg) const { return seg != 0; }
  __device__ bool b_kcontig(int seg) const { return seg != 0; }
  __device__ float a(int seg, int m, int k) const {
    if (seg == 0) return dg[(int64_t)k * p.Q + m];
    int h = g * p.hpg + seg - 1;
    float send = p.Sv(bb, h, cc, p.Q - 1);
    return p.x[(t0 + m) * p.ldx + h * p.P + k] * p.dtv(t0 + m, h) * expf(send - p.Sv(bb, h, cc, m));
  }
  __device__ float b(int seg, int k, int n) const {
    if (seg == 0) return p.c[(t0 + k) * p.ldbc + g * p.N + n];
    int h = g * p.hpg + seg - 1;
    return p.dh[((((int64_t)bb * p.nc + cc) * p.H + h) * p.N + n) * p.P + k];
  }
  __device__ float seg_scale(int, int, int) const { return 1.0f; }
  __device__ void store(int m, int n, float v) const {
    if (nsplit > 1) pout[(int64_t)m * Ndim + n] = v; else p.db[(t0 + m) * p.lddbc + g * p.N + n] = v;
  }
};

// ---------------------------------------------------------------------------------------------
// Small kernels
// ---------------------------------------------------------------------------------------------

// S[b,h,c*Q+q] = inclusive cumsum over q of a.  One warp per (b,c,h).  With raw.dt_raw the warp first forms
// dt = softplus(dt_raw + bias) (written out for the later kernels) and A = -exp(a_log).
struct CumsumRaw { const float* dt_raw; int64_t ld_raw; const float* dt_bias; const float* a_log; float* dt_out; float* A_out; };
__global__ void chunk_cumsum_kernel(SsdP p, CumsumRaw raw) {
  int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  int total = p.B * p.nc * p.H;
  if (w >= total) return;
  int h = w % p.H, bc = w / p.H, cc = bc % p.nc, bb = bc / p.nc;
  float carry = 0.0f;
  float* out = p.S + ((int64_t)bb * p.H + h) * p.T + (int64_t)cc * p.Q;
  // the strided loads of up to 8 rounds are requested together, ahead of the dependent scan chain
  constexpr int AHEAD = 8;
  const float Ah = raw.dt_raw ? -expf(raw.a_log[h]) : (p.dt ? p.A[h] : 1.0f);
  const float bias = raw.dt_raw ? raw.dt_bias[h] : 0.0f;
  if (raw.dt_raw && bc == 0 && lane == 0) raw.A_out[h] = Ah;
  const float* srcv = p.dt ? p.dt : p.a;
  float pre[AHEAD];
  for (int q0 = 0; q0 < p.Q; q0 += 32) {
    const int r = (q0 >> 5) % AHEAD;
    if (r == 0) {
#pragma unroll
      for (int j = 0; j < AHEAD; ++j) {
        const int qq = q0 + 32 * j + lane;
        pre[j] = 0.0f;
        if (qq < p.Q) {
          const int64_t tk = p.tok(bb, cc, qq);
          if (raw.dt_raw) {
            const float dtv = softplus_acc(raw.dt_raw[tk * raw.ld_raw + h] + bias);
            raw.dt_out[tk * p.H + h] = dtv;
            pre[j] = Ah * dtv;
          } else {
            pre[j] = Ah * srcv[tk * p.H + h];
          }
        }
      }
    }
    int q = q0 + lane;
    float v = 0.0f;
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) if (j == r) v = pre[j];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      float u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    v += carry;
    if (q < p.Q) out[q] = v;
    carry = __shfl_sync(0xffffffffu, v, 31);
  }
}

// Fused variant for the tensor-core path, one 256-thread block per (b,c,h): the same cumsum (with dt and A formed
// here when raw inputs are given), then xs[t,:] = x[t,:] * dt_t * exp(S_end - S_t), the operand that the chunk-state
// and dB contractions share.  S and dt of the chunk stay in shared memory between the two phases.
constexpr int PREP_THREADS = 256, PREP_MAX_Q = 1024;
__global__ void __launch_bounds__(PREP_THREADS) chunk_prepare_kernel(SsdP p, CumsumRaw raw, float* __restrict__ xs,
                                                                     uint16_t* __restrict__ xt_hi, uint16_t* __restrict__ xt_lo,
                                                                     uint16_t* __restrict__ xs_hi, uint16_t* __restrict__ xs_lo) {
  __shared__ float sS[PREP_MAX_Q], sdt[PREP_MAX_Q], wsum[PREP_THREADS / 32];
  // gridDim.y CTAs share one (b,c,h): each repeats the short cumulative sum (same order, same values) and takes its
  // slice of the rows in the second phase; the first of them writes dt, A and S
  const int w = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const bool writer = blockIdx.y == 0;
  const int h = w % p.H, bc = w / p.H, cc = bc % p.nc, bb = bc / p.nc;
  const float Ah = raw.dt_raw ? -expf(raw.a_log[h]) : (p.dt ? p.A[h] : 1.0f);
  const float bias = raw.dt_raw ? raw.dt_bias[h] : 0.0f;
  if (raw.dt_raw && bc == 0 && tid == 0 && writer) raw.A_out[h] = Ah;
  float* Sout = p.S + ((int64_t)bb * p.H + h) * p.T + (int64_t)cc * p.Q;
  float carry = 0.0f;
  for (int q0 = 0; q0 < p.Q; q0 += PREP_THREADS) {
    const int q = q0 + tid;
    float v = 0.0f, dtv = 1.0f;
    if (q < p.Q) {
      const int64_t tk = p.tok(bb, cc, q);
      if (raw.dt_raw) { dtv = softplus_acc(raw.dt_raw[tk * raw.ld_raw + h] + bias); if (writer) raw.dt_out[tk * p.H + h] = dtv; v = Ah * dtv; }
      else if (p.dt) { dtv = p.dt[tk * p.H + h]; v = Ah * dtv; }
      else v = p.a[tk * p.H + h];
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const float u = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += u; }
    if (lane == 31) wsum[wid] = v;
    __syncthreads();
    float off = carry;
    for (int j = 0; j < wid; ++j) off += wsum[j];          // fixed order: the same sums for every launch
    v += off;
    if (q < p.Q) { sS[q] = v; sdt[q] = dtv; if (writer) Sout[q] = v; }
    float tot = carry;
    for (int j = 0; j < PREP_THREADS / 32; ++j) tot += wsum[j];
    carry = tot;
    __syncthreads();
  }
  const float send = sS[p.Q - 1];
  const int P4 = p.P >> 2;
  const int rows_per = (p.Q + (int)gridDim.y - 1) / (int)gridDim.y;        // this CTA's rows [r0, r1) of the chunk
  const int r0 = (int)blockIdx.y * rows_per, r1 = min(p.Q, r0 + rows_per);
  const int total = r1 * P4;
  const int64_t tok0 = p.tok(bb, cc, 0);
  constexpr int U = 4;
  for (int i0 = r0 * P4 + tid; i0 < total; i0 += U * PREP_THREADS) {
    float4 v[U]; float f[U], fd[U]; int tt[U], jj[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * PREP_THREADS;
      tt[u] = i / P4; jj[u] = i % P4;
      if (i < total) {
        v[u] = reinterpret_cast<const float4*>(p.x + (tok0 + tt[u]) * p.ldx + h * p.P)[jj[u]];
        fd[u] = sdt[tt[u]];
        f[u] = __expf(send - sS[tt[u]]) * fd[u];
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * PREP_THREADS;
      if (i < total) {
        const int64_t o = (tok0 + tt[u]) * (int64_t)(p.H * p.P) + h * p.P + 4 * jj[u];
        if (xs_hi) store_pair4(xs_hi + o, xs_lo ? xs_lo + o : nullptr, v[u].x * f[u], v[u].y * f[u], v[u].z * f[u], v[u].w * f[u]);
        else *reinterpret_cast<float4*>(xs + o) = make_float4(v[u].x * f[u], v[u].y * f[u], v[u].z * f[u], v[u].w * f[u]);
        // x~ = x dt as a bf16 pair: the V operand of the fused intra-chunk kernel
        if (xt_hi) store_pair4(xt_hi + o, xt_lo ? xt_lo + o : nullptr, v[u].x * fd[u], v[u].y * fd[u], v[u].z * fd[u], v[u].w * fd[u]);
      }
    }
  }
}

// Exclusive scan over chunks, in place, forward or reverse.  One thread owns VEC adjacent p of one (b,h,n).
//   forward: buf[c] holds states[c] on entry and h_prev[c] (state entering chunk c) on exit; last = final state.
//            run_{c+1} = exp(S_end[c]) run_c + states[c],  run_0 = init (or 0)
//   reverse: buf[c] holds contrib[c] on entry and dh[c] (adjoint of the state leaving chunk c) on exit.
//            run_{c-1} = exp(S_end[c]) run_c + contrib[c], run_{nc-1} = 0
// The chunk values are fetched four at a time before the dependent chain so the loads overlap.
template <int VEC>
__global__ void __launch_bounds__(256) state_scan_kernel(SsdP p, float* __restrict__ buf, const float* __restrict__ init,
                                                         float* __restrict__ last, int reverse,
                                                         uint16_t* __restrict__ pair_hi, uint16_t* __restrict__ pair_lo) {
  const int64_t NP = (int64_t)p.N * p.P;
  const int64_t per = NP / VEC;
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)p.B * p.H * per) return;
  const int64_t e = (i % per) * VEC; const int64_t bh = i / per; const int h = (int)(bh % p.H); const int bb = (int)(bh / p.H);
  float run[VEC];
#pragma unroll
  for (int v = 0; v < VEC; ++v) run[v] = (init && !reverse) ? init[bh * NP + e + v] : 0.0f;
  const float* send = p.S + ((int64_t)bb * p.H + h) * p.T + p.Q - 1;
  for (int c0 = 0; c0 < p.nc; c0 += 4) {
    float tmp[4][VEC]; float dec[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int cc = reverse ? p.nc - 1 - (c0 + j) : c0 + j;
      if (c0 + j < p.nc) {
        const float* slot = buf + (((int64_t)bb * p.nc + cc) * p.H + h) * NP + e;
        if (VEC == 4) { float4 q = *reinterpret_cast<const float4*>(slot); tmp[j][0] = q.x; tmp[j][1 % VEC] = q.y; tmp[j][2 % VEC] = q.z; tmp[j][3 % VEC] = q.w; }
        else tmp[j][0] = slot[0];
        dec[j] = expf(send[(int64_t)cc * p.Q]);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int cc = reverse ? p.nc - 1 - (c0 + j) : c0 + j;
      if (c0 + j < p.nc) {
        float* slot = buf + (((int64_t)bb * p.nc + cc) * p.H + h) * NP + e;
        if (VEC == 4) {
          *reinterpret_cast<float4*>(slot) = make_float4(run[0], run[1 % VEC], run[2 % VEC], run[3 % VEC]);
          // the same values as a bf16 pair: the state operand of the fused intra-chunk kernel
          if (pair_hi) store_pair4(pair_hi + (slot - buf), pair_lo ? pair_lo + (slot - buf) : nullptr, run[0], run[1 % VEC], run[2 % VEC], run[3 % VEC]);
        }
        else slot[0] = run[0];
#pragma unroll
        for (int v = 0; v < VEC; ++v) run[v] = fmaf(dec[j], run[v], tmp[j][v]);
      }
    }
  }
  if (last && !reverse) {
#pragma unroll
    for (int v = 0; v < VEC; ++v) last[bh * NP + e + v] = run[v];
  }
}

// dsend[b,c,h] = <dh[c], h_next[c]> with h_next[c] = h_prev[c+1], or the final state for the last chunk.
// own_state != 0: <dh[c], h_prev[c]> instead (the fused backward adds the other part of <dh, h_next> from the very
// values that enter dS, see chunk_rows_finish_w_kernel).
__global__ void __launch_bounds__(256) state_dot_kernel(SsdP p, float* __restrict__ dsend, int own_state) {
  __shared__ float red[32];
  const int bch = blockIdx.x;
  const int h = bch % p.H; const int bc = bch / p.H; const int cc = bc % p.nc; const int bb = bc / p.nc;
  const int NP = p.N * p.P;
  const float* a = p.dh + (int64_t)bch * NP;
  const float* b = own_state ? p.hprev + (int64_t)bch * NP : (cc + 1 < p.nc) ? p.hprev + (((int64_t)bb * p.nc + cc + 1) * p.H + h) * NP : p.hlast + ((int64_t)bb * p.H + h) * NP;
  float dot = 0.0f;
  for (int e = threadIdx.x; e < NP; e += blockDim.x) dot = fmaf(a[e], b[e], dot);
  float tot = block_sum(dot, red);
  if (threadIdx.x == 0) dsend[bch] = tot;
}

// Reverse scan and d[b,c,h] = <dh[c], h_prev[c]> in one launch for the pair path: one CTA per (b,h), a thread owns
// ITEMS groups of four adjacent p; the chunk values are fetched four chunks at a time before the dependent chain.
// Per-chunk dot products: warp sums into shared memory, then one thread per chunk adds the warps in order.
constexpr int SCAN_DOT_MAX_NC = 64;
template <int ITEMS>
__global__ void __launch_bounds__(1024) state_scan_rev_dot_kernel(SsdP p, float* __restrict__ buf, uint16_t* __restrict__ pair_hi,
                                                                  uint16_t* __restrict__ pair_lo, float* __restrict__ dsend) {
  __shared__ float wdot[SCAN_DOT_MAX_NC][32];
  const int bh = blockIdx.x, h = bh % p.H, bb = bh / p.H;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nth = blockDim.x;
  const int64_t NP = (int64_t)p.N * p.P;
  const float* send = p.S + ((int64_t)bb * p.H + h) * p.T + p.Q - 1;
  float4 run[ITEMS];
#pragma unroll
  for (int it = 0; it < ITEMS; ++it) run[it] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (int c0 = 0; c0 < p.nc; c0 += 4) {
    float4 q[4][ITEMS], hv[4][ITEMS]; float dec[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int cc = p.nc - 1 - (c0 + j);
      if (cc >= 0) {
        const int64_t base = (((int64_t)bb * p.nc + cc) * p.H + h) * NP;
#pragma unroll
        for (int it = 0; it < ITEMS; ++it) {
          const int64_t e = ((int64_t)it * nth + tid) * 4;
          if (e < NP) { q[j][it] = *reinterpret_cast<const float4*>(buf + base + e); hv[j][it] = *reinterpret_cast<const float4*>(p.hprev + base + e); }
        }
        dec[j] = expf(send[(int64_t)cc * p.Q]);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int cc = p.nc - 1 - (c0 + j);
      if (cc >= 0) {
        const int64_t base = (((int64_t)bb * p.nc + cc) * p.H + h) * NP;
        float dot = 0.0f;
#pragma unroll
        for (int it = 0; it < ITEMS; ++it) {
          const int64_t e = ((int64_t)it * nth + tid) * 4;
          if (e < NP) {
            const float4 r = run[it];
            *reinterpret_cast<float4*>(buf + base + e) = r;
            store_pair4(pair_hi + base + e, pair_lo ? pair_lo + base + e : nullptr, r.x, r.y, r.z, r.w);
            dot = fmaf(r.x, hv[j][it].x, fmaf(r.y, hv[j][it].y, fmaf(r.z, hv[j][it].z, fmaf(r.w, hv[j][it].w, dot))));
            run[it] = make_float4(fmaf(dec[j], r.x, q[j][it].x), fmaf(dec[j], r.y, q[j][it].y), fmaf(dec[j], r.z, q[j][it].z), fmaf(dec[j], r.w, q[j][it].w));
          }
        }
        dot = warp_sum(dot);
        if (lane == 0) wdot[cc][wid] = dot;
      }
    }
  }
  __syncthreads();
  if (tid < p.nc) {
    float tot = 0.0f;
    for (int j = 0; j < (nth >> 5); ++j) tot += wdot[tid][j];
    dsend[((int64_t)bb * p.nc + tid) * p.H + h] = tot;
  }
}

// true when the merged kernel took the launch
static bool launch_state_scan_rev_dot(cudaStream_t st, const SsdP& p, float* buf, uint16_t* pair_hi, uint16_t* pair_lo, float* dsend) {
  const int64_t quads = (int64_t)p.N * p.P / 4;
  if ((p.P & 3) || !pair_hi || !p.hprev || p.nc > SCAN_DOT_MAX_NC || quads > 4 * 1024) return false;
  const int items = quads <= 1024 ? 1 : (quads <= 2048 ? 2 : 4);
  const unsigned threads = (unsigned)(((quads + items - 1) / items + 31) / 32 * 32);
  const unsigned grid = (unsigned)(p.B * p.H);
  if (items == 1) state_scan_rev_dot_kernel<1><<<grid, threads, 0, st>>>(p, buf, pair_hi, pair_lo, dsend);
  else if (items == 2) state_scan_rev_dot_kernel<2><<<grid, threads, 0, st>>>(p, buf, pair_hi, pair_lo, dsend);
  else state_scan_rev_dot_kernel<4><<<grid, threads, 0, st>>>(p, buf, pair_hi, pair_lo, dsend);
  return true;
}

static pmb_status launch_state_scan(cudaStream_t st, const SsdP& p, float* buf, const float* init, float* last, int reverse,
                                    uint16_t* pair_hi = nullptr, uint16_t* pair_lo = nullptr) {
  const int64_t NP = (int64_t)p.N * p.P;
  const bool vec = (p.P % 4 == 0);
  const int64_t n = (int64_t)p.B * p.H * (vec ? NP / 4 : NP);
  if (vec) state_scan_kernel<4><<<(unsigned)cdiv(n, 256), 256, 0, st>>>(p, buf, init, last, reverse, pair_hi, pair_lo);
  else state_scan_kernel<1><<<(unsigned)cdiv(n, 256), 256, 0, st>>>(p, buf, init, last, reverse, nullptr, nullptr);
  PMB_LAUNCHED();
  return PMB_OK;
}

// fp32 blocks outside of a model take <dY, y - D x> except in rows (one token and head) that this holds for: there D x is more than 48 times what
// the scan adds per unit of dt (of dt, because heads with a small dt have a small y on any input), and the difference has lost most of y.
// Inputs of unit size have next to no such rows and keep their results, which <dY, y> throughout would move by up to 8e-4 in d(a_log) and
// d(dt_bias).  From fp64 those two are off by (8 heads of 64 x 64, 2 x 1000 tokens; y - D x everywhere / in the other rows): inputs
// of size 1: 6.7e-4 / 5.9e-4; 0.5: 2.8e-3 / 2.9e-3; 0.2: 2.6e-2 / 2.6e-3; 0.1: 0.10 / 2.2e-4; 0.02: 0.78 / 7.8e-5.
__device__ __forceinline__ bool outweighed(float skip_sq, float y_sq, float dt) { return skip_sq * dt * dt > 48.0f * 48.0f * y_sq; }

// One warp per (b,t,h): row dot products and dx.
//   ddt_x = <dx~, x>;  dS = <dY, Y - D x> - dt * ddt_x;  dDrow = <dY, x>;  dx = dx~ * dt + D * dY
__global__ void ssd_rowdots_kernel(SsdP p, float* __restrict__ dx, int64_t lddx, float* __restrict__ ddt_x,
                                   float* __restrict__ dS, float* __restrict__ dDrow) {
  int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  int64_t total = (int64_t)p.B * p.T * p.H;
  if (w >= total) return;
  int h = (int)(w % p.H); int64_t tk = w / p.H;
  float dtv = p.dtv(tk, h), Dv = p.D ? p.D[h] : 0.0f, Dy = p.skip_in_y ? Dv : 0.0f;
  float s1 = 0.0f, s2 = 0.0f, s3 = 0.0f, s2p = 0.0f, yy = 0.0f, kk = 0.0f;
  for (int pp = lane; pp < p.P; pp += 32) {
    float xv = p.x[tk * p.ldx + h * p.P + pp];
    float dxt = p.dxt[tk * (int64_t)(p.H * p.P) + h * p.P + pp];
    float dyv = p.dy[tk * p.lddy + h * p.P + pp];
    float yv = p.y[tk * p.ldy + h * p.P + pp] - Dy * xv;
    s1 = fmaf(dxt, xv, s1);
    s2 = fmaf(dyv, yv, s2);
    s3 = fmaf(dyv, xv, s3);
    if (p.yp) {
      const float q = p.yp[(tk * p.H + h) * p.P + pp], k = Dv * xv;
      s2p = fmaf(dyv, q, s2p); yy = fmaf(q, q, yy); kk = fmaf(k, k, kk);
    }
    dx[tk * lddx + h * p.P + pp] = fmaf(dxt, dtv, Dv * dyv);
  }
  s1 = warp_sum(s1); s2 = warp_sum(s2); s3 = warp_sum(s3);
  if (p.yp) {
    s2p = warp_sum(s2p); yy = warp_sum(yy); kk = warp_sum(kk);
    if (outweighed(kk, yy, dtv)) s2 = s2p;
  }
  if (lane == 0) {
    ddt_x[w] = s1;
    dS[w] = s2 - dtv * s1;
    dDrow[w] = s3;
  }
}

// One warp per (b,c,h): da = reverse inclusive cumsum of dS (dS[Q-1] += dsend).
// a-mode (dt == NULL): writes da.  dt-mode: ddt = ddt_x + A da; partial sums of da*dt and dDrow per chunk.
__global__ void ssd_chunk_finish_kernel(SsdP p, const float* __restrict__ ddt_x, const float* __restrict__ dS,
                                        const float* __restrict__ dDrow, const float* __restrict__ dsend,
                                        float* __restrict__ da_out, float* __restrict__ ddt_out, float* __restrict__ part) {
  int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  int total = p.B * p.nc * p.H;
  if (w >= total) return;
  int h = w % p.H, bc = w / p.H, cc = bc % p.nc, bb = bc / p.nc;
  float carry = 0.0f, pA = 0.0f, pD = 0.0f;
  float Ah = p.dt ? p.A[h] : 0.0f;
  int nblk = (p.Q + 31) / 32;
  // the strided loads of up to 8 rounds are requested together, ahead of the dependent scan chain
  constexpr int AHEAD = 8;
  float pre[AHEAD];
  const float send = dsend[w];
  for (int blk = nblk - 1; blk >= 0; --blk) {
    const int r = (nblk - 1 - blk) % AHEAD;
    if (r == 0) {
#pragma unroll
      for (int j = 0; j < AHEAD; ++j) {
        const int qq = (blk - j) * 32 + lane;
        pre[j] = (blk - j >= 0 && qq < p.Q) ? dS[p.tok(bb, cc, qq) * p.H + h] : 0.0f;
      }
    }
    int q = blk * 32 + lane;
    float v = 0.0f;
    int64_t idx = 0;
#pragma unroll
    for (int j = 0; j < AHEAD; ++j) if (j == r) v = pre[j];
    if (q < p.Q) {
      idx = p.tok(bb, cc, q) * p.H + h;
      if (q == p.Q - 1) v += send;
    } else {
      v = 0.0f;
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      float u = __shfl_down_sync(0xffffffffu, v, o);
      if (lane + o < 32) v += u;
    }
    v += carry;
    if (q < p.Q) {
      if (p.dt) {
        ddt_out[idx] = fmaf(Ah, v, ddt_x[idx]);
        pA = fmaf(v, p.dt[idx], pA);
        pD += dDrow[idx];
      } else {
        da_out[idx] = v;
      }
    }
    carry = __shfl_sync(0xffffffffu, v, 0);
  }
  if (p.dt) {
    pA = warp_sum(pA); pD = warp_sum(pD);
    if (lane == 0) {
      part[(int64_t)bc * p.H + h] = pA;
      part[(int64_t)p.B * p.nc * p.H + (int64_t)bc * p.H + h] = pD;
    }
  }
}

// Fused variant of the two kernels above, one 256-thread block per (b,c,h), for launches whose blocks fit the
// machine at once: the row dot products stay in shared memory and feed the reverse cumsum directly.
__global__ void __launch_bounds__(PREP_THREADS) chunk_rows_finish_kernel(SsdP p, float* __restrict__ dx, int64_t lddx,
                                                                         const float* __restrict__ dsend, float* __restrict__ da_out,
                                                                         float* __restrict__ ddt_out, float* __restrict__ part) {
  __shared__ float s_ddtx[PREP_MAX_Q], s_dS[PREP_MAX_Q], s_dD[PREP_MAX_Q], s_dt[PREP_MAX_Q], wsum[PREP_THREADS / 32], red[32];
  const int w = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int h = w % p.H, bc = w / p.H, cc = bc % p.nc, bb = bc / p.nc;
  const float Dv = p.D ? p.D[h] : 0.0f, Dy = p.skip_in_y ? Dv : 0.0f;
  const int64_t tok0 = p.tok(bb, cc, 0);
  const int P4 = p.P >> 2;
  // phase 1: a half-warp per row, float4 lanes (P <= 64) or strided lanes beyond
  const int sub = lane >> 4, l16 = lane & 15;
  for (int t0 = wid * 2; t0 < p.Q; t0 += (PREP_THREADS / 32) * 2) {
    const int t = t0 + sub;
    float s1 = 0.0f, s2 = 0.0f, s3 = 0.0f, s2p = 0.0f, yy = 0.0f, kk = 0.0f, dtv = 1.0f;
    if (t < p.Q) {
      const int64_t tk = tok0 + t;
      dtv = p.dtv(tk, h);
      for (int j = l16; j < P4; j += 16) {
        const float4 xv = reinterpret_cast<const float4*>(p.x + tk * p.ldx + h * p.P)[j];
        const float4 dxt = reinterpret_cast<const float4*>(p.dxt + tk * (int64_t)(p.H * p.P) + h * p.P)[j];
        const float4 dyv = reinterpret_cast<const float4*>(p.dy + tk * p.lddy + h * p.P)[j];
        float4 yv = reinterpret_cast<const float4*>(p.y + tk * p.ldy + h * p.P)[j];
        if (p.yp) {
          const float4 q = reinterpret_cast<const float4*>(p.yp + (tk * p.H + h) * p.P)[j];
          const float4 k = make_float4(Dv * xv.x, Dv * xv.y, Dv * xv.z, Dv * xv.w);
          s2p = fmaf(dyv.x, q.x, fmaf(dyv.y, q.y, fmaf(dyv.z, q.z, fmaf(dyv.w, q.w, s2p))));
          yy = fmaf(q.x, q.x, fmaf(q.y, q.y, fmaf(q.z, q.z, fmaf(q.w, q.w, yy))));
          kk = fmaf(k.x, k.x, fmaf(k.y, k.y, fmaf(k.z, k.z, fmaf(k.w, k.w, kk))));
        }
        yv.x -= Dy * xv.x; yv.y -= Dy * xv.y; yv.z -= Dy * xv.z; yv.w -= Dy * xv.w;
        s1 = fmaf(dxt.x, xv.x, fmaf(dxt.y, xv.y, fmaf(dxt.z, xv.z, fmaf(dxt.w, xv.w, s1))));
        s2 = fmaf(dyv.x, yv.x, fmaf(dyv.y, yv.y, fmaf(dyv.z, yv.z, fmaf(dyv.w, yv.w, s2))));
        s3 = fmaf(dyv.x, xv.x, fmaf(dyv.y, xv.y, fmaf(dyv.z, xv.z, fmaf(dyv.w, xv.w, s3))));
        reinterpret_cast<float4*>(dx + tk * lddx + h * p.P)[j] =
            make_float4(fmaf(dxt.x, dtv, Dv * dyv.x), fmaf(dxt.y, dtv, Dv * dyv.y), fmaf(dxt.z, dtv, Dv * dyv.z), fmaf(dxt.w, dtv, Dv * dyv.w));
      }
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {        // sums within each half-warp
      s1 += __shfl_xor_sync(0xffffffffu, s1, o); s2 += __shfl_xor_sync(0xffffffffu, s2, o); s3 += __shfl_xor_sync(0xffffffffu, s3, o);
    }
    if (p.yp) {
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        s2p += __shfl_xor_sync(0xffffffffu, s2p, o); yy += __shfl_xor_sync(0xffffffffu, yy, o); kk += __shfl_xor_sync(0xffffffffu, kk, o);
      }
      if (outweighed(kk, yy, dtv)) s2 = s2p;
    }
    if (t < p.Q && l16 == 0) { s_ddtx[t] = s1; s_dS[t] = s2 - dtv * s1; s_dD[t] = s3; s_dt[t] = dtv; }
  }
  __syncthreads();
  if (tid == 0) s_dS[p.Q - 1] += dsend[w];
  __syncthreads();
  // phase 2: reverse inclusive cumsum of dS over the chunk, rounds of 256 from the end
  const float Ah = p.dt ? p.A[h] : 0.0f;
  float carry = 0.0f, pA = 0.0f, pD = 0.0f;
  for (int r0 = 0; r0 < p.Q; r0 += PREP_THREADS) {
    const int q = p.Q - 1 - (r0 + tid);                 // thread 0 owns the last element of the chunk
    float v = q >= 0 ? s_dS[q] : 0.0f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const float u = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += u; }
    if (lane == 31) wsum[wid] = v;
    __syncthreads();
    float off = carry;
    for (int j = 0; j < wid; ++j) off += wsum[j];
    v += off;
    if (q >= 0) {
      const int64_t idx = (tok0 + q) * p.H + h;
      if (p.dt) { ddt_out[idx] = fmaf(Ah, v, s_ddtx[q]); pA = fmaf(v, s_dt[q], pA); pD += s_dD[q]; }
      else da_out[idx] = v;
    }
    float tot = carry;
    for (int j = 0; j < PREP_THREADS / 32; ++j) tot += wsum[j];
    carry = tot;
    __syncthreads();
  }
  if (p.dt) {
    const float tA = block_sum(pA, red);
    const float tD = block_sum(pD, red);
    if (tid == 0) {
      part[(int64_t)bc * p.H + h] = tA;
      part[(int64_t)p.B * p.nc * p.H + (int64_t)bc * p.H + h] = tD;
    }
  }
}

// Row sums and the reverse cumulative sum for the fused backward, one 256-thread block per (b,c,h).
// The gradient w.r.t. the in-chunk cumulative sum S is assembled from terms that were each formed once:
//   dS_t = r_t - c_t + f_t - e_t,      dS_{Q-1} += sum_s e_s + exp(S_end) <dh, h_prev>
//   r_t = sum_{s<t} W[t,s], c_t = sum_{u>t} W[u,t]   (W = dM o G o L, both sums from the same registers of the fused kernel)
//   f_t = <dY_t, exp(S_t) C_t h_prev>                 (the carried-state part of y, kept by the forward kernel)
//   e_s = exp(S_end - S_s) <x~_s, B_s dh>             (from the fused kernel's epilogue)
// so the cancellation inside sum_t S_t dS_t (the gradient of A) is between identically rounded numbers and never
// goes through y - D x or through two separately rounded matrix products.  da = reverse cumsum(dS);
// ddt = <dx~, x> + A da;  dx = dx~ dt + D dY;  per-chunk partials of dA and dD.
struct WSums { const float* rpart; const float* csum; const float* esum; const float* yoff; int nb; };
// A half-warp takes one row per pass and asks for its next one before (cp.async, slots of the thread's own, no barrier); five CTAs share an
// SM: while one sums over its chunk another streams.  Bound by HBM, rows of 256 bytes of four tensors (16384 tokens, 24 heads, 500 MB): 159 us
// with two rows per pass in registers and two CTAs, 127 with three; two rows ahead in shared memory and three CTAs 116, one row and three
// CTAs 122, four 106, five 107 (8192 tokens: 46, 43, 43, 45, 44).
constexpr int ROWS_THREADS = 256;
__global__ void __launch_bounds__(ROWS_THREADS, 5) chunk_rows_finish_w_kernel(SsdP p, WSums ws, float* __restrict__ dx, int64_t lddx,
                                                                           const float* __restrict__ dd, float* __restrict__ da_out,
                                                                           float* __restrict__ ddt_out, float* __restrict__ part,
                                                                           SsdGrads::RawDt raw) {
  __shared__ float wsum[ROWS_THREADS / 32], red[32];
  constexpr int NHW = ROWS_THREADS / 16;
  const int w = blockIdx.x, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int h = w % p.H, bc = w / p.H, cc = bc % p.nc, bb = bc / p.nc;
  const float Dv = p.D ? p.D[h] : 0.0f;
  const int64_t tok0 = p.tok(bb, cc, 0);
  const int P4 = p.P >> 2;
  const int hw = tid >> 4, l16 = lane & 15;
  const int64_t hp = (int64_t)p.H * p.P;
  extern __shared__ __align__(16) float4 rring[];           // [pass % 2][x, dx~, dY, yoff][thread], then five values per row of the chunk
  float4* const own = rring + tid;
  float* const s_ddtx = reinterpret_cast<float*>(rring + 8 * ROWS_THREADS);
  float *const s_dS = s_ddtx + p.Q, *const s_dD = s_dS + p.Q, *const s_dt = s_dD + p.Q, *const s_e = s_dt + p.Q;
  auto fetch = [&](int t) {
    if (t < p.Q && l16 < P4) {
      const int64_t tk = tok0 + t;
      const uint32_t d = (uint32_t)__cvta_generic_to_shared(own + (t / NHW % 2) * 4 * ROWS_THREADS);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(p.x + tk * p.ldx + h * p.P + 4 * l16) : "memory");
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16 * ROWS_THREADS), "l"(p.dxt + tk * hp + h * p.P + 4 * l16) : "memory");
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 32 * ROWS_THREADS), "l"(p.dy + tk * p.lddy + h * p.P + 4 * l16) : "memory");
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 48 * ROWS_THREADS), "l"(ws.yoff + tk * hp + h * p.P + 4 * l16) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(hw);
  for (int tb = 0; tb < p.Q; tb += NHW) {
    const int t = tb + hw;
    const int64_t tk = tok0 + t;
    float s1 = 0.0f, s2 = 0.0f, s3 = 0.0f, dtv = 1.0f, rr = 0.0f, cs = 0.0f, es = 0.0f;
    if (t < p.Q) {
      dtv = p.dtv(tk, h);
      if (l16 == 0) {
        const int64_t idx = tk * p.H + h;
        for (int rb = 0; rb <= t / 128; ++rb) rr += ws.rpart[((int64_t)w * ws.nb + rb) * p.Q + t];   // row blocks whose rows s can be < t
        cs = ws.csum[idx]; es = ws.esum[idx];
      }
    }
    fetch(t + NHW);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    if (t < p.Q && l16 < P4) {
      const float4* const in = own + (t / NHW % 2) * 4 * ROWS_THREADS;
      const float4 xv = in[0], dxt = in[ROWS_THREADS], dyv = in[2 * ROWS_THREADS], yo = in[3 * ROWS_THREADS];
      s1 = fmaf(dxt.x, xv.x, fmaf(dxt.y, xv.y, fmaf(dxt.z, xv.z, dxt.w * xv.w)));
      s2 = fmaf(dyv.x, yo.x, fmaf(dyv.y, yo.y, fmaf(dyv.z, yo.z, dyv.w * yo.w)));
      s3 = fmaf(dyv.x, xv.x, fmaf(dyv.y, xv.y, fmaf(dyv.z, xv.z, dyv.w * xv.w)));
      reinterpret_cast<float4*>(dx + tk * lddx + h * p.P)[l16] =
          make_float4(fmaf(dxt.x, dtv, Dv * dyv.x), fmaf(dxt.y, dtv, Dv * dyv.y), fmaf(dxt.z, dtv, Dv * dyv.z), fmaf(dxt.w, dtv, Dv * dyv.w));
    }
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      s1 += __shfl_xor_sync(0xffffffffu, s1, o); s2 += __shfl_xor_sync(0xffffffffu, s2, o); s3 += __shfl_xor_sync(0xffffffffu, s3, o);
    }
    if (t < p.Q && l16 == 0) {
      s_ddtx[t] = s1; s_dD[t] = s3; s_dt[t] = dtv; s_e[t] = es;
      s_dS[t] = ((rr - cs) + s2) - es;
    }
  }
  __syncthreads();
  // sum of e over the chunk in a fixed order, then the terms that belong to the last position
  float ep = 0.0f;
  for (int q = tid; q < p.Q; q += ROWS_THREADS) ep += s_e[q];
  const float esum = block_sum(ep, red);
  if (tid == 0) {
    const float send = p.S[((int64_t)bb * p.H + h) * p.T + (int64_t)cc * p.Q + p.Q - 1];
    s_dS[p.Q - 1] += esum + expf(send) * dd[w];
  }
  __syncthreads();
  const float Ah = p.dt ? p.A[h] : 0.0f;
  float carry = 0.0f, pA = 0.0f, pD = 0.0f, pB = 0.0f;
  for (int r0 = 0; r0 < p.Q; r0 += ROWS_THREADS) {
    const int q = p.Q - 1 - (r0 + tid);
    float v = q >= 0 ? s_dS[q] : 0.0f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) { const float u = __shfl_up_sync(0xffffffffu, v, o); if (lane >= o) v += u; }
    if (lane == 31) wsum[wid] = v;
    __syncthreads();
    float off = carry;
    for (int j = 0; j < wid; ++j) off += wsum[j];
    v += off;
    if (q >= 0) {
      const int64_t idx = (tok0 + q) * p.H + h;
      if (p.dt) {
        const float ddt = fmaf(Ah, v, s_ddtx[q]);
        ddt_out[idx] = ddt; pA = fmaf(v, s_dt[q], pA); pD += s_dD[q];
        if (raw.hi) {      // through the softplus: d softplus(u) / du = sigmoid(u) = 1 - exp(-softplus(u))
          const float gr = ddt * (-expm1f(-s_dt[q]));
          const int64_t o = (tok0 + q) * raw.ld + raw.col0 + h;
          uint32_t hh, ll;
          split_bf16_pair(gr, hh, ll);
          raw.hi[o] = (uint16_t)hh;
          if (raw.lo) raw.lo[o] = (uint16_t)ll;
          pB += gr;
        }
      }
      else da_out[idx] = v;
    }
    float tot = carry;
    for (int j = 0; j < ROWS_THREADS / 32; ++j) tot += wsum[j];
    carry = tot;
    __syncthreads();
  }
  if (p.dt) {
    const float tA = block_sum(pA, red);
    const float tD = block_sum(pD, red);
    const float tB = block_sum(pB, red);
    if (tid == 0) {
      part[(int64_t)bc * p.H + h] = tA;
      part[(int64_t)p.B * p.nc * p.H + (int64_t)bc * p.H + h] = tD;
      part[2 * (int64_t)p.B * p.nc * p.H + (int64_t)bc * p.H + h] = tB;
    }
  }
}

// The per-head sums of the pair path in one launch: one warp per head adds the partials of dA, dD and (when asked for) d_dt_bias in a
// fixed order; d_a_log = A dA.  (One thread per head walked the rows in 16 us at 64 rows.)
__global__ void __launch_bounds__(128) head_finish_kernel(const float* __restrict__ part, int rows, int H, const float* __restrict__ A, float* __restrict__ dA,
                                   float* __restrict__ dD, float* __restrict__ d_dt_bias, float* __restrict__ d_a_log) {
  pdl_launch();
  pdl_wait();
  const int h = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (h >= H) return;
  float a = 0.0f, d = 0.0f, b = 0.0f;
  for (int r = lane; r < rows; r += 32) {
    a += part[(int64_t)r * H + h];
    d += part[((int64_t)rows + r) * H + h];
    b += part[(2 * (int64_t)rows + r) * H + h];
  }
  a = warp_sum(a); d = warp_sum(d); b = warp_sum(b);
  if (lane > 0) return;
  dA[h] = a;
  if (dD) dD[h] = d;
  if (d_dt_bias) d_dt_bias[h] = b;
  if (d_a_log) d_a_log[h] = A[h] * a;
}

pmb_status ssd_head_finish(cudaStream_t st, const float* part, int rows, int H, const float* A, float* dA, float* dD, float* d_dt_bias, float* d_a_log) {
  PMB_TRY(launch_pdl(st, head_finish_kernel, dim3((unsigned)cdiv(H, 4)), 128, 0, part, rows, H, A, dA, dD, d_dt_bias, d_a_log));
  return PMB_OK;
}

// Sums the split-K partial tiles in a fixed order.  mode 0: dG (lower-triangular 64x64 tiles only, the
// others were never produced); mode 1/2: dC/dB rows go to out + token * ld + g * cols.  A block has 256 x V adjacent elements of one batch
// (blockIdx.y and z): V = 4 where rows and destinations allow 16-byte accesses.  With an element per thread and 64-bit divisions to find its place
// two slabs of 16384 x 64 took 12.6 us, 4.2 now.
constexpr int REDUCE_Y = 65535;
template <int V>
__global__ void __launch_bounds__(256) splitk_reduce_kernel(const float* __restrict__ part, int nsplit, int rows, int cols, int mode, int G, int Q,
                                                            float* __restrict__ out, int64_t ld, int64_t batches, int tile,
                                                            uint16_t* __restrict__ pair_hi, uint16_t* __restrict__ pair_lo) {
  const int64_t mn = (int64_t)rows * cols, r = ((int64_t)blockIdx.x * 256 + threadIdx.x) * V, batch = blockIdx.y + (int64_t)blockIdx.z * REDUCE_Y;
  if (r >= mn || batch >= batches) return;
  const int m = mn >> 32 ? (int)(r / cols) : (int)((uint32_t)r / (uint32_t)cols), n = (int)(r - (int64_t)m * cols);
  if (mode == 0 && n / tile > m / tile) return;   // tiles above the diagonal were never produced (a tile's width is a multiple of V)
  float s[V];
#pragma unroll
  for (int e = 0; e < V; ++e) s[e] = 0.0f;
  const float* p = part + batch * nsplit * mn + r;
#pragma unroll 4
  for (int k = 0; k < nsplit; ++k, p += mn) {
    if (V == 4) {
      const float4 v = *reinterpret_cast<const float4*>(p);
      s[0] += v.x; s[1 % V] += v.y; s[2 % V] += v.z; s[3 % V] += v.w;
    } else s[0] += *p;
  }
  if (mode == 0 && pair_hi) {       // dG as a bf16 pair: it is only ever an operand of the dC / dB contractions
    if (V == 4) store_pair4(pair_hi + batch * mn + r, pair_lo ? pair_lo + batch * mn + r : nullptr, s[0], s[1 % V], s[2 % V], s[3 % V]);
    else {
      uint32_t h, l;
      split_bf16_pair(s[0], h, l);
      pair_hi[batch * mn + r] = (uint16_t)h;
      if (pair_lo) pair_lo[batch * mn + r] = (uint16_t)l;
    }
    return;
  }
  float* o = out + (mode == 0 ? batch * mn + r : (batch / G * Q + m) * ld + batch % G * cols + n);
  if (V == 4) *reinterpret_cast<float4*>(o) = make_float4(s[0], s[1 % V], s[2 % V], s[3 % V]);
  else *o = s[0];
}

static int pick_nsplit(int batches, int tiles, int hpg) {
  int want = (int)cdiv(2 * 148, (int64_t)batches * tiles);
  if (want < 1) want = 1;
  return want > hpg ? hpg : want;
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
static bool fused_enabled();

// Buffers of one scan.  part bit 0: what the forward writes and the backward reads (kept per forward slot by the
// block workspace); bit 1: what only the backward touches (one copy).  Fields of the other part are left alone.
// plain16: the products read plain bf16 operands and ssd_dx.cu has the backward (ssd_plain16_shape), which needs neither the carried part of y nor sums of W.
void ssd_ws_take(Arena& ar, int B, int T, int H, int P, int N, int G, int Q, SsdWs* wp, int part, bool plain16) {
  SsdWs& w = *wp;
  const int nc = T / Q;
  const bool tcshape = Q % 64 == 0 && N % 32 == 0 && P % 64 == 0;
  const bool fz = ssd_fused_supported(P, N, Q) && fused_enabled();
  const size_t hp = (size_t)B * T * H * P, gn = (size_t)B * T * 2 * G * N, stn = (size_t)B * nc * H * N * P, qq = (size_t)B * nc * G * Q * Q;
  if (part & 1) {
    w.S = ar.take<float>((size_t)B * H * T);
    w.hprev = ar.take<float>(stn);
    w.hlast = ar.take<float>((size_t)B * H * N * P);
    if (!fz) w.CB = ar.take<float>(qq);
    w.xs = ar.take<float>((tcshape && !fz) ? hp : 0);
    w.xs_hi = fz ? ar.take<uint16_t>(hp) : nullptr; w.xs_lo = fz ? ar.take<uint16_t>(hp) : nullptr;
    // bf16 (hi, lo) pairs of the operands of the fused intra-chunk kernels, and the carried-state part of y
    w.xt_hi = fz ? ar.take<uint16_t>(hp) : nullptr; w.xt_lo = fz ? ar.take<uint16_t>(hp) : nullptr;
    w.bc_hi = fz ? ar.take<uint16_t>(gn) : nullptr; w.bc_lo = fz ? ar.take<uint16_t>(gn) : nullptr;
    w.hp_hi = fz ? ar.take<uint16_t>(stn) : nullptr; w.hp_lo = fz ? ar.take<uint16_t>(stn) : nullptr;
    w.yoff = fz && !plain16 ? ar.take<float>(hp) : nullptr;
  }
  if (part & 2) {
    if (fz) w.CB = ar.take<float>(qq);     // only for a backward that cannot take the fused kernel after a forward that did
    w.dh = ar.take<float>(stn);
    w.dG = ar.take<float>(qq);
    w.dxt = ar.take<float>(hp);
    w.rows = ar.take<float>((size_t)4 * B * T * H);
    w.part = ar.take<float>((size_t)B * nc * 3 * H);
    {
      int nbcg = B * nc * G, hpg = H / G, qt = (int)cdiv(Q, BM);
      size_t a = (size_t)pick_nsplit(nbcg, qt * (qt + 1) / 2, hpg) * nbcg * Q * Q;
      size_t b = (size_t)pick_nsplit(nbcg, qt * (int)cdiv(N, BN), hpg) * nbcg * Q * N;
      size_t need = a > b ? a : b;
      if (tcshape) {
        // tensor-core path: the head-split dB / dC partial tiles
        size_t dbc = (size_t)ssd_tc_dbc_nsplit_dims(B, T, H, N, G, Q) * nbcg * Q * N;
        if (dbc > need) need = dbc;
        size_t dgp = (size_t)ssd_tc_dg_nsplit_dims(B, T, H, G, Q) * nbcg * Q * Q;
        if (dgp > need) need = dgp;
      }
      if (fz) {
        // pair path: dC and dB run side by side, each with its own partial tiles
        size_t dbc2 = (size_t)2 * ssd_pairs_dbc_nsplit(B, T, H, N, G, Q) * nbcg * Q * N;
        if (dbc2 > need) need = dbc2;
        size_t dgp2 = (size_t)ssd_dg_nsplit(B, T, H, G, Q) * nbcg * Q * Q;
        if (dgp2 > need) need = dgp2;
      }
      w.splitk = ar.take<float>(need);
    }
    w.dys = ar.take<float>((tcshape && !fz) ? hp : 0);
    w.dys_hi = fz ? ar.take<uint16_t>(hp) : nullptr; w.dys_lo = fz ? ar.take<uint16_t>(hp) : nullptr;
    w.dg_hi = fz ? ar.take<uint16_t>(qq) : nullptr; w.dg_lo = fz ? ar.take<uint16_t>(qq) : nullptr;
    w.dy_hi = fz ? ar.take<uint16_t>(hp) : nullptr; w.dy_lo = fz ? ar.take<uint16_t>(hp) : nullptr;
    w.dh_hi = fz ? ar.take<uint16_t>(stn) : nullptr; w.dh_lo = fz ? ar.take<uint16_t>(stn) : nullptr;
    // the sums of W that the fused backward kernel leaves for the row-sum kernel
    w.csum = fz && !plain16 ? ar.take<float>((size_t)B * T * H) : nullptr;
    w.esum = fz && !plain16 ? ar.take<float>((size_t)B * T * H) : nullptr;
    w.rpart = fz ? ar.take<float>((size_t)B * T * H * (Q / 128)) : nullptr;
  }
}

size_t ssd_ws_layout(int B, int T, int H, int P, int N, int G, int Q, void* base, size_t bytes, SsdWs* out) {
  Arena ar(base, bytes);
  SsdWs w{};
  ssd_ws_take(ar, B, T, H, P, N, G, Q, &w, 3);
  if (out) *out = w;
  return ar.ok ? ar.used() : 0;
}

static pmb_status fill_params(const SsdIn& in, const SsdWs& ws, SsdP* pp) {
  if (in.Q <= 0 || in.T % in.Q != 0) return fail(PMB_ERR_SHAPE, "ssd: T=%d is not a multiple of block_len=%d", in.T, in.Q);
  if (!(in.G == 1 || in.G == in.H)) return fail(PMB_ERR_SHAPE, "ssd: n_groups must be 1 or n_heads");
  SsdP p{};
  p.B = in.B; p.T = in.T; p.H = in.H; p.P = in.P; p.N = in.N; p.G = in.G; p.Q = in.Q; p.nc = in.T / in.Q; p.hpg = in.H / in.G;
  p.x = in.x; p.ldx = in.ldx; p.dt = in.dt; p.A = in.A; p.a = in.a; p.b = in.b; p.c = in.c; p.ldbc = in.ldbc; p.D = in.D;
  p.S = ws.S; p.hprev = ws.hprev; p.hlast = ws.hlast; p.CB = ws.CB; p.dh = ws.dh; p.dG = ws.dG; p.dxt = ws.dxt;
  *pp = p;
  return PMB_OK;
}

template <class Op>
static pmb_status run_op(cudaStream_t st, const char* name, const Op& op, int batches, double flops) {
  ProfScope prof(st, name, flops, 0.0);
  return launch_bgemm(st, op, batches);
}

template <class Op>
static Op make_op(const SsdP& p, int Mdim, int Ndim) {
  Op op{};
  op.p = p; op.Mdim = Mdim; op.Ndim = Ndim;
  return op;
}

// ---------------------------------------------------------------------------------------------
// Independent kernels of one scan run side by side.  At training sizes of a few thousand tokens every kernel
// of the scan occupies the GPU for tens of microseconds with one or two ragged waves of latency-bound CTAs, so
// the chains that do not depend on each other (forward: C B^T next to x~ -> chunk states -> state pass;
// backward: dG -> dC -> dB next to dstates -> reverse pass -> dx~ -> row sums) go to two streams joined by events.
// One side stream and a handful of events per device, created on first use (make the first call outside stream
// capture).  PMB_SSD_CONCURRENT=0 keeps everything on the caller's stream.
// ---------------------------------------------------------------------------------------------
// lane 0 serves the backward, lane 2 the forward: a recompute may be in flight on another stream while the
// backward of the block above it runs, and the two must not share events
static pmb_status side_lane(int idx, SideLane** out) {
  static const int on = [] { const char* e = getenv("PMB_SSD_CONCURRENT"); return (e && e[0] == '0') ? 0 : 1; }();
  *out = nullptr;
  if (!on) return PMB_OK;
  return get_side_lane(idx, out);
}
static bool fused_enabled() {
  static const int on = [] { const char* e = getenv("PMB_SSD_FUSED"); return (e && e[0] == '0') ? 0 : 1; }();
  return on != 0;
}

bool ssd_chain_enabled() {
  static const bool simt = [] { const char* e = getenv("PMB_SSD_ENGINE"); return e && strcmp(e, "simt") == 0; }();
  return fused_enabled() && !simt;
}
bool ssd_wants_plain_y(int P, int N, int Q) { return !(ssd_chain_enabled() && ssd_fused_supported(P, N, Q)); }
bool ssd_plain16_shape(int P, int N, int Q) { return P == 64 && N == 64 && (Q == 128 || Q == 256); }

// x~[b,t,h,:] = x[b,t,h,:] * dt[b,t,h] as a bf16 pair (only when the fused cumsum kernel did not already write it)
__global__ void __launch_bounds__(256) xt_pair_kernel(const float* __restrict__ x, int64_t ldx, const float* __restrict__ dt,
                                                      uint16_t* __restrict__ hi, uint16_t* __restrict__ lo, int64_t rows, int H, int P,
                                                      const float* __restrict__ S, int T, int Q, uint16_t* __restrict__ xs_hi, uint16_t* __restrict__ xs_lo) {
  const int P4 = P >> 2;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * H * P4) return;
  const int j = (int)(i % P4); const int64_t w = i / P4; const int h = (int)(w % H); const int64_t tk = w / H;
  const float f = dt ? dt[tk * H + h] : 1.0f;
  const float4 v = reinterpret_cast<const float4*>(x + tk * ldx + h * P)[j];
  const int64_t o = (tk * H + h) * (int64_t)P + 4 * j;
  store_pair4(hi + o, lo ? lo + o : nullptr, v.x * f, v.y * f, v.z * f, v.w * f);      // (lo == NULL: the hi halves alone are read)
  // xs = x~ exp(S_end - S_t): the operand of the chunk-state and dB contractions
  const int b = (int)(tk / T), t = (int)(tk % T);
  const float* sp = S + ((int64_t)b * H + h) * T;
  const float f2 = f * __expf(sp[(t / Q) * Q + Q - 1] - sp[t]);
  store_pair4(xs_hi + o, xs_lo ? xs_lo + o : nullptr, v.x * f2, v.y * f2, v.z * f2, v.w * f2);
}

// The B and C columns (adjacent in the caller's buffer when it is the block's activation buffer, else two arrays)
// as bf16 pairs with row pitch 2*G*N: B in columns [0, G*N), C in [G*N, 2*G*N).
static pmb_status fused_operand_pairs(cudaStream_t st, const SsdIn& in, const SsdWs& ws, bool want_xt) {
  const int64_t rows = (int64_t)in.B * in.T;
  const int gn = in.G * in.N;
  if (in.bc_pair_ready) {
    // written by the producer of B and C
  } else if (in.c == in.b + gn) {
    PMB_TRY(split_pair16(st, in.b, rows, 2 * gn, in.ldbc, ws.bc_hi, ws.bc_lo, 2 * gn));
  } else {
    ProfScope prof(st, "split_f32_bf16x2", 0.0, 16.0 * rows * gn);
    PMB_TRY(split_pair16_strided(st, in.b, rows, gn, in.ldbc, ws.bc_hi, ws.bc_lo, 2 * gn));
    PMB_TRY(split_pair16_strided(st, in.c, rows, gn, in.ldbc, ws.bc_hi + gn, ws.bc_lo + gn, 2 * gn));
  }
  if (want_xt) {
    ProfScope prof(st, "ssd_xt_pair", 0.0, (in.plain16 ? 8.0 : 12.0) * rows * in.H * in.P);
    xt_pair_kernel<<<(unsigned)cdiv(rows * in.H * (in.P / 4), 256), 256, 0, st>>>(in.x, in.ldx, in.dt, ws.xt_hi, in.plain16 ? nullptr : ws.xt_lo, rows,
                                                                                  in.H, in.P, ws.S, in.T, in.Q, ws.xs_hi, in.plain16 ? nullptr : ws.xs_lo);
    PMB_LAUNCHED();
  }
  return PMB_OK;
}

static FusedArgs fused_args(const SsdIn& in, const SsdWs& ws) {
  FusedArgs fa{};
  fa.B = in.B; fa.T = in.T; fa.H = in.H; fa.P = in.P; fa.N = in.N; fa.G = in.G; fa.Q = in.Q;
  fa.S = ws.S;
  const int64_t pitch = 2 * (int64_t)in.G * in.N;
  const bool pairs = ws.bc_lo && !in.plain16;
  fa.b = Op16{ws.bc_hi, pairs ? ws.bc_lo : nullptr, pitch};
  fa.c = Op16{ws.bc_hi + in.G * in.N, pairs ? ws.bc_lo + in.G * in.N : nullptr, pitch};
  return fa;
}

static pmb_status ssd_fwd_on_lanes(cudaStream_t st, const SsdIn& in, const float* init_state, float* y, int64_t ldy, float* final_state,
                                   const SsdWs& ws) {
  SsdP p;
  PMB_TRY(fill_params(in, ws, &p));
  p.yout = y; p.ldyo = ldy; p.yplain = in.y_plain;
  int nbch = p.B * p.nc * p.H, nbcg = p.B * p.nc * p.G;
  const double tok = (double)p.B * p.T;
  const bool tc = ssd_tc_supported(in) && (ldy % 4 == 0) && (reinterpret_cast<uintptr_t>(y) % 16 == 0);
  // the intra-chunk chain C B^T -> mask -> x x~ (+ the carried-state term) as one tcgen05 kernel on bf16 pairs
  const bool fz = tc && fused_enabled() && ssd_fused_supported(p.P, p.N, p.Q);
  SsdIn in_tc = in;
  bool xt_ready = false;
  {
    CumsumRaw raw{in.dt_raw, in.ld_raw, in.dt_bias, in.a_log, const_cast<float*>(in.dt), const_cast<float*>(in.A)};
    if (in.dt_raw && (!in.dt || !in.A || !in.dt_bias || !in.a_log)) return fail(PMB_ERR_ARG, "ssd: dt_raw needs dt, A, dt_bias and a_log");
    // (one block per (b,c,h): worth it while those blocks fit the machine at once; beyond that the two separate,
    // finer-grained kernels use the memory system better)
    if (tc && nbch <= 4 * 148 && p.Q <= PREP_MAX_Q && (in.ldx % 4 == 0) && (reinterpret_cast<uintptr_t>(in.x) % 16 == 0)) {
      ProfScope prof(st, "ssd_chunk_prepare", 0.0, 8.0 * tok * p.H * (1.0 + p.P));
      // at a few hundred (b,c,h) the second phase (the only one with real traffic) is short of threads: split its rows
      const unsigned ysplit = nbch <= 148 ? 4u : (nbch <= 2 * 148 ? 2u : 1u);
      chunk_prepare_kernel<<<dim3((unsigned)nbch, ysplit), PREP_THREADS, 0, st>>>(p, raw, ws.xs, fz ? ws.xt_hi : nullptr, in.plain16 ? nullptr : ws.xt_lo, fz ? ws.xs_hi : nullptr,
                                                                                  in.plain16 ? nullptr : ws.xs_lo);
      PMB_LAUNCHED();
      in_tc.xs_ready = true;
      xt_ready = fz;
    } else {
      ProfScope prof(st, "ssd_chunk_cumsum", 0.0, 8.0 * tok * p.H);
      chunk_cumsum_kernel<<<(unsigned)cdiv((int64_t)nbch * 32, 256), 256, 0, st>>>(p, raw);
      PMB_LAUNCHED();
    }
  }
  SideLane* lane = nullptr;
  if (tc && !fz) PMB_TRY(side_lane(2, &lane));      // (the pair path is one chain: nothing to run beside it)
  if (fz) {
    // every contraction reads bf16 pairs: B | C and x~ / xs come from their producers, or are split here
    if (!in.bc_pair_ready || !xt_ready) PMB_TRY(fused_operand_pairs(st, in, ws, !xt_ready));
    PMB_TRY(ssd_pairs_state(st, in, ws, 0));
  } else if (tc) {
    cudaStream_t sb = lane ? lane->s : st;
    if (lane) PMB_TRY(order_after(st, lane->ev[0], sb));     // S is ready
    PMB_TRY(ssd_tc_cb(sb, in, ws));
    PMB_TRY(ssd_tc_state(st, in_tc, ws));
  } else {
    PMB_TRY(run_op(st, "ssd_cb", make_op<OpCB>(p, p.Q, p.Q), nbcg, 2.0 * tok * p.Q * p.N * p.G));
    PMB_TRY(run_op(st, "ssd_chunk_state", make_op<OpState>(p, p.N, p.P), nbch, 2.0 * tok * p.H * p.N * p.P));
  }
  int64_t nel = (int64_t)p.B * p.H * p.N * p.P;
  {
    ProfScope prof(st, "ssd_state_pass", 0.0, 8.0 * nel * p.nc);
    PMB_TRY(launch_state_scan(st, p, p.hprev, init_state, p.hlast, 0, fz ? ws.hp_hi : nullptr, in.plain16 ? nullptr : ws.hp_lo));
  }
  if (lane) PMB_TRY(order_after(lane->s, lane->ev[1], st));   // C B^T (or the operand pairs) are ready
  if (fz) {
    FusedArgs fa = fused_args(in, ws);
    fa.v = Op16{ws.xt_hi, in.plain16 ? nullptr : ws.xt_lo, (int64_t)p.H * p.P};
    fa.state = Op16{ws.hp_hi, in.plain16 ? nullptr : ws.hp_lo, p.P};
    fa.out = y; fa.ldo = ldy; fa.x = in.x; fa.ldx = in.ldx; fa.D = in.D;
    fa.off_out = in.plain16 ? nullptr : ws.yoff;
    PMB_TRY(ssd_fused(st, 0, fa));
  }
  else if (tc) PMB_TRY(ssd_tc_scan(st, in, y, ldy, ws));
  else PMB_TRY(run_op(st, "ssd_chunk_scan", make_op<OpScan>(p, p.Q, p.P), nbch, 2.0 * tok * p.H * p.P * (p.Q + p.N)));
  if (final_state) PMB_CUDA(cudaMemcpyAsync(final_state, ws.hlast, (size_t)nel * sizeof(float), cudaMemcpyDeviceToDevice, st));
  return PMB_OK;
}

pmb_status ssd_fwd(cudaStream_t st, const SsdIn& in, const float* init_state, float* y, int64_t ldy, float* final_state,
                   const SsdWs& ws) {
  return lanes_joined(st, ssd_fwd_on_lanes(st, in, init_state, y, ldy, final_state, ws));
}

// dYs[b,t,h,:] = dY[b,t,h,:] exp(S[b,h,t]) as a bf16 pair (when the producer of dY did not already write it)
__global__ void __launch_bounds__(256) dys_pair_kernel(const float* __restrict__ dy, int64_t lddy, const float* __restrict__ S,
                                                       uint16_t* __restrict__ hi, uint16_t* __restrict__ lo, int64_t rows, int T, int H, int P) {
  const int P4 = P >> 2;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * H * P4) return;
  const int j = (int)(i % P4); const int64_t w = i / P4; const int h = (int)(w % H); const int64_t tk = w / H;
  const float f = __expf(S[((tk / T) * H + h) * T + tk % T]);
  const float4 v = reinterpret_cast<const float4*>(dy + tk * lddy + h * P)[j];
  const int64_t o = (tk * H + h) * (int64_t)P + 4 * j;
  store_pair4(hi + o, lo ? lo + o : nullptr, v.x * f, v.y * f, v.z * f, v.w * f);
}

bool ssd_bwd_takes_pairs(const SsdIn& in, const float* dy, int64_t lddy, const SsdGrads& g) {
  const bool tc = ssd_tc_supported(in) && (lddy % 4 == 0) && (reinterpret_cast<uintptr_t>(dy) % 16 == 0) && (g.lddbc % 4 == 0) &&
                  ((reinterpret_cast<uintptr_t>(g.db) | reinterpret_cast<uintptr_t>(g.dc)) % 16 == 0);
  return tc && fused_enabled() && ssd_fused_supported(in.P, in.N, in.Q) && (g.lddx % 4 == 0) && (reinterpret_cast<uintptr_t>(g.dx) % 16 == 0);
}

static pmb_status ssd_bwd_on_lanes(cudaStream_t st, const SsdIn& in, const float* y, int64_t ldy, const float* dy, int64_t lddy,
                                   const SsdGrads& g, const SsdWs& ws) {
  SsdP p;
  PMB_TRY(fill_params(in, ws, &p));
  const bool plain = in.y_plain && !in.y_plain_rarely;
  p.y = plain ? in.y_plain : y; p.ldy = plain ? (int64_t)in.H * in.P : ldy; p.skip_in_y = in.D && !plain; p.yp = plain ? nullptr : in.y_plain; p.dy = dy; p.lddy = lddy; p.db = g.db; p.dc = g.dc; p.lddbc = g.lddbc;
  int nbch = p.B * p.nc * p.H, nbcg = p.B * p.nc * p.G;
  int64_t rows = (int64_t)p.B * p.T * p.H;
  float* ddt_x = ws.rows; float* dS = ws.rows + rows; float* dDrow = ws.rows + 2 * rows; float* dsend = ws.rows + 3 * rows;
  const double tok = (double)p.B * p.T;
  const bool tc = ssd_tc_supported(in) && (lddy % 4 == 0) && (reinterpret_cast<uintptr_t>(dy) % 16 == 0) && (g.lddbc % 4 == 0) &&
                  ((reinterpret_cast<uintptr_t>(g.db) | reinterpret_cast<uintptr_t>(g.dc)) % 16 == 0);
  const bool tc_group = tc;
  const bool fz = ssd_bwd_takes_pairs(in, dy, lddy, g);
  SideLane* lane = nullptr;
  if (tc) PMB_TRY(side_lane(0, &lane));
  cudaStream_t sb = lane ? lane->s : st;                      // stream of the dG -> dC -> dB chain
  if (fz) {
    // both chains read dY (and dY exp(S)) as bf16 pairs: written by the producer of dY, or here
    const int64_t tokens = (int64_t)p.B * p.T;
    if (!in.dy_pair_ready) PMB_TRY(split_pair16(st, dy, tokens, p.H * p.P, lddy, ws.dy_hi, ws.dy_lo, (int64_t)p.H * p.P));
    if (!in.dys_ready) {
      ProfScope prof(st, "ssd_prescale_dy", 0.0, 8.0 * tokens * p.H * p.P);
      dys_pair_kernel<<<(unsigned)cdiv(tokens * p.H * (p.P / 4), 256), 256, 0, st>>>(dy, lddy, ws.S, ws.dys_hi, ws.dys_lo, tokens, p.T, p.H, p.P);
      PMB_LAUNCHED();
    }
  }
  if (lane) PMB_TRY(order_after(st, lane->ev[0], sb));        // inputs of the scan are ready
  if (fz) {
    PMB_TRY(ssd_pairs_state(st, in, ws, 1));
  } else if (tc) {
    PMB_TRY(ssd_tc_dstate(st, in, dy, lddy, ws));
  } else {
    PMB_TRY(run_op(st, "ssd_bwd_dstate", make_op<OpDstate>(p, p.N, p.P), nbch, 2.0 * tok * p.H * p.N * p.P));
  }
  if (lane) PMB_CUDA(cudaEventRecord(lane->ev[1], st));       // dY exp(S) is ready (dC reads it)
  {
    ProfScope prof(st, "ssd_bwd_state_pass", 0.0, 12.0 * p.B * p.H * p.N * p.P * p.nc);
    uint16_t* const dh_lo = in.plain16 ? nullptr : ws.dh_lo;
    if (fz && launch_state_scan_rev_dot(st, p, p.dh, ws.dh_hi, dh_lo, dsend)) {
      PMB_LAUNCHED();
    } else {
      PMB_TRY(launch_state_scan(st, p, p.dh, nullptr, nullptr, 1, fz ? ws.dh_hi : nullptr, dh_lo));
      state_dot_kernel<<<(unsigned)nbch, 256, 0, st>>>(p, dsend, fz ? 1 : 0);
      PMB_LAUNCHED();
    }
  }
  if (lane) PMB_CUDA(cudaEventRecord(lane->ev[2], st));       // dh is ready (dB reads it)
  if (fz && in.plain16) {
    // (the B / C / x~ operands were written by the forward of this scan and are still in the workspace)
    const FusedArgs fa = fused_args(in, ws);
    DxArgs da{};
    da.B = in.B; da.T = in.T; da.H = in.H; da.P = in.P; da.N = in.N; da.G = in.G; da.Q = in.Q;
    da.S = ws.S; da.dt = in.dt; da.A = in.A; da.D = in.D; da.b = fa.b; da.c = fa.c;
    da.xt = ws.xt_hi; da.dy16 = ws.dy_hi; da.hp = ws.hp_hi; da.dh = ws.dh_hi;
    da.x = in.x; da.ldx = in.ldx; da.dy = dy; da.lddy = lddy; da.dx = g.dx; da.lddx = g.lddx;
    da.dd = dsend; da.rpart = ws.rpart; da.sums = p.dxt; da.part = ws.part; da.raw = g.raw;
    PMB_TRY(ssd_dx(st, da));
  } else if (fz) {
    // dY as a bf16 pair (the B / C / x~ pairs were written by the forward of this scan and are still in the workspace)
    FusedArgs fa = fused_args(in, ws);
    fa.v = Op16{ws.dy_hi, ws.dy_lo, (int64_t)p.H * p.P};
    fa.state = Op16{ws.dh_hi, ws.dh_lo, p.P};
    fa.out = p.dxt; fa.ldo = (int64_t)p.H * p.P;
    fa.xt = Op16{ws.xt_hi, ws.xt_lo, (int64_t)p.H * p.P};
    fa.csum = ws.csum; fa.esum = ws.esum; fa.rpart = ws.rpart;
    PMB_TRY(ssd_fused(st, 1, fa));
  }
  else if (tc) {
    // (a forward that took the fused kernel left no C B^T behind: form it now)
    if (fused_enabled() && ssd_fused_supported(p.P, p.N, p.Q)) PMB_TRY(ssd_tc_cb(st, in, ws));
    PMB_TRY(ssd_tc_dx(st, in, dy, lddy, ws));
  }
  else PMB_TRY(run_op(st, "ssd_bwd_dx", make_op<OpDx>(p, p.Q, p.P), nbch, 2.0 * tok * p.H * p.P * (p.Q + p.N)));
  if (!(fz && in.plain16)) {
    ProfScope prof(st, "ssd_bwd_rows", 0.0, 4.0 * tok * p.H * (5.0 * p.P + 8.0));
    const bool vec_ok = (p.P % 4 == 0) && (p.ldx % 4 == 0) && (p.ldy % 4 == 0) && (p.lddy % 4 == 0) && (g.lddx % 4 == 0) &&
                        ((reinterpret_cast<uintptr_t>(p.x) | reinterpret_cast<uintptr_t>(p.y) | reinterpret_cast<uintptr_t>(p.dy) |
                          reinterpret_cast<uintptr_t>(g.dx) | reinterpret_cast<uintptr_t>(p.dxt)) % 16 == 0);
    if (fz) {
      WSums wsm{ws.rpart, ws.csum, ws.esum, ws.yoff, p.Q / 128};
      const int ring = 8 * 16 * ROWS_THREADS + 5 * 4 * p.Q;
      PMB_SMEM_OPT_IN(8 * 16 * ROWS_THREADS + 5 * 4 * PREP_MAX_Q, chunk_rows_finish_w_kernel);
      chunk_rows_finish_w_kernel<<<(unsigned)nbch, ROWS_THREADS, ring, st>>>(p, wsm, g.dx, g.lddx, dsend, g.da, g.ddt, ws.part, in.dt ? g.raw : SsdGrads::RawDt{});
      PMB_LAUNCHED();
    } else if (vec_ok && nbch <= 4 * 148 && p.Q <= PREP_MAX_Q) {
      chunk_rows_finish_kernel<<<(unsigned)nbch, PREP_THREADS, 0, st>>>(p, g.dx, g.lddx, dsend, g.da, g.ddt, ws.part);
      PMB_LAUNCHED();
    } else {
      ssd_rowdots_kernel<<<(unsigned)cdiv(rows * 32, 256), 256, 0, st>>>(p, g.dx, g.lddx, ddt_x, dS, dDrow);
      PMB_LAUNCHED();
      ssd_chunk_finish_kernel<<<(unsigned)cdiv((int64_t)nbch * 32, 256), 256, 0, st>>>(p, ddt_x, dS, dDrow, dsend, g.da, g.ddt, ws.part);
      PMB_LAUNCHED();
    }
  }
  auto head_sums = [&](cudaStream_t s) -> pmb_status {   // part = [dA partials (B*nc,H)] [dD partials (B*nc,H)] [d_dt_bias partials]
    if (!in.dt) return PMB_OK;
    if (fz) {
      PMB_TRY(launch_pdl(s, head_finish_kernel, dim3((unsigned)cdiv(p.H, 4)), 128, 0, ws.part, p.B * p.nc, p.H, in.A, g.dA, g.dD, g.raw.hi ? g.raw.d_dt_bias : nullptr,
                                                                  g.raw.hi ? g.raw.d_a_log : nullptr));
      return PMB_OK;
    }
    PMB_TRY(column_sum(s, ws.part, (int64_t)p.B * p.nc, p.H, g.dA));
    if (g.dD) PMB_TRY(column_sum(s, ws.part + (int64_t)p.B * p.nc * p.H, (int64_t)p.B * p.nc, p.H, g.dD));
    return PMB_OK;
  };
  // the two tiny per-head reductions ride at the end of the side chain instead of holding up the caller's stream
  if (lane && tc_group) PMB_CUDA(cudaEventRecord(lane->ev[4], st));
  else PMB_TRY(head_sums(st));
  // The three per-group contractions sum over the heads of the group; with few (batch, chunk) pairs the
  // head loop is split across CTAs and the partial tiles are summed in a fixed order afterwards.
  const int qt = (int)cdiv(p.Q, BM);
  auto reduce = [&](int nsplit, int cols, int mode, float* out, int64_t ld, int tile = BM, cudaStream_t rs = nullptr,
                    const float* part = nullptr) -> pmb_status {
    if (nsplit <= 1) return PMB_OK;
    const float* from = part ? part : ws.splitk;
    const bool vec = cols % 4 == 0 && tile % 4 == 0 && (mode == 0 || ld % 4 == 0) && aligned16(out) && aligned16(from);
    const int64_t batches = nbcg, blocks = cdiv((int64_t)p.Q * cols, vec ? 1024 : 256);
    const dim3 grid((unsigned)blocks, (unsigned)(batches < REDUCE_Y ? batches : REDUCE_Y), (unsigned)cdiv(batches, REDUCE_Y));
    (vec ? splitk_reduce_kernel<4> : splitk_reduce_kernel<1>)<<<grid, 256, 0, rs ? rs : (tc_group ? sb : st)>>>(from, nsplit, p.Q, cols, mode, p.G, p.Q, out, ld, batches, tile,
                                                                                                           (mode == 0 && fz) ? ws.dg_hi : nullptr, ws.dg_lo);
    PMB_LAUNCHED();
    return PMB_OK;
  };
  if (fz) {
    {
      ProfScope prof(sb, "ssd_bwd_dg_pair", 2.0 * tok * p.H * p.Q * p.P, 0.0);
      const int nsg = ssd_dg_nsplit(p.B, p.T, p.H, p.G, p.Q);
      PMB_TRY(ssd_dg(sb, in, ws, nsg));
      PMB_TRY(reduce(nsg, p.Q, 0, ws.dG, 0, 128));
    }
    const int ns = ssd_pairs_dbc_nsplit(p.B, p.T, p.H, p.N, p.G, p.Q);
    // dC and dB both wait for dG only: they run side by side, each with its own partial tiles
    SideLane* lane_b = nullptr;
    if (lane) PMB_TRY(side_lane(5, &lane_b));
    if (lane_b) PMB_CUDA(cudaEventRecord(lane->ev[5], sb));               // dG and its pair are ready
    {
      if (lane) PMB_CUDA(cudaStreamWaitEvent(sb, lane->ev[1], 0));       // (the forward's h_prev pair is long there)
      ProfScope prof(sb, "ssd_bwd_dc_pair", 2.0 * tok * p.N * (p.G * p.Q + (double)p.H * p.P), 0.0);
      PMB_TRY(ssd_pairs_dbc(sb, in, ws, 0, g.dc, g.lddbc, ns, ws.splitk));
      PMB_TRY(reduce(ns, p.N, 1, g.dc, g.lddbc));
    }
    {
      cudaStream_t sdb = lane_b ? lane_b->s : sb;
      float* part_b = lane_b ? ws.splitk + (size_t)ns * nbcg * p.Q * p.N : ws.splitk;
      if (lane_b) PMB_CUDA(cudaStreamWaitEvent(sdb, lane->ev[5], 0));
      if (lane) PMB_CUDA(cudaStreamWaitEvent(sdb, lane->ev[2], 0));      // dh and its pair are ready
      ProfScope prof(sdb, "ssd_bwd_db_pair", 2.0 * tok * p.N * (p.G * p.Q + (double)p.H * p.P), 0.0);
      PMB_TRY(ssd_pairs_dbc(sdb, in, ws, 1, g.db, g.lddbc, ns, part_b));
      PMB_TRY(reduce(ns, p.N, 2, g.db, g.lddbc, BM, sdb, part_b));
    }
    if (lane_b) PMB_TRY(order_after(lane_b->s, lane_b->ev[0], sb));
    if (lane) {
      PMB_CUDA(cudaStreamWaitEvent(sb, lane->ev[4], 0));
      PMB_TRY(head_sums(sb));
      PMB_TRY(order_after(sb, lane->ev[3], st));               // join
    }
    return PMB_OK;
  }
  if (tc_group) {
    {
      ProfScope prof(sb, "ssd_bwd_dg_tc", 2.0 * tok * p.H * p.Q * p.P, 0.0);
      const int nsg = ssd_tc_dg_nsplit_dims(p.B, p.T, p.H, p.G, p.Q);
      PMB_TRY(ssd_tc_dg(sb, in, dy, lddy, ws, nsg));
      PMB_TRY(reduce(nsg, p.Q, 0, ws.dG, 0, 128));
    }
    const int ns = ssd_tc_dbc_nsplit(in);
    {
      if (lane) PMB_CUDA(cudaStreamWaitEvent(sb, lane->ev[1], 0));
      ProfScope prof(sb, "ssd_bwd_dc_tc", 2.0 * tok * p.N * (p.G * p.Q + (double)p.H * p.P), 0.0);
      PMB_TRY(ssd_tc_dc(sb, in, g.dc, g.lddbc, ws, ns));
      PMB_TRY(reduce(ns, p.N, 1, g.dc, g.lddbc));
    }
    {
      if (lane) PMB_CUDA(cudaStreamWaitEvent(sb, lane->ev[2], 0));
      ProfScope prof(sb, "ssd_bwd_db_tc", 2.0 * tok * p.N * (p.G * p.Q + (double)p.H * p.P), 0.0);
      PMB_TRY(ssd_tc_db(sb, in, g.db, g.lddbc, ws, ns));
      PMB_TRY(reduce(ns, p.N, 2, g.db, g.lddbc));
    }
    if (lane) {
      PMB_CUDA(cudaStreamWaitEvent(sb, lane->ev[4], 0));
      PMB_TRY(head_sums(sb));
      PMB_TRY(order_after(sb, lane->ev[3], st));               // join
    }
    return PMB_OK;
  }
  {
    OpDG op = make_op<OpDG>(p, p.Q, p.Q);
    op.nsplit = pick_nsplit(nbcg, qt * (qt + 1) / 2, p.hpg); op.part = ws.splitk;
    ProfScope prof(st, "ssd_bwd_dg", 2.0 * tok * p.H * p.Q * p.P, 0.0);
    PMB_TRY(launch_bgemm(st, op, nbcg * op.nsplit));
    PMB_TRY(reduce(op.nsplit, p.Q, 0, ws.dG, 0));
  }
  {
    OpDC op = make_op<OpDC>(p, p.Q, p.N);
    op.nsplit = pick_nsplit(nbcg, qt * (int)cdiv(p.N, BN), p.hpg); op.part = ws.splitk;
    ProfScope prof(st, "ssd_bwd_dc", 2.0 * tok * p.N * (p.G * p.Q + (double)p.H * p.P), 0.0);
    PMB_TRY(launch_bgemm(st, op, nbcg * op.nsplit));
    PMB_TRY(reduce(op.nsplit, p.N, 1, g.dc, g.lddbc));
  }
  {
    OpDB op = make_op<OpDB>(p, p.Q, p.N);
    op.nsplit = pick_nsplit(nbcg, qt * (int)cdiv(p.N, BN), p.hpg); op.part = ws.splitk;
    ProfScope prof(st, "ssd_bwd_db", 2.0 * tok * p.N * (p.G * p.Q + (double)p.H * p.P), 0.0);
    PMB_TRY(launch_bgemm(st, op, nbcg * op.nsplit));
    PMB_TRY(reduce(op.nsplit, p.N, 2, g.db, g.lddbc));
  }
  return PMB_OK;
}

pmb_status ssd_bwd(cudaStream_t st, const SsdIn& in, const float* y, int64_t ldy, const float* dy, int64_t lddy,
                   const SsdGrads& g, const SsdWs& ws) {
  return lanes_joined(st, ssd_bwd_on_lanes(st, in, y, ldy, dy, lddy, g, ws));
}

// ---------------------------------------------------------------------------------------------
// The scan on bf16 inputs as they are (mamba2/block.rs:203-208: x, B, C in bf16, the recurrence in fp32).  x, B, C and dY go to
// the tensor cores as plain bf16 operands, a, S, the states and every accumulator stay fp32, y and the gradients leave the kernels
// as bf16.  On whole chunks of 128 or 256 tokens at d_head 64 (ssd16_plain) the operands formed on the way (masked tiles, scaled x and
// dY, states) are rounded to bf16 too; on every other shape they are (hi, lo) pairs, so that nothing but the outputs is rounded to bf16.
// Measured, forward and backward: 16 x 8192 tokens, 32 heads of 128 x 64: 7.01 ms chunk by chunk (16 launches), 3.22 ms as chains (5);
// 5 x 1474 tokens, 16 heads: 4443 us widened to fp32 for the FMA contractions, 234 us.
// ---------------------------------------------------------------------------------------------

// Whole chunks of 128 tokens at d_head 64: the callers' tensors must be 16-byte aligned.  (More than 64 chunks were never part of this:
// such sequences keep pairs of what is formed on the way, and with them da at 1.5e-6 instead of 4e-4.)
static bool ssd16_whole(int T, int P, int N, int Q) {
  return P == 64 && (N == 64 || N == 128) && Q % 128 == 0 && Q <= PREP_MAX_Q && T / Q <= SCAN_DOT_MAX_NC;
}
// Rounds what is formed on the way to bf16.  A state enters the products of every step of 128 tokens, not of every chunk, and each time
// its rounding adds to da (fp32; everything else leaves as bf16 and does not notice): with k steps to a chunk the error is up to sqrt(k) of
// what rounding once per chunk leaves, and a sequence of one chunk has no need of any.  Error of da against fp64, 8 heads of 64 x 64, rounded
// once per chunk / once per step / on pairs: 256 tokens in one chunk 2.4e-6 / 2.3e-4 / 1.5e-6; two chunks of 256 2.6e-4 / 3.7e-4 /
// 1.5e-6; four 3.2e-4 / 4.2e-4 / 1.5e-6, and 1.25 times as large on longer sequences; eight chunks of 512 2.4e-4 / 4.2e-4 / 1.5e-6.  Pairs take
// 13 to 37 % longer (2 x 512 tokens, 8 heads of 64 x 64: 64 -> 72 us; 16 x 8192, 32 heads of 128 x 64: 3.15 -> 4.31 ms).  They serve
// chunks of more than two steps and sequences of at most two chunks of two steps; the others stay within 1.4 of one rounding per chunk.
static bool ssd16_plain(int T, int P, int N, int Q) {
  return ssd16_whole(T, P, N, Q) && (Q == SCAN_STEP || (Q == 2 * SCAN_STEP && T / Q > 2));
}
bool ssd16_supported(int B, int T, int H, int P, int N, int G, int Q) {
  return ssd_chain_enabled() && ssd_chain_shape(P, N) && (int64_t)B * T < (1LL << 31) && (int64_t)B * cdiv(T, SCAN_STEP) < (1LL << 31);
}

size_t ssd16_ws_layout(int B, int T, int H, int P, int N, int G, int Q, void* base, size_t bytes, Scan16Ws* out) {
  Arena ar(base, bytes);
  Scan16Ws w{};
  const size_t hp = (size_t)B * T * H * P, gn = (size_t)B * T * G * N, np = (size_t)B * H * N * P, stn = np * cdiv(T, SCAN_STEP);
  w.whole = ssd16_whole(T, P, N, Q);
  w.plain = ssd16_plain(T, P, N, Q);
  w.S = ar.take<float>((size_t)B * T * H);
  w.x = ar.take<uint16_t>(hp);
  w.b = ar.take<uint16_t>(gn); w.c = ar.take<uint16_t>(gn);
  w.hp_hi = ar.take<uint16_t>(stn); w.dh_hi = ar.take<uint16_t>(stn);
  if (!w.plain) { w.hp_lo = ar.take<uint16_t>(stn); w.dh_lo = ar.take<uint16_t>(stn); }
  if (!w.whole) {
    w.t0 = ar.take<uint16_t>(hp); w.t1 = ar.take<uint16_t>(hp); w.g0 = ar.take<uint16_t>(gn); w.g1 = ar.take<uint16_t>(gn);
  }
  w.init = ar.take<float>(np); w.last = ar.take<float>(w.whole ? np : 0);
  w.seg = ar.take<float>(ssd_chain_seg_floats(B, T, H, P, N));
  w.part = ar.take<float>(ssd_heads_part_floats(B, T, H, N, G));
  if (out) *out = w;
  return ar.ok ? ar.used() : 0;
}

// The state after the last token, in fp32 throughout: h <- exp(S_end) h + sum_t exp(S_end - S_t) B_t x_t, step by step.  The chain kernel's
// state carries the rounding of its scaled x to a pair (2e-6 of its norm from fp64); shapes off the whole chunks, whose inputs were widened
// to fp32 before, keep 5e-8 to 6e-7 this way.  A CTA owns 32 rows of one (batch, head)'s state, 4 x 4 of them per thread, and takes 32 tokens
// at a time through shared memory, the next 32 on their way.  Bound by its multiply-adds (about half of their rate); it runs where the caller
// asks for the state.  Measured at 5 x 1474 tokens, 16 heads of 64 x 64: 67 us next to 61 for the rest of the call (1220 when all of it
// ran on FMA); at 2 x 100, 32 heads of 128 x 64: 10 next to 15.
constexpr int FS_TOK = 32, FS_ROWS = 32, FS_THREADS = 128;
__global__ void __launch_bounds__(FS_THREADS) scan16_final_state_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ b, const float* __restrict__ S,
                                                                        const float* __restrict__ init, float* __restrict__ last, int T, int H, int G, int P, int N) {
  __shared__ __align__(16) float sb[FS_TOK][FS_ROWS], sx[FS_TOK][64];
  const int bh = blockIdx.x, bb = bh / H, h = bh % H, g = h / (H / G), n0 = blockIdx.y * FS_ROWS;
  const int tp = 4 * (threadIdx.x & 15), tn = 4 * (threadIdx.x >> 4);
  const bool mine = n0 + tn < N && tp < P;                 // (N and P are multiples of 8)
  const float* Sr = S + (int64_t)bh * T;
  const int64_t at = ((int64_t)bh * N + n0 + tn) * P + tp;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = mine && init ? init[at + (int64_t)i * P + j] : 0.0f;
  // what a thread brings of each tile: eight n of one token of B, eight p of two tokens of x (16-byte pieces; rows start on such)
  const int bk = threadIdx.x >> 2, bn = 8 * (threadIdx.x & 3), xk = threadIdx.x >> 3, xp = 8 * (threadIdx.x & 7);
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  uint4 bq = zero, xq[2] = {zero, zero};
  float sq[2] = {0.0f, 0.0f};
  auto request = [&](int tt) {
    bq = tt + bk < T && n0 + bn < N ? *reinterpret_cast<const uint4*>(b + (((int64_t)bb * T + tt + bk) * G + g) * N + n0 + bn) : zero;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int t = tt + xk + 16 * u;
      xq[u] = t < T && xp < P ? *reinterpret_cast<const uint4*>(x + (((int64_t)bb * T + t) * H + h) * P + xp) : zero;
      sq[u] = Sr[t < T ? t : T - 1];
    }
  };
  auto put = [&](float* dst, const uint4& q, float f) {
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int e = 0; e < 2; ++e)
      *reinterpret_cast<float4*>(dst + 4 * e) = make_float4(f * __uint_as_float(w[2 * e] << 16), f * __uint_as_float(w[2 * e] & 0xffff0000u),
                                                            f * __uint_as_float(w[2 * e + 1] << 16), f * __uint_as_float(w[2 * e + 1] & 0xffff0000u));
  };
  request(0);
  for (int t0 = 0; t0 < T; t0 += SCAN_STEP) {
    const int t1 = min(t0 + SCAN_STEP, T);
    const float send = Sr[t1 - 1], dec = expf(send);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] *= dec;
    for (int tt = t0; tt < t1; tt += FS_TOK) {
      __syncthreads();
      put(&sb[bk][bn], bq, 1.0f);
#pragma unroll
      for (int u = 0; u < 2; ++u) put(&sx[xk + 16 * u][xp], xq[u], expf(send - sq[u]));      // (zeros past the end: the factor is 1 there)
      __syncthreads();
      request(tt + FS_TOK);                                // (lands under the products)
#pragma unroll 8
      for (int k = 0; k < FS_TOK; ++k) {
        const float4 bv = *reinterpret_cast<const float4*>(&sb[k][tn]), xv = *reinterpret_cast<const float4*>(&sx[k][tp]);
        const float br[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          acc[i][0] = fmaf(br[i], xv.x, acc[i][0]); acc[i][1] = fmaf(br[i], xv.y, acc[i][1]);
          acc[i][2] = fmaf(br[i], xv.z, acc[i][2]); acc[i][3] = fmaf(br[i], xv.w, acc[i][3]);
        }
      }
    }
  }
  if (mine) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) last[at + (int64_t)i * P + j] = acc[i][j];
  }
}

static pmb_status copy16(cudaStream_t st, void* dst, const void* src, size_t bytes) {
  PMB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, st));
  return PMB_OK;
}

pmb_status ssd16_fwd(cudaStream_t st, int B, int T, int H, int P, int N, int G, const uint16_t* x, const float* a,
                     const uint16_t* b, const uint16_t* c, const float* init_state, uint16_t* y, float* final_state, const Scan16Ws& ws) {
  const size_t hp = (size_t)B * T * H * P * 2, gn = (size_t)B * T * G * N * 2, np = (size_t)B * H * N * P * 4;
  {
    // (the backward is not handed the inputs again: B and C are copied here, x by the kernel)
    ProfScope prof(st, "ssd16_keep_bc", 0.0, 4.0 * gn);
    PMB_TRY(copy16(st, ws.b, b, gn));
    PMB_TRY(copy16(st, ws.c, c, gn));
  }
  ChainArgs k{};
  k.B = B; k.T = T; k.H = H; k.P = P; k.N = N; k.G = G; k.exact = !ws.plain;
  k.b = Op16{ws.b, nullptr, (int64_t)G * N}; k.c = Op16{ws.c, nullptr, (int64_t)G * N};
  k.x16 = x; k.x_keep = ws.x; k.ldx = k.ldy = (int64_t)H * P; k.a = a;
  if (!aligned16(x)) { PMB_TRY(copy16(st, ws.x, x, hp)); k.x16 = ws.x; k.x_keep = nullptr; }
  k.init = init_state;
  if (init_state && !aligned16(init_state)) { PMB_TRY(copy16(st, ws.init, init_state, np)); k.init = ws.init; }
  k.y16 = aligned16(y) ? y : ws.t0;
  k.last = !ws.whole ? nullptr : final_state && !aligned16(final_state) ? ws.last : final_state;
  k.S_out = ws.S; k.hp_hi = ws.hp_hi; k.hp_lo = ws.hp_lo; k.seg = ws.seg;
  PMB_TRY(ssd_chain_fwd(st, k));
  if (k.y16 != y) PMB_TRY(copy16(st, y, k.y16, hp));
  if (final_state && !ws.whole) {
    ProfScope prof(st, "ssd16_final_state", 2.0 * B * T * H * N * P, 0.0);
    scan16_final_state_kernel<<<dim3((unsigned)(B * H), (unsigned)cdiv(N, FS_ROWS)), FS_THREADS, 0, st>>>(ws.x, ws.b, ws.S, init_state, final_state, T, H, G, P, N);
    PMB_LAUNCHED();
  } else if (k.last != final_state) PMB_TRY(copy16(st, final_state, k.last, np));
  return PMB_OK;
}

pmb_status ssd16_bwd(cudaStream_t st, int B, int T, int H, int P, int N, int G, const uint16_t* dy, uint16_t* dx, float* da, uint16_t* db,
                     uint16_t* dc, const Scan16Ws& ws) {
  const size_t hp = (size_t)B * T * H * P * 2, gn = (size_t)B * T * G * N * 2;
  const int64_t ldp = (int64_t)H * P, ldn = (int64_t)G * N;
  if (!aligned16(dy)) { PMB_TRY(copy16(st, ws.t0, dy, hp)); dy = ws.t0; }
  ChainBwdArgs k{};
  k.B = B; k.T = T; k.H = H; k.P = P; k.N = N; k.G = G;
  k.b = Op16{ws.b, nullptr, ldn}; k.c = Op16{ws.c, nullptr, ldn};
  k.hp_hi = ws.hp_hi; k.hp_lo = ws.hp_lo; k.S = ws.S; k.x16 = ws.x; k.dy16 = dy; k.ldx = k.lddy = k.lddx = ldp;
  k.dx16 = aligned16(dx) ? dx : ws.t1; k.dh_hi = ws.dh_hi; k.dh_lo = ws.dh_lo; k.da = da; k.seg = ws.seg;
  PMB_TRY(ssd_chain_bwd(st, k));
  if (k.dx16 != dx) PMB_TRY(copy16(st, dx, k.dx16, hp));
  HeadsArgs h{};
  h.B = B; h.T = T; h.H = H; h.P = P; h.N = N; h.G = G; h.b = k.b; h.c = k.c; h.dy = Op16{dy, nullptr, ldp}; h.xt = Op16{ws.x, nullptr, ldp};
  h.hp_hi = ws.hp_hi; h.hp_lo = ws.hp_lo; h.dh_hi = ws.dh_hi; h.dh_lo = ws.dh_lo; h.S = ws.S; h.ld = ldn; h.part = ws.part;
  h.dc16 = aligned16(dc) ? dc : ws.g0; h.db16 = aligned16(db) ? db : ws.g1;
  PMB_TRY(ssd_heads(st, h));
  if (h.dc16 != dc) PMB_TRY(copy16(st, dc, h.dc16, gn));
  if (h.db16 != db) PMB_TRY(copy16(st, db, h.db16, gn));
  return PMB_OK;
}

}  // namespace pmb

// HBM-bound kernels of the Mamba2 block: causal depthwise conv1d + bias + SiLU, dt softplus,
// gated RMSNorm, their backward passes, and small deterministic reductions.
#include "common.cuh"
#include "kernels.h"

namespace pmb {

constexpr int COLSUM_LANES = 32;
__global__ void column_sum_kernel(const float* __restrict__ partial, int64_t rows, int cols, float* __restrict__ out, const float* __restrict__ more, int more_cols, float* __restrict__ more_out);
static unsigned column_blocks(int cols) { return (unsigned)cdiv(cols, 32); }

// ---------------------------------------------------------------------------------------------
// conv1d (causal, depthwise) + bias + SiLU.   u[t,c] = b[c] + sum_k w[c,k] * xbc[t-(K-1)+k, c]
// Layout stays (B,T,channels): a thread owns VEC adjacent channels and walks a run of time steps with the K-1 previous inputs in
// registers and the next CONV_AHEAD rows on their way, so that every global access is a coalesced vector access and each input
// row is read (run+K-1)/run times.  Bound by HBM.  A CTA of the vector kernels is 16 runs of 8 channel quads (128-byte strips of
// its rows): no thread is idle for any channel count that is a multiple of 32.
// Measured at 8 x 2048 tokens of 1664 channels: forward 68 us with runs of 8 all requested up front, 49 with the next four rows in registers,
// 43 now: they wait in shared memory (cp.async), which leaves room for more CTAs (eight rows and pairs of channels no better); at 8 x 1024 22;
// backward (plain bf16 result) 131 us, 110 with four channels per thread and the next four rows in registers (170 of them, three CTAs per SM), 82 with
// two channels and the next eight rows in shared memory, 60 now: that one was bound by issue (87 warp instructions per element in 79 % of the
// issue slots), so four channels go as two pairs of packed fp32 operations, with the next four rows in shared memory (128 registers); its bytes
// alone take 42.  At 8 x 1024 36, at 4 x 512 with a (hi, lo) result 19 and 15, at 2 x 128 of 544 channels 6 either way.  Sigmoids stay
// scalar: an exponential of pairs was faster but 12 % further from fp64, and its flipped roundings grew through 24 layers of bf16 storage until a
// step's gradients had moved by more than 2e-2 of their norm.
// ---------------------------------------------------------------------------------------------
constexpr int CONV_AHEAD = 4;
constexpr int CONV_SLICES = 16;
constexpr int CONV_STRIP_THREADS = CONV_SLICES * 8;

// Steps per run: 32 where that still gives eight CTAs per SM (the halo of K - 1 rows is then a tenth), else 16 or 8.
static int conv_run(const Dims& d) {
  for (int run = 32; run > 8; run >>= 1)
    if (cdiv(d.X, 32) * d.B * cdiv(d.T, CONV_SLICES * run) >= 148 * 8) return run;
  return 8;
}

// weights and bias of channels [c, c + 4), as two pairs
template <int K>
__device__ __forceinline__ void conv_weights(const float* __restrict__ w, const float* __restrict__ bias, int c, F2 (&wr)[2][K], F2 (&br)[2]) {
#pragma unroll
  for (int v = 0; v < 2; ++v) {
    br[v] = bias ? pack2(bias[c + 2 * v], bias[c + 2 * v + 1]) : 0;
#pragma unroll
    for (int k = 0; k < K; ++k) wr[v][k] = pack2(w[(c + 2 * v) * K + k], w[(c + 2 * v + 1) * K + k]);
  }
}

template <int VEC>
__device__ __forceinline__ void conv_load(const float* p, float (&o)[VEC]) {
  if (VEC == 4) { const float4 q = *reinterpret_cast<const float4*>(p); o[0] = q.x; o[1 % VEC] = q.y; o[2 % VEC] = q.z; o[3 % VEC] = q.w; }
  else o[0] = *p;
}

// channels [c, c + VEC) of batch b, time steps [t0, t1)
template <int K, int VEC>
__device__ __forceinline__ void conv_fwd_thread(const float* __restrict__ xzd, int64_t ldx, int col0, const float* __restrict__ w,
                                                const float* __restrict__ bias, float* __restrict__ act, int X, int T,
                                                const ConvPairOut& po, int c, int b, int t0, int t1, uint32_t slots = 0) {
  float wr[VEC][K], br[VEC], win[VEC][K];
#pragma unroll
  for (int v = 0; v < VEC; ++v) {
    br[v] = bias ? bias[c + v] : 0.0f;
#pragma unroll
    for (int k = 0; k < K; ++k) wr[v][k] = w[(c + v) * K + k];
  }
  const float* src = xzd + (int64_t)b * T * ldx + col0 + c;
#pragma unroll
  for (int k = 0; k < K - 1; ++k) {
    const int t = t0 - (K - 1) + k;
    float o[VEC];
#pragma unroll
    for (int v = 0; v < VEC; ++v) o[v] = 0.0f;
    if (t >= 0) conv_load<VEC>(src + (int64_t)t * ldx, o);
#pragma unroll
    for (int v = 0; v < VEC; ++v) win[v][k] = o[v];
  }
  // four channels: the next rows wait in slots of the thread's own in shared memory (cp.async, no barrier) and not in registers
  constexpr bool STAGED = VEC == 4;
  constexpr uint32_t PITCH = CONV_STRIP_THREADS * 16;
  float ring[STAGED ? 1 : CONV_AHEAD][VEC];
  uint32_t slot = slots;
  const float* nx = src + (int64_t)t0 * ldx;                  // the next row to request
  auto request = [&](int t, int q) {
    if (STAGED) {
      if (t < t1) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(slot), "l"(nx) : "memory");
      asm volatile("cp.async.commit_group;" ::: "memory");
      slot = slot + PITCH == slots + CONV_AHEAD * PITCH ? slots : slot + PITCH;
    } else if (t < t1) conv_load<VEC>(nx, ring[q]);
    nx += ldx;
  };
#pragma unroll
  for (int q = 0; q < CONV_AHEAD; ++q) request(t0 + q, q);
  float* dst = act + ((int64_t)b * T + t0) * X + c;
  int64_t o16 = ((int64_t)b * T + t0) * po.width + (c - po.col0);
  const bool pair = VEC == 4 && po.hi && c >= po.col0;        // the B | C columns also go out as a bf16 pair (operands of the scan)
  for (int tb = t0; tb < t1; tb += CONV_AHEAD) {
#pragma unroll
    for (int q = 0; q < CONV_AHEAD; ++q) {
      const int t = tb + q;
      if (t >= t1) break;
      float o[VEC];
      if (STAGED) {                                          // (the slot that is due is the one to request into)
        asm volatile("cp.async.wait_group %0;" ::"n"(CONV_AHEAD - 1) : "memory");
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(o[0]), "=f"(o[1 % VEC]), "=f"(o[2 % VEC]), "=f"(o[3 % VEC]) : "r"(slot) : "memory");
      }
#pragma unroll
      for (int v = 0; v < VEC; ++v) win[v][K - 1] = STAGED ? o[v] : ring[STAGED ? 0 : q][v];
      request(t + CONV_AHEAD, q);
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        float u = br[v];
#pragma unroll
        for (int k = 0; k < K; ++k) u = fmaf(wr[v][k], win[v][k], u);
        o[v] = u * sigmoid_acc(u);
#pragma unroll
        for (int k = 0; k < K - 1; ++k) win[v][k] = win[v][k + 1];
      }
      if (VEC == 4) *reinterpret_cast<float4*>(dst) = make_float4(o[0], o[1 % VEC], o[2 % VEC], o[3 % VEC]);
      else *dst = o[0];
      if (pair) store_pair4(po.hi + o16, po.lo ? po.lo + o16 : nullptr, o[0], o[1 % VEC], o[2 % VEC], o[3 % VEC]);
      dst += X; o16 += po.width;
    }
  }
}

template <int K>
__global__ void __launch_bounds__(CONV_STRIP_THREADS) conv_silu_fwd_strip_kernel(const float* __restrict__ xzd, int64_t ldx, int col0,
                                                                                 const float* __restrict__ w, const float* __restrict__ bias,
                                                                                 float* __restrict__ act, int X, int T, int run, ConvPairOut po) {
  pdl_launch();
  pdl_wait();
  __shared__ __align__(16) float4 rows[CONV_AHEAD][CONV_STRIP_THREADS];
  if (po.clear && blockIdx.x == 0 && blockIdx.y == 0)
    for (int i = threadIdx.x; i < CONV_CLEAR_WORDS; i += CONV_STRIP_THREADS) po.clear[i] = 0;
  const int c = (blockIdx.x * 8 + (threadIdx.x & 7)) * 4;
  const int tblocks = (T + CONV_SLICES * run - 1) / (CONV_SLICES * run);
  const int b = blockIdx.y / tblocks, t0 = (blockIdx.y % tblocks) * (CONV_SLICES * run) + (threadIdx.x >> 3) * run;
  if (c < X && t0 < T)
    conv_fwd_thread<K, 4>(xzd, ldx, col0, w, bias, act, X, T, po, c, b, t0, min(t0 + run, T), (uint32_t)__cvta_generic_to_shared(&rows[0][threadIdx.x]));
}
// any channel count and alignment
template <int K>
__global__ void __launch_bounds__(128) conv_silu_fwd_kernel(const float* __restrict__ xzd, int64_t ldx, int col0, const float* __restrict__ w,
                                                            const float* __restrict__ bias, float* __restrict__ act, int X, int T, int run) {
  pdl_launch();
  pdl_wait();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int tblocks = (T + run - 1) / run;
  const int b = blockIdx.y / tblocks, t0 = (blockIdx.y % tblocks) * run;
  if (c < X) conv_fwd_thread<K, 1>(xzd, ldx, col0, w, bias, act, X, T, ConvPairOut{}, c, b, t0, min(t0 + run, T));
}

__global__ void dt_softplus_kernel(const float* __restrict__ xzd, int64_t ldx, int col0, const float* __restrict__ dt_bias,
                                   float* __restrict__ dt, int64_t rows, int H) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * H) return;
  int64_t r = i / H;
  int h = (int)(i % H);
  dt[i] = softplus_acc(xzd[r * ldx + col0 + h] + dt_bias[h]);
}

template <int K>
static pmb_status launch_conv_fwd_k(cudaStream_t st, const Dims& d, const float* xzd, const float* w, const float* b, float* act,
                                    ConvPairOut* pair) {
  const int run = conv_run(d);
  bool vec = (d.X % 4 == 0) && (d.J % 4 == 0) && (d.I % 4 == 0) && ((reinterpret_cast<uintptr_t>(xzd) | reinterpret_cast<uintptr_t>(act)) % 16 == 0);
  ConvPairOut po{};
  if (pair) {
    if (vec && pair->hi && ((reinterpret_cast<uintptr_t>(pair->hi) | reinterpret_cast<uintptr_t>(pair->lo)) % 8 == 0) && pair->width % 4 == 0) po = *pair;
    else pair->hi = nullptr;       // tells the caller that the pair was not written
  }
  if (vec) {
    dim3 grid((unsigned)cdiv(d.X, 32), (unsigned)(d.B * cdiv(d.T, CONV_SLICES * run)));
    PMB_TRY(launch_pdl(st, conv_silu_fwd_strip_kernel<K>, grid, CONV_STRIP_THREADS, 0, xzd, d.J, d.I, w, b, act, d.X, d.T, run, po));
  } else {
    dim3 grid((unsigned)cdiv(d.X, 128), (unsigned)(d.B * cdiv(d.T, run)));
    PMB_TRY(launch_pdl(st, conv_silu_fwd_kernel<K>, grid, 128, 0, xzd, d.J, d.I, w, b, act, d.X, d.T, run));
  }
  return PMB_OK;
}

pmb_status conv_silu_dt_fwd(cudaStream_t st, const Dims& d, const float* xzd, const float* w, const float* b,
                            const float* dt_bias, float* act, float* dt, ConvPairOut* pair) {
  ProfScope prof(st, "conv_silu_dt_fwd", 0.0, 4.0 * d.M * (2.0 * d.X + 2.0 * d.H));
  switch (d.K) {
    case 2: PMB_TRY(launch_conv_fwd_k<2>(st, d, xzd, w, b, act, pair)); break;
    case 3: PMB_TRY(launch_conv_fwd_k<3>(st, d, xzd, w, b, act, pair)); break;
    case 4: PMB_TRY(launch_conv_fwd_k<4>(st, d, xzd, w, b, act, pair)); break;
    case 5: PMB_TRY(launch_conv_fwd_k<5>(st, d, xzd, w, b, act, pair)); break;
    case 6: PMB_TRY(launch_conv_fwd_k<6>(st, d, xzd, w, b, act, pair)); break;
    case 7: PMB_TRY(launch_conv_fwd_k<7>(st, d, xzd, w, b, act, pair)); break;
    case 8: PMB_TRY(launch_conv_fwd_k<8>(st, d, xzd, w, b, act, pair)); break;
    default: return fail(PMB_ERR_SHAPE, "d_conv %d unsupported", d.K);
  }
  if (dt) {
    int64_t n = d.M * d.H;
    dt_softplus_kernel<<<(unsigned)cdiv(n, 256), 256, 0, st>>>(xzd, d.J, d.I + d.X, dt_bias, dt, d.M, d.H);
    PMB_LAUNCHED();
  }
  return PMB_OK;
}

// ---------------------------------------------------------------------------------------------
// conv backward.  du = dact * silu'(u) with u recomputed from the pre-conv window;
// dxbc[t',c] = sum_k w[c,k] du[t'+(K-1)-k, c];  dw[c,k] = sum_{b,t} du[t,c] xbc[t-(K-1)+k,c];  db = sum du.
// Partial dw/db go to `partial` (rows = gridDim.y, K+1 values per channel) and are summed by column_sum_kernel (fixed order).
// ---------------------------------------------------------------------------------------------
// The work of one thread: channels [c, c + VEC) of batch b, time steps [t0, t1); writes its rows of the data gradient
// and leaves its share of the parameter gradients in dwacc / dbacc.
template <int K, int VEC>
__device__ __forceinline__ void conv_bwd_thread(const float* __restrict__ xzd, int64_t ldx, int col0, const float* __restrict__ w,
                                                const float* __restrict__ bias, const float* __restrict__ dact,
                                                float* __restrict__ dxzd, int X, int T, uint16_t* __restrict__ pair_hi,
                                                uint16_t* __restrict__ pair_lo, int c, int b, int t0, int t1,
                                                float (&dwacc)[VEC][K], float (&dbacc)[VEC]) {
  float wr[VEC][K], br[VEC];
#pragma unroll
  for (int v = 0; v < VEC; ++v) {
    br[v] = bias ? bias[c + v] : 0.0f;
#pragma unroll
    for (int k = 0; k < K; ++k) wr[v][k] = w[(c + v) * K + k];
  }
  const float* src = xzd + (int64_t)b * T * ldx + col0 + c;
  // xin holds xbc[t-(K-1) .. t]; dus holds du[t-(K-1) .. t] for the current t.
  float xin[VEC][K], dus[VEC][K];
#pragma unroll
  for (int v = 0; v < VEC; ++v) {
    dbacc[v] = 0.0f;
#pragma unroll
    for (int k = 0; k < K; ++k) { dwacc[v][k] = 0.0f; dus[v][k] = 0.0f; xin[v][k] = 0.0f; }
  }
#pragma unroll
  for (int k = 0; k < K - 1; ++k) {
    int t = t0 - (K - 1) + k;
    float o[VEC];
#pragma unroll
    for (int v = 0; v < VEC; ++v) o[v] = 0.0f;
    if (t >= 0) conv_load<VEC>(src + (int64_t)t * ldx, o);
#pragma unroll
    for (int v = 0; v < VEC; ++v) xin[v][k + 1] = o[v];
  }
  // Walk t from t0 to t1-1+(K-1): du[t] is needed by dxbc[t-(K-1) .. t]; du beyond the sequence end is 0.
  const int tend = t1 + K - 1;
  const int tl = min(tend, T);                                 // rows that exist
  float xr[CONV_AHEAD][VEC], dr[CONV_AHEAD][VEC];
  const float* nx = src + (int64_t)t0 * ldx;
  const float* nd = dact + ((int64_t)b * T + t0) * X + c;
  auto request = [&](int t, int q) {
    if (t < tl) { conv_load<VEC>(nx, xr[q]); conv_load<VEC>(nd, dr[q]); }
    nx += ldx; nd += X;
  };
#pragma unroll
  for (int q = 0; q < CONV_AHEAD; ++q) request(t0 + q, q);
  int64_t off = ((int64_t)b * T + t0 - (K - 1)) * ldx + col0 + c;      // of row t - (K - 1)
  for (int tb = t0; tb < tend; tb += CONV_AHEAD) {
#pragma unroll
    for (int q = 0; q < CONV_AHEAD; ++q) {
      const int t = tb + q;
      if (t >= tend) break;
      float xn[VEC], dn[VEC], g[VEC];
#pragma unroll
      for (int v = 0; v < VEC; ++v) { xn[v] = xr[q][v]; dn[v] = dr[q][v]; }
      request(t + CONV_AHEAD, q);
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
#pragma unroll
        for (int k = 0; k < K - 1; ++k) { xin[v][k] = xin[v][k + 1]; dus[v][k] = dus[v][k + 1]; }
        float du = 0.0f;
        if (t < T) {
          xin[v][K - 1] = xn[v];
          float u = br[v];
#pragma unroll
          for (int k = 0; k < K; ++k) u = fmaf(wr[v][k], xin[v][k], u);
          float s = sigmoid_acc(u);
          du = dn[v] * (s + u * s * (1.0f - s));
          if (t < t1) {  // this run owns the parameter-gradient contribution of t in [t0,t1)
            dbacc[v] += du;
#pragma unroll
            for (int k = 0; k < K; ++k) dwacc[v][k] = fmaf(du, xin[v][k], dwacc[v][k]);
          }
        }
        dus[v][K - 1] = du;
        float acc = 0.0f;   // dxbc[tp] = sum_k w[k] * du[tp + (K-1) - k] = sum_k w[k] * dus[K-1-k]
#pragma unroll
        for (int k = 0; k < K; ++k) acc = fmaf(wr[v][k], dus[v][K - 1 - k], acc);
        g[v] = acc;
      }
      if (t - (K - 1) >= t0) {
        if (pair_hi) {       // the gradient is only a GEMM operand: write it as a (hi, lo) bf16 pair with the same pitch
          if (VEC == 4) store_pair4(pair_hi + off, pair_lo ? pair_lo + off : nullptr, g[0], g[1 % VEC], g[2 % VEC], g[3 % VEC]);
          else { uint32_t h, l; split_bf16_pair(g[0], h, l); pair_hi[off] = (uint16_t)h; if (pair_lo) pair_lo[off] = (uint16_t)l; }
        } else if (VEC == 4) *reinterpret_cast<float4*>(dxzd + off) = make_float4(g[0], g[1 % VEC], g[2 % VEC], g[3 % VEC]);
        else dxzd[off] = g[0];
      }
      off += ldx;
    }
  }
}

// partial = [gridDim.y rows of X*K weight partials][gridDim.y rows of X bias partials]
// One thread = VEC channels and a run of time steps, its own partial row (any shape, any alignment).
template <int K, int VEC>
__global__ void __launch_bounds__(128) conv_silu_bwd_kernel(const float* __restrict__ xzd, int64_t ldx, int col0,
                                                            const float* __restrict__ w, const float* __restrict__ bias,
                                                            const float* __restrict__ dact, float* __restrict__ dxzd,
                                                            float* __restrict__ partial, int X, int T, int run,
                                                            uint16_t* __restrict__ pair_hi, uint16_t* __restrict__ pair_lo) {
  pdl_launch();
  pdl_wait();
  int c = (blockIdx.x * blockDim.x + threadIdx.x) * VEC;
  if (c >= X) return;
  int tblocks = (T + run - 1) / run;
  int b = blockIdx.y / tblocks;
  int t0 = (blockIdx.y % tblocks) * run;
  float dwacc[VEC][K], dbacc[VEC];
  conv_bwd_thread<K, VEC>(xzd, ldx, col0, w, bias, dact, dxzd, X, T, pair_hi, pair_lo, c, b, t0, min(t0 + run, T), dwacc, dbacc);
  float* prow = partial + (int64_t)blockIdx.y * X * K;
  float* pbias = partial + (int64_t)gridDim.y * X * K + (int64_t)blockIdx.y * X;
#pragma unroll
  for (int v = 0; v < VEC; ++v) {
#pragma unroll
    for (int k = 0; k < K; ++k) prow[(int64_t)(c + v) * K + k] = dwacc[v][k];
    pbias[c + v] = dbacc[v];
  }
}

// The same work on four channels as two pairs, up to four taps, with the parameter-gradient partials summed inside the CTA: one partial row
// entry per channel and CTA instead of one per thread, which at a few thousand tokens moved more partial sums than data.  Sums run in a
// fixed order (shuffles, then the warps in order).
template <int K>
__global__ void __launch_bounds__(CONV_STRIP_THREADS, 4) conv_silu_bwd_strip_kernel(const float* __restrict__ xzd, int64_t ldx, int col0,
                                                                  const float* __restrict__ w, const float* __restrict__ bias,
                                                                  const float* __restrict__ dact, float* __restrict__ dxzd,
                                                                  float* __restrict__ partial, int X, int T, int run,
                                                                  uint16_t* __restrict__ pair_hi, uint16_t* __restrict__ pair_lo) {
  pdl_launch();
  pdl_wait();
  constexpr int NV = 4 * K + 4, NW = CONV_STRIP_THREADS / 32;
  __shared__ float red[NW][8][NV];
  __shared__ __align__(16) float4 stage[CONV_AHEAD][2][CONV_STRIP_THREADS];
  const int tx = threadIdx.x & 7, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = (blockIdx.x * 8 + tx) * 4;
  const int tblocks = (T + CONV_SLICES * run - 1) / (CONV_SLICES * run);
  const int b = blockIdx.y / tblocks;
  const int t0 = (blockIdx.y % tblocks) * (CONV_SLICES * run) + (threadIdx.x >> 3) * run;
  F2 dwacc[2][K], dbacc[2] = {0, 0};
#pragma unroll
  for (int k = 0; k < K; ++k) dwacc[0][k] = dwacc[1][k] = 0;
  if (c < X && t0 < T) {
    const int t1 = min(t0 + run, T), tend = t1 + K - 1, tl = min(tend, T);      // rows [t0, tl) are read: du[t] is needed by dxbc[t-(K-1) .. t]
    F2 wr[2][K], br[2], xin[2][K], dus[2][K];                // xbc and du of [t-(K-1), t]
    conv_weights<K>(w, bias, c, wr, br);
    const float* src = xzd + (int64_t)b * T * ldx + col0 + c;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int t = t0 - K + k;
      const Quad v = k > 0 && t >= 0 ? load_quad(src + (int64_t)t * ldx) : Quad{0, 0};
      xin[0][k] = v.a; xin[1][k] = v.b;
      dus[0][k] = dus[1][k] = 0;
    }
    // the next rows wait in slots of the thread's own in shared memory (cp.async, no barrier) and not in registers
    constexpr uint32_t HALF = CONV_STRIP_THREADS * 16, PITCH = 2 * HALF;
    const uint32_t slots = (uint32_t)__cvta_generic_to_shared(&stage[0][0][threadIdx.x]);
    const float *nx = src + (int64_t)t0 * ldx, *nd = dact + ((int64_t)b * T + t0) * X + c;
    auto request = [&](int t, uint32_t slot) {
      if (t < tl) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(slot), "l"(nx) : "memory");
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(slot + HALF), "l"(nd) : "memory");
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      nx += ldx; nd += X;
    };
#pragma unroll
    for (int q = 0; q < CONV_AHEAD; ++q) request(t0 + q, slots + q * PITCH);
    int64_t off = ((int64_t)b * T + t0 - (K - 1)) * ldx + col0 + c;      // of row t - (K - 1)
    const F2 one = pack2(1.0f, 1.0f), neg = pack2(-1.0f, -1.0f);
    for (int tb = t0; tb < tend; tb += CONV_AHEAD) {
#pragma unroll
      for (int q = 0; q < CONV_AHEAD; ++q) {
        const int t = tb + q;
        if (t >= tend) break;
        const uint32_t slot = slots + q * PITCH;              // (the slot that is due is the one to request into)
        F2 xn[2], dn[2];
        asm volatile("cp.async.wait_group %0;" ::"n"(CONV_AHEAD - 1) : "memory");
        asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(xn[0]), "=l"(xn[1]) : "r"(slot) : "memory");
        asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(dn[0]), "=l"(dn[1]) : "r"(slot + HALF) : "memory");
        request(t + CONV_AHEAD, slot);
        Quad g;
        F2* const gv[2] = {&g.a, &g.b};
#pragma unroll
        for (int v = 0; v < 2; ++v) {
#pragma unroll
          for (int k = 0; k < K - 1; ++k) { xin[v][k] = xin[v][k + 1]; dus[v][k] = dus[v][k + 1]; }
          xin[v][K - 1] = xn[v];
          F2 u = br[v];
#pragma unroll
          for (int k = 0; k < K; ++k) u = fma2(wr[v][k], xin[v][k], u);
          const float2 uv = unpack2(u);
          const F2 s = pack2(sigmoid_acc(uv.x), sigmoid_acc(uv.y));
          F2 du = mul2(dn[v], fma2(mul2(u, s), fma2(s, neg, one), s));      // silu'(u) = s + u s (1 - s)
          if (t >= T) du = 0;                                 // (rows past the end: what lies in the slot is an older row)
          if (t < t1) {                                       // this run owns the parameter gradients' share of its own rows
            dbacc[v] = add2(dbacc[v], du);
#pragma unroll
            for (int k = 0; k < K; ++k) dwacc[v][k] = fma2(du, xin[v][k], dwacc[v][k]);
          }
          dus[v][K - 1] = du;
          F2 acc = 0;                                         // dxbc[tp] = sum_k w[k] du[tp + (K-1) - k]
#pragma unroll
          for (int k = 0; k < K; ++k) acc = fma2(wr[v][k], dus[v][K - 1 - k], acc);
          *gv[v] = acc;
        }
        if (t - (K - 1) >= t0) {
          if (pair_hi) store_pair4(pair_hi + off, pair_lo ? pair_lo + off : nullptr, g);      // the gradient is only a GEMM operand
          else store_quad(dxzd + off, g);
        }
        off += ldx;
      }
    }
  }
  float vals[NV];                                             // [channel][tap], [channel]
#pragma unroll
  for (int v = 0; v < 2; ++v) {
#pragma unroll
    for (int k = 0; k < K; ++k) { const float2 d = unpack2(dwacc[v][k]); vals[2 * v * K + k] = d.x; vals[(2 * v + 1) * K + k] = d.y; }
    const float2 d = unpack2(dbacc[v]);
    vals[4 * K + 2 * v] = d.x; vals[4 * K + 2 * v + 1] = d.y;
  }
#pragma unroll
  for (int i = 0; i < NV; ++i) {                              // the four time slices of a warp
    vals[i] += __shfl_xor_sync(0xffffffffu, vals[i], 16);
    vals[i] += __shfl_xor_sync(0xffffffffu, vals[i], 8);
  }
  if (lane < 8) {
#pragma unroll
    for (int i = 0; i < NV; ++i) red[warp][tx][i] = vals[i];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 8 * NV; e += CONV_STRIP_THREADS) {
    const int q = e / NV, i = e % NV;
    const int cc = (blockIdx.x * 8 + q) * 4;
    if (cc < X) {
      float tot = 0.0f;
#pragma unroll
      for (int wv = 0; wv < NW; ++wv) tot += red[wv][q][i];
      if (i < 4 * K) partial[(int64_t)blockIdx.y * X * K + (int64_t)cc * K + i] = tot;      // (cc + channel) * K + tap
      else partial[(int64_t)gridDim.y * X * K + (int64_t)blockIdx.y * X + cc + (i - 4 * K)] = tot;
    }
  }
}

size_t conv_bwd_ws_bytes(const Dims& d) {
  return align_up((size_t)d.B * cdiv(d.T, conv_run(d)) * d.X * (d.K + 1) * sizeof(float), 256);
}

// Rows of `partial` the launch below writes (what column_sum has to add up).
static int64_t conv_bwd_partial_rows(const Dims& d, bool strip) {
  return (int64_t)d.B * cdiv(d.T, (strip ? CONV_SLICES : 1) * conv_run(d));
}
static bool conv_bwd_strip_ok(const Dims& d, const float* xzd, const float* dact, const float* dxzd) {
  return (d.X % 4 == 0) && (d.J % 4 == 0) && (d.I % 4 == 0) && d.K <= 4 &&
         ((reinterpret_cast<uintptr_t>(xzd) | reinterpret_cast<uintptr_t>(dact) | reinterpret_cast<uintptr_t>(dxzd)) % 16 == 0);
}

template <int K>
static pmb_status launch_conv_bwd_k(cudaStream_t st, const Dims& d, const float* xzd, const float* w, const float* b,
                                    const float* dact, float* dxzd, float* partial, uint16_t* pair_hi, uint16_t* pair_lo) {
  const bool strip = conv_bwd_strip_ok(d, xzd, dact, dxzd);
  bool vec = (d.X % 4 == 0) && (d.J % 4 == 0) && (d.I % 4 == 0) &&
             ((reinterpret_cast<uintptr_t>(xzd) | reinterpret_cast<uintptr_t>(dact) | reinterpret_cast<uintptr_t>(dxzd)) % 16 == 0);
  const unsigned rows = (unsigned)conv_bwd_partial_rows(d, strip);
  const int run = conv_run(d);
  if (strip) {
    if constexpr (K <= 4)
      PMB_TRY(launch_pdl(st, conv_silu_bwd_strip_kernel<K>, dim3((unsigned)cdiv(d.X, 32), rows), CONV_STRIP_THREADS, 0, xzd, d.J, d.I, w, b, dact, dxzd, partial, d.X, d.T, run, pair_hi, pair_lo));
  } else if (vec) {
    PMB_TRY(launch_pdl(st, conv_silu_bwd_kernel<K, 4>, dim3((unsigned)cdiv(d.X / 4, 128), rows), 128, 0, xzd, d.J, d.I, w, b, dact, dxzd, partial, d.X, d.T, run, pair_hi, pair_lo));
  } else {
    PMB_TRY(launch_pdl(st, conv_silu_bwd_kernel<K, 1>, dim3((unsigned)cdiv(d.X, 128), rows), 128, 0, xzd, d.J, d.I, w, b, dact, dxzd, partial, d.X, d.T, run, pair_hi, pair_lo));
  }
  return PMB_OK;
}

pmb_status conv_silu_bwd(cudaStream_t st, const Dims& d, const float* xzd, const float* w, const float* b,
                         const float* dact, float* dxzd, float* dw, float* db, void* ws, size_t ws_bytes, SideLane* red,
                         uint16_t* pair_hi, uint16_t* pair_lo) {
  if (ws_bytes < conv_bwd_ws_bytes(d)) return fail(PMB_ERR_WORKSPACE, "conv bwd workspace too small");
  float* partial = static_cast<float*>(ws);
  ProfScope prof(st, "conv_silu_bwd", 0.0, 4.0 * d.M * 3.0 * d.X);
  switch (d.K) {
    case 2: PMB_TRY(launch_conv_bwd_k<2>(st, d, xzd, w, b, dact, dxzd, partial, pair_hi, pair_lo)); break;
    case 3: PMB_TRY(launch_conv_bwd_k<3>(st, d, xzd, w, b, dact, dxzd, partial, pair_hi, pair_lo)); break;
    case 4: PMB_TRY(launch_conv_bwd_k<4>(st, d, xzd, w, b, dact, dxzd, partial, pair_hi, pair_lo)); break;
    case 5: PMB_TRY(launch_conv_bwd_k<5>(st, d, xzd, w, b, dact, dxzd, partial, pair_hi, pair_lo)); break;
    case 6: PMB_TRY(launch_conv_bwd_k<6>(st, d, xzd, w, b, dact, dxzd, partial, pair_hi, pair_lo)); break;
    case 7: PMB_TRY(launch_conv_bwd_k<7>(st, d, xzd, w, b, dact, dxzd, partial, pair_hi, pair_lo)); break;
    case 8: PMB_TRY(launch_conv_bwd_k<8>(st, d, xzd, w, b, dact, dxzd, partial, pair_hi, pair_lo)); break;
    default: return fail(PMB_ERR_SHAPE, "d_conv %d unsupported", d.K);
  }
  const int64_t rows = conv_bwd_partial_rows(d, conv_bwd_strip_ok(d, xzd, dact, dxzd));
  cudaStream_t rs = st;
  if (red) { PMB_TRY(order_after(st, red->ev[4], red->s)); rs = red->s; }
  PMB_TRY(launch_pdl(rs, column_sum_kernel, dim3(column_blocks(d.X * d.K) + column_blocks(d.X)), 32 * COLSUM_LANES, 0, partial, rows, d.X * d.K, dw, partial + rows * d.X * d.K, d.X, db));
  return PMB_OK;
}

// ---------------------------------------------------------------------------------------------
// gated RMSNorm.  g = y * z * sigmoid(z); r = rsqrt(mean(g^2)+eps); out = g * r * w.
// One 256-thread block per row; the row stays in registers between the two passes.
// ---------------------------------------------------------------------------------------------
constexpr int NORM_THREADS = 256;
constexpr int NORM_MAX_PER_THREAD = 8;   // width <= 2048 (registers hold a whole row)

__global__ void __launch_bounds__(NORM_THREADS) gated_rmsnorm_fwd_kernel(const float* __restrict__ y, const float* __restrict__ z,
                                                                         int64_t ldz, const float* __restrict__ w,
                                                                         float* __restrict__ out, float* __restrict__ rstd,
                                                                         int width, float eps, uint16_t* __restrict__ out_hi,
                                                                         uint16_t* __restrict__ out_lo) {
  pdl_launch();
  pdl_wait();
  __shared__ float red[32];
  int64_t row = blockIdx.x;
  const float* yr = y + row * width;
  const float* zr = z + row * ldz;
  float g[NORM_MAX_PER_THREAD];
  float ss = 0.0f;
#pragma unroll
  for (int n = 0; n < NORM_MAX_PER_THREAD; ++n) {
    int i = threadIdx.x + n * NORM_THREADS;
    if (i < width) {
      float zv = zr[i];
      float gv = yr[i] * zv * sigmoid_acc(zv);
      g[n] = gv;
      ss = fmaf(gv, gv, ss);
    }
  }
  float tot = block_sum(ss, red);
  float r = 1.0f / sqrtf(tot / (float)width + eps);
  if (threadIdx.x == 0 && rstd) rstd[row] = r;
#pragma unroll
  for (int n = 0; n < NORM_MAX_PER_THREAD; ++n) {
    int i = threadIdx.x + n * NORM_THREADS;
    if (i < width) {
      float v = g[n] * r * w[i];
      if (out) out[row * width + i] = v;
      if (out_hi) {   // (hi, lo) bf16 pair of v for the pair GEMM: hi = bf16(v), lo = bf16(v - hi), round to nearest even
        uint32_t u = __float_as_uint(v);
        uint32_t h = (u + 0x7fffu + ((u >> 16) & 1u)) >> 16;
        float rem = v - __uint_as_float(h << 16);
        uint32_t ul = __float_as_uint(rem);
        out_hi[row * width + i] = (uint16_t)h;
        if (out_lo) out_lo[row * width + i] = (uint16_t)((ul + 0x7fffu + ((ul >> 16) & 1u)) >> 16);
      }
    }
  }
}

// Sum over the block with one barrier: every warp adds up the warps' sums itself (the same tree in each, the one of block_sum).
// `red` alternates between two buffers from call to call, so that no second barrier keeps a fast warp out.
__device__ __forceinline__ float block_sum_once(float v, float* red) {
  const int lane = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  if (lane == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  return warp_sum(lane < nw ? red[lane] : 0.0f);
}

// float4 variant: width % 4 == 0, 16-byte aligned rows.  PER float4 per thread, blockDim.x * PER >= width / 4.  Bound by HBM; a block
// walks `nrows` rows and requests the next one before it reduces the current one.  Measured at 16384 rows of 1536 with a bf16 output
// (250 MB): 51 us with a block per row, 44 now.
template <int PER>
__global__ void __launch_bounds__(NORM_THREADS) gated_rmsnorm_fwd_vec_kernel(const float* __restrict__ y, const float* __restrict__ z,
                                                                             int64_t ldz, const float* __restrict__ w,
                                                                             float* __restrict__ out, float* __restrict__ rstd,
                                                                             int width, float eps, uint16_t* __restrict__ out_hi,
                                                                             uint16_t* __restrict__ out_lo, int64_t rows, int nrows) {
  pdl_launch();
  pdl_wait();
  __shared__ float red[2][32];
  const int nvec = width >> 2;
  const int64_t r0 = (int64_t)blockIdx.x * nrows;
  const int64_t r1 = r0 + nrows < rows ? r0 + nrows : rows;
  float4 yn[PER], zn[PER];
  auto request = [&](int64_t row) {
#pragma unroll
    for (int n = 0; n < PER; ++n) {
      const int i = threadIdx.x + n * blockDim.x;
      yn[n] = zn[n] = make_float4(0, 0, 0, 0);
      if (i < nvec) { yn[n] = reinterpret_cast<const float4*>(y + row * width)[i]; zn[n] = reinterpret_cast<const float4*>(z + row * ldz)[i]; }
    }
  };
  if (r0 < r1) request(r0);
  for (int64_t row = r0; row < r1; ++row) {
  float4 g[PER];
  float ss = 0.0f;
#pragma unroll
  for (int n = 0; n < PER; ++n) {
    const float4 yv = yn[n], zv = zn[n];
    g[n] = make_float4(yv.x * zv.x * sigmoid_acc(zv.x), yv.y * zv.y * sigmoid_acc(zv.y), yv.z * zv.z * sigmoid_acc(zv.z),
                       yv.w * zv.w * sigmoid_acc(zv.w));
    ss = fmaf(g[n].x, g[n].x, fmaf(g[n].y, g[n].y, fmaf(g[n].z, g[n].z, fmaf(g[n].w, g[n].w, ss))));
  }
  if (row + 1 < r1) request(row + 1);
  const float tot = block_sum_once(ss, red[row & 1]);
  const float r = 1.0f / sqrtf(tot / (float)width + eps);
  if (threadIdx.x == 0 && rstd) rstd[row] = r;
#pragma unroll
  for (int n = 0; n < PER; ++n) {
    const int i = threadIdx.x + n * blockDim.x;
    if (i < nvec) {
      const float4 wv = reinterpret_cast<const float4*>(w)[i];
      const float4 v = make_float4(g[n].x * r * wv.x, g[n].y * r * wv.y, g[n].z * r * wv.z, g[n].w * r * wv.w);
      if (out) reinterpret_cast<float4*>(out + row * width)[i] = v;
      if (out_hi) store_pair4(out_hi + row * width + 4 * i, out_lo ? out_lo + row * width + 4 * i : nullptr, v.x, v.y, v.z, v.w);
    }
  }
  }
}

// threads per block for the float4 kernels: every thread owns exactly `per` float4 when width/4 divides evenly
static inline int norm_vec_threads(int width, int* per) {
  const int nvec = width / 4;
  *per = (nvec + NORM_THREADS - 1) / NORM_THREADS;
  int t = (nvec + *per - 1) / *per;
  return ((t + 31) / 32) * 32;
}
static inline bool norm_vec_ok(int width, int64_t ldz, const void* a, const void* b, const void* c, const void* d2 = nullptr, const void* e2 = nullptr) {
  auto al = [](const void* p) { return p == nullptr || (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  return (width % 4 == 0) && (ldz % 4 == 0) && width / 4 <= 2 * NORM_THREADS && al(a) && al(b) && al(c) && al(d2) && al(e2);
}

pmb_status gated_rmsnorm_fwd(cudaStream_t st, int64_t rows, int width, float eps, const float* y, const float* z, int64_t ldz,
                             const float* w, float* out, float* rstd, uint16_t* out_hi, uint16_t* out_lo) {
  if (width > NORM_THREADS * NORM_MAX_PER_THREAD) return fail(PMB_ERR_SHAPE, "rmsnorm width %d > %d", width, NORM_THREADS * NORM_MAX_PER_THREAD);
  ProfScope prof(st, "gated_rmsnorm_fwd", 0.0, 4.0 * rows * 3.0 * width);
  if (norm_vec_ok(width, ldz, y, z, w, out, out_hi) && (!out_lo || (reinterpret_cast<uintptr_t>(out_lo) & 15) == 0)) {
    int per = 1;
    const int threads = norm_vec_threads(width, &per);
    // four to eight blocks share an SM; with fewer rows than fill it that way every row has a block
    const int nr = (int)cdiv(rows, 148 * 6);
    const unsigned nblk = (unsigned)cdiv(rows, nr);
    if (per == 1) PMB_TRY(launch_pdl(st, gated_rmsnorm_fwd_vec_kernel<1>, dim3((unsigned)nblk), threads, 0, y, z, ldz, w, out, rstd, width, eps, out_hi, out_lo, rows, nr));
    else PMB_TRY(launch_pdl(st, gated_rmsnorm_fwd_vec_kernel<2>, dim3((unsigned)nblk), threads, 0, y, z, ldz, w, out, rstd, width, eps, out_hi, out_lo, rows, nr));
    return PMB_OK;
  }
  PMB_TRY(launch_pdl(st, gated_rmsnorm_fwd_kernel, dim3((unsigned)rows), NORM_THREADS, 0, y, z, ldz, w, out, rstd, width, eps, out_hi, out_lo));
  return PMB_OK;
}

// Backward.  dg = w r dout - g r^3 (sum_j dout_j g_j w_j)/I;  dy = dg z sig(z);
// dz = dg y (sig + z sig (1-sig));  dw_i = sum_rows dout_i g_i r.
// A block handles NORM_ROWS consecutive rows so the dw partial stays in registers across them.
constexpr int NORM_ROWS = 4;

__global__ void __launch_bounds__(NORM_THREADS) gated_rmsnorm_bwd_kernel(const float* __restrict__ dout, const float* __restrict__ y,
                                                                         const float* __restrict__ z, int64_t ldz,
                                                                         const float* __restrict__ w, const float* __restrict__ rstd,
                                                                         float* __restrict__ dy, float* __restrict__ dz, int64_t lddz,
                                                                         float* __restrict__ dw_partial, int64_t rows, int width) {
  pdl_launch();
  pdl_wait();
  __shared__ float red[32];
  float dwacc[NORM_MAX_PER_THREAD];
#pragma unroll
  for (int n = 0; n < NORM_MAX_PER_THREAD; ++n) dwacc[n] = 0.0f;
  int64_t r0 = (int64_t)blockIdx.x * NORM_ROWS;
  for (int rr = 0; rr < NORM_ROWS; ++rr) {
    int64_t row = r0 + rr;
    if (row >= rows) break;  // uniform across the block
    float r = rstd[row];
    // pass 1: load the row once, keep it in registers
    float zv[NORM_MAX_PER_THREAD], yv[NORM_MAX_PER_THREAD], dn[NORM_MAX_PER_THREAD];
    float dot = 0.0f;
#pragma unroll
    for (int n = 0; n < NORM_MAX_PER_THREAD; ++n) {
      int i = threadIdx.x + n * NORM_THREADS;
      if (i < width) {
        zv[n] = z[row * ldz + i]; yv[n] = y[row * width + i]; dn[n] = dout[row * width + i];
        float gv = yv[n] * zv[n] * sigmoid_acc(zv[n]);
        dot = fmaf(dn[n] * gv, w[i], dot);
      }
    }
    float tot = block_sum(dot, red);
    float coef = r * r * r * tot / (float)width;
#pragma unroll
    for (int n = 0; n < NORM_MAX_PER_THREAD; ++n) {
      int i = threadIdx.x + n * NORM_THREADS;
      if (i < width) {
        float s = sigmoid_acc(zv[n]);
        float gv = yv[n] * zv[n] * s;
        float dg = w[i] * r * dn[n] - gv * coef;
        dwacc[n] = fmaf(dn[n] * gv, r, dwacc[n]);
        dy[row * width + i] = dg * zv[n] * s;
        dz[row * lddz + i] = dg * yv[n] * (s + zv[n] * s * (1.0f - s));
      }
    }
  }
#pragma unroll
  for (int n = 0; n < NORM_MAX_PER_THREAD; ++n) {
    int i = threadIdx.x + n * NORM_THREADS;
    if (i < width) dw_partial[(int64_t)blockIdx.x * width + i] = dwacc[n];
  }
}

// float4 variant of the backward.  Optional extras (see NormBwdExtra): dz as a (hi, lo) bf16 pair instead of fp32, and dY exp(S) for
// the scan backward.  Bound by HBM (reads of dout, y, z, writes of dy and the bf16 copies).  A block walks `nrows` rows
// with its share of dw in registers: few long blocks leave few partial sums (one row of them per block), and the blocks that share an SM
// cover each other's loads; the next row is asked for before this one's sum (in registers, with room for two blocks: 145 us).
// Measured at 16384 rows of 1536 with plain bf16 copies (550 MB): 136 us + 60 us of partial sums with four rows per block, 117 us + 3 with
// fourteen, 97 now with the next row in shared memory (104 when registers are held to four blocks; one row more ahead 114); 8192 rows: 39 and 32.
template <int PER>
__global__ void __launch_bounds__(NORM_THREADS, 3) gated_rmsnorm_bwd_vec_kernel(const float* __restrict__ dout, const float* __restrict__ y,
                                                                             const float* __restrict__ z, int64_t ldz,
                                                                             const float* __restrict__ w, const float* __restrict__ rstd,
                                                                             float* __restrict__ dy, float* __restrict__ dz, int64_t lddz,
                                                                             float* __restrict__ dw_partial, int64_t rows, int width, int nrows,
                                                                             NormBwdExtra ex) {
  pdl_launch();
  pdl_wait();
  __shared__ float red[2][32];
  const int nvec = width >> 2;
  float4 dwacc[PER], wv[PER];
#pragma unroll
  for (int n = 0; n < PER; ++n) {
    const int i = threadIdx.x + n * blockDim.x;
    dwacc[n] = make_float4(0, 0, 0, 0);
    wv[n] = i < nvec ? reinterpret_cast<const float4*>(w)[i] : make_float4(0, 0, 0, 0);
  }
  const int64_t r0 = (int64_t)blockIdx.x * nrows;
  const int64_t r1 = r0 + nrows < rows ? r0 + nrows : rows;
  // the next row waits in slots of the thread's own (cp.async, no barrier): [z, y, dout][PER][thread]
  __shared__ __align__(16) float4 next[3 * PER * NORM_THREADS];
  float4* const own = next + threadIdx.x;
  auto fetch = [&](int64_t row) {
#pragma unroll
    for (int n = 0; n < PER; ++n) {
      const int i = threadIdx.x + n * blockDim.x;
      if (i >= nvec || row >= r1) continue;
      const uint32_t d = (uint32_t)__cvta_generic_to_shared(own + n * NORM_THREADS);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(z + row * ldz + 4 * i) : "memory");
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16 * PER * NORM_THREADS), "l"(y + row * width + 4 * i) : "memory");
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 32 * PER * NORM_THREADS), "l"(dout + row * width + 4 * i) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  fetch(r0);
  float rnext = r0 < r1 ? rstd[r0] : 0.0f;
  for (int64_t row = r0; row < r1; ++row) {
    const float r = rnext;
    if (row + 1 < r1) rnext = rstd[row + 1];
    float4 zv[PER], yv[PER], dn[PER], gv[PER], sv[PER];
    float dot = 0.0f;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int n = 0; n < PER; ++n) {
      zv[n] = yv[n] = dn[n] = make_float4(0, 0, 0, 0);
      if (threadIdx.x + n * blockDim.x < nvec) { zv[n] = own[n * NORM_THREADS]; yv[n] = own[(PER + n) * NORM_THREADS]; dn[n] = own[(2 * PER + n) * NORM_THREADS]; }
    }
    fetch(row + 1);
#pragma unroll
    for (int n = 0; n < PER; ++n) {
      sv[n] = make_float4(sigmoid_acc(zv[n].x), sigmoid_acc(zv[n].y), sigmoid_acc(zv[n].z), sigmoid_acc(zv[n].w));
      gv[n] = make_float4(yv[n].x * zv[n].x * sv[n].x, yv[n].y * zv[n].y * sv[n].y, yv[n].z * zv[n].z * sv[n].z, yv[n].w * zv[n].w * sv[n].w);
      dot = fmaf(dn[n].x * gv[n].x, wv[n].x, fmaf(dn[n].y * gv[n].y, wv[n].y, fmaf(dn[n].z * gv[n].z, wv[n].z, fmaf(dn[n].w * gv[n].w, wv[n].w, dot))));
    }
    const float tot = block_sum_once(dot, red[row & 1]);
    const float coef = r * r * r * tot / (float)width;
#pragma unroll
    for (int n = 0; n < PER; ++n) {
      const int i = threadIdx.x + n * blockDim.x;
      if (i < nvec) {
        float4 dg, o_dy, o_dz;
#define PMB_NORM_LANE(c)                                                        \
        dg.c = wv[n].c * r * dn[n].c - gv[n].c * coef;                           \
        dwacc[n].c = fmaf(dn[n].c * gv[n].c, r, dwacc[n].c);                     \
        o_dy.c = dg.c * zv[n].c * sv[n].c;                                       \
        o_dz.c = dg.c * yv[n].c * (sv[n].c + zv[n].c * sv[n].c * (1.0f - sv[n].c));
        PMB_NORM_LANE(x) PMB_NORM_LANE(y) PMB_NORM_LANE(z) PMB_NORM_LANE(w)
#undef PMB_NORM_LANE
        reinterpret_cast<float4*>(dy + row * width)[i] = o_dy;
        if (ex.dz_hi) store_pair4(ex.dz_hi + row * lddz + 4 * i, ex.dz_lo ? ex.dz_lo + row * lddz + 4 * i : nullptr, o_dz.x, o_dz.y, o_dz.z, o_dz.w);
        else reinterpret_cast<float4*>(dz + row * lddz)[i] = o_dz;
        if (ex.dy_hi) store_pair4(ex.dy_hi + row * width + 4 * i, ex.dy_lo ? ex.dy_lo + row * width + 4 * i : nullptr, o_dy.x, o_dy.y, o_dy.z, o_dy.w);
        if (ex.dys_hi) {   // the same, as a bf16 pair (operand of the pair contractions of the scan backward)
          const int h = (4 * i) / ex.P;
          const int64_t bb = row / ex.T, tt = row % ex.T;
          const float f = __expf(ex.S[(bb * ex.H + h) * ex.T + tt]);
          store_pair4(ex.dys_hi + row * width + 4 * i, ex.dys_lo ? ex.dys_lo + row * width + 4 * i : nullptr, o_dy.x * f, o_dy.y * f, o_dy.z * f, o_dy.w * f);
        }
        if (ex.dys) {    // dys[t, h, :] = dy[t, h, :] * exp(S[b, h, t]) for the scan backward (head width ex.P is a multiple of 4)
          const int h = (4 * i) / ex.P;
          const int64_t bb = row / ex.T, tt = row % ex.T;
          const float f = __expf(ex.S[(bb * ex.H + h) * ex.T + tt]);
          reinterpret_cast<float4*>(ex.dys + row * width)[i] = make_float4(o_dy.x * f, o_dy.y * f, o_dy.z * f, o_dy.w * f);
        }
      }
    }
  }
#pragma unroll
  for (int n = 0; n < PER; ++n) {
    const int i = threadIdx.x + n * blockDim.x;
    if (i < nvec) reinterpret_cast<float4*>(dw_partial + (int64_t)blockIdx.x * width)[i] = dwacc[n];
  }
}

// out[j] = sum_r partial[r*cols + j]; blocks past the columns' do the same for a second matrix of as many rows.  Block = 32 columns x COLSUM_LANES
// row lanes; each lane sums rows ty, ty + COLSUM_LANES, ... and the lanes' sums are added in a fixed order (deterministic).  The columns alone
// give few blocks, so what counts is the length of a lane's chain of loads: 1171 rows of 1536 columns 10.9 us with four of them in
// flight, 5.9 with COLSUM_AHEAD.
constexpr int COLSUM_AHEAD = 12;
__global__ void __launch_bounds__(32 * COLSUM_LANES) column_sum_kernel(const float* __restrict__ partial, int64_t rows, int cols, float* __restrict__ out,
                                                                       const float* __restrict__ more, int more_cols, float* __restrict__ more_out) {
  pdl_launch();
  pdl_wait();
  __shared__ float sh[COLSUM_LANES][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, first = (cols + 31) >> 5;
  int j = blockIdx.x * 32 + tx;
  if ((int)blockIdx.x >= first) { j -= first * 32; partial = more; cols = more_cols; out = more_out; }
  float s = 0.0f;
  if (j < cols) {
    const float* p = partial + (int64_t)ty * cols + j;
    const int64_t step = (int64_t)COLSUM_LANES * cols;
    int64_t left = (rows - ty + COLSUM_LANES - 1) / COLSUM_LANES;
    for (; left > 0; left -= COLSUM_AHEAD, p += COLSUM_AHEAD * step) {
      float v[COLSUM_AHEAD];
#pragma unroll
      for (int u = 0; u < COLSUM_AHEAD; ++u) v[u] = u < left ? p[u * step] : 0.0f;
#pragma unroll
      for (int u = 0; u < COLSUM_AHEAD; ++u) s += v[u];
    }
  }
  sh[ty][tx] = s;
  __syncthreads();
  if (ty == 0 && j < cols) {
    float t = 0.0f;
#pragma unroll
    for (int k = 0; k < COLSUM_LANES; ++k) t += sh[k][tx];
    out[j] = t;
  }
}

size_t gated_rmsnorm_bwd_ws_bytes(int64_t rows, int width) {
  return align_up((size_t)cdiv(rows, NORM_ROWS) * width * sizeof(float), 256);
}

pmb_status gated_rmsnorm_bwd(cudaStream_t st, int64_t rows, int width, const float* dout, const float* y, const float* z, int64_t ldz,
                             const float* w, const float* rstd, float* dy, float* dz, int64_t lddz, float* dw, void* ws, size_t ws_bytes,
                             SideLane* red, const NormBwdExtra* extra) {
  NormBwdExtra ex{};
  if (extra) ex = *extra;
  if (width > NORM_THREADS * NORM_MAX_PER_THREAD) return fail(PMB_ERR_SHAPE, "rmsnorm width %d too large", width);
  if (ws_bytes < gated_rmsnorm_bwd_ws_bytes(rows, width)) return fail(PMB_ERR_WORKSPACE, "rmsnorm bwd workspace too small");
  float* partial = static_cast<float*>(ws);
  ProfScope prof(st, "gated_rmsnorm_bwd", 0.0, 4.0 * rows * 5.0 * width);
  int64_t nblk = cdiv(rows, NORM_ROWS);
  const bool vec_ok = norm_vec_ok(width, ldz, dout, y, z, w, dy) && (lddz % 4 == 0) &&
                      ((reinterpret_cast<uintptr_t>(dz) | reinterpret_cast<uintptr_t>(partial)) & 15) == 0;
  if ((ex.dz_hi || ex.dys || ex.dy_hi || ex.dys_hi) && !vec_ok) return fail(PMB_ERR_UNSUPPORTED, "gated_rmsnorm_bwd: pair / scaled outputs need the vector kernel's alignment");
  if (vec_ok) {
    int per = 1;
    const int threads = norm_vec_threads(width, &per);
    // two waves of the blocks that fit; below four rows each the partial sums would outgrow the workspace's rows
    int64_t nr = cdiv(rows, 8 * 148);
    if (nr < NORM_ROWS) nr = NORM_ROWS;
    nblk = cdiv(rows, nr);
    if (per == 1) PMB_TRY(launch_pdl(st, gated_rmsnorm_bwd_vec_kernel<1>, dim3((unsigned)nblk), threads, 0, dout, y, z, ldz, w, rstd, dy, dz, lddz, partial, rows, width, (int)nr, ex));
    else PMB_TRY(launch_pdl(st, gated_rmsnorm_bwd_vec_kernel<2>, dim3((unsigned)nblk), threads, 0, dout, y, z, ldz, w, rstd, dy, dz, lddz, partial, rows, width, (int)nr, ex));
  } else {
    PMB_TRY(launch_pdl(st, gated_rmsnorm_bwd_kernel, dim3((unsigned)nblk), NORM_THREADS, 0, dout, y, z, ldz, w, rstd, dy, dz, lddz, partial, rows, width));
  }
  cudaStream_t rs = st;
  if (red) { PMB_TRY(order_after(st, red->ev[4], red->s)); rs = red->s; }
  PMB_TRY(launch_pdl(rs, column_sum_kernel, dim3(column_blocks(width)), 32 * COLSUM_LANES, 0, partial, nblk, width, dw, nullptr, 0, nullptr));
  return PMB_OK;
}

// ---------------------------------------------------------------------------------------------
// Gated RMSNorm backward for callers that cannot allocate device memory.
//
// Some hosts may not call cudaMalloc at the point where they need this kernel: a trainer that handed the
// whole device to its own pool at start-up and has nothing left to carve a workspace from, or a
// latency-bound serving loop that must stay out of the driver's allocator.  For them the per-row-block
// weight-gradient partials live in the array below, which is part of the library image: every GPU that
// loads the library holds these 4 MiB until the process exits.
//
// In host code `g_static_scratch` names a host-side shadow of the symbol, not device memory; the device
// address is looked up once per device with cudaGetSymbolAddress (with that device current) and cached.
// That lookup happens on the first call on a device, so make that first call outside any stream capture.
// Nothing has to be zeroed between calls: each call overwrites the rows of the array it later reads.
// All calls share the one array, so two calls whose kernels may overlap on the GPU (different streams
// without an ordering between them) race on it; serialise them.
// ---------------------------------------------------------------------------------------------
constexpr size_t STATIC_SCRATCH_BYTES = 4u << 20;
static __device__ __align__(256) float g_static_scratch[STATIC_SCRATCH_BYTES / sizeof(float)];
constexpr int STATIC_SCRATCH_MAX_DEVICES = 64;
static float* g_static_scratch_addr[STATIC_SCRATCH_MAX_DEVICES] = {nullptr};

static pmb_status static_scratch_for_current_device(float** out) {
  int dev = -1;
  PMB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= STATIC_SCRATCH_MAX_DEVICES) return fail(PMB_ERR_UNSUPPORTED, "device ordinal %d is outside 0..%d", dev, STATIC_SCRATCH_MAX_DEVICES - 1);
  if (!g_static_scratch_addr[dev]) {
    void* p = nullptr;
    PMB_CUDA(cudaGetSymbolAddress(&p, g_static_scratch));
    g_static_scratch_addr[dev] = static_cast<float*>(p);
  }
  *out = g_static_scratch_addr[dev];
  return PMB_OK;
}

pmb_status gated_rmsnorm_bwd_static(cudaStream_t st, int64_t rows, int width, const float* dout, const float* y, const float* z,
                                    int64_t ldz, const float* w, const float* rstd, float* dy, float* dz, int64_t lddz, float* dw) {
  size_t need = gated_rmsnorm_bwd_ws_bytes(rows, width);
  if (need > STATIC_SCRATCH_BYTES)
    return fail(PMB_ERR_SHAPE, "gated_rmsnorm_bwd_static: rows=%lld x width=%d needs %zu bytes of scratch, the built-in array holds %zu "
                "(ceil(rows/%d) * width * 4 must not exceed it); use pmb_gated_rmsnorm_bwd with a caller workspace",
                (long long)rows, width, need, STATIC_SCRATCH_BYTES, NORM_ROWS);
  float* scratch = nullptr;
  PMB_TRY(static_scratch_for_current_device(&scratch));
  return gated_rmsnorm_bwd(st, rows, width, dout, y, z, ldz, w, rstd, dy, dz, lddz, dw, scratch, STATIC_SCRATCH_BYTES);
}

pmb_status column_sum(cudaStream_t st, const float* partial, int64_t rows, int cols, float* out) {
  PMB_TRY(launch_pdl(st, column_sum_kernel, dim3(column_blocks(cols)), 32 * COLSUM_LANES, 0, partial, rows, cols, out, nullptr, 0, nullptr));
  return PMB_OK;
}

}  // namespace pmb

extern "C" size_t pmb_gated_rmsnorm_bwd_static_max_bytes(void) { return pmb::STATIC_SCRATCH_BYTES; }

extern "C" pmb_status pmb_gated_rmsnorm_bwd_static(void* stream, int64_t rows, int32_t width,
                                                   const float* d_dout, const float* d_y, const float* d_z, int64_t ldz,
                                                   const float* d_w, const float* d_rstd,
                                                   float* d_dy, float* d_dz, int64_t lddz, float* d_dw) {
  using namespace pmb;
  if (rows <= 0 || width <= 0 || ldz < width || lddz < width) return fail(PMB_ERR_SHAPE, "gated_rmsnorm_bwd_static: bad shape");
  if (!d_dout || !d_y || !d_z || !d_w || !d_rstd || !d_dy || !d_dz || !d_dw) return fail(PMB_ERR_ARG, "gated_rmsnorm_bwd_static: NULL argument");
  return gated_rmsnorm_bwd_static(static_cast<cudaStream_t>(stream), rows, width, d_dout, d_y, d_z, ldz, d_w, d_rstd, d_dy, d_dz, lddz, d_dw);
}

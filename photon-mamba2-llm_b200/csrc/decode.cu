// One-token recurrent decode (Mamba2Block::step, crates/pm-core/src/mamba2/block.rs:278-417):
// rolling conv window + h <- exp(A dt) h + dt (B (x) x), y = C h + D x, gate, norm, out_proj.
//
// The weights (fp32) and the state are read once per token and that is most of the cost at both ends, so no pass copies them: up to 16
// sequences the projections are FMA kernels that stream the weight rows (three launches: in_proj + conv step + dt, state
// step + gate, norm + out_proj), beyond that a tensor-core kernel that turns each weight tile into a bf16 pair on its way
// through shared memory.  The launches are chained with programmatic dependent launch: a kernel is placed while its predecessor
// runs, requests the weights or state it will need, and only then waits.  (A kernel that waits does so for everything enqueued
// before, because its predecessor did.)  What is requested early has to be older than the step: so in_proj, which may follow any kernel
// and be placed while several are at work, reads nothing before its wait, and the kernel in front of the state step lets that one in only
// after its own wait.
// Measured: 1 sequence at d_model 768, 24 heads of 64 x 64: 71 -> 16 -> 14.2 us a step, which is the host's time for it (splitting both
// weights into pairs on every call and GEMM tiles of 128 rows before; 10.1 when replayed from a graph); 256 at d_model 2048, 32 heads of 64 x 128: 228 -> 145 -> 127 us, of which the
// state takes 81 (537 MB, 6.6 TB/s).
#include <cuda_bf16.h>
#include "common.cuh"
#include "kernels.h"
#include "tc_common.cuh"

namespace pmb {

static __device__ unsigned int g_decode_status = 0;

pmb_status read_clear_device_status_decode(unsigned int* word) {
  unsigned int zero = 0;
  PMB_CUDA(cudaMemcpyFromSymbol(word, g_decode_status, sizeof(unsigned int)));
  if (*word) PMB_CUDA(cudaMemcpyToSymbol(g_decode_status, &zero, sizeof(unsigned int)));
  return PMB_OK;
}

namespace dec {


// conv window (B,X,K-1) fp32: oldest column first (state.rs:31-51).  Shifts the window and returns silu(conv).
__device__ __forceinline__ float conv_step(float* __restrict__ win, const float* __restrict__ w, float bias, float xn, int K) {
  float u = bias;
  for (int k = 0; k < K - 1; ++k) {
    const float v = win[k];
    u = fmaf(w[k], v, u);
    if (k > 0) win[k - 1] = v;
  }
  u = fmaf(w[K - 1], xn, u);
  win[K - 2] = xn;
  return u * sigmoid_acc(u);
}

struct StepIn {           // columns of in_proj: z | xBC | dt
  int B, D, I, X, J, H, G, N, P, K;
  const float* conv_w; const float* conv_b; const float* dt_bias;
  float* window;
  float* z; int64_t ldz;          // (B, I) rows of pitch ldz
  float* act; float* dt;          // (B, X) silu(conv), (B, H) softplus
};
// one column j of in_proj's result for sequence b
__device__ __forceinline__ void in_proj_column(const StepIn& s, int b, int j, float v) {
  if (j < s.I) { s.z[b * s.ldz + j] = v; return; }
  const int c = j - s.I;
  if (c < s.X) s.act[(int64_t)b * s.X + c] = conv_step(s.window + ((int64_t)b * s.X + c) * (s.K - 1), s.conv_w + c * s.K, s.conv_b ? s.conv_b[c] : 0.0f, v, s.K);
  else s.dt[(int64_t)b * s.H + c - s.X] = softplus_acc(v + s.dt_bias[c - s.X]);
}

// ---- up to 16 sequences: out[b, j] = sum_k in[b, k] W[k, j] on FMA ------------------------------------------------------------
// CTA = 4 CW columns: CW lanes x 16 bytes across a weight row, a thread takes four adjacent rows at a time (one 16-byte read of a
// sequence's inputs, which sit in shared memory as they lie in memory, serves 16 products) and has GV_GROUPS such groups in flight.
// What bounds it is the chain launch, inputs, weights, reduction, and beyond four sequences the fetching of the inputs by every CTA.
// Inputs interleaved by sequence, stored a float at a time 8 or 16 ways to a bank, and tiles of 32 columns took, in us per step (24 heads
// of 64 x 64 at d_model 768): 2 sequences 20.5, 4: 25.2, 8: 36.2, 16: 56.7; now 14.1, 14.6, 18.4, 27.2 (32 heads of 64 x 128 at 2048: 1 sequence 31.6 -> 21.1, 8: 60.8 -> 31.4, 16: 94.7 -> 48.1).
// OUT = 0: in_proj with the conv step and softplus in the epilogue.
// OUT = 1: out_proj of the gated, normalised y (g = y silu(z) and its per-head sums of squares come from the state kernel; the row's
// rstd is one factor of the result).
constexpr int GV_THREADS = 256, GV_GROUPS = 3;
struct GemvArgs {
  int B, K, N; const float* W; int64_t ldw;
  const float* in;                                       // OUT 0: x_t (B, K); OUT 1: g
  bool in_vec;                                           // `in` (and norm_w) can be read 16 bytes at a time
  const float* ss; int H; const float* norm_w; float eps;   // OUT 1
  float* out; StepIn st;
};
template <int BT, int OUT, int CW>
__global__ void __launch_bounds__(GV_THREADS) gemv_kernel(const GemvArgs a) {
  constexpr int COLS = 4 * CW, PASS = 4 * (GV_THREADS / CW);                 // columns; weight rows of one group of all threads
  extern __shared__ __align__(16) float sx[];             // [BT][K], then the partial sums [8][BT][COLS]
  __shared__ float rs[16];
  const int tid = threadIdx.x, tx = tid % CW, k4 = 4 * (tid / CW), warp = tid >> 5, lane = tid & 31;
  const int j = blockIdx.x * COLS + 4 * tx;
  const bool jin = j < a.N;                               // (N and K are multiples of 4)
  const float* wp = a.W + (int64_t)k4 * a.ldw + (jin ? j : 0);
  float4 w[GV_GROUPS][4];
  auto request = [&](int u, int k0) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
      w[u][r] = jin && k0 + k4 < a.K ? __ldg(reinterpret_cast<const float4*>(wp + (int64_t)(k0 + r) * a.ldw)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  };
  // in_proj follows whatever the caller put in the stream, which may have written the weights and the state: it waits first, and only
  // then lets the state kernel in, which reads the state before its own wait.  What out_proj requests is older than the step.
  if (OUT == 0) { pdl_wait(); pdl_launch(); }
#pragma unroll
  for (int u = 0; u < GV_GROUPS; ++u) request(u, u * PASS);
  if (OUT == 1) { pdl_launch(); pdl_wait(); }
  const int kq = a.K >> 2;
#pragma unroll 4
  for (int i = tid; i < kq * BT; i += GV_THREADS) {
    const int b = BT == 1 ? 0 : i / kq, k = 4 * (i - b * kq);
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (b < a.B) {
      const float* p = a.in + (int64_t)b * a.K + k;
      float4 n = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
      if (a.in_vec) {
        v = *reinterpret_cast<const float4*>(p);
        if (OUT == 1) n = __ldg(reinterpret_cast<const float4*>(a.norm_w + k));
      } else {
        v = make_float4(p[0], p[1], p[2], p[3]);
        if (OUT == 1) n = make_float4(a.norm_w[k], a.norm_w[k + 1], a.norm_w[k + 2], a.norm_w[k + 3]);
      }
      if (OUT == 1) { v.x *= n.x; v.y *= n.y; v.z *= n.z; v.w *= n.w; }
    }
    *reinterpret_cast<float4*>(sx + b * a.K + k) = v;
  }
  if (OUT == 1) {
    for (int b = warp; b < a.B; b += GV_THREADS / 32) {
      float t = 0.0f;
      for (int h = lane; h < a.H; h += 32) t += a.ss[(int64_t)b * a.H + h];
      t = warp_sum(t);
      if (lane == 0) rs[b] = 1.0f / sqrtf(t / (float)a.K + a.eps);
    }
  }
  __syncthreads();
  float acc[BT][4];
#pragma unroll
  for (int b = 0; b < BT; ++b)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[b][e] = 0.0f;
  for (int k0 = 0; k0 < a.K; k0 += GV_GROUPS * PASS) {
#pragma unroll
    for (int u = 0; u < GV_GROUPS; ++u) {
      const int k = k0 + u * PASS + k4;
      if (k < a.K) {
#pragma unroll
        for (int b = 0; b < BT; ++b) {
          const float4 xv = *reinterpret_cast<const float4*>(sx + b * a.K + k);
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const float xr = r == 0 ? xv.x : (r == 1 ? xv.y : (r == 2 ? xv.z : xv.w));
            acc[b][0] = fmaf(xr, w[u][r].x, acc[b][0]); acc[b][1] = fmaf(xr, w[u][r].y, acc[b][1]);
            acc[b][2] = fmaf(xr, w[u][r].z, acc[b][2]); acc[b][3] = fmaf(xr, w[u][r].w, acc[b][3]);
          }
        }
      }
      request(u, k0 + (GV_GROUPS + u) * PASS);
    }
  }
#pragma unroll
  for (int b = 0; b < BT; ++b)
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int m = CW; m < 32; m *= 2) acc[b][e] += __shfl_xor_sync(0xffffffffu, acc[b][e], m);
  __syncthreads();
  float* red = sx;
  if (lane < CW) {
#pragma unroll
    for (int b = 0; b < BT; ++b) *reinterpret_cast<float4*>(red + (warp * BT + b) * COLS + 4 * lane) = make_float4(acc[b][0], acc[b][1], acc[b][2], acc[b][3]);
  }
  __syncthreads();
  for (int i = tid; i < BT * COLS; i += GV_THREADS) {
    const int b = i / COLS, col = blockIdx.x * COLS + i % COLS;
    if (b >= a.B || col >= a.N) continue;
    float v = 0.0f;
#pragma unroll
    for (int q = 0; q < 8; ++q) v += red[(q * BT + b) * COLS + i % COLS];
    if (OUT == 0) in_proj_column(a.st, b, col, v);
    else a.out[(int64_t)b * a.N + col] = v * rs[b];
  }
}

// ---- state step + gate: one CTA per (b, h), state (B,H,N,P) ------------------------------------------------------------------
// A thread owns 4 adjacent p and every (256 / (P/4))-th state row; all its rows (ITER of them) are requested before the wait for
// in_proj, so that 268 MB of state at batch 256 stream with every load of a CTA in flight.  Writes g = (C h + D x) silu(z)
// and the sum of g^2 over the head.
constexpr int STEP_THREADS = 256;
// floats that B and C take in front of the partial outputs, which are stored 16 bytes at a time
__host__ __device__ constexpr int bc_floats(int N) { return (2 * N + 3) & ~3; }
struct StateArgs {
  const float* act; const float* dt; const float* z; int64_t ldz; const float* a_log; const float* D;
  const float* norm_w;
  float* state; float* g; uint16_t* hi; uint16_t* lo; float* ss; int H, G, N, P, X, I;      // hi: g norm_w as a (hi, lo) pair instead of g
};
// the gated output of one (b, i)
__device__ __forceinline__ void store_gated(const StateArgs& s, int b, int i, float gv) {
  const int64_t o = (int64_t)b * s.I + i;
  if (!s.hi) { s.g[o] = gv; return; }
  uint32_t h, l;
  split_bf16_pair(gv * s.norm_w[i], h, l);
  s.hi[o] = (uint16_t)h; s.lo[o] = (uint16_t)l;
}
template <int ITER>
__global__ void __launch_bounds__(STEP_THREADS) state_step_kernel(const StateArgs s) {
  extern __shared__ __align__(16) float sh[];             // B (N), C (N), partial outputs (rows x P)
  __shared__ float red[32];
  const int bh = blockIdx.x, h = bh % s.H, b = bh / s.H, g = h / (s.H / s.G);
  float* Bs = sh; float* Cs = sh + s.N; float* part = sh + bc_floats(s.N);
  const int pw = s.P / 4, nsl = STEP_THREADS / pw, p4 = threadIdx.x % pw, sl = threadIdx.x / pw;
  float4* st = reinterpret_cast<float4*>(s.state + (int64_t)bh * s.N * s.P);
  float4 hv[ITER];
#pragma unroll
  for (int i = 0; i < ITER; ++i) {
    const int n = sl + i * nsl;
    if (sl < nsl && n < s.N) hv[i] = __ldcs(st + (int64_t)n * pw + p4);
  }
  const float A = -expf(s.a_log[h]), Dh = s.D[h];
  pdl_launch();
  pdl_wait();
  const float* arow = s.act + (int64_t)b * s.X;
  for (int n = threadIdx.x; n < s.N; n += STEP_THREADS) {
    Bs[n] = arow[s.I + g * s.N + n];
    Cs[n] = arow[s.I + s.G * s.N + g * s.N + n];
  }
  const float dt = s.dt[(int64_t)b * s.H + h];
  const float decay = expf(A * dt);
  __syncthreads();
  if (sl < nsl) {
    const float4 xv = *reinterpret_cast<const float4*>(arow + h * s.P + 4 * p4);
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < ITER; ++i) {
      const int n = sl + i * nsl;
      if (n < s.N) {
        const float bx = dt * Bs[n], cn = Cs[n];
        float4 v = hv[i];
        v.x = fmaf(decay, v.x, bx * xv.x); v.y = fmaf(decay, v.y, bx * xv.y); v.z = fmaf(decay, v.z, bx * xv.z); v.w = fmaf(decay, v.w, bx * xv.w);
        __stcs(st + (int64_t)n * pw + p4, v);
        acc.x = fmaf(cn, v.x, acc.x); acc.y = fmaf(cn, v.y, acc.y); acc.z = fmaf(cn, v.z, acc.z); acc.w = fmaf(cn, v.w, acc.w);
      }
    }
    *reinterpret_cast<float4*>(part + sl * s.P + 4 * p4) = acc;
  }
  __syncthreads();
  float q = 0.0f;
  for (int p = threadIdx.x; p < s.P; p += STEP_THREADS) {
    float y = 0.0f;
    for (int k = 0; k < nsl; ++k) y += part[k * s.P + p];
    y = fmaf(Dh, arow[h * s.P + p], y);
    const float zv = s.z[b * s.ldz + h * s.P + p];
    const float gv = y * zv * sigmoid_acc(zv);
    store_gated(s, b, h * s.P + p, gv);
    q = fmaf(gv, gv, q);
  }
  const float tot = block_sum(q, red);
  if (threadIdx.x == 0) s.ss[bh] = tot;
}

// Any P and N: one block per (b,h); thread = (p, n-slice).
__global__ void __launch_bounds__(STEP_THREADS) state_step_any_kernel(const StateArgs s) {
  extern __shared__ __align__(16) float sh[];
  __shared__ float red[32];
  const int bh = blockIdx.x, h = bh % s.H, b = bh / s.H, g = h / (s.H / s.G);
  float* Bs = sh; float* Cs = sh + s.N; float* part = sh + 2 * s.N;
  pdl_launch();
  pdl_wait();
  const float* arow = s.act + (int64_t)b * s.X;
  for (int n = threadIdx.x; n < s.N; n += STEP_THREADS) {
    Bs[n] = arow[s.I + g * s.N + n];
    Cs[n] = arow[s.I + s.G * s.N + g * s.N + n];
  }
  __syncthreads();
  const float dt = s.dt[(int64_t)b * s.H + h];
  const float decay = expf(-expf(s.a_log[h]) * dt);
  const int pw = s.P < STEP_THREADS ? s.P : STEP_THREADS, nsl = STEP_THREADS / pw, p0 = threadIdx.x % pw, sl = threadIdx.x / pw;
  float* st = s.state + (int64_t)bh * s.N * s.P;
  if (sl < nsl) {
    for (int p = p0; p < s.P; p += pw) {
      const float xv = arow[h * s.P + p];
      float acc = 0.0f;
      for (int n = sl; n < s.N; n += nsl) {
        const float hv = fmaf(decay, st[(int64_t)n * s.P + p], dt * Bs[n] * xv);
        st[(int64_t)n * s.P + p] = hv;
        acc = fmaf(Cs[n], hv, acc);
      }
      part[sl * s.P + p] = acc;
    }
  }
  __syncthreads();
  float q = 0.0f;
  for (int p = threadIdx.x; p < s.P; p += STEP_THREADS) {
    float y = 0.0f;
    for (int k = 0; k < nsl; ++k) y += part[k * s.P + p];
    y = fmaf(s.D[h], arow[h * s.P + p], y);
    const float zv = s.z[b * s.ldz + h * s.P + p];
    const float gv = y * zv * sigmoid_acc(zv);
    store_gated(s, b, h * s.P + p, gv);
    q = fmaf(gv, gv, q);
  }
  const float tot = block_sum(q, red);
  if (threadIdx.x == 0) s.ss[bh] = tot;
}

// ---- more than 16 sequences: slab[ks][b, j] = sum over K part ks of x[b, k] W[k, j] on tcgen05 -------------------------------------
// The product is formed transposed: a CTA owns 128 columns j of W (the MMA's M) and NB sequences (its N), so a weight is read
// once per NB sequences.  Eight warps load the fp32 weight tile (64 k x 128 j, whole 512-byte rows, the next tile requested
// while this one is converted), split it into a bf16 pair and store it as the MN-major operand; x arrives as a pair by TMA.
// lo*hi + hi*lo + hi*hi as in every fp32 product here.  K is split over CTAs so that the launch fills the machine once.
// XC: x in fp32, converted by the same warps, for in_proj up to 64 sequences; a launch and a pass less (17 sequences, 24 heads: 25.3 -> 20.5 us a
// step together with the norm's, which out_finish_kernel took over).  With more sequences the conversion in every CTA would cost more
// than the pass: it grows with the tile, the weights' does not.
using namespace tcx;
constexpr int SK_BK = 64, SK_CONV = 8, SK_THREADS = 64 + 32 * SK_CONV, SK_STAGES = 2;
template <int NB> struct SkGeo {
  static constexpr int WT = 128 * SK_BK * 2, XT = NB * SK_BK * 2;         // one part of the W / x tile
  static constexpr int STAGE = 2 * WT + 2 * XT;
  static constexpr int SMEM = SK_STAGES * STAGE + 1024 + 256;
};
struct SkMaps { CUtensorMap x[2]; };
__device__ __forceinline__ void pairs8(const float4 (&w)[2], uint32_t (&hi)[4], uint32_t (&lo)[4]) {
  const float v[8] = {w[0].x, w[0].y, w[0].z, w[0].w, w[1].x, w[1].y, w[1].z, w[1].w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const __nv_bfloat162 hh = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
    const float2 hf = __bfloat1622float2(hh);
    const __nv_bfloat162 ll = __floats2bfloat162_rn(v[2 * e] - hf.x, v[2 * e + 1] - hf.y);
    hi[e] = *reinterpret_cast<const uint32_t*>(&hh); lo[e] = *reinterpret_cast<const uint32_t*>(&ll);
  }
}
struct SkArgs { const float* W; int64_t ldw; const float* x; int K, J, B, kt_per; bool early; float* slab; unsigned int* status; };    // early: W is older than the kernel before

template <int NB, bool XC>
__global__ void __launch_bounds__(SK_THREADS, 1) skinny_gemm_kernel(const __grid_constant__ SkMaps maps, const SkArgs a) {
  using GE = SkGeo<NB>;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u, bars = base + SK_STAGES * GE::STAGE;
  uint8_t* bar_ptr = smem_raw + (bars - raw);
  enum { XFULL = 0, WFULL = 2, EMPTY = 4, ACC = 6, NBAR };
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bar_ptr + 8 * NBAR);
  volatile uint32_t* abort_flag = tmem_slot + 1;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;    // (uniform to the compiler)
  const int j0 = (int)blockIdx.x * 128, b0 = (int)blockIdx.z * NB;
  const int kt_all = (a.K + SK_BK - 1) / SK_BK, kt0 = (int)blockIdx.y * a.kt_per, kt1 = min(kt_all, kt0 + a.kt_per);
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(bar(XFULL + i), 1); mbar_init(bar(WFULL + i), SK_CONV); mbar_init(bar(EMPTY + i), 1); }
    mbar_init(bar(ACC), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "n"(NB) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  pdl_launch();
  auto wait = [&](int b, uint32_t parity, unsigned int code) -> bool {
    if (*abort_flag) return false;
    if (mbar_wait(bar(b), parity & 1u)) return true;
    atomicOr(a.status, code);
    *abort_flag = 1;
    return false;
  };
  if (warp == 0) {
    if (!XC && lane == 0) {
      pdl_wait();                                          // (x comes from the kernel before)
      int issued = 0;
      for (int kt = kt0; kt < kt1; ++kt) {
        const int it = kt - kt0, s = it % SK_STAGES;
        if (!wait(EMPTY + s, (uint32_t)(it / SK_STAGES) ^ 1u, 1u)) break;
        mbar_expect_tx(bar(XFULL + s), 2 * GE::XT);
        const uint32_t dst = base + s * GE::STAGE + 2 * GE::WT;
        tma_load_2d(dst, &maps.x[0], kt * SK_BK, b0, bar(XFULL + s));
        tma_load_2d(dst + GE::XT, &maps.x[1], kt * SK_BK, b0, bar(XFULL + s));
        issued = it + 1;
      }
      if (*abort_flag)
        for (int it = (issued > SK_STAGES ? issued - SK_STAGES : 0); it < issued; ++it) mbar_wait(bar(XFULL + it % SK_STAGES), (uint32_t)((it / SK_STAGES) & 1));
    }
  } else if (warp == 1) {
    const uint32_t dh = desc_hi(1024, 2), idesc = idesc_bf16(1, 0, 128, NB);
    for (int kt = kt0; kt < kt1; ++kt) {
      const int it = kt - kt0, s = it % SK_STAGES;
      const uint32_t ph = (uint32_t)(it / SK_STAGES);
      if (!__all_sync(0xffffffffu, (XC || wait(XFULL + s, ph, 2u)) && wait(WFULL + s, ph, 2u))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (elect_one()) {
        const uint32_t st = base + s * GE::STAGE;
        const uint32_t w0 = desc_lo(st, 64 * 128), x0 = desc_lo(st + 2 * GE::WT, 16);
#pragma unroll
        for (int k = 0; k < SK_BK / 16; ++k) {
          const uint32_t wo = w0 + ((uint32_t)(k * 2048) >> 4), xo = x0 + ((uint32_t)(k * 32) >> 4);
          mma_f16_h(tmem, wo + (GE::WT >> 4), dh, xo, dh, idesc, (it | k) ? 1u : 0u);
          mma_f16_h(tmem, wo, dh, xo + (GE::XT >> 4), dh, idesc, 1u);
          mma_f16_h(tmem, wo, dh, xo, dh, idesc, 1u);
        }
        umma_commit(bar(EMPTY + s));
        if (kt + 1 == kt1) umma_commit(bar(ACC));
      }
      __syncwarp();
    }
  } else {
    const int ct = threadIdx.x - 64, jq = ct & 15, kr = ct >> 4;       // eight columns, rows kr + 16 i
    const int j = j0 + 8 * jq;
    const bool in0 = j < a.J, in1 = j + 4 < a.J;                       // (J is a multiple of 4)
    float4 wa[4][2], wb[4][2];                                         // two tiles in flight
    auto request = [&](int kt, float4 (&w)[4][2]) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = kt * SK_BK + kr + 16 * i;
        const float* src = a.W + (int64_t)k * a.ldw + j;
        const bool in = kt < kt1 && k < a.K;
        w[i][0] = in && in0 ? __ldcs(reinterpret_cast<const float4*>(src)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        w[i][1] = in && in1 ? __ldcs(reinterpret_cast<const float4*>(src + 4)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
    };
    constexpr int XR = XC ? NB / 32 : 1;                               // x: eight columns k of rows xr + 32 i
    const int xq = ct & 7, xr = ct >> 3;
    float4 xa[XR][2], xb[XR][2];
    auto request_x = [&](int kt, float4 (&x)[XR][2]) {
#pragma unroll
      for (int i = 0; i < XR; ++i) {
        const int b = b0 + xr + 32 * i, k = kt * SK_BK + 8 * xq;       // (K is a multiple of 8)
        const float* src = a.x + (int64_t)b * a.K + k;
        const bool in = kt < kt1 && k < a.K && b < a.B;
        x[i][0] = in ? *reinterpret_cast<const float4*>(src) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        x[i][1] = in ? *reinterpret_cast<const float4*>(src + 4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
    };
    bool ok = true;
    // converts one tile into its stage and requests the tile two further on into the registers it came from
    auto convert = [&](int kt, float4 (&w)[4][2], float4 (&x)[XR][2]) {
      const int it = kt - kt0, s = it % SK_STAGES;
      uint32_t hi[4][4], lo[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        pairs8(w[i], hi[i], lo[i]);
      }
      uint32_t xh[XR][4], xl[XR][4];
      if (XC) {
#pragma unroll
        for (int i = 0; i < XR; ++i) pairs8(x[i], xh[i], xl[i]);
        request_x(kt + 2, x);
      }
      request(kt + 2, w);
      ok = __all_sync(0xffffffffu, ok && wait(EMPTY + s, (uint32_t)(it / SK_STAGES) ^ 1u, 4u));
      if (!ok) return;
      const uint32_t dst = base + s * GE::STAGE + (uint32_t)((jq >> 3) * 64 * 128);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = kr + 16 * i;
        const uint32_t o = dst + (uint32_t)(k * 128 + (((jq & 7) ^ (k & 7)) << 4));
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(o), "r"(hi[i][0]), "r"(hi[i][1]), "r"(hi[i][2]), "r"(hi[i][3]) : "memory");
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(o + GE::WT), "r"(lo[i][0]), "r"(lo[i][1]), "r"(lo[i][2]), "r"(lo[i][3]) : "memory");
      }
      if (XC) {
#pragma unroll
        for (int i = 0; i < XR; ++i) {
          const int r = xr + 32 * i;
          const uint32_t o = base + s * GE::STAGE + 2 * GE::WT + (uint32_t)(r * 128 + ((xq ^ (r & 7)) << 4));
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(o), "r"(xh[i][0]), "r"(xh[i][1]), "r"(xh[i][2]), "r"(xh[i][3]) : "memory");
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(o + GE::XT), "r"(xl[i][0]), "r"(xl[i][1]), "r"(xl[i][2]), "r"(xl[i][3]) : "memory");
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(WFULL + s));
    };
    if (XC || !a.early) pdl_wait();
    request(kt0, wa);
    request(kt0 + 1, wb);
    if (XC) { request_x(kt0, xa); request_x(kt0 + 1, xb); }
    for (int kt = kt0; kt < kt1 && ok; kt += 2) {
      convert(kt, wa, xa);
      if (kt + 1 < kt1 && ok) convert(kt + 1, wb, xb);
    }
    ok = __all_sync(0xffffffffu, ok && wait(ACC, 0u, 8u));
    if (ok) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int quarter = warp & 3, half = (warp - 2) >> 2;
      const int jr = j0 + quarter * 32 + lane;
      float* out = a.slab + (int64_t)blockIdx.y * a.B * a.J + jr;
#pragma unroll 1
      for (int c0 = 32 * half; c0 < NB && b0 + c0 < a.B; c0 += 64) {
        uint32_t r[32];
        tmem_ld32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0, r);
        if (jr < a.J) {
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (b0 + c0 + e < a.B) out[(int64_t)(b0 + c0 + e) * a.J] = __uint_as_float(r[e]);
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(NB) : "memory");
  }
}

// adds the slabs of in_proj and runs the per-column work of the step on the sums (grid: columns x sequences, which go on in z where y
// ends; a linear grid costs a division, 0.5 us of 30 at 24 sequences)
constexpr int FINISH_Y = 65535;
__global__ void __launch_bounds__(256) in_proj_finish_kernel(const float* __restrict__ slab, int n, StepIn s) {
  pdl_wait();
  pdl_launch();                                            // (in this order: the state step reads the state before it waits)
  const int j = (int)(blockIdx.x * blockDim.x + threadIdx.x), b = (int)(blockIdx.y + blockIdx.z * FINISH_Y);
  if (j >= s.J || b >= s.B) return;
  // what the column's conv step needs is requested with the slabs (11.7 -> 10.7 us for 256 sequences, 2304 channels)
  const int c = j - s.I;
  const bool conv4 = s.K == 4 && c >= 0 && c < s.X;
  float* win = s.window + ((int64_t)b * s.X + (conv4 ? c : 0)) * (s.K - 1);
  float t3[3], w4[4], bias = 0.0f;
  if (conv4) {
#pragma unroll
    for (int k = 0; k < 3; ++k) t3[k] = win[k];
#pragma unroll
    for (int k = 0; k < 4; ++k) w4[k] = __ldg(s.conv_w + 4 * c + k);
    if (s.conv_b) bias = __ldg(s.conv_b + c);
  }
  const float* p = slab + (int64_t)b * s.J + j;
  const int64_t pitch = (int64_t)s.B * s.J;
  float v = 0.0f;
  for (int q = 0; q < n; q += 4) {
    float t[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) t[u] = q + u < n ? p[(q + u) * pitch] : 0.0f;
#pragma unroll
    for (int u = 0; u < 4; ++u) v += t[u];
  }
  if (conv4) {
    win[0] = t3[1]; win[1] = t3[2]; win[2] = v;
    const float u = fmaf(w4[3], v, fmaf(w4[2], t3[2], fmaf(w4[1], t3[1], fmaf(w4[0], t3[0], bias))));
    s.act[(int64_t)b * s.X + c] = u * sigmoid_acc(u);
    return;
  }
  in_proj_column(s, b, j, v);
}

// The same with four adjacent columns per thread, all of one part of in_proj's columns, four taps: whole 16-byte accesses throughout.  A thread per
// column took four waves of short blocks, with the window's twelve bytes per thread: a step of 256 sequences, 32 heads of 64 x 128, 134.0 us, 132.2 now.
constexpr int FINISH4_THREADS = 128;
__global__ void __launch_bounds__(FINISH4_THREADS) in_proj_finish4_kernel(const float* __restrict__ slab, int n, StepIn s) {
  pdl_wait();
  pdl_launch();                                            // (in this order: the state step reads the state before it waits)
  const int j = 4 * (int)(blockIdx.x * FINISH4_THREADS + threadIdx.x), b = (int)(blockIdx.y + blockIdx.z * FINISH_Y);
  if (j >= s.J || b >= s.B) return;
  const int c = j - s.I;
  const bool conv = c >= 0 && c < s.X;
  float4* const win = reinterpret_cast<float4*>(s.window + ((int64_t)b * s.X + (conv ? c : 0)) * 3);
  float4 t[3], w[4], bias = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (conv) {
#pragma unroll
    for (int k = 0; k < 3; ++k) t[k] = win[k];
#pragma unroll
    for (int u = 0; u < 4; ++u) w[u] = __ldg(reinterpret_cast<const float4*>(s.conv_w + 4 * (c + u)));
    if (s.conv_b) bias = make_float4(__ldg(s.conv_b + c), __ldg(s.conv_b + c + 1), __ldg(s.conv_b + c + 2), __ldg(s.conv_b + c + 3));
  }
  const float* p = slab + (int64_t)b * s.J + j;
  const int64_t pitch = (int64_t)s.B * s.J;
  float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  for (int q = 0; q < n; q += 4) {
    float4 f[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) f[u] = q + u < n ? *reinterpret_cast<const float4*>(p + (q + u) * pitch) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int u = 0; u < 4; ++u) { v.x += f[u].x; v.y += f[u].y; v.z += f[u].z; v.w += f[u].w; }
  }
  if (c < 0) { *reinterpret_cast<float4*>(s.z + b * s.ldz + j) = v; return; }
  if (!conv) {
    const float o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int u = 0; u < 4; ++u) in_proj_column(s, b, j + u, o[u]);
    return;
  }
  // the window's channels: (x y z) (w | x y) (z w | x) (y z w)
  win[0] = make_float4(t[0].y, t[0].z, v.x, t[1].x);
  win[1] = make_float4(t[1].y, v.y, t[1].w, t[2].x);
  win[2] = make_float4(v.z, t[2].z, t[2].w, v.w);
  auto act = [](const float4& k, float a, float b2, float c2, float x, float bi) {
    const float u = fmaf(k.w, x, fmaf(k.z, c2, fmaf(k.y, b2, fmaf(k.x, a, bi))));
    return u * sigmoid_acc(u);
  };
  *reinterpret_cast<float4*>(s.act + (int64_t)b * s.X + c) = make_float4(act(w[0], t[0].x, t[0].y, t[0].z, v.x, bias.x), act(w[1], t[0].w, t[1].x, t[1].y, v.y, bias.y),
                                                                        act(w[2], t[1].z, t[1].w, t[2].x, v.z, bias.z), act(w[3], t[2].y, t[2].z, t[2].w, v.w, bias.w));
}

// g rstd w, for the general product
__global__ void __launch_bounds__(256) norm_kernel(const float* __restrict__ g, const float* __restrict__ ss, const float* __restrict__ w, float* __restrict__ out, int I, int H,
                                                   float eps) {
  __shared__ float rs;
  const int64_t b = blockIdx.x;
  pdl_launch();
  pdl_wait();
  if (threadIdx.x == 0) {
    float t = 0.0f;
    for (int h = 0; h < H; ++h) t += ss[b * H + h];
    rs = 1.0f / sqrtf(t / (float)I + eps);
  }
  __syncthreads();
  const float r = rs;
  for (int i = threadIdx.x; i < I; i += blockDim.x) out[b * I + i] = g[b * I + i] * r * w[i];
}

// y[b] = rstd[b] (sum of out_proj's slabs); grid: sequences x 1024 columns (D is a multiple of 8).  The state step writes the pair of
// g norm_w, so that no pass stands between it and out_proj (5.6 us of 138 at 256 sequences, 32 heads of 64 x 128).
__global__ void __launch_bounds__(256) out_finish_kernel(const float* __restrict__ slab, int n, const float* __restrict__ ss, float* __restrict__ y, bool vec, int64_t BD, int D,
                                                         int I, int H, float eps) {
  const int64_t b = blockIdx.x;
  const int j = (int)(blockIdx.y * 1024 + 4 * threadIdx.x);
  pdl_launch();
  pdl_wait();
  const bool in = j < D;
  const float* p = slab + b * D + (in ? j : 0);
  float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float t = 0.0f;
  for (int h = threadIdx.x & 31; h < H; h += 32) t += ss[b * H + h];
  for (int q = 0; q < n; q += 4) {
    float4 f[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) f[u] = q + u < n ? *reinterpret_cast<const float4*>(p + (q + u) * BD) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int u = 0; u < 4; ++u) { v.x += f[u].x; v.y += f[u].y; v.z += f[u].z; v.w += f[u].w; }
  }
  const float r = 1.0f / sqrtf(warp_sum(t) / (float)I + eps);
  if (!in) return;
  float* o = y + b * D + j;
  if (vec) *reinterpret_cast<float4*>(o) = make_float4(v.x * r, v.y * r, v.z * r, v.w * r);
  else { o[0] = v.x * r; o[1] = v.y * r; o[2] = v.z * r; o[3] = v.w * r; }
}

}  // namespace dec
}  // namespace pmb

using namespace pmb;

struct StepWs {
  float *z, *act, *dt, *g, *ss;
  float* slab;                        // in_proj / out_proj results per K split
  uint16_t *x_hi, *x_lo, *n_hi, *n_lo;
  float* normed;
};

// Sequences per tile of the tensor-core projection.  128 where the SMs are shared by K splits: two tiles of 128 take half the splits of one
// of 256, so half the sums go through memory.  256 where there is one split either way and tiles of 128 need a second round, and where they
// leave one split of 24 k-tiles or more.  Each weight is converted once per tile.  What 256 gives of a step in us, for in_proj and out_proj
// by tiles of 128 (k-tiles): 24 heads of 64 x 64 at d_model 768, 256 sequences -1.5 with 52 (12), -2.4 with 12 (24); 640 -5.4 with 130,
// -3.3 with 30; 768 +6.1 with 156; 2048 (417) +4.1 with 416, +6.1 with 96; 32 heads of 64 x 128 at 2048, 256 sequences -2.9 with 70 (32), -4.5
// with 32 (32); 512 -0.5 with 140, -0.6 with 64; 768 (357) +11.8 with 210, +7.4 with 96; 8 heads of 64 x 64 at 256, 1024 sequences -2.3 with 80
// (4); 2048 +2.7 with 160.  (64 at 256 sequences: 67.5, 145 and 31.5 where 128 took 65.4, 127.1 and 33.1.)
static int64_t skinny_tile(int64_t B, int64_t J, int64_t K) {
  const int64_t tiles = cdiv(J, 128) * cdiv(B, 128);
  if (B > 128 && (tiles > 148 || (tiles > 74 && K >= 24 * dec::SK_BK))) return 256;
  return B > 64 ? 128 : (B > 32 ? 64 : 32);
}
// K splits: one wave of CTAs, at least two k-tiles each
static int skinny_splits(int64_t B, int64_t J, int64_t K) {
  const int64_t nb = skinny_tile(B, J, K);
  const int64_t ctas = cdiv(J, 128) * cdiv(B, nb), kt = cdiv(K, dec::SK_BK);
  int64_t sp = 148 / ctas;
  if (sp > kt / 2) sp = kt / 2;
  if (sp < 1) sp = 1;
  return (int)cdiv(kt, cdiv(kt, sp));           // (no empty split)
}

static size_t step_ws_layout(const Dims& d, void* base, size_t bytes, StepWs* out) {
  Arena ar(base, bytes);
  StepWs w;
  w.z = ar.take<float>((size_t)d.B * d.I);
  w.act = ar.take<float>((size_t)d.B * d.X);
  w.dt = ar.take<float>((size_t)d.B * d.H);
  w.g = ar.take<float>((size_t)d.B * d.I);
  w.ss = ar.take<float>((size_t)d.B * d.H);
  const size_t a = (size_t)skinny_splits(d.B, d.J, d.D) * d.B * d.J, b = (size_t)skinny_splits(d.B, d.D, d.I) * d.B * d.D;
  w.slab = ar.take<float>(a > b ? a : b);
  w.x_hi = ar.take<uint16_t>((size_t)d.B * d.D); w.x_lo = ar.take<uint16_t>((size_t)d.B * d.D);
  w.n_hi = ar.take<uint16_t>((size_t)d.B * d.I); w.n_lo = ar.take<uint16_t>((size_t)d.B * d.I);
  w.normed = ar.take<float>((size_t)d.B * d.I);
  if (out) *out = w;
  return ar.ok ? ar.used() : 0;
}

extern "C" size_t pmb_mamba2_step_workspace_bytes(const pmb_mamba2_config* cfg, int32_t batch) {
  Dims d;
  if (make_dims(cfg, batch, 1, &d) != PMB_OK) return 0;
  return step_ws_layout(d, nullptr, 0, nullptr);
}

constexpr size_t GEMV_MAX_SMEM = 200 * 1024;
static int gemv_tile(int B) { return B > 8 ? 16 : (B > 4 ? 8 : (B > 2 ? 4 : (B > 1 ? 2 : 1))); }
static size_t gemv_smem(int B, int K) {
  const size_t bt = (size_t)gemv_tile(B), a = (size_t)K * bt, b = 8 * bt * 32;      // (32: the widest tile's columns)
  return (a > b ? a : b) * sizeof(float);
}
template <int BT, int OUT, int CW>
static pmb_status gemv_cw(cudaStream_t st, const dec::GemvArgs& a) {
  PMB_SMEM_OPT_IN(GEMV_MAX_SMEM, dec::gemv_kernel<BT, OUT, CW>);
  return launch_pdl(st, dec::gemv_kernel<BT, OUT, CW>, dim3((unsigned)cdiv(a.N, 4 * CW)), dec::GV_THREADS, gemv_smem(a.B, a.K), a);
}
template <int OUT>
static pmb_status gemv(cudaStream_t st, const dec::GemvArgs& a) {
  // Tiles of 16 columns for in_proj and of 8 for out_proj, which has fewer and longer ones: more CTAs, and most or all of a thread's
  // weights requested at once.  With 16 sequences a CTA holds 64 bytes of inputs per k, which every CTA has to fetch: twice the width.
  // us per step with tiles of 32/32, 32/16, 16/16, 16/8, 8/8 (24 heads of 64 x 64 at d_model 768): 4 sequences 17.3, 16.1, 15.6, 14.6, 16.1;
  // 8: 23.0, 20.4, 18.8, 18.4, 22.5; 16: 30.0, 27.1, 29.8, 28.3, 32.4; (32 heads of 64 x 128 at 2048) 1: 23.7, 22.4, 20.6, 21.0, 22.9;
  // 8: 38.7, 35.4, 34.2, 31.4, 38.1; 16: 53.1, 48.2, 53.3, 65.1, 78.6.
  switch (gemv_tile(a.B)) {
    case 1: return gemv_cw<1, OUT, OUT ? 2 : 4>(st, a);
    case 2: return gemv_cw<2, OUT, OUT ? 2 : 4>(st, a);
    case 4: return gemv_cw<4, OUT, OUT ? 2 : 4>(st, a);
    case 8: return gemv_cw<8, OUT, OUT ? 2 : 4>(st, a);
    default: return gemv_cw<16, OUT, OUT ? 4 : 8>(st, a);
  }
}

namespace pmb { namespace hb { pmb_status pair_operand_map(CUtensorMap* map, const uint16_t* base, int64_t inner, int64_t outer, int64_t ld, int box_inner, int box_outer); } }

// x in fp32 (K a multiple of 8, on the 16-byte grid) or, x == NULL, as the pair (hi, lo)
template <int NB, bool XC>
static pmb_status skinny_nb(cudaStream_t st, const float* x, const uint16_t* hi, const uint16_t* lo, int64_t B, int64_t K, int64_t J, const float* W, bool early, float* slab, int splits) {
  static unsigned int* known[PMB_MAX_DEVICES] = {nullptr};
  unsigned int* status = tcx::status_address(g_decode_status, known);
  if (!status) return fail(PMB_ERR_CUDA, "decode: no status word on this device");
  dec::SkMaps ms{};
  if (!XC) {
    PMB_TRY(hb::pair_operand_map(&ms.x[0], hi, K, B, K, dec::SK_BK, NB));
    PMB_TRY(hb::pair_operand_map(&ms.x[1], lo, K, B, K, dec::SK_BK, NB));
  }
  dec::SkArgs a{W, J, x, (int)K, (int)J, (int)B, (int)cdiv(cdiv(K, dec::SK_BK), splits), early, slab, status};
  PMB_SMEM_OPT_IN(dec::SkGeo<NB>::SMEM, dec::skinny_gemm_kernel<NB, XC>);
  ProfScope prof(st, "decode_gemm", 2.0 * B * K * J, 4.0 * ((double)K * J + (double)splits * B * J));
  return launch_pdl(st, dec::skinny_gemm_kernel<NB, XC>, dim3((unsigned)cdiv(J, 128), (unsigned)splits, (unsigned)cdiv(B, NB)), dec::SK_THREADS, dec::SkGeo<NB>::SMEM, ms, a);
}
static pmb_status skinny(cudaStream_t st, const float* x, const uint16_t* hi, const uint16_t* lo, int64_t B, int64_t K, int64_t J, const float* W, bool early, float* slab, int splits) {
  const int64_t nb = skinny_tile(B, J, K);
  if (nb == 256) return skinny_nb<256, false>(st, nullptr, hi, lo, B, K, J, W, early, slab, splits);
  if (nb == 128) return skinny_nb<128, false>(st, nullptr, hi, lo, B, K, J, W, early, slab, splits);
  if (nb == 64) return x ? skinny_nb<64, true>(st, x, hi, lo, B, K, J, W, early, slab, splits) : skinny_nb<64, false>(st, x, hi, lo, B, K, J, W, early, slab, splits);
  return x ? skinny_nb<32, true>(st, x, hi, lo, B, K, J, W, early, slab, splits) : skinny_nb<32, false>(st, x, hi, lo, B, K, J, W, early, slab, splits);
}

static pmb_status launch_state_step(cudaStream_t st, const Dims& d, const dec::StateArgs& s) {
  const bool vec4 = (d.P % 4 == 0) && (d.P / 4 <= dec::STEP_THREADS) && (dec::STEP_THREADS % (d.P / 4) == 0) && (d.X % 4 == 0) && (d.I % 4 == 0) &&
                    (reinterpret_cast<uintptr_t>(s.state) % 16 == 0);
  const int pw = vec4 ? d.P / 4 : (d.P < dec::STEP_THREADS ? d.P : dec::STEP_THREADS), nsl = dec::STEP_THREADS / pw;
  const size_t shm = (size_t)((vec4 ? dec::bc_floats(d.N) : 2 * d.N) + nsl * d.P) * sizeof(float);
  if (shm > 48 * 1024) return fail(PMB_ERR_SHAPE, "mamba2_step: d_state/d_head too large for the step kernel");
  const int iter = (int)cdiv(d.N, nsl);
  ProfScope prof(st, "decode_ssm_step", 0.0, 8.0 * d.B * d.H * d.N * d.P);
  void (*k)(const dec::StateArgs) = dec::state_step_any_kernel;
  if (vec4 && iter <= 2) k = dec::state_step_kernel<2>;
  else if (vec4 && iter <= 4) k = dec::state_step_kernel<4>;
  else if (vec4 && iter <= 8) k = dec::state_step_kernel<8>;
  return launch_pdl(st, k, dim3((unsigned)(d.B * d.H)), dec::STEP_THREADS, shm, s);
}

extern "C" pmb_status pmb_mamba2_step(void* stream, const pmb_mamba2_config* cfg, const pmb_block_params* p,
                                      int32_t batch, const float* d_x_t, float* d_ssm_state, float* d_conv_window,
                                      float* d_y_t, void* d_ws, size_t ws_bytes) {
  Dims d;
  PMB_TRY(make_dims(cfg, batch, 1, &d));
  if (!p || !d_x_t || !d_ssm_state || !d_conv_window || !d_y_t || !d_ws) return fail(PMB_ERR_ARG, "mamba2_step: NULL argument");
  StepWs w;
  if (step_ws_layout(d, d_ws, ws_bytes, &w) == 0) return fail(PMB_ERR_WORKSPACE, "mamba2_step: workspace too small");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto al = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  const bool vec = d.J % 4 == 0 && d.D % 4 == 0 && d.I % 4 == 0 && al(p->in_proj_weight) && al(p->out_proj_weight);
  const bool fma = vec && d.B <= 16 && gemv_smem(d.B, d.D) <= GEMV_MAX_SMEM && gemv_smem(d.B, d.I) <= GEMV_MAX_SMEM;
  const bool tc = !fma && vec && d.D % 8 == 0 && d.I % 8 == 0;
  dec::StepIn si{d.B, d.D, d.I, d.X, d.J, d.H, d.G, d.N, d.P, d.K, p->conv1d_weight, p->conv1d_bias, p->dt_bias, d_conv_window, w.z, d.I, w.act, w.dt};
  const dec::StateArgs sa{w.act, w.dt, w.z, d.I, p->a_log, p->d_skip, p->norm_weight, d_ssm_state, w.g, tc ? w.n_hi : nullptr, w.n_lo, w.ss, d.H, d.G, d.N, d.P, d.X, d.I};
  // Up to 16 sequences the products are fp32 FMA (y 2e-7 of its norm from fp64), beyond on bf16 pairs (7e-6).  Where the line
  // lies is a matter of that precision, not of time.  us per step, FMA / tensor cores (24 heads of 64 x 64 at d_model 768; 32 of 64 x 128
  // at d_model 2048): 1 sequence 14.2 / 19.0, 21.1 / 26.6; 2: 14.1 / 19.8, 23.9 / 28.3; 4: 14.6 / 20.3, 28.3 / 28.4; 8: 18.4 / 22.1, 31.4 / 29.0;
  // 16: 27.2 / 22.6, 48.1 / 31.1; 17: 22.9 and 31.6 (20.5 and 30.4 since that side's steps take two launches less).
  if (fma) {
    dec::GemvArgs a{};
    a.B = d.B; a.K = d.D; a.N = d.J; a.W = p->in_proj_weight; a.ldw = d.J; a.in = d_x_t; a.in_vec = al(d_x_t); a.st = si;
    { ProfScope prof(st, "decode_in_proj", 2.0 * d.B * d.D * d.J, 4.0 * d.D * d.J); PMB_TRY(gemv<0>(st, a)); }
    PMB_TRY(launch_state_step(st, d, sa));
    dec::GemvArgs o{};
    o.B = d.B; o.K = d.I; o.N = d.D; o.W = p->out_proj_weight; o.ldw = d.D; o.in = w.g; o.in_vec = al(w.g) && al(p->norm_weight); o.ss = w.ss; o.H = d.H; o.norm_w = p->norm_weight; o.eps = d.eps; o.out = d_y_t;
    ProfScope prof(st, "decode_out_proj", 2.0 * d.B * d.D * d.I, 4.0 * d.D * d.I);
    return gemv<1>(st, o);
  }
  int n_in = 1;
  if (tc) {
    n_in = skinny_splits(d.B, d.J, d.D);
    const bool x32 = d.B <= 64 && al(d_x_t);
    if (!x32) PMB_TRY(split_pair16(st, d_x_t, d.B, d.D, d.D, w.x_hi, w.x_lo, d.D));
    PMB_TRY(skinny(st, x32 ? d_x_t : nullptr, w.x_hi, w.x_lo, d.B, d.D, d.J, p->in_proj_weight, false, w.slab, n_in));
  } else {
    PMB_TRY(gemm(st, 0, 0, d.B, d.J, d.D, d_x_t, d.D, p->in_proj_weight, d.J, w.slab, d.J, nullptr, 0));
  }
  { ProfScope prof(st, "decode_conv_step", 0.0, 4.0 * d.B * d.J * (n_in + 1.0));
  const dim3 rows(1, (unsigned)(d.B < dec::FINISH_Y ? d.B : dec::FINISH_Y), (unsigned)cdiv(d.B, dec::FINISH_Y));
  const bool quads = tc && d.K == 4 && d.X % 4 == 0 && al(d_conv_window) && al(p->conv1d_weight);      // (tc: J and I are multiples of 4)
  if (quads) PMB_TRY(launch_pdl(st, dec::in_proj_finish4_kernel, dim3((unsigned)cdiv(d.J, 4 * dec::FINISH4_THREADS), rows.y, rows.z), dec::FINISH4_THREADS, 0, static_cast<const float*>(w.slab), n_in, si));
  else PMB_TRY(launch_pdl(st, dec::in_proj_finish_kernel, dim3((unsigned)cdiv(d.J, 256), rows.y, rows.z), 256, 0, static_cast<const float*>(w.slab), n_in, si));
  }
  PMB_TRY(launch_state_step(st, d, sa));
  if (!tc) {
    { ProfScope prof(st, "decode_norm", 0.0, 8.0 * d.B * d.I);
    PMB_TRY(launch_pdl(st, dec::norm_kernel, dim3((unsigned)d.B), 256, 0, static_cast<const float*>(w.g), static_cast<const float*>(w.ss), p->norm_weight, w.normed, d.I, d.H, d.eps)); }
    return gemm(st, 0, 0, d.B, d.D, d.I, w.normed, d.I, p->out_proj_weight, d.D, d_y_t, d.D, nullptr, 0);
  }
  const int n_out = skinny_splits(d.B, d.D, d.I);
  PMB_TRY(skinny(st, nullptr, w.n_hi, w.n_lo, d.B, d.I, d.D, p->out_proj_weight, true, w.slab, n_out));
  ProfScope prof(st, "decode_out_sum", 0.0, 4.0 * d.B * d.D * (n_out + 1.0));
  return launch_pdl(st, dec::out_finish_kernel, dim3((unsigned)d.B, (unsigned)cdiv(d.D, 1024)), 256, 0, static_cast<const float*>(w.slab), n_out, static_cast<const float*>(w.ss), d_y_t,
                    al(d_y_t), (int64_t)d.B * d.D, d.D, d.I, d.H, d.eps);
}

// Fused global-norm gradient clipping + AdamW over a flat fp32 parameter buffer.
// Mirrors crates/pm-train/src/clip.rs:13-53 (global L2 norm, scale by max_norm / norm when above it) and
// crates/pm-train/src/optim.rs:104-157 (decoupled weight decay applied to the parameter first, then the moment
// updates, bias corrections as 1/(1-beta^t) factors, update = m_hat / (sqrt(v_hat) + eps)).
// The reference spends ~12 Ops calls and two assigns per parameter tensor and one host sync for the norm; here the
// norm stays on the device (two-pass, fixed order) and one kernel updates every parameter.
#include "common.cuh"
#include "kernels.h"

namespace pmb {

constexpr int SUMSQ_BLOCKS = 1024;

// Both kernels are bound by HBM (one element of arithmetic per 4 to 28 bytes moved), so what matters is bytes in
// flight: 16-byte accesses, four independent ones per thread.  At 126 M elements norm + update take 623 us, the
// 28 bytes per element of the update alone 547 us at the copy rate (scalar accesses: 102 + 651 us, 742 us together).
// VEC = 1 serves buffers whose base is not 16-byte aligned.
template <int VEC>
__global__ void __launch_bounds__(256) sumsq_partial_kernel(const float* __restrict__ g, int64_t n, float* __restrict__ partial) {
  __shared__ float red[32];
  float s = 0.0f;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (VEC == 4) {
    constexpr int U = 4;
    const int64_t n4 = n >> 2;
    const float4* g4 = reinterpret_cast<const float4*>(g);
    float t[U] = {0.0f, 0.0f, 0.0f, 0.0f};
    int64_t i = i0;
    for (; i + (U - 1) * stride < n4; i += U * stride) {
      float4 v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = g4[i + u * stride];
#pragma unroll
      for (int u = 0; u < U; ++u) t[u] = fmaf(v[u].x, v[u].x, fmaf(v[u].y, v[u].y, fmaf(v[u].z, v[u].z, fmaf(v[u].w, v[u].w, t[u]))));
    }
    for (; i < n4; i += stride) {
      const float4 v = g4[i];
      t[0] = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, t[0]))));
    }
    s = (t[0] + t[1]) + (t[2] + t[3]);
    if (i0 < (n & 3)) s = fmaf(g[4 * n4 + i0], g[4 * n4 + i0], s);
  } else {
    for (int64_t i = i0; i < n; i += stride) s = fmaf(g[i], g[i], s);
  }
  float tot = block_sum(s, red);
  if (threadIdx.x == 0) partial[blockIdx.x] = tot;
}

__global__ void __launch_bounds__(256) sumsq_final_kernel(const float* __restrict__ partial, int nblocks, float* __restrict__ out) {
  __shared__ float red[32];
  float s = 0.0f;
  for (int i = threadIdx.x; i < nblocks; i += blockDim.x) s += partial[i];
  float tot = block_sum(s, red);
  if (threadIdx.x == 0) *out = tot;
}

struct AdamWArgs { float lr, beta1, beta2, eps, wd, inv_bc1, inv_bc2, scale; };
__device__ __forceinline__ void adamw_element(float& p, float g, float& m, float& v, const AdamWArgs& a) {
  const float gi = g * a.scale;
  float pi = p;
  if (a.wd > 0.0f) pi *= (1.0f - a.lr * a.wd);
  m = a.beta1 * m + (1.0f - a.beta1) * gi;
  v = a.beta2 * v + (1.0f - a.beta2) * (gi * gi);
  p = pi - a.lr * ((m * a.inv_bc1) / (sqrtf(v * a.inv_bc2) + a.eps));
}

// The blocks walk the buffer from its end: the norm has just read the gradients front to back, so their last part is
// still in L2 and is taken from there before the update's own traffic pushes it out.  Parameters and moments are
// read and written once (streaming hints), which leaves that part of L2 to the gradients a little longer.
template <int VEC>
__global__ void __launch_bounds__(256) adamw_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                                                    int64_t n, AdamWArgs a, float max_norm, const float* __restrict__ sumsq) {
  a.scale = 1.0f;
  if (max_norm > 0.0f && sumsq) {
    const float norm = sqrtf(*sumsq);
    if (norm > max_norm && norm > 0.0f) a.scale = max_norm / norm;
  }
  const int64_t blk = (int64_t)gridDim.x - 1 - blockIdx.x;
  if (VEC == 4) {
    const int64_t n4 = n >> 2, i = blk * blockDim.x + threadIdx.x;
    if (i < n4) {
      const float4 gv = reinterpret_cast<const float4*>(g)[i];
      float4 pv = __ldcs(reinterpret_cast<const float4*>(p) + i);
      float4 mv = __ldcs(reinterpret_cast<const float4*>(m) + i);
      float4 vv = __ldcs(reinterpret_cast<const float4*>(v) + i);
      adamw_element(pv.x, gv.x, mv.x, vv.x, a);
      adamw_element(pv.y, gv.y, mv.y, vv.y, a);
      adamw_element(pv.z, gv.z, mv.z, vv.z, a);
      adamw_element(pv.w, gv.w, mv.w, vv.w, a);
      __stcs(reinterpret_cast<float4*>(p) + i, pv);
      __stcs(reinterpret_cast<float4*>(m) + i, mv);
      __stcs(reinterpret_cast<float4*>(v) + i, vv);
    } else if (i - n4 < (n & 3)) {
      const int64_t e = 4 * n4 + (i - n4);
      adamw_element(p[e], g[e], m[e], v[e], a);
    }
  } else {
    const int64_t i = blk * blockDim.x + threadIdx.x;
    if (i < n) adamw_element(p[i], g[i], m[i], v[i], a);
  }
}

}  // namespace pmb

using namespace pmb;

extern "C" size_t pmb_grad_sumsq_workspace_bytes(void) { return SUMSQ_BLOCKS * sizeof(float); }

extern "C" pmb_status pmb_grad_sumsq(void* stream, int64_t n, const float* d_grads, float* d_sumsq_out, void* d_ws, size_t ws_bytes) {
  if (n <= 0 || !d_grads || !d_sumsq_out || !d_ws) return fail(PMB_ERR_ARG, "grad_sumsq: bad argument");
  if (ws_bytes < SUMSQ_BLOCKS * sizeof(float)) return fail(PMB_ERR_WORKSPACE, "grad_sumsq: workspace too small");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int blocks = (int)(cdiv(n, 1024) < SUMSQ_BLOCKS ? cdiv(n, 1024) : SUMSQ_BLOCKS);
  ProfScope prof(st, "grad_sumsq", 0.0, 4.0 * n);
  if (reinterpret_cast<uintptr_t>(d_grads) & 15) sumsq_partial_kernel<1><<<blocks, 256, 0, st>>>(d_grads, n, static_cast<float*>(d_ws));
  else sumsq_partial_kernel<4><<<blocks, 256, 0, st>>>(d_grads, n, static_cast<float*>(d_ws));
  PMB_LAUNCHED();
  sumsq_final_kernel<<<1, 256, 0, st>>>(static_cast<float*>(d_ws), blocks, d_sumsq_out);
  PMB_LAUNCHED();
  return PMB_OK;
}

extern "C" pmb_status pmb_adamw_step(void* stream, int64_t n, float* d_params, const float* d_grads, float* d_m, float* d_v,
                                     float lr, float beta1, float beta2, float eps, float weight_decay, int32_t step,
                                     float max_norm, const float* d_sumsq) {
  if (n <= 0 || !d_params || !d_grads || !d_m || !d_v || step <= 0) return fail(PMB_ERR_ARG, "adamw_step: bad argument");
  if (max_norm > 0.0f && !d_sumsq) return fail(PMB_ERR_ARG, "adamw_step: clipping needs the squared gradient norm (pmb_grad_sumsq)");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  float bc1 = 1.0f - powf(beta1, (float)step), bc2 = 1.0f - powf(beta2, (float)step);
  ProfScope prof(st, "adamw_step", 0.0, 28.0 * n);
  const AdamWArgs a{lr, beta1, beta2, eps, weight_decay, 1.0f / bc1, 1.0f / bc2, 1.0f};
  const bool vec = ((reinterpret_cast<uintptr_t>(d_params) | reinterpret_cast<uintptr_t>(d_grads) | reinterpret_cast<uintptr_t>(d_m) | reinterpret_cast<uintptr_t>(d_v)) & 15) == 0;
  if (vec) adamw_kernel<4><<<(unsigned)cdiv(n / 4 + (n & 3), 256), 256, 0, st>>>(d_params, d_grads, d_m, d_v, n, a, max_norm, d_sumsq);
  else adamw_kernel<1><<<(unsigned)cdiv(n, 256), 256, 0, st>>>(d_params, d_grads, d_m, d_v, n, a, max_norm, d_sumsq);
  PMB_LAUNCHED();
  return PMB_OK;
}

// The library's host code on a CUDA runtime that launches nothing: it keeps, for every stream, which launches are ordered before the stream's next one.
// Each call below is made once for every launch it consists of, with that launch failing, and must leave the caller's stream ordered after all that it had
// launched by then.  Prints, per call: name, launches, calls that left work behind.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <set>
#include <vector>
#include <cuda.h>
#include <cuda_runtime_api.h>
#include "pm_b200.h"

using Work = std::set<int>;
static std::map<cudaStream_t, Work> before;
static std::map<cudaEvent_t, Work> recorded;
static int launches, fail_at, streams;
static cudaError_t last = cudaSuccess;
static uintptr_t next_addr = 0x7000000000;

static cudaError_t launch(cudaStream_t s) {
  if (++launches == fail_at) return last = cudaErrorInvalidConfiguration;
  before[s].insert(launches);
  return cudaSuccess;
}
static struct { dim3 g, b; size_t smem; cudaStream_t s; } config;

extern "C" {
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) { config = {g, b, smem, s}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) { *g = config.g; *b = config.b; *smem = config.smem; *static_cast<cudaStream_t*>(s) = config.s; return cudaSuccess; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t s) { return launch(s); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void*, void**) { return launch(c->stream); }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t s) { return launch(s); }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t s) { return launch(s); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { recorded[e] = before[s]; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { before[s].insert(recorded[e].begin(), recorded[e].end()); return cudaSuccess; }
cudaError_t cudaStreamGetCaptureInfo_v2(cudaStream_t, cudaStreamCaptureStatus* st, unsigned long long*, cudaGraph_t*, const cudaGraphNode_t**, size_t*) { *st = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* st) { *st = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int) { *s = reinterpret_cast<cudaStream_t>((uintptr_t)(0x1000 + ++streams)); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = reinterpret_cast<cudaEvent_t>((uintptr_t)(0x100000 + ++streams)); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.0f; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = reinterpret_cast<void*>(next_addr); next_addr += (n + 1023) / 1024 * 1024; return cudaSuccess; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaMemset(void*, int, size_t) { return cudaSuccess; }
cudaError_t cudaMemcpy(void*, const void*, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemcpyFromSymbol(void* p, const void*, size_t n, size_t, cudaMemcpyKind) { memset(p, 0, n); return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = reinterpret_cast<void*>((uintptr_t)0x6000); return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* greatest) { *least = 0; *greatest = -5; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
static CUresult encode(CUtensorMap* m) { memset(m, 0, sizeof *m); return CUDA_SUCCESS; }
cudaError_t cudaGetDriverEntryPointByVersion(const char* name, void** f, unsigned, unsigned long long, cudaDriverEntryPointQueryResult* r) {
  const bool known = strcmp(name, "cuTensorMapEncodeTiled") == 0;
  *f = known ? reinterpret_cast<void*>(encode) : nullptr;
  if (r) *r = known ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
  return cudaSuccess;
}
}

static const cudaStream_t USER = reinterpret_cast<cudaStream_t>((uintptr_t)0x500);
template <class T = float> static T* mem() { void* p; cudaMalloc(&p, (size_t)1 << 32); return static_cast<T*>(p); }

static void check(const char* name, const std::function<pmb_status()>& call) {
  int left = 0;
  for (fail_at = 1;; ++fail_at) {
    before.clear(); recorded.clear(); launches = 0;
    const pmb_status s = call();
    Work all;
    for (auto& b : before) all.insert(b.second.begin(), b.second.end());
    left += before[USER] != all;
    if (launches < fail_at) {
      if (s != PMB_OK) { fprintf(stderr, "%s: %s\n", name, pmb_last_error()); exit(1); }
      break;
    }
    if (s == PMB_OK) { fprintf(stderr, "%s: the failed launch %d went unnoticed\n", name, fail_at); exit(1); }
  }
  printf("%s %d %d\n", name, fail_at - 1, left);
}

static pmb_block_params params() { return {mem(), mem(), mem(), mem(), mem(), mem(), mem(), mem()}; }
static pmb_block_grads grads() { return {mem(), mem(), mem(), mem(), mem(), mem(), mem(), mem()}; }

int main() {
  const size_t WS = (size_t)1 << 38;
  float *x = mem(), *y = mem(), *z = mem(), *ws = mem();
  uint16_t *x16 = mem<uint16_t>(), *y16 = mem<uint16_t>(), *z16 = mem<uint16_t>(), *w0 = mem<uint16_t>(), *w1 = mem<uint16_t>();
  next_addr += WS;
  void* const st = USER;
  const pmb_mamba2_config small{128, 16, 32, 8, 1, 4, 64, 1e-5f}, wide{768, 64, 64, 24, 1, 4, 256, 1e-5f}, states{768, 128, 64, 24, 1, 4, 256, 1e-5f}, odd{60, 7, 5, 3, 1, 4, 32, 1e-5f};
  const pmb_block_params p = params();
  const pmb_block_grads g = grads();
  auto block = [&](const char* name, const pmb_mamba2_config& c, int B, int T) {
    check(name, [&, B, T] { return pmb_mamba2_block_bwd(st, &c, &p, B, T, x, y, nullptr, z, &g, ws, WS); });
  };
  auto block16 = [&](const char* name, const pmb_mamba2_config& c, int B, int T) {
    check(name, [&, B, T] { return pmb_mamba2_block_bwd_bf16(st, &c, &p, w0, w1, B, T, x16, y16, nullptr, z16, &g, ws, WS); });
  };
  block("small", small, 2, 128);
  block("wide", wide, 4, 512);
  block("segments", wide, 1, 1024);
  block("states", states, 2, 512);
  block("odd", odd, 2, 100);
  block16("bf16", wide, 2, 512);
  block16("bf16_long", wide, 8, 2048);
  block16("bf16_ragged", wide, 2, 1000);
  const std::vector<pmb_block_params> ps(3, p);
  const std::vector<pmb_block_grads> gs(3, g);
  check("stack", [&] { return pmb_stack_bwd(st, &small, 3, ps.data(), gs.data(), 2, 128, x, y, ws, WS, nullptr, nullptr); });
  check("stack_wide", [&] { return pmb_stack_bwd(st, &wide, 3, ps.data(), gs.data(), 2, 384, x, y, ws, WS, nullptr, nullptr); });
  check("stack_narrow_ws", [&] { return pmb_stack_bwd(st, &small, 3, ps.data(), gs.data(), 2, 128, x, y, ws, pmb_mamba2_block_workspace_bytes(&small, 2, 128), nullptr, nullptr); });
  float *a = mem(), *b = mem(), *c = mem(), *dy = mem(), *da = mem(), *db = mem(), *dc = mem();
  for (int N : {64, 128}) {
    check(N == 64 ? "scan_fwd" : "scan_fwd_states", [&] { return pmb_ssd_scan_fwd(st, 2, 512, 8, 64, N, 1, 128, x, 512, a, b, c, N, nullptr, y, 512, nullptr, ws, WS); });
    check(N == 64 ? "scan_bwd" : "scan_bwd_states",
          [&] { return pmb_ssd_scan_bwd(st, 2, 512, 8, 64, N, 1, 128, x, 512, a, b, c, N, y, 512, dy, 512, z, 512, da, db, dc, N, ws, WS); });
  }
  int64_t *ids = mem<int64_t>(), *targets = mem<int64_t>();
  for (int bf16 : {0, 1}) {
    pmb_lm* lm = nullptr;
    fail_at = 0;
    if (pmb_lm_create_dtype(&wide, 2, 1000, 2, 512, bf16, &lm) != PMB_OK) { fprintf(stderr, "%s\n", pmb_last_error()); return 1; }
    check(bf16 ? "lm_bf16" : "lm", [&] { return pmb_lm_step_device(lm, st, ids, targets, nullptr, nullptr); });
    pmb_lm_destroy(lm);
  }
}

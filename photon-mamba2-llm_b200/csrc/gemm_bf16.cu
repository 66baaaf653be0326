// bf16 GEMM on tcgen05 (kind::f16, fp32 accumulation in TMEM) for the bf16-storage configurations:
// C = op(A) op(B) (+ R), A and B bf16 in HBM, C (and R) fp32 or bf16.
//
// CTA = one 128x128 output tile; warp 0 = TMA producer, warp 1 = MMA issuer, warps 2..5 = epilogue.
// bf16 operands need no in-smem processing, so a stage is just the two landed tiles (128 x 64 bf16 each,
// 32 KiB per stage) and the ring is 6 deep.  K-major tiles: 128-byte rows, 128-byte swizzle.  MN-major
// tiles: blocks of 64 elements along M/N, 64 k-rows of 128 bytes per block, same swizzle.
// Every mbarrier wait is bounded; on expiry the kernel raises the device status word and drains.
#include <algorithm>
#include <climits>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>
#include "tc_common.cuh"
#include "kernels.h"

namespace pmb {

static __device__ unsigned int g_bf16_status = 0;

namespace hb { static void sched_reset_current_device(); }

pmb_status read_clear_device_status_bf16(unsigned int* word) {
  unsigned int zero = 0;
  PMB_CUDA(cudaMemcpyFromSymbol(word, g_bf16_status, sizeof(unsigned int)));
  if (*word) {
    PMB_CUDA(cudaMemcpyToSymbol(g_bf16_status, &zero, sizeof(unsigned int)));
    hb::sched_reset_current_device();      // a kernel that gave up may have left its tile-ticket counter out of step
  }
  return PMB_OK;
}

namespace hb {

using namespace tcx;

constexpr int TBM = 128, TBN = 128, TBK = 64;
constexpr int TILE_BYTES = TBM * TBK * 2;   // 16 KiB
// SPLIT = false: plain bf16 operands, a stage holds A and B (32 KiB), 6 stages.
// SPLIT = true : every operand is a pair (hi, lo) of bf16 arrays with hi + lo ~= an fp32 value (16 mantissa bits);
//                a stage holds A_hi, B_hi, A_lo, B_lo (64 KiB), 3 stages, and each k-step issues hi*hi + lo*hi + hi*lo.
template <bool SPLIT> struct Cfg {
  static constexpr int STAGES = SPLIT ? 3 : 6;
  static constexpr int STAGE_BYTES = (SPLIT ? 4 : 2) * TILE_BYTES;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 4 * 2 * 4096 + 1024 + 512;   // + the epilogue's staging slots, barriers and the tile queue
};
constexpr int NTHREADS = 192;
constexpr int TMEM_COLS = 256;               // two 128-column accumulators
constexpr int EPI_SLOT_BYTES = 32 * 32 * 4;  // 32 rows x 32 fp32 columns
constexpr int EPI_BYTES = 4 * 2 * EPI_SLOT_BYTES;
constexpr int NQ = 4;                       // depth of the tile-id queue inside a CTA

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

struct Params {
  int M, N, K;
  int a_mn_major, b_mn_major;
  void* C; int64_t ldc; const void* R; int out_bf16;
  int tma_out;     // result (and residual) meet the TMA rules: the epilogue stores through shared memory
  int red;         // fp32 result added onto C: the TMA store adds in L2 and no residual block is loaded
  int bn;          // width of the persistent CTA-pair kernel's tiles (256 or 128)
  int pairs;       // operands are (hi, lo) pairs
  uint16_t* e_hi; uint16_t* e_lo; int64_t lde;   // optional second output: the result as a bf16 pair (TMA-store epilogue only)
  // split K: tiles of split i cover k-tiles [i * kt_per, (i + 1) * kt_per) and go to rows i * slab_rows .. of C, whose
  // slabs the caller adds up (kt_per covers all of K when there is one split)
  int kt_per, slab_rows;
};

__device__ __forceinline__ float bf16_bits_to_float(uint16_t b) { return __uint_as_float((uint32_t)b << 16); }
__device__ __forceinline__ uint16_t float_to_bf16_bits(float f) {   // round to nearest even
  uint32_t u = __float_as_uint(f);
  if ((u & 0x7fffffffu) > 0x7f800000u) return (uint16_t)((u >> 16) | 0x40);
  u += 0x7fffu + ((u >> 16) & 1u);
  return (uint16_t)(u >> 16);
}

// Epilogue of one 32-column piece of an output row: adds R when given and stores fp32 or bf16, 16-byte vectors
// when the row is aligned and the piece lies inside the matrix, element by element otherwise.
__device__ __forceinline__ void store_row_piece(const Params& p, int m, int nb, const uint32_t (&r)[32]) {
  if (p.out_bf16) {
    uint16_t* crow = static_cast<uint16_t*>(p.C) + (int64_t)m * p.ldc + nb;
    const uint16_t* rrow = p.R ? static_cast<const uint16_t*>(p.R) + (int64_t)m * p.ldc + nb : nullptr;
    const bool vec = (nb + 32 <= p.N) && ((p.ldc & 7) == 0) && ((reinterpret_cast<uintptr_t>(p.C) & 15) == 0) &&
                     (!p.R || (reinterpret_cast<uintptr_t>(p.R) & 15) == 0);
    if (vec) {
#pragma unroll
      for (int j = 0; j < 32; j += 8) {
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(r[j + e]);
        if (rrow) {
          uint4 q = *reinterpret_cast<const uint4*>(rrow + j);
          const uint32_t qq[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) { v[2 * e] += __uint_as_float(qq[e] << 16); v[2 * e + 1] += __uint_as_float(qq[e] & 0xffff0000u); }
        }
        uint4 o;
        o.x = (uint32_t)float_to_bf16_bits(v[0]) | ((uint32_t)float_to_bf16_bits(v[1]) << 16);
        o.y = (uint32_t)float_to_bf16_bits(v[2]) | ((uint32_t)float_to_bf16_bits(v[3]) << 16);
        o.z = (uint32_t)float_to_bf16_bits(v[4]) | ((uint32_t)float_to_bf16_bits(v[5]) << 16);
        o.w = (uint32_t)float_to_bf16_bits(v[6]) | ((uint32_t)float_to_bf16_bits(v[7]) << 16);
        *reinterpret_cast<uint4*>(crow + j) = o;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (nb + j < p.N) crow[j] = float_to_bf16_bits(__uint_as_float(r[j]) + (rrow ? bf16_bits_to_float(rrow[j]) : 0.0f));
    }
  } else {
    float* crow = static_cast<float*>(p.C) + (int64_t)m * p.ldc + nb;
    const float* rrow = p.R ? static_cast<const float*>(p.R) + (int64_t)m * p.ldc + nb : nullptr;
    const bool vec = (nb + 32 <= p.N) && ((p.ldc & 3) == 0) && ((reinterpret_cast<uintptr_t>(p.C) & 15) == 0) &&
                     (!p.R || (reinterpret_cast<uintptr_t>(p.R) & 15) == 0);
    if (vec) {
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        float4 v = make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]));
        if (rrow) {
          float4 q = *reinterpret_cast<const float4*>(rrow + j);
          v.x += q.x; v.y += q.y; v.z += q.z; v.w += q.w;
        }
        *reinterpret_cast<float4*>(crow + j) = v;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (nb + j < p.N) crow[j] = __uint_as_float(r[j]) + (rrow ? rrow[j] : 0.0f);
    }
  }
}

// One launch carries up to MAX_GROUP independent products: CTAs [0, pr[0].tiles) work on the first, the next
// pr[1].tiles on the second, and so on (unused entries have tiles == 0).
// Two products whose tile counts each fill the 148 SMs badly (weight-gradient and data-gradient of one projection)
// then share the machine instead of running as two ragged waves.
// (On the CTA-pair kernel a product can be two problems: columns from n_begin up to n_end each, in tiles of their own width.)
struct Problem { CUtensorMap mA, mB, mAlo, mBlo, mC, mR; Params p; int tiles_n; int tiles_mn; int tiles; int n_begin, n_end; };
constexpr int MAX_GROUP = 4;
// Order of the tiles on the persistent CTA-pair kernel.  lead == 0: cluster c takes tiles c, c + clusters, ...  lead > 0 (fewer
// than the clusters): the first `lead` tiles are the long ones (weight gradients: K is the token count) and take one cluster
// each; meanwhile the other clusters take `rounds` of the short tiles each, and what is left goes round all of them.
// (Round-robin alone would give the clusters with a long tile their full share of the short ones on top.)
struct Group { Problem pr[MAX_GROUP]; int lead, rounds; };
__host__ __device__ __forceinline__ int pair_tile_at(const Group& g, int c, int clusters, int j) {
  if (g.lead == 0) return c + j * clusters;
  const int f = clusters - g.lead;
  if (c < g.lead) return j == 0 ? c : g.lead + f * g.rounds + (j - 1) * clusters + c;
  return j < g.rounds ? g.lead + j * f + (c - g.lead) : g.lead + f * g.rounds + (j - g.rounds) * clusters + c;
}
// split of one tile of a problem and its k-tiles; `tile` becomes the tile's index inside the split's slab of C
__device__ __forceinline__ int split_of(const Problem& q, int* tile, int* kt0, int* kt1) {
  const int sp = *tile / q.tiles_mn, num_kt = (q.p.K + TBK - 1) / TBK;
  *tile -= sp * q.tiles_mn;
  *kt0 = sp * q.p.kt_per;
  *kt1 = min(num_kt, *kt0 + q.p.kt_per);
  return sp;
}
__device__ __forceinline__ int pick_problem(const Group& g, int id, int* local) {
  int which = 0, base = 0;
#pragma unroll
  for (int i = 0; i + 1 < MAX_GROUP; ++i) if (id >= base + g.pr[i].tiles && which == i) { base += g.pr[i].tiles; which = i + 1; }
  *local = id - base;
  return which;
}

// TMA store of one 32 x 32 fp32 block (128-byte rows, 128-byte swizzle) and its bookkeeping
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(src) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// Epilogue of one tile for one epilogue warp: its 32 rows (row0 ..) x `ncols` columns (n0 ..) of the accumulator at
// `tmem_acc` (lane offset included).  fp32 results that meet the TMA rules go out from the accumulator's fragments as whole 32-byte
// sectors, and so do their bf16 pairs; the residual's fragments are in registers, the first 32 columns' requested by prefetch() while
// the products still run, the others 32 columns ahead.  (Through one staging slot per warp the second block's residual waited for the first
// one's store: 2048 x 768 x 1536 on pairs with residual and pair output, a tile per cluster, 28 us, 17.6 without either.)  bf16 results
// and fp32 ones that are added onto C leave through the warp's NSLOT swizzled staging slots of 32 rows of 128 bytes (32 fp32 or 64 bf16
// columns) and TMA stores; a bf16 residual is TMA-loaded into the slots: the first NSLOT blocks of a tile by prefetch(), further
// ones as soon as a slot's store has read it.  Everything else is stored row by row.  `pc` and `rph` carry the slot in turn and the
// residual barriers' phases across tiles.
__device__ __forceinline__ void tma_add_2d(const CUtensorMap* map, uint32_t src, int c0, int c1) {
  asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2}], [%3];"
               ::"l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(src) : "memory");
}
template <int NSLOT>
struct Epilogue {
  uint32_t slot0, rbar0;                     // the warp's slots and their residual barriers (8 bytes apart)
  uint32_t pc = 0, rph = 0, loading = 0;     // (loading: lane 0's record of the slots with a load in flight)
  uint2 rr[16];                              // fp32 residual of the next 32 columns, as fragments
  __device__ __forceinline__ bool loads(const Params& p) const { return p.tma_out && p.R && p.out_bf16; }
  // residual fragments of 32 columns from c0 on (rows and columns outside of the matrix: zeros)
  __device__ __forceinline__ void fetch(const Params& p, int row0, int n0, int c0, int lane) {
    const int r = row0 + (lane >> 2), c = n0 + c0 + (lane & 3) * 2;
    const float* base = static_cast<const float*>(p.R) + (int64_t)r * p.ldc + c;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int dr = 16 * (i >> 1) + 8 * (e & 1), dc = 16 * (i & 1) + 8 * (e >> 1);
        const float* at = base + (int64_t)dr * p.ldc + dc;
        uint2 v = make_uint2(0u, 0u);
        if (r + dr < p.M && c + dc + 1 < p.N) v = *reinterpret_cast<const uint2*>(at);
        else if (r + dr < p.M && c + dc < p.N) v.x = __float_as_uint(*at);
        rr[4 * i + e] = v;
      }
  }
  __device__ __forceinline__ void load(const Problem& q, uint32_t slot, int c, int row0) {
    mbar_expect_tx(rbar0 + 8u * slot, EPI_SLOT_BYTES);
    tma_load_2d(slot0 + slot * EPI_SLOT_BYTES, &q.mR, c, row0, rbar0 + 8u * slot);
    loading |= 1u << slot;
  }
  __device__ __forceinline__ void prefetch(const Problem& q, const Params& p, int row0, int n0, int ncols, int lane) {
    if (p.tma_out && p.R && !p.out_bf16 && !p.red) { fetch(p, row0, n0, 0, lane); return; }
    if (!loads(p) || row0 >= p.M || n0 >= p.N || lane != 0) return;
    const int bw = 64, end = min(ncols, p.N - n0);
    bulk_wait_read<0>();
    for (int i = 0; i < NSLOT && i * bw < end; ++i) load(q, (pc + i) % NSLOT, n0 + i * bw, row0);
  }
  // before the CTA leaves: stores have been written, loads (of a tile that was given up) have landed or are given up on
  __device__ __forceinline__ void drain(int lane) {
    if (lane != 0) return;
    for (int i = 0; i < NSLOT; ++i) if ((loading >> i) & 1u) mbar_wait(rbar0 + 8u * i, (rph >> i) & 1u);
    bulk_wait_all();
  }
  __device__ __forceinline__ void run(const Problem& q, const Params& p, uint32_t tmem_acc, int row0, int rowoff, int n0, int ncols, int lane, volatile uint32_t* abort_flag) {
    if (!p.tma_out) {
      const int m = row0 + lane;
#pragma unroll 1
      for (int c0 = 0; c0 < ncols; c0 += 32) {
        uint32_t r[32];
        tmem_ld32(tmem_acc + (uint32_t)c0, r);
        if (m < p.M) store_row_piece(p, rowoff + m, n0 + c0, r);
      }
      return;
    }
    if (row0 >= p.M) return;
    const bool res = loads(p);
    if (!p.red && !p.out_bf16) {
      // 16 x 8 fragments go out as they are, a quad of lanes one whole 32-byte sector, and nobody waits
      const int r = row0 + (lane >> 2), c = n0 + (lane & 3) * 2;
      float* base = static_cast<float*>(p.C) + (int64_t)(rowoff + r) * p.ldc + c;
#pragma unroll 1
      for (int c0 = 0; c0 < ncols && n0 + c0 < p.N; c0 += 32) {
        uint32_t v[4][8];
#pragma unroll
        for (int i = 0; i < 4; ++i) tmem_ld16x256_x2(tmem_acc + ((uint32_t)(16 * (i >> 1)) << 16) + (uint32_t)(c0 + 16 * (i & 1)), v[i]);
        tmem_wait_ld();
        if (p.R) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              uint32_t* w = &v[i][4 * (e >> 1) + 2 * (e & 1)];
              w[0] = __float_as_uint(__uint_as_float(w[0]) + __uint_as_float(rr[4 * i + e].x));
              w[1] = __float_as_uint(__uint_as_float(w[1]) + __uint_as_float(rr[4 * i + e].y));
            }
          if (c0 + 32 < ncols && n0 + c0 + 32 < p.N) fetch(p, row0, n0, c0 + 32, lane);
        }
        const bool whole = row0 + 32 <= p.M && n0 + c0 + 32 <= p.N;
        auto put = [&](bool inside) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) {                   // e & 1: row + 8, e >> 1: columns + 8
              const int dr = 16 * (i >> 1) + 8 * (e & 1), dc = c0 + 16 * (i & 1) + 8 * (e >> 1);
              const uint2 o = make_uint2(v[i][4 * (e >> 1) + 2 * (e & 1)], v[i][4 * (e >> 1) + 2 * (e & 1) + 1]);
              float* at = base + (int64_t)dr * p.ldc + dc;
              if (inside || (r + dr < p.M && c + dc + 1 < p.N)) *reinterpret_cast<uint2*>(at) = o;
              else if (r + dr < p.M && c + dc < p.N) *at = __uint_as_float(o.x);
            }
        };
        if (whole) put(true); else put(false);
        if (p.e_hi) {
          // the same values as a (hi, lo) bf16 pair: neighbouring lanes swap halves, so that a lane has four columns of one of two octets
          const bool odd = lane & 1;
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int row = r + 16 * (i >> 1) + 8 * e, c16 = n0 + c0 + 16 * (i & 1);
              uint32_t h0, l0, h1, l1;
              split2(__uint_as_float(v[i][2 * e]), __uint_as_float(v[i][2 * e + 1]), h0, l0, true);
              split2(__uint_as_float(v[i][4 + 2 * e]), __uint_as_float(v[i][4 + 2 * e + 1]), h1, l1, true);
              const uint32_t gh = __shfl_xor_sync(0xffffffffu, odd ? h0 : h1, 1), gl = __shfl_xor_sync(0xffffffffu, odd ? l0 : l1, 1);
              const uint2 h = odd ? make_uint2(gh, h1) : make_uint2(h0, gh), l = odd ? make_uint2(gl, l1) : make_uint2(l0, gl);
              const int col = c16 + ((lane & 3) * 2) + (odd ? 6 : 0);      // first of the lane's four columns
              if (row >= p.M) continue;
              uint16_t* eh = p.e_hi + (int64_t)row * p.lde + col;
              uint16_t* el = p.e_lo + (int64_t)row * p.lde + col;
              if (whole || col + 4 <= p.N) { *reinterpret_cast<uint2*>(eh) = h; *reinterpret_cast<uint2*>(el) = l; }
              else
                for (int j = 0; j < 4 && col + j < p.N; ++j) {
                  eh[j] = (uint16_t)((j < 2 ? h.x : h.y) >> (16 * (j & 1))); el[j] = (uint16_t)((j < 2 ? l.x : l.y) >> (16 * (j & 1)));
                }
            }
        }
      }
      return;
    }
    const int bw = p.out_bf16 ? 64 : 32, end = min(ncols, p.N - n0);
#pragma unroll 1
    for (int c0 = 0; c0 < end; c0 += bw) {
      const uint32_t slot = pc % NSLOT, sbase = slot0 + slot * EPI_SLOT_BYTES + (uint32_t)lane * 128u;
      bool landed = res;
      if (res) {
        landed = __all_sync(0xffffffffu, mbar_wait(rbar0 + 8u * slot, (rph >> slot) & 1u));
        rph ^= 1u << slot;
        loading &= ~(1u << slot);
        if (!landed && lane == 0) { atomicOr(&g_bf16_status, 16u); *abort_flag = 1; }
      }
#pragma unroll 1
      for (int half = 0; 32 * half < bw; ++half) {
        uint32_t r[32];
        tmem_ld32(tmem_acc + (uint32_t)(c0 + 32 * half), r);
        if (p.out_bf16) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const uint32_t at = sbase + (uint32_t)(((4 * half + j) ^ (lane & 7)) * 16);
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(r[8 * j + e]);
            if (landed) {
              uint32_t w[4];
              asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(at));
#pragma unroll
              for (int e = 0; e < 4; ++e) { v[2 * e] += __uint_as_float(w[e] << 16); v[2 * e + 1] += __uint_as_float(w[e] & 0xffff0000u); }
            }
            uint32_t o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = bf16_of_two(v[2 * e], v[2 * e + 1]);
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
          }
          continue;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(sbase + (uint32_t)((j ^ (lane & 7)) * 16)),
                       "r"(r[4 * j]), "r"(r[4 * j + 1]), "r"(r[4 * j + 2]), "r"(r[4 * j + 3]) : "memory");
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      ++pc;
      if (lane == 0) {
        if (p.red) tma_add_2d(&q.mC, slot0 + slot * EPI_SLOT_BYTES, n0 + c0, rowoff + row0);
        else tma_store_2d(&q.mC, slot0 + slot * EPI_SLOT_BYTES, n0 + c0, rowoff + row0);
        bulk_commit();
        if (res && c0 + NSLOT * bw < end) {
          bulk_wait_read<0>();
          load(q, slot, n0 + c0 + NSLOT * bw, row0);
        } else {
          bulk_wait_read<NSLOT - 1>();       // the next slot's last store has read its data
        }
      }
      __syncwarp();
    }
  }
};

// Persistent: CTA b works on tiles b, b + gridDim.x, ... of the group.  The operand ring and its phases run on
// across tiles, so the producer is already loading the next tile while the last k-tiles of this one are
// multiplied; the accumulator alternates between two 128-column TMEM buffers, so the epilogue warps drain tile i
// while the tensor core fills tile i + 1.
//   full[s] / empty[s]        operand stage s landed / consumed
//   acc_full[b] / acc_empty[b] accumulator b complete / drained by all four epilogue warps
//   rbar[w][slot]             residual block landed in epilogue warp w's staging slot
// fp32 results leave through shared memory: each epilogue warp writes its 32 rows x 32 columns into a swizzled
// 4 KiB slot (conflict-free 16-byte stores) and one lane hands the slot to a TMA store, which writes whole
// 128-byte row segments and clips at the matrix edge; two slots per warp, so a store is in flight while the next
// block is formed.  The residual block, when there is one, is loaded into the slot first and added in place.
template <bool SPLIT>
__global__ void __launch_bounds__(NTHREADS, 1)
gemm_bf16_kernel(const __grid_constant__ Group g, const int total_tiles, unsigned long long* __restrict__ sched, const unsigned long long ticket0) {
  constexpr int STAGES = Cfg<SPLIT>::STAGES;
  constexpr int STAGE_BYTES = Cfg<SPLIT>::STAGE_BYTES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t tiles = (raw + 1023u) & ~1023u;
  uint8_t* tiles_ptr = smem_raw + (tiles - raw);
  const uint32_t epi = tiles + STAGES * STAGE_BYTES;                 // 4 warps x 2 slots x 4 KiB
  const uint32_t bars = epi + EPI_BYTES;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
  auto acc_full = [&](int b) { return bars + 8u * (2 * STAGES + b); };
  auto acc_empty = [&](int b) { return bars + 8u * (2 * STAGES + 2 + b); };
  auto r_bar = [&](int w, int slot) { return bars + 8u * (2 * STAGES + 4 + 2 * w + slot); };
  auto tq_full = [&](int i) { return bars + 8u * (2 * STAGES + 12 + i); };
  auto tq_empty = [&](int i) { return bars + 8u * (2 * STAGES + 12 + NQ + i); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(tiles_ptr + STAGES * STAGE_BYTES + EPI_BYTES + 8 * (2 * STAGES + 12 + 2 * NQ));
  volatile uint32_t* abort_flag = tmem_slot + 1;
  volatile int* tile_q = reinterpret_cast<volatile int*>(tmem_slot + 2);      // NQ tile ids handed from the producer to the other roles
  // CTA b starts with tile b; every further tile is handed out by a device-wide ticket counter (*sched), so a CTA
  // that starts late (its SM was busy with another stream's kernel) finds the rest of the work already taken instead
  // of holding its share back.  A launch draws exactly total_tiles tickets (one per processed tile), so the counter
  // is never reset: ticket t stands for tile gridDim.x + (t - ticket0) % total_tiles, where ticket0 is the counter's
  // value before the launch (launches outside stream capture) or 0 (a captured launch, which owns its counter and
  // advances it by total_tiles per replay).  sched == NULL: CTA b takes tiles b, b + gridDim.x, ...
  auto ticket_tile = [&](unsigned long long t) { return (int)gridDim.x + (int)((t - ticket0) % (unsigned long long)total_tiles); };

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 4); }
    for (int w = 0; w < 4; ++w) { mbar_init(r_bar(w, 0), 1); mbar_init(r_bar(w, 1), 1); }
    for (int i = 0; i < NQ; ++i) { mbar_init(tq_full(i), 1); mbar_init(tq_empty(i), 5); }    // readers: the MMA thread + four epilogue warps
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // The producer needs the barriers (its own thread initialised them) but not the TMEM address: warp 0 only arrives at
  // the set-up barrier and starts loading while warp 1's TMEM allocation is still under way; the other warps wait.
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  if (warp == 0) { __syncwarp(); asm volatile("bar.arrive 1, %0;" ::"n"(NTHREADS) : "memory"); }
  else asm volatile("bar.sync 1, %0;" ::"n"(NTHREADS) : "memory");
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = warp == 0 ? 0u : *tmem_slot;
  pdl_launch();
  pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      int s = 0; uint32_t ph = 0;
      int in_flight = 0;                       // stages armed and possibly not yet landed (for the abort drain)
      bool stop = false;
      int tid = (int)blockIdx.x;
      for (int it = 0; !stop; ++it) {
        // publish this tile (or the end mark) to the MMA and epilogue roles
        const int qs = it % NQ;
        if (!mbar_wait(tq_empty(qs), (((uint32_t)(it / NQ)) & 1u) ^ 1u)) { atomicOr(&g_bf16_status, 32u); *abort_flag = 1; break; }
        tile_q[qs] = tid < total_tiles ? tid : -1;
        mbar_arrive(tq_full(qs));
        if (tid >= total_tiles) break;
        // the next ticket is requested now and used after this tile's loads
        unsigned long long next_ticket = 0;
        if (sched) next_ticket = atomicAdd(sched, 1ull);
        int tile;
        const Problem& q = g.pr[pick_problem(g, tid, &tile)];
        const Params& p = q.p;
        int kt0, kt1;
        split_of(q, &tile, &kt0, &kt1);
        const int m0 = (tile / q.tiles_n) * TBM, n0 = (tile % q.tiles_n) * TBN;
        for (int kt = kt0; kt < kt1; ++kt) {
          if (!mbar_wait(empty_bar(s), ph ^ 1u)) { atomicOr(&g_bf16_status, 1u); *abort_flag = 1; stop = true; break; }
          if (*abort_flag) { stop = true; break; }
          const uint32_t a_dst = tiles + s * STAGE_BYTES, b_dst = a_dst + TILE_BYTES;
          mbar_expect_tx(full_bar(s), STAGE_BYTES);
          const int k0 = kt * TBK;
          if (!p.a_mn_major) {
            tma_load_2d(a_dst, &q.mA, k0, m0, full_bar(s));
          } else {
#pragma unroll
            for (int j = 0; j < TBM / 64; ++j) tma_load_2d(a_dst + j * (TBK * 128), &q.mA, m0 + 64 * j, k0, full_bar(s));
          }
          if (!p.b_mn_major) {
            tma_load_2d(b_dst, &q.mB, k0, n0, full_bar(s));
          } else {
#pragma unroll
            for (int j = 0; j < TBN / 64; ++j) tma_load_2d(b_dst + j * (TBK * 128), &q.mB, n0 + 64 * j, k0, full_bar(s));
          }
          if (SPLIT) {
            const uint32_t al_dst = a_dst + 2 * TILE_BYTES, bl_dst = al_dst + TILE_BYTES;
            if (!p.a_mn_major) {
              tma_load_2d(al_dst, &q.mAlo, k0, m0, full_bar(s));
            } else {
#pragma unroll
              for (int j = 0; j < TBM / 64; ++j) tma_load_2d(al_dst + j * (TBK * 128), &q.mAlo, m0 + 64 * j, k0, full_bar(s));
            }
            if (!p.b_mn_major) {
              tma_load_2d(bl_dst, &q.mBlo, k0, n0, full_bar(s));
            } else {
#pragma unroll
              for (int j = 0; j < TBN / 64; ++j) tma_load_2d(bl_dst + j * (TBK * 128), &q.mBlo, n0 + 64 * j, k0, full_bar(s));
            }
          }
          if (in_flight < STAGES) ++in_flight;
          if (++s == STAGES) { s = 0; ph ^= 1u; }
        }
        tid = sched ? ticket_tile(next_ticket) : tid + (int)gridDim.x;
      }
      if (*abort_flag) {
        // the copies already issued still land in this CTA's shared memory: wait (bounded) for each before leaving
        for (int i = 0; i < in_flight; ++i) {
          if (--s < 0) { s = STAGES - 1; ph ^= 1u; }
          mbar_wait(full_bar(s), ph);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t d_hi = desc_hi(1024, 2);
      constexpr uint32_t LO_OFF = (2 * TILE_BYTES) >> 4;        // from the hi tiles of a stage to its lo tiles
      int s = 0; uint32_t ph = 0;
      bool stop = false;
      for (int it = 0; !stop; ++it) {
        const int qs = it % NQ;
        if (!mbar_wait(tq_full(qs), ((uint32_t)(it / NQ)) & 1u)) { atomicOr(&g_bf16_status, 64u); *abort_flag = 1; break; }
        const int tid = tile_q[qs];
        mbar_arrive(tq_empty(qs));
        if (tid < 0) break;
        int tile;
        const Problem& q = g.pr[pick_problem(g, tid, &tile)];
        const Params& p = q.p;
        int kt0, kt1;
        split_of(q, &tile, &kt0, &kt1);
        // kind::f16 descriptor: fp32 accumulate (bit 4), A/B format bf16 (=1) at bits 7 and 10, majorness, N, M
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)p.a_mn_major << 15) | ((uint32_t)p.b_mn_major << 16) |
                               ((uint32_t)(TBN >> 3) << 17) | ((uint32_t)(TBM >> 4) << 24);
        // K-major: 8-row groups 1024 B apart, one MMA (K=16) advances 32 B inside the 128-byte row.
        // MN-major: blocks of 64 elements TBK*128 B apart (LBO), 8-k-row groups 1024 B apart (SBO); K=16 spans two groups.
        const uint32_t a_lbo = p.a_mn_major ? TBK * 128 : 16, b_lbo = p.b_mn_major ? TBK * 128 : 16;
        const uint32_t a_step = (p.a_mn_major ? 2048u : 32u) >> 4, b_step = (p.b_mn_major ? 2048u : 32u) >> 4;
        const int b = it & 1;
        if (!mbar_wait(acc_empty(b), (((uint32_t)it >> 1) & 1u) ^ 1u)) { atomicOr(&g_bf16_status, 4u); *abort_flag = 1; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem_acc = tmem_base + (uint32_t)(b * TBN);
        for (int kt = kt0; kt < kt1; ++kt) {
          if (!mbar_wait(full_bar(s), ph)) { atomicOr(&g_bf16_status, 2u); *abort_flag = 1; stop = true; break; }
          if (*abort_flag) { stop = true; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_s = tiles + s * STAGE_BYTES;
          uint32_t al = desc_lo(a_s, a_lbo), bl = desc_lo(a_s + TILE_BYTES, b_lbo);
#pragma unroll
          for (int k = 0; k < TBK / 16; ++k) {
            const uint32_t acc = (kt > kt0 || k > 0) ? 1u : 0u;
            if (SPLIT) {
              mma_f16_h(tmem_acc, al + LO_OFF, d_hi, bl, d_hi, idesc, acc);
              mma_f16_h(tmem_acc, al, d_hi, bl + LO_OFF, d_hi, idesc, 1u);
              mma_f16_h(tmem_acc, al, d_hi, bl, d_hi, idesc, 1u);
            } else {
              mma_f16_h(tmem_acc, al, d_hi, bl, d_hi, idesc, acc);
            }
            al += a_step; bl += b_step;
          }
          umma_commit(empty_bar(s));
          if (++s == STAGES) { s = 0; ph ^= 1u; }
        }
        if (!stop) umma_commit(acc_full(b));
      }
    }
  } else {
    const int ew = warp - 2;                       // staging slots and residual barriers of this warp
    const int quarter = warp & 3;                  // the TMEM lanes this warp may read
    Epilogue<2> est{epi + (uint32_t)ew * (2 * EPI_SLOT_BYTES), r_bar(ew, 0)};
    for (int it = 0;; ++it) {
      const int qs = it % NQ;
      const bool have = __all_sync(0xffffffffu, mbar_wait_idle(tq_full(qs), ((uint32_t)(it / NQ)) & 1u));
      if (!have) { if (lane == 0) { atomicOr(&g_bf16_status, 128u); *abort_flag = 1; } break; }
      const int tid = tile_q[qs];
      __syncwarp();
      if (lane == 0) mbar_arrive(tq_empty(qs));
      if (tid < 0) break;
      int tile;
      const Problem& q = g.pr[pick_problem(g, tid, &tile)];
      const Params& p = q.p;
      int kt0, kt1;
      const int rowoff = split_of(q, &tile, &kt0, &kt1) * p.slab_rows;
      const int m0 = (tile / q.tiles_n) * TBM, n0 = (tile % q.tiles_n) * TBN;
      const int b = it & 1;
      est.prefetch(q, p, m0 + quarter * 32, n0, TBN, lane);
      const bool acc_ok = __all_sync(0xffffffffu, mbar_wait_idle(acc_full(b), ((uint32_t)it >> 1) & 1u));
      if (!acc_ok && lane == 0) { atomicOr(&g_bf16_status, 8u); *abort_flag = 1; }
      if (!acc_ok || __any_sync(0xffffffffu, *abort_flag != 0)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tmem_acc = tmem_base + (uint32_t)(b * TBN) + ((uint32_t)(quarter * 32) << 16);
      const int row0 = m0 + quarter * 32;
      est.run(q, p, tmem_acc, row0, rowoff, n0, TBN, lane, abort_flag);
      // every TMEM read of this warp has completed (tcgen05.wait::ld): hand the accumulator back
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty(b));
    }
    est.drain(lane);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// ---- CTA-pair variant ------------------------------------------------------------------------------------
// Two CTAs of a cluster (a CTA pair) own one 256x256 output tile.  Each loads its 128 rows of A and its 128
// columns of B (64 KiB per k-tile with pairs, 32 KiB without, exactly what a 128x128 single-CTA tile loads) and
// the leader issues tcgen05.mma.cta_group::2 with M = 256, N = 256: each SM multiplies its A rows by the B
// columns of both, so a byte fetched from L2 feeds twice the tensor work.  The 128x128 kernel above is bound by
// L2 -> shared-memory traffic at these shapes; this one halves that traffic per flop.
//   full_bar[s]  (leader's copy): both CTAs' loads complete their bytes on it
//   empty_bar[s] (one per CTA):   the leader commits the k-tile's MMAs to both, freeing the stage in both CTAs
//   accum_bar    (one per CTA):   the leader commits the last MMAs to both; each CTA drains its own 128 TMEM lanes
// Every wait is bounded; a CTA that gives up records it, stops issuing work and still joins the closing
// cluster barrier, so its peer never waits for it unboundedly.
// stage = A tile (128 x 64) + B tile (BN2/2 x 64), twice that with pairs; as many stages as fit in 192 KiB
template <bool SPLIT, int BN2> struct PairCfg {
  static constexpr int STAGE_BYTES = (SPLIT ? 2 : 1) * (TILE_BYTES + (BN2 / 2) * TBK * 2);
  static constexpr int STAGES = (192 * 1024) / STAGE_BYTES > 8 ? 8 : (192 * 1024) / STAGE_BYTES;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
};
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t map_to_cta(uint32_t saddr, uint32_t rank) {
  uint32_t r; asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank)); return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// tile load issued by either CTA of the pair, completing bytes on a barrier given as a cluster address
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar_cluster_addr) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(bar_cluster_addr)
      : "memory");
}
__device__ __forceinline__ void mma_bf16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}
__device__ __forceinline__ void umma_commit_pair(uint32_t bar_cluster_addr) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_cluster_addr) : "memory");
}

// the same to the barrier at this offset in both CTAs of the pair
__device__ __forceinline__ void umma_commit_both(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}

// BN2 = width of the pair's tile (256 or 128); each CTA loads BN2/2 columns of B.
template <bool SPLIT, int BN2>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NTHREADS, 1)
gemm_bf16_pair_kernel(const __grid_constant__ Group g) {
  const uint32_t rank = cluster_rank();
  const int cluster_id = (int)(blockIdx.x >> 1);
  int tile;
  const int which = pick_problem(g, cluster_id, &tile);
  const Problem& q = g.pr[which];
  const Params& p = q.p;
  constexpr int BNH = BN2 / 2;                       // B columns (rows of the K-major tile) per CTA
  constexpr int TILE_B = BNH * TBK * 2;
  constexpr int HALF_BYTES = TILE_BYTES + TILE_B;    // one A tile + one B tile
  constexpr int STAGE_BYTES = PairCfg<SPLIT, BN2>::STAGE_BYTES;
  constexpr int STAGES = PairCfg<SPLIT, BN2>::STAGES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t tiles = (raw + 1023u) & ~1023u;
  uint8_t* tiles_ptr = smem_raw + (tiles - raw);
  const uint32_t bars = tiles + STAGES * STAGE_BYTES;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
  const uint32_t accum_bar = bars + 8u * (2 * STAGES);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(tiles_ptr + STAGES * STAGE_BYTES + 8 * (2 * STAGES + 1));
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int m0 = (tile / q.tiles_n) * 256 + (int)rank * TBM;     // this CTA's rows of A and of the output
  const int n0 = (tile % q.tiles_n) * BN2;                      // the pair's columns; this CTA loads B columns n0 + rank*128 ..
  const int nb0 = n0 + (int)rank * BNH;
  const int num_kt = (p.K + TBK - 1) / TBK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    mbar_init(accum_bar, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "r"(BN2) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();     // both CTAs' barriers are initialised before either signals the other's
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_acc = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int armed = 0;
      for (int kt = 0; kt < num_kt; ++kt) {
        const int s = kt % STAGES;
        const uint32_t ph = (kt / STAGES) & 1;
        if (!mbar_wait(empty_bar(s), ph ^ 1u)) { atomicOr(&g_bf16_status, 1u); *abort_flag = 1; break; }
        if (*abort_flag) break;
        const uint32_t a_dst = tiles + s * STAGE_BYTES, b_dst = a_dst + TILE_BYTES;
        const uint32_t fb = map_to_cta(full_bar(s), 0);            // the leader's barrier collects both CTAs' bytes
        if (rank == 0) mbar_expect_tx(full_bar(s), 2 * STAGE_BYTES);
        const int k0 = kt * TBK;
        if (!p.a_mn_major) {
          tma_load_2d_pair(a_dst, &q.mA, k0, m0, fb);
        } else {
#pragma unroll
          for (int j = 0; j < TBM / 64; ++j) tma_load_2d_pair(a_dst + j * (TBK * 128), &q.mA, m0 + 64 * j, k0, fb);
        }
        if (!p.b_mn_major) {
          tma_load_2d_pair(b_dst, &q.mB, k0, nb0, fb);
        } else {
#pragma unroll
          for (int j = 0; j < BNH / 64; ++j) tma_load_2d_pair(b_dst + j * (TBK * 128), &q.mB, nb0 + 64 * j, k0, fb);
        }
        if (SPLIT) {
          const uint32_t al_dst = a_dst + HALF_BYTES, bl_dst = al_dst + TILE_BYTES;
          if (!p.a_mn_major) {
            tma_load_2d_pair(al_dst, &q.mAlo, k0, m0, fb);
          } else {
#pragma unroll
            for (int j = 0; j < TBM / 64; ++j) tma_load_2d_pair(al_dst + j * (TBK * 128), &q.mAlo, m0 + 64 * j, k0, fb);
          }
          if (!p.b_mn_major) {
            tma_load_2d_pair(bl_dst, &q.mBlo, k0, nb0, fb);
          } else {
#pragma unroll
            for (int j = 0; j < BNH / 64; ++j) tma_load_2d_pair(bl_dst + j * (TBK * 128), &q.mBlo, nb0 + 64 * j, k0, fb);
          }
        }
        armed = kt + 1;
      }
      // after giving up, the leader still waits (bounded) for the loads both CTAs have in flight
      if (*abort_flag && rank == 0)
        for (int kt = max(0, armed - STAGES); kt < armed; ++kt) mbar_wait(full_bar(kt % STAGES), (kt / STAGES) & 1);
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      // M = 256 (two CTAs x 128 rows), N = 256
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)p.a_mn_major << 15) | ((uint32_t)p.b_mn_major << 16) |
                             ((uint32_t)(BN2 >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
      const uint32_t a_lbo = p.a_mn_major ? TBK * 128 : 16, b_lbo = p.b_mn_major ? TBK * 128 : 16;
      const uint32_t d_hi = desc_hi(1024, 2);
      const uint32_t a_step = (p.a_mn_major ? 2048u : 32u) >> 4, b_step = (p.b_mn_major ? 2048u : 32u) >> 4;
      constexpr uint32_t LO_OFF = HALF_BYTES >> 4;
      // the barriers of both CTAs as cluster addresses, once
      uint32_t eb0[STAGES], eb1[STAGES];
#pragma unroll
      for (int i = 0; i < STAGES; ++i) { eb0[i] = map_to_cta(empty_bar(i), 0); eb1[i] = map_to_cta(empty_bar(i), 1); }
      int s = 0; uint32_t ph = 0;
      for (int kt = 0; kt < num_kt; ++kt) {
        if (!mbar_wait(full_bar(s), ph)) { atomicOr(&g_bf16_status, 2u); *abort_flag = 1; break; }
        if (*abort_flag) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t a_s = tiles + s * STAGE_BYTES;
        uint32_t al = desc_lo(a_s, a_lbo), bl = desc_lo(a_s + TILE_BYTES, b_lbo);
#pragma unroll
        for (int k = 0; k < TBK / 16; ++k) {
          const uint32_t acc = (kt > 0 || k > 0) ? 1u : 0u;
          if (SPLIT) {
            mma_f16_pair_h(tmem_acc, al + LO_OFF, d_hi, bl, d_hi, idesc, acc);
            mma_f16_pair_h(tmem_acc, al, d_hi, bl + LO_OFF, d_hi, idesc, 1u);
            mma_f16_pair_h(tmem_acc, al, d_hi, bl, d_hi, idesc, 1u);
          } else {
            mma_f16_pair_h(tmem_acc, al, d_hi, bl, d_hi, idesc, acc);
          }
          al += a_step; bl += b_step;
        }
        // the commits go through a switch on the stage so that the cluster addresses stay in registers
#pragma unroll
        for (int i = 0; i < STAGES; ++i)
          if (i == s) { umma_commit_pair(eb0[i]); umma_commit_pair(eb1[i]); }
        if (++s == STAGES) { s = 0; ph ^= 1u; }
      }
      umma_commit_pair(map_to_cta(accum_bar, 0));
      umma_commit_pair(map_to_cta(accum_bar, 1));
    }
  } else {
    const bool acc_ok = __all_sync(0xffffffffu, mbar_wait_idle(accum_bar, 0));
    if (!acc_ok && lane == 0) { atomicOr(&g_bf16_status, 8u); *abort_flag = 1; }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const bool aborted = __any_sync(0xffffffffu, *abort_flag != 0);
    if (acc_ok && !aborted) {
      const int lane_base = (warp & 3) * 32;
      const int m = m0 + lane_base + lane;
#pragma unroll 1
      for (int c0 = 0; c0 < BN2; c0 += 32) {
        if (n0 + c0 >= p.N) break;      // uniform
        uint32_t r[32];
        tmem_ld32(tmem_acc + ((uint32_t)lane_base << 16) + (uint32_t)c0, r);
        if (m < p.M) store_row_piece(p, m, n0 + c0, r);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();     // neither CTA leaves (or frees TMEM) while the other may still read its shared memory or signal its barriers
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_acc), "r"(BN2) : "memory");
  }
}

// ---- persistent CTA-pair variant ----------------------------------------------------------------------------
// (BN2 = the widest tile; a problem may ask for 128-wide ones, see choose_widths.)
// What bounds it: at long K the tensor cores under the power limit (8192^3 plain: 946 us when single lanes issued loads and MMAs from
// inside `if (lane == 0)`, 791 us = 1390 TFLOP/s with one elected lane of a converged warp and one commit for both CTAs); at K = 768 the
// 256 KB of fp32 that a tile writes.  Four epilogue warps were the limit there: products with a bf16 residual 67 -> 40 us, the two
// gradients of in_proj at 16384 tokens 165 -> 129, of the tied head per 1024 rows 339 -> 254.
// The warp index is a shuffle's result, so that the roles' branches are uniform to the compiler: 2 % of the training steps' products.
// Plain products of 16384 x 4096 x 768 take 65 us without an epilogue, 66 with the accumulators read, 82 with bf16 results, 104 with fp32
// ones: the results' bytes at HBM's rate on top of the products, however they leave (fragments, slots and TMA, whole lines through shared
// memory) and whenever (paced over the next tile, clusters staggered).  Tiles of 512 columns, one pass over A for both accumulators: 107 and 130.
// The CTA-pair kernel above as a tile loop: cluster c works on tiles c, c + clusters, ...; the operand ring keeps
// running across tiles; the accumulator alternates between two TMEM buffers of BN2 columns, so each CTA drains its
// 128 rows of tile i (through the same TMA-store epilogue as the single-CTA kernel) while the leader issues tile
// i + 1.  The epilogue warps of BOTH CTAs hand a buffer back by arriving on the leader's acc_empty barrier.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}
template <bool SPLIT, int BN2> struct PairPCfg {
  static constexpr int STAGE_BYTES = PairCfg<SPLIT, BN2>::STAGE_BYTES;
  // eight epilogue warps (two per TMEM quarter, half of the columns each) with a staging slot each
  static constexpr int EPI_WARPS = 8, THREADS = 32 * (2 + EPI_WARPS);
  static constexpr int NSLOT = 1, RING = 192 * 1024;
  static constexpr int STAGES = RING / STAGE_BYTES > 8 ? 8 : RING / STAGE_BYTES;
  static constexpr int EPI = EPI_WARPS * NSLOT * EPI_SLOT_BYTES;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI + 1024 + 512;
  static constexpr int TMEM = 2 * BN2;
};

template <bool SPLIT, int BN2>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairPCfg<SPLIT, BN2>::THREADS, 1)
gemm_bf16_pairp_kernel(const __grid_constant__ Group g, const int total_tiles) {
  const uint32_t rank = cluster_rank();
  const int cluster_id = (int)(blockIdx.x >> 1), nclusters = (int)(gridDim.x >> 1);
  constexpr int BNH = BN2 / 2;
  constexpr int TILE_B = BNH * TBK * 2;
  constexpr int HALF_BYTES = TILE_BYTES + TILE_B;
  constexpr int STAGE_BYTES = PairPCfg<SPLIT, BN2>::STAGE_BYTES;
  constexpr int STAGES = PairPCfg<SPLIT, BN2>::STAGES, NSLOT = PairPCfg<SPLIT, BN2>::NSLOT, EPI = PairPCfg<SPLIT, BN2>::EPI;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t tiles = (raw + 1023u) & ~1023u;
  uint8_t* tiles_ptr = smem_raw + (tiles - raw);
  const uint32_t epi = tiles + STAGES * STAGE_BYTES;
  const uint32_t bars = epi + EPI;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
  auto acc_full = [&](int b) { return bars + 8u * (2 * STAGES + b); };
  auto acc_empty = [&](int b) { return bars + 8u * (2 * STAGES + 2 + b); };
  auto r_bar = [&](int w, int slot) { return bars + 8u * (2 * STAGES + 4 + NSLOT * w + slot); };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(tiles_ptr + STAGES * STAGE_BYTES + EPI + 8 * (2 * STAGES + 4 + PairPCfg<SPLIT, BN2>::EPI_WARPS * NSLOT));
  volatile uint32_t* abort_flag = tmem_slot + 1;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(acc_full(b), 1); mbar_init(acc_empty(b), 2 * PairPCfg<SPLIT, BN2>::EPI_WARPS); }
    for (int w = 0; w < PairPCfg<SPLIT, BN2>::EPI_WARPS * NSLOT; ++w) mbar_init(r_bar(0, w), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "n"(PairPCfg<SPLIT, BN2>::TMEM) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();     // both CTAs' barriers are initialised before either signals the other's
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch();
  pdl_wait();

  if (warp == 0) {
    // (the whole warp waits, one elected lane issues)
    int s = 0; uint32_t ph = 0;
    int in_flight = 0;
    bool stop = false;
    const uint32_t fb0 = map_to_cta(full_bar(0), 0);               // the leader's barriers collect both CTAs' bytes
    for (int j = 0; !stop; ++j) {
      const int tid = pair_tile_at(g, cluster_id, nclusters, j);
      if (tid >= total_tiles) break;
      int tile, kt0, kt1;
      const Problem& q = g.pr[pick_problem(g, tid, &tile)];
      const Params& p = q.p;
      split_of(q, &tile, &kt0, &kt1);
      const int m0 = (tile / q.tiles_n) * 256 + (int)rank * TBM, bnh = p.bn >> 1;      // (tiles of bn <= BN2 columns)
      const int nb0 = q.n_begin + (tile % q.tiles_n) * p.bn + (int)rank * bnh;
      const uint32_t tx = 2u * (uint32_t)(STAGE_BYTES - (SPLIT ? 2 : 1) * (BNH - bnh) * TBK * 2);
      const bool amn = p.a_mn_major, bmn = p.b_mn_major, wide = BNH > 64 && bnh > 64;
      for (int kt = kt0; kt < kt1; ++kt) {
        const bool got = __all_sync(0xffffffffu, mbar_wait(empty_bar(s), ph ^ 1u));
        if (!got && lane == 0) { atomicOr(&g_bf16_status, 1u); *abort_flag = 1; }
        if (!got || __any_sync(0xffffffffu, *abort_flag != 0)) { stop = true; break; }
        const uint32_t a_dst = tiles + s * STAGE_BYTES, b_dst = a_dst + TILE_BYTES, fb = fb0 + 8u * s;
        const int k0 = kt * TBK;
        if (elect_one()) {
          if (rank == 0) mbar_expect_tx(full_bar(s), tx);
          auto load = [&](uint32_t dst, const CUtensorMap* map, bool mn, int row0, bool two) {
            if (!mn) { tma_load_2d_pair(dst, map, k0, row0, fb); return; }
            tma_load_2d_pair(dst, map, row0, k0, fb);
            if (two) tma_load_2d_pair(dst + TBK * 128, map, row0 + 64, k0, fb);
          };
          load(a_dst, &q.mA, amn, m0, true);
          load(b_dst, &q.mB, bmn, nb0, wide);
          if (SPLIT) {
            load(a_dst + HALF_BYTES, &q.mAlo, amn, m0, true);
            load(b_dst + HALF_BYTES, &q.mBlo, bmn, nb0, wide);
          }
        }
        __syncwarp();
        if (in_flight < STAGES) ++in_flight;
        if (++s == STAGES) { s = 0; ph ^= 1u; }
      }
    }
    // after giving up, the leader still waits (bounded) for the loads both CTAs have in flight
    if (*abort_flag && rank == 0 && lane == 0) {
      for (int i = 0; i < in_flight; ++i) {
        if (--s < 0) { s = STAGES - 1; ph ^= 1u; }
        mbar_wait(full_bar(s), ph);
      }
    }
  } else if (warp == 1) {
    // The whole warp of the leader waits and one elected lane issues: descriptors then stay in uniform registers, and a k-tile's
    // commit reaches both CTAs as one instruction (see the comment above the kernel for what that gave).
    if (rank == 0) {
      const uint32_t d_hi = desc_hi(1024, 2);
      constexpr uint32_t LO_OFF = HALF_BYTES >> 4;
      int s = 0; uint32_t ph = 0;
      bool stop = false;
      for (int it = 0; !stop; ++it) {
        const int tid = pair_tile_at(g, cluster_id, nclusters, it);
        if (tid >= total_tiles) break;
        int tile, kt0, kt1;
        const Problem& q = g.pr[pick_problem(g, tid, &tile)];
        const Params& p = q.p;
        split_of(q, &tile, &kt0, &kt1);
        // M = 256 (two CTAs x 128 rows), N = bn
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)p.a_mn_major << 15) | ((uint32_t)p.b_mn_major << 16) |
                               ((uint32_t)(p.bn >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
        const uint32_t a_lbo = p.a_mn_major ? TBK * 128 : 16, b_lbo = p.b_mn_major ? TBK * 128 : 16;
        const uint32_t a_step = (p.a_mn_major ? 2048u : 32u) >> 4, b_step = (p.b_mn_major ? 2048u : 32u) >> 4;
        const int b = it & 1;
        if (!__all_sync(0xffffffffu, mbar_wait(acc_empty(b), (((uint32_t)it >> 1) & 1u) ^ 1u))) {
          if (lane == 0) { atomicOr(&g_bf16_status, 4u); *abort_flag = 1; }
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tmem_acc = tmem_base + (uint32_t)(b * BN2);
        for (int kt = kt0; kt < kt1; ++kt) {
          const bool got = __all_sync(0xffffffffu, mbar_wait(full_bar(s), ph));
          if (!got && lane == 0) { atomicOr(&g_bf16_status, 2u); *abort_flag = 1; }
          if (!got || __any_sync(0xffffffffu, *abort_flag != 0)) { stop = true; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_s = tiles + s * STAGE_BYTES;
          const uint32_t al0 = desc_lo(a_s, a_lbo), bl0 = desc_lo(a_s + TILE_BYTES, b_lbo);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < TBK / 16; ++k) {
              const uint32_t acc = (kt > kt0 || k > 0) ? 1u : 0u, al = al0 + k * a_step, bl = bl0 + k * b_step;
              if (SPLIT) {
                mma_f16_pair_h(tmem_acc, al + LO_OFF, d_hi, bl, d_hi, idesc, acc);
                mma_f16_pair_h(tmem_acc, al, d_hi, bl + LO_OFF, d_hi, idesc, 1u);
                mma_f16_pair_h(tmem_acc, al, d_hi, bl, d_hi, idesc, 1u);
              } else {
                mma_f16_pair_h(tmem_acc, al, d_hi, bl, d_hi, idesc, acc);
              }
            }
            umma_commit_both(empty_bar(s));
          }
          __syncwarp();
          if (++s == STAGES) { s = 0; ph ^= 1u; }
        }
        if (!stop && elect_one()) umma_commit_both(acc_full(b));
        __syncwarp();
      }
    }
  } else {
    const int ew = warp - 2;
    const int quarter = warp & 3, chalf = ew >> 2;             // this warp's TMEM lanes and half of the columns
    Epilogue<NSLOT> est{epi + (uint32_t)ew * (NSLOT * EPI_SLOT_BYTES), r_bar(ew, 0)};
    const uint32_t ae[2] = {map_to_cta(acc_empty(0), 0), map_to_cta(acc_empty(1), 0)};      // the leader's barriers
    int it = 0;
    for (;; ++it) {
      const int tid = pair_tile_at(g, cluster_id, nclusters, it);
      if (tid >= total_tiles) break;
      int tile, kt0, kt1;
      const Problem& q = g.pr[pick_problem(g, tid, &tile)];
      const Params& p = q.p;
      const int rowoff = split_of(q, &tile, &kt0, &kt1) * p.slab_rows;
      const int m0 = (tile / q.tiles_n) * 256 + (int)rank * TBM, cw = p.bn >> 1, n0 = q.n_begin + (tile % q.tiles_n) * p.bn + chalf * cw;
      const int b = it & 1;
      est.prefetch(q, p, m0 + quarter * 32, n0, cw, lane);
      const bool acc_ok = __all_sync(0xffffffffu, mbar_wait_idle(acc_full(b), ((uint32_t)it >> 1) & 1u));
      if (!acc_ok && lane == 0) { atomicOr(&g_bf16_status, 8u); *abort_flag = 1; }
      if (!acc_ok || __any_sync(0xffffffffu, *abort_flag != 0)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tmem_acc = tmem_base + (uint32_t)(b * BN2 + chalf * cw) + ((uint32_t)(quarter * 32) << 16);
      const int row0 = m0 + quarter * 32;
      est.run(q, p, tmem_acc, row0, rowoff, n0, cw, lane, abort_flag);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(ae[b]);
    }
    est.drain(lane);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();     // neither CTA leaves (or frees TMEM) while the other may still read its shared memory or signal its barriers
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "n"(PairPCfg<SPLIT, BN2>::TMEM) : "memory");
  }
}

struct MapKey {
  const void* base; int64_t inner, outer, ld; int bi, bo, f32;
  bool operator<(const MapKey& o) const {
    return std::tie(base, inner, outer, ld, bi, bo, f32) < std::tie(o.base, o.inner, o.outer, o.ld, o.bi, o.bo, o.f32);
  }
};
static std::map<MapKey, CUtensorMap> g_cache;   // shared by every device and host thread: guarded by g_cache_mu
static std::mutex g_cache_mu;

static pmb_status make_map(CUtensorMap* map, const void* base, int64_t inner, int64_t outer, int64_t ld, int box_inner, int box_outer,
                           bool f32 = false) {
  MapKey key{base, inner, outer, ld, box_inner, box_outer, f32 ? 1 : 0};
  std::lock_guard<std::mutex> lock(g_cache_mu);
  auto it = g_cache.find(key);
  if (it == g_cache.end()) {
    if (g_cache.size() > 8192) g_cache.clear();
    EncodeTiledFn enc = get_encode();
    if (!enc) return fail(PMB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer};
    cuuint64_t strides[1] = {(cuuint64_t)ld * (f32 ? 4 : 2)};
    cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer};
    cuuint32_t estr[2] = {1, 1};
    CUtensorMap m;
    CUresult r = enc(&m, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(PMB_ERR_CUDA, "cuTensorMapEncodeTiled (%s) failed with code %d", f32 ? "fp32" : "bf16", (int)r);
    it = g_cache.emplace(key, m).first;
  }
  *map = it->second;
  return PMB_OK;
}

// bf16 operand map for other translation units (128-byte swizzle)
pmb_status pair_operand_map(CUtensorMap* map, const uint16_t* base, int64_t inner, int64_t outer, int64_t ld, int box_inner, int box_outer) {
  return make_map(map, base, inner, outer, ld, box_inner, box_outer);
}

// Maps for the epilogue of the single-CTA kernel: 32 x 32 fp32 blocks of C (and of R, which shares C's pitch).
// (32 x 64 of a bf16 result: row by row, a thread's 64 bytes apart from its neighbour's, the bf16 results with a residual took longer
// than their products: out_proj at 16384 tokens 67 us, 48 this way, 40 with
// eight epilogue warps.)  Leaves tma_out = 0 when a TMA rule is broken (a store
// clips a row at whole 16 bytes, so a width that ends inside them would reach into the pitch); the kernel then stores row by row.
static pmb_status make_out_maps(Problem* q, int slabs = 1) {
  Params& p = q->p;
  p.tma_out = p.red = 0;
  if (p.out_bf16) {
    if (slabs > 1 || (p.N & 7) || (p.ldc & 7) || (reinterpret_cast<uintptr_t>(p.C) & 15) || (p.R && (reinterpret_cast<uintptr_t>(p.R) & 15))) return PMB_OK;
    PMB_TRY(make_map(&q->mC, p.C, p.N, p.M, p.ldc, 64, 32));
    if (p.R) PMB_TRY(make_map(&q->mR, p.R, p.N, p.M, p.ldc, 64, 32));
    p.tma_out = 1;
    return PMB_OK;
  }
  if ((p.ldc & 3) || (p.R && (p.N & 3)) || (reinterpret_cast<uintptr_t>(p.C) & 15) || (p.R && (reinterpret_cast<uintptr_t>(p.R) & 15))) return PMB_OK;
  PMB_TRY(make_map(&q->mC, p.C, p.N, slabs > 1 ? (int64_t)slabs * p.slab_rows : p.M, p.ldc, 32, 32, true));
  // (one addend per element and launch, so the order of the additions is as it was: C, then the product)
  p.red = p.R == p.C && slabs == 1 && !p.e_hi;
  p.tma_out = 1;
  return PMB_OK;
}

// Ticket counters of the persistent kernel (64-bit, never reset; see the kernel).  Launches outside stream capture
// share EAGER_SLOTS counters round-robin and are told the counter's value before the launch, which the host tracks
// (a launch draws exactly `tiles` tickets); a captured launch keeps a counter of its own for the life of the graph,
// from a range that is never recycled.  Returns NULL (static tile order) when that range is used up, the counters
// cannot be allocated, or PMB_GEMM_SCHED=0.
constexpr unsigned EAGER_SLOTS = 4096, GRAPH_SLOTS = 61440;
static unsigned long long* g_sched_base[PMB_MAX_DEVICES] = {};
static std::vector<unsigned long long> g_sched_shadow[PMB_MAX_DEVICES];
static std::mutex g_sched_mu;

// After a kernel gave up on a bounded wait it may have drawn fewer tickets than its launch was accounted for: put
// every counter of the current device (and the host's record of them) back to zero, so that later launches start
// from a consistent state.  Called when the status word is read and found raised.
static void sched_reset_current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= PMB_MAX_DEVICES) return;
  std::lock_guard<std::mutex> lock(g_sched_mu);
  if (!g_sched_base[dev]) return;
  cudaMemset(g_sched_base[dev], 0, (size_t)(EAGER_SLOTS + GRAPH_SLOTS) * sizeof(unsigned long long));
  g_sched_shadow[dev].assign(EAGER_SLOTS, 0ull);
}

static unsigned long long* sched_counter(cudaStream_t st, int64_t tiles, unsigned long long* ticket0) {
  unsigned long long** base = g_sched_base;
  std::vector<unsigned long long>* shadow = g_sched_shadow;
  std::mutex& mu = g_sched_mu;
  static bool failed[PMB_MAX_DEVICES] = {};
  static unsigned eager_next[PMB_MAX_DEVICES] = {}, graph_next[PMB_MAX_DEVICES] = {};
  static const int on = [] { const char* e = getenv("PMB_GEMM_SCHED"); return (e && e[0] == '0') ? 0 : 1; }();   // 0: static tile order
  *ticket0 = 0;
  if (!on) return nullptr;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= PMB_MAX_DEVICES) return nullptr;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cap) != cudaSuccess) { cudaGetLastError(); return nullptr; }
  std::lock_guard<std::mutex> lock(mu);
  if (!base[dev]) {
    if (failed[dev] || cap != cudaStreamCaptureStatusNone) return nullptr;      // (first use must be outside capture)
    const size_t bytes = (size_t)(EAGER_SLOTS + GRAPH_SLOTS) * sizeof(unsigned long long);
    if (cudaMalloc(&base[dev], bytes) != cudaSuccess || cudaMemset(base[dev], 0, bytes) != cudaSuccess) {
      cudaGetLastError(); failed[dev] = true; base[dev] = nullptr; return nullptr;
    }
    shadow[dev].assign(EAGER_SLOTS, 0ull);
  }
  if (cap == cudaStreamCaptureStatusNone) {
    const unsigned slot = eager_next[dev]++ % EAGER_SLOTS;
    *ticket0 = shadow[dev][slot];
    shadow[dev][slot] += (unsigned long long)tiles;
    return base[dev] + slot;
  }
  if (graph_next[dev] >= GRAPH_SLOTS) return nullptr;
  return base[dev] + EAGER_SLOTS + graph_next[dev]++;
}

// One persistent CTA per SM, fewer when there are fewer tiles.
static unsigned persistent_grid(int64_t tiles) {
  static int sms[PMB_MAX_DEVICES] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  int n = 148;
  if (dev >= 0 && dev < PMB_MAX_DEVICES) {
    if (!sms[dev]) { int v = 0; if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && v > 0) sms[dev] = v; else sms[dev] = 148; }
    n = sms[dev];
  }
  return (unsigned)(tiles < n ? tiles : n);
}

}  // namespace hb

namespace hb {

static int64_t ktiles(int64_t K) { return cdiv(K, TBK); }

// What a tile of the CTA-pair kernel costs, in k-tiles of 256 columns: a 128-wide one has half the columns, but with one MMA per product
// hardly less than the time (311 ns against 299 per k-tile; the loads and barriers of a k-tile set the pace), with three 0.6 of it.
static double tile_cost(const Problem& q) { return (double)q.p.kt_per * (q.p.bn == 256 ? 1.0 : q.p.pairs ? 0.6 : 0.9) + 1.0; }

// Long tiles first on the pair kernel (Group): the leading problems whose tiles cost at least twice those of the last one, when they
// have fewer tiles than there are clusters.
static void set_lead(Group* g, int n, int clusters) {
  g->lead = g->rounds = 0;
  if (n < 2) return;
  const Problem& last = g->pr[n - 1];
  const double b = tile_cost(last);
  int64_t lead = 0;
  double a = 0.0;
  for (int i = 0; i + 1 < n; ++i) { lead += g->pr[i].tiles; const double c = tile_cost(g->pr[i]); if (c > a) a = c; }
  if (lead >= clusters || a < 2.0 * b) return;
  g->lead = (int)lead; g->rounds = (int)(a / b);
}

static void set_tiles(Problem* q, int bn) {
  const int splits = (int)cdiv(ktiles(q->p.K), q->p.kt_per);
  q->p.bn = bn;
  if (q->n_end == 0) q->n_end = q->p.N;
  q->tiles_n = (int)cdiv(q->n_end - q->n_begin, bn);
  q->tiles_mn = (int)(cdiv(q->p.M, 256) * q->tiles_n);
  q->tiles = q->tiles_mn * splits;
}

// The longest cluster's work for the widths that are set.
static double makespan(Group* g, int n, int slots) {
  int64_t tiles = 0;
  double total = 0.0, most = 0.0;
  for (int i = 0; i < n; ++i) {
    const double c = tile_cost(g->pr[i]);
    tiles += g->pr[i].tiles; total += c * g->pr[i].tiles;
    if (c > most) most = c;
  }
  const int clusters = (int)(tiles < slots ? tiles : slots);
  set_lead(g, n, clusters);
  if (tiles > 8 * slots) return total / clusters > most ? total / clusters : most;
  // the first cluster of the round (and the first one without a long tile) has the most to do: tiles are in order of their length
  double worst = 0.0;
  for (int i = 0; i < 2; ++i) {
    const int c = i ? g->lead : 0;
    if (i && (c == 0 || c >= clusters)) continue;
    double t = 0.0;
    for (int j = 0;; ++j) {
      const int id = pair_tile_at(*g, c, clusters, j);
      if (id >= tiles) break;
      int base = 0, k = 0;
      while (id >= base + g->pr[k].tiles) base += g->pr[k++].tiles;
      t += tile_cost(g->pr[k]);
    }
    if (t > worst) worst = t;
  }
  return worst;
}

// Tile widths of the products of a launch: 256 columns, or 128 where the shorter tiles bring the longest cluster down by a tenth (few
// tiles: 2048 x 768 outputs are 24 tiles of 256 columns; on pairs with K = 1536 they took 44 us, 48 tiles of 128 columns 28).  Every sum runs over K in the same order at either width.
static void choose_widths(Group* g, int n, int slots) {
  double best = 0.0;
  int pick = 0;
  for (int mask = 0; mask < (1 << n); ++mask) {
    for (int i = 0; i < n; ++i) set_tiles(&g->pr[i], (mask >> i) & 1 ? 128 : 256);
    const double t = makespan(g, n, slots);
    if (mask == 0 || t < 0.9 * best) { best = t; pick = mask; }
  }
  for (int i = 0; i < n; ++i) set_tiles(&g->pr[i], (pick >> i) & 1 ? 128 : 256);
}

// The longest cluster's work, cluster by cluster.
static double makespan_exact(Group* g, int n, int slots) {
  int tiles = 0;
  for (int i = 0; i < n; ++i) tiles += g->pr[i].tiles;
  const int clusters = tiles < slots ? tiles : slots;
  set_lead(g, n, clusters);
  double worst = 0.0;
  for (int c = 0; c < clusters; ++c) {
    double t = 0.0;
    for (int j = 0;; ++j) {
      const int id = pair_tile_at(*g, c, clusters, j);
      if (id >= tiles) break;
      int base = 0, k = 0;
      while (id >= base + g->pr[k].tiles) base += g->pr[k++].tiles;
      t += tile_cost(g->pr[k]);
    }
    if (t > worst) worst = t;
  }
  return worst;
}

// A few rounds of tiles leave the last one partly empty whatever the width: one product's columns then go to tiles of 256 up to a column and
// of 128 from there on, where that brings the longest cluster down by a fourteenth (2048 x 3224 x 768 on pairs: 104 tiles of 256 columns are
// two rounds on 74 clusters, 30.1 us; 64 and 80 of 128 are one and a half).  The answer depends on the shapes alone and is kept (256 of
// them).  Returns the number of problems.
struct CutKey {
  int n, slots; int64_t v[3 * MAX_GROUP];
  bool operator<(const CutKey& o) const { return n != o.n ? n < o.n : slots != o.slots ? slots < o.slots : std::lexicographical_compare(v, v + 3 * MAX_GROUP, o.v, o.v + 3 * MAX_GROUP); }
};
struct Cut { int which, at; };
static int cut_widths(Group* g, int n, int slots) {
  int64_t tiles = 0;
  for (int i = 0; i < n; ++i) tiles += g->pr[i].tiles;
  if (n >= MAX_GROUP || tiles <= slots || tiles > 4 * slots) return n;
  static std::map<CutKey, Cut> known;
  static std::mutex mu;
  CutKey key{};
  key.n = n; key.slots = slots;
  for (int i = 0; i < n; ++i) { key.v[3 * i] = g->pr[i].p.M; key.v[3 * i + 1] = g->pr[i].p.N; key.v[3 * i + 2] = (int64_t)g->pr[i].p.kt_per << 32 | g->pr[i].p.K; }
  auto apply = [&](const Cut& c, Group* to) {
    for (int i = n; i > c.which; --i) to->pr[i] = to->pr[i - 1];
    Problem &a = to->pr[c.which], &b = to->pr[c.which + 1];
    a.n_begin = 0; a.n_end = c.at; b.n_begin = c.at; b.n_end = b.p.N;
    set_tiles(&a, 256); set_tiles(&b, 128);
  };
  Cut best{-1, 0};
  {
    std::lock_guard<std::mutex> lock(mu);
    const auto it = known.find(key);
    if (it != known.end()) best = it->second;
    else {
      double t0 = makespan_exact(g, n, slots) * (13.0 / 14.0);
      for (int i = 0; i < n; ++i)
        for (int at = 256; at < g->pr[i].p.N; at += 256) {
          Group h = *g;
          apply(Cut{i, at}, &h);
          const double t = makespan_exact(&h, n + 1, slots);
          if (t < t0) { t0 = t; best = Cut{i, at}; }
        }
      if (known.size() >= 256) known.clear();
      known.emplace(key, best);
    }
  }
  if (best.which < 0) return n;
  apply(best, g);
  return n + 1;
}

}  // namespace hb

// Splits of K for a product that shares a launch with `other_tiles` tiles of `other_kt` k-tiles: as many as bring its tiles down
// to an even share of the launch's k-tiles per cluster (a weight gradient has few tiles as long as the token count: at 16384 tokens
// 18 of them kept 18 of the 74 clusters busy four times as long as the rest of the launch needed), at most 8.
int gemm_bf16_ksplit(int64_t M, int64_t N, int64_t K, int64_t other_tiles, int64_t other_kt) {
  const int64_t tiles = cdiv(M, 256) * cdiv(N, 256), kt = hb::ktiles(K);
  const int64_t share = cdiv(tiles * kt + other_tiles * other_kt, 74);
  int64_t sp = cdiv(kt, share > 8 ? share : 8);
  if (sp > 8) sp = 8;
  return (int)cdiv(kt, cdiv(kt, sp));          // (no empty split)
}

// C = op(A) op(B) (+ R) on bf16 operands, up to MAX_GROUP independent products in one launch (the ones with the longest K first).
// Row pitches must be multiples of 8 elements (16 bytes) and the bases 16-byte aligned (TMA rules).  ksplit > 1: C is fp32 and
// receives ksplit slabs of slab_rows rows (a multiple of 256, at least M), which the caller adds up.
pmb_status gemm_bf16_group(cudaStream_t st, const PlainGemm* gs, int n, int max_clusters) {
  using namespace hb;
  if (n < 1 || n > MAX_GROUP) return fail(PMB_ERR_ARG, "gemm_bf16_group: 1 to %d products per launch", MAX_GROUP);
  PMB_SMEM_OPT_IN(Cfg<false>::SMEM_BYTES, gemm_bf16_kernel<false>);
  Group g{};
  double flops = 0.0, bytes = 0.0;
  int64_t clusters = 0, tiles = 0;
  bool tall = true;
  for (int i = 0; i < n; ++i) {
    const PlainGemm& e = gs[i];
    if (e.M <= 0 || e.N <= 0 || e.K <= 0) return fail(PMB_ERR_SHAPE, "gemm_bf16: non-positive dimension");
    if ((reinterpret_cast<uintptr_t>(e.A) & 15) || (reinterpret_cast<uintptr_t>(e.B) & 15) || (e.lda & 7) || (e.ldb & 7))
      return fail(PMB_ERR_SHAPE, "gemm_bf16: operands need 16-byte aligned bases and row pitches that are multiples of 8 elements");
    if (e.ksplit > 1 && (e.out_bf16 || e.R || e.slab_rows < e.M || e.slab_rows % 256)) return fail(PMB_ERR_ARG, "gemm_bf16: split products go to fp32 slabs");
    Problem& q = g.pr[i];
    if (!e.ta) PMB_TRY(make_map(&q.mA, e.A, e.K, e.M, e.lda, TBK, TBM)); else PMB_TRY(make_map(&q.mA, e.A, e.M, e.K, e.lda, 64, TBK));
    if (e.tb) PMB_TRY(make_map(&q.mB, e.B, e.K, e.N, e.ldb, TBK, TBN)); else PMB_TRY(make_map(&q.mB, e.B, e.N, e.K, e.ldb, 64, TBK));
    Params& p = q.p;
    p.M = (int)e.M; p.N = (int)e.N; p.K = (int)e.K;
    p.a_mn_major = e.ta ? 1 : 0; p.b_mn_major = e.tb ? 0 : 1;
    p.C = e.C; p.ldc = e.ldc; p.R = e.R; p.out_bf16 = e.out_bf16;
    const int sp = e.ksplit > 1 ? e.ksplit : 1;
    p.kt_per = (int)cdiv(ktiles(e.K), sp); p.slab_rows = sp > 1 ? (int)e.slab_rows : 0;
    const int splits = (int)cdiv(ktiles(e.K), p.kt_per);
    if (splits < sp) return fail(PMB_ERR_ARG, "gemm_bf16: more splits than k-tiles");
    PMB_TRY(make_out_maps(&q, sp));
    clusters += cdiv(e.M, 256) * cdiv(e.N, 256) * sp;
    tiles += cdiv(e.M, TBM) * cdiv(e.N, TBN) * sp;
    tall = tall && e.M > 128;
    flops += 2.0 * e.M * e.N * e.K;
    bytes += 2.0 * ((double)e.M * e.K + (double)e.K * e.N) + (e.out_bf16 ? 2.0 : 4.0) * e.M * e.N * (e.R ? 2 : 1);
  }
  if (tiles > 0x7fffffff) return fail(PMB_ERR_SHAPE, "gemm_bf16: too many tiles");
  static const int env = [] { const char* e = getenv("PMB_GEMM_PAIR"); return e ? atoi(e) : -1; }();
  static const int min_clusters = [] { const char* e = getenv("PMB_GEMM_PAIR_MIN"); return e ? atoi(e) : 4; }();
  const bool pair = env >= 0 ? env != 0 : (tall && clusters >= min_clusters);      // see pick_pair_mode
  for (int i = 0; i < n; ++i) {
    Problem& q = g.pr[i];
    const int64_t tm = pair ? cdiv(gs[i].M, 256) : cdiv(gs[i].M, TBM), tn = pair ? cdiv(gs[i].N, 256) : cdiv(gs[i].N, TBN);
    q.tiles_n = (int)tn; q.tiles_mn = (int)(tm * tn); q.tiles = q.tiles_mn * (gs[i].ksplit > 1 ? gs[i].ksplit : 1);
  }
  for (int i = n; i < MAX_GROUP; ++i) { g.pr[i].tiles_n = g.pr[i].tiles_mn = 1; g.pr[i].tiles = 0; }
  ProfScope prof(st, "gemm_bf16", flops, bytes);
  if (pair) {
    PMB_SMEM_OPT_IN((PairPCfg<false, 256>::SMEM_BYTES), gemm_bf16_pairp_kernel<false, 256>);
    int64_t slots = persistent_grid(148) / 2;
    if (max_clusters > 0 && slots > max_clusters) slots = max_clusters;
    choose_widths(&g, n, (int)slots);
    clusters = 0;
    for (int i = 0; i < n; ++i) {
      clusters += g.pr[i].tiles;
      if (gs[i].tb) PMB_TRY(make_map(&g.pr[i].mB, gs[i].B, gs[i].K, gs[i].N, gs[i].ldb, TBK, g.pr[i].p.bn / 2));
    }
    const unsigned grid = 2u * (unsigned)(clusters < slots ? clusters : slots);
    set_lead(&g, n, (int)(grid / 2));
    PMB_TRY(launch_pdl(st, gemm_bf16_pairp_kernel<false, 256>, grid, (PairPCfg<false, 256>::THREADS), PairPCfg<false, 256>::SMEM_BYTES, g, (int)clusters));
  } else {
    unsigned long long t0 = 0;
    unsigned long long* sc = sched_counter(st, tiles, &t0);
    PMB_TRY(launch_pdl(st, gemm_bf16_kernel<false>, dim3((unsigned)(persistent_grid(tiles))), NTHREADS, Cfg<false>::SMEM_BYTES, g, (int)tiles, sc, t0));
  }
  return PMB_OK;
}

pmb_status gemm_bf16(cudaStream_t st, int ta, int tb, int64_t M, int64_t N, int64_t K, const void* A, int64_t lda,
                     const void* B, int64_t ldb, void* C, int64_t ldc, const void* R, int out_bf16) {
  const PlainGemm e{ta, tb, M, N, K, A, lda, B, ldb, C, ldc, R, out_bf16};
  return gemm_bf16_group(st, &e, 1);
}

// out = sum of n slabs, fixed order; `pitch` elements apart, `elems` each; out fp32 or bf16
__global__ void __launch_bounds__(256) sum_slabs_kernel(const float* __restrict__ part, int n, int64_t pitch, int64_t elems, void* __restrict__ out, int out_bf16) {
  pdl_launch();
  pdl_wait();
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i >= elems) return;
  float4 a = *reinterpret_cast<const float4*>(part + i);
#pragma unroll 4
  for (int s = 1; s < n; ++s) {
    const float4 b = *reinterpret_cast<const float4*>(part + (int64_t)s * pitch + i);
    a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
  }
  if (out_bf16) store_pair4(static_cast<uint16_t*>(out) + i, nullptr, a.x, a.y, a.z, a.w);
  else *reinterpret_cast<float4*>(static_cast<float*>(out) + i) = a;
}
pmb_status sum_slabs(cudaStream_t st, const float* part, int n, int64_t pitch, int64_t elems, void* out, int out_bf16) {
  if (elems & 3) return fail(PMB_ERR_SHAPE, "sum_slabs: the element count must be a multiple of 4");
  ProfScope prof(st, "splitk_sum", 0.0, (4.0 * n + (out_bf16 ? 2.0 : 4.0)) * elems);
  PMB_TRY(launch_pdl(st, sum_slabs_kernel, dim3((unsigned)cdiv(elems / 4, 256)), 256, 0, part, n, pitch, elems, out, out_bf16));
  return PMB_OK;
}

// ---- fp32 GEMM through bf16 pairs ------------------------------------------------------------------
// a = hi + lo with hi = bf16(a), lo = bf16(a - hi): 16 mantissa bits, relative representation error <= 2^-17.
// One thread = 4 consecutive columns of the pair; columns in [cols, ld16) are written as zero.
__global__ void split_pair16_kernel(const float* __restrict__ src, int64_t rows, int64_t cols, int64_t ld,
                                    uint16_t* __restrict__ hi, uint16_t* __restrict__ lo, int64_t ld16, int vec) {
  pdl_launch();
  pdl_wait();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t c4 = ld16 / 4;
  if (i >= rows * c4) return;
  int64_t r = i / c4, c = (i % c4) * 4;
  float f[4];
  if (vec && c + 4 <= cols) {
    float4 v = *reinterpret_cast<const float4*>(src + r * ld + c);
    f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e) f[e] = (c + e < cols) ? src[r * ld + c + e] : 0.0f;
  }
  uint32_t h[4], l[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    h[e] = hb::float_to_bf16_bits(f[e]);
    l[e] = hb::float_to_bf16_bits(f[e] - hb::bf16_bits_to_float((uint16_t)h[e]));
  }
  *reinterpret_cast<uint2*>(hi + r * ld16 + c) = make_uint2(h[0] | (h[1] << 16), h[2] | (h[3] << 16));
  *reinterpret_cast<uint2*>(lo + r * ld16 + c) = make_uint2(l[0] | (l[1] << 16), l[2] | (l[3] << 16));
}

pmb_status split_pair16(cudaStream_t st, const float* src, int64_t rows, int64_t cols, int64_t ld, uint16_t* hi, uint16_t* lo,
                        int64_t ld16) {
  if ((ld16 & 7) || ld16 < cols || ((reinterpret_cast<uintptr_t>(hi) | reinterpret_cast<uintptr_t>(lo)) & 15))
    return fail(PMB_ERR_ARG, "split_pair16: the pair needs 16-byte aligned bases and a row pitch that is a multiple of 8");
  const int vec = ((reinterpret_cast<uintptr_t>(src) & 15) == 0 && (ld & 3) == 0) ? 1 : 0;
  ProfScope prof(st, "split_f32_bf16x2", 0.0, 8.0 * rows * cols);
  PMB_TRY(launch_pdl(st, split_pair16_kernel, dim3((unsigned)cdiv(rows * (ld16 / 4), 256)), 256, 0, src, rows, cols, ld, hi, lo, ld16, vec));
  return PMB_OK;
}

// Contiguous arrays, several to a launch: blocks of 256 U quads, each of one array.  Bound by HBM for the parameters of a model (126 M
// elements: 148 us, 6.8 TB/s, against 230 through the rows-and-columns kernel above with its division per quad), by the launch for a small block's operands
// (which is why they share one).
struct SplitGroup { SplitItem it[4]; int first[4]; };      // first[i]: block at which item i starts
template <int U>
__global__ void __launch_bounds__(256) split_flat_kernel(const SplitGroup g) {
  pdl_launch();
  pdl_wait();
  int w = 0;
#pragma unroll
  for (int i = 1; i < 4; ++i) if ((int)blockIdx.x >= g.first[i]) w = i;
  const SplitItem it = g.it[w];
  const int64_t q0 = (int64_t)((int)blockIdx.x - g.first[w]) * (256 * U) + threadIdx.x, n4 = it.n >> 2;
  const bool vec = (reinterpret_cast<uintptr_t>(it.src) & 15) == 0;
  float4 v[U];
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int64_t q = q0 + 256 * u;
    if (q < n4) {
      if (vec) v[u] = reinterpret_cast<const float4*>(it.src)[q];
      else v[u] = make_float4(it.src[4 * q], it.src[4 * q + 1], it.src[4 * q + 2], it.src[4 * q + 3]);
    }
  }
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int64_t q = q0 + 256 * u;
    if (q < n4) store_pair4(it.hi + 4 * q, it.lo + 4 * q, v[u].x, v[u].y, v[u].z, v[u].w);
  }
}

pmb_status split_pairs_flat(cudaStream_t st, const SplitItem* items, int n) {
  if (n < 1 || n > 4) return fail(PMB_ERR_ARG, "split_pairs_flat: one to four arrays");
  int64_t total = 0;
  for (int i = 0; i < n; ++i) {
    if ((items[i].n & 3) || ((reinterpret_cast<uintptr_t>(items[i].hi) | reinterpret_cast<uintptr_t>(items[i].lo)) & 7))
      return fail(PMB_ERR_ARG, "split_pairs_flat: lengths must be multiples of 4 and the pair arrays 8-byte aligned");
    total += items[i].n;
  }
  const int U = total >= (int64_t)4 << 20 ? 4 : 1;         // (below, more and shorter blocks fill the machine)
  SplitGroup g{};
  int64_t blocks = 0;
  for (int i = 0; i < 4; ++i) {
    g.first[i] = (int)blocks;
    if (i < n) { g.it[i] = items[i]; blocks += cdiv(items[i].n >> 2, 256 * U); } else g.first[i] = 0x7fffffff;
  }
  if (blocks > 0x7ffffffe) return fail(PMB_ERR_SHAPE, "split_pairs_flat: too large");
  ProfScope prof(st, "split_f32_bf16x2", 0.0, 8.0 * total);
  if (U == 4) PMB_TRY(launch_pdl(st, split_flat_kernel<4>, dim3((unsigned)blocks), 256, 0, g));
  else PMB_TRY(launch_pdl(st, split_flat_kernel<1>, dim3((unsigned)blocks), 256, 0, g));
  return PMB_OK;
}

// Columns [0, cols) of each row only (cols a multiple of 4); the rest of the destination pitch is left alone, so two
// sources can share one pair buffer side by side.
__global__ void split_pair16_cols_kernel(const float* __restrict__ src, int64_t rows, int64_t cols, int64_t ld,
                                         uint16_t* __restrict__ hi, uint16_t* __restrict__ lo, int64_t ld16) {
  pdl_launch();
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t c4 = cols / 4;
  if (i >= rows * c4) return;
  const int64_t r = i / c4, c = (i % c4) * 4;
  const float* s = src + r * ld + c;
  store_pair4(hi + r * ld16 + c, lo ? lo + r * ld16 + c : nullptr, s[0], s[1], s[2], s[3]);
}

pmb_status split_pair16_strided(cudaStream_t st, const float* src, int64_t rows, int64_t cols, int64_t ld, uint16_t* hi, uint16_t* lo,
                                int64_t ld16) {
  if ((cols & 3) || (ld16 & 3) || ld16 < cols || ((reinterpret_cast<uintptr_t>(hi) | reinterpret_cast<uintptr_t>(lo)) & 7))
    return fail(PMB_ERR_ARG, "split_pair16_strided: column count and pitch must be multiples of 4, destinations 8-byte aligned");
  PMB_TRY(launch_pdl(st, split_pair16_cols_kernel, dim3((unsigned)cdiv(rows * (cols / 4), 256)), 256, 0, src, rows, cols, ld, hi, lo, ld16));
  return PMB_OK;
}

bool gemm_pairs_enabled() {
  static const int on = [] { const char* e = getenv("PMB_GEMM_ENGINE"); return (e && (strcmp(e, "tf32") == 0 || strcmp(e, "simt") == 0)) ? 0 : 1; }();
  return on != 0;
}

// Tile shape of the pair GEMM: 0 = 128x128 single-CTA tiles, 1 = 256x128 CTA-pair tiles, 2 = 256x256 CTA-pair tiles.
// `tile_mode` >= 0 (engines 4 / 5 / 6 of the public GEMM entry) or PMB_GEMM_PAIR=0/1/2 force it.
static int pick_pair_mode(const PairGemm* gs, int n, int tile_mode) {
  static const int env = [] { const char* e = getenv("PMB_GEMM_PAIR"); return e ? atoi(e) : -1; }();
  const int forced = tile_mode >= 0 ? tile_mode : env;
  if (forced >= 0 && forced <= 4) return forced;          // 3 / 4: the persistent CTA-pair kernel with 256x128 / 256x256 tiles
  // CTA-pair tiles fetch half the operand bytes per flop, read half as much shared memory per MMA, and come 256 or 128 columns
  // wide (choose_widths); below four clusters per product too few SMs take part.  Residual stack of four layers at 2 x 384 tokens of
  // d_model 768: 1226 us with the line at 18 clusters, 1150 at 9 and at 4; training step at 2 x 512: 1240, 1154, 1153; prefill of
  // 160 tokens at d_model 1024: 99, 97, 89; the smallest block is 5 % slower without a line.  PMB_GEMM_PAIR_MIN overrides it.
  static const int half_wave = [] { const char* e = getenv("PMB_GEMM_PAIR_MIN"); return e ? atoi(e) : 4; }();
  for (int i = 0; i < n; ++i) {
    if (gs[i].M <= 128) return 0;        // a pair tile would be half empty
    if (cdiv(gs[i].M, 256) * cdiv(gs[i].N, 256) * (gs[i].ksplit > 1 ? gs[i].ksplit : 1) < half_wave) return 0;
  }
  return 4;
}

// C (fp32) = op(A) op(B) (+ R) with both operands given as bf16 pairs: three kind::f16 MMAs per k-step.
// Relative accuracy ~1e-5 of the result's scale; twice the tensor-core rate and less than half the shared-memory
// traffic of the 3xTF32 kernel.  Up to two independent products go out as one launch; the tiles of g[0] are
// scheduled first, so put the product with the longer K there.
pmb_status gemm_pairs_group(cudaStream_t st, const PairGemm* gs, int n, int tile_mode) {
  using namespace hb;
  if (n < 1 || n > MAX_GROUP) return fail(PMB_ERR_ARG, "gemm_pairs_group: 1 to %d products per launch", MAX_GROUP);
  PMB_SMEM_OPT_IN(Cfg<true>::SMEM_BYTES, gemm_bf16_kernel<true>);
  Group g{};
  for (int i = 1; i < MAX_GROUP; ++i) { g.pr[i].tiles_n = g.pr[i].tiles_mn = 1; g.pr[i].tiles = 0; }
  double flops = 0.0, bytes = 0.0;
  int64_t total = 0;
  for (int i = 0; i < n; ++i) {
    const PairGemm& e = gs[i];
    const int64_t M = e.M, N = e.N, K = e.K;
    if (M <= 0 || N <= 0 || K <= 0) return fail(PMB_ERR_SHAPE, "gemm_pairs: M, N, K must be positive");
    if ((e.A.ld & 7) || (e.B.ld & 7) ||
        ((reinterpret_cast<uintptr_t>(e.A.hi) | reinterpret_cast<uintptr_t>(e.A.lo) | reinterpret_cast<uintptr_t>(e.B.hi) | reinterpret_cast<uintptr_t>(e.B.lo)) & 15))
      return fail(PMB_ERR_UNSUPPORTED, "gemm_pairs: operands need 16-byte aligned bases and row pitches that are multiples of 8");
    Problem& q = g.pr[i];
    if (!e.ta) { PMB_TRY(make_map(&q.mA, e.A.hi, K, M, e.A.ld, TBK, TBM)); PMB_TRY(make_map(&q.mAlo, e.A.lo, K, M, e.A.ld, TBK, TBM)); }
    else { PMB_TRY(make_map(&q.mA, e.A.hi, M, K, e.A.ld, 64, TBK)); PMB_TRY(make_map(&q.mAlo, e.A.lo, M, K, e.A.ld, 64, TBK)); }
    if (e.tb) { PMB_TRY(make_map(&q.mB, e.B.hi, K, N, e.B.ld, TBK, TBN)); PMB_TRY(make_map(&q.mBlo, e.B.lo, K, N, e.B.ld, TBK, TBN)); }
    else { PMB_TRY(make_map(&q.mB, e.B.hi, N, K, e.B.ld, 64, TBK)); PMB_TRY(make_map(&q.mBlo, e.B.lo, N, K, e.B.ld, 64, TBK)); }
    Params& p = q.p;
    p.M = (int)M; p.N = (int)N; p.K = (int)K;
    p.a_mn_major = e.ta ? 1 : 0; p.b_mn_major = e.tb ? 0 : 1;
    p.C = e.C; p.ldc = e.ldc; p.R = e.R; p.out_bf16 = 0; p.pairs = 1;
    const int sp = e.ksplit > 1 ? e.ksplit : 1;
    if (sp > 1 && (e.R || e.emit.hi || e.slab_rows < M || e.slab_rows % 256)) return fail(PMB_ERR_ARG, "gemm_pairs: split products go to fp32 slabs");
    p.kt_per = (int)cdiv(ktiles(K), sp); p.slab_rows = sp > 1 ? (int)e.slab_rows : 0;
    if (cdiv(ktiles(K), p.kt_per) < sp) return fail(PMB_ERR_ARG, "gemm_pairs: more splits than k-tiles");
    p.e_hi = const_cast<uint16_t*>(e.emit.hi); p.e_lo = const_cast<uint16_t*>(e.emit.lo); p.lde = e.emit.ld;   // (Pair16 is declared for reading; this one is written)
    PMB_TRY(make_out_maps(&q, sp));
    if (p.e_hi && (!p.tma_out || !p.e_lo || (p.lde & 7) || ((reinterpret_cast<uintptr_t>(p.e_hi) | reinterpret_cast<uintptr_t>(p.e_lo)) & 15)))
      return fail(PMB_ERR_UNSUPPORTED, "gemm_pairs: the pair output needs the TMA-store epilogue, 16-byte aligned arrays and a pitch that is a multiple of 8");
    q.tiles_n = (int)cdiv(N, TBN);
    q.tiles_mn = (int)(cdiv(M, TBM) * cdiv(N, TBN));
    const int64_t t = (int64_t)q.tiles_mn * sp;
    total += t;
    if (total > 0x7fffffff) return fail(PMB_ERR_UNSUPPORTED, "gemm_pairs: too many tiles");
    q.tiles = (int)t;
    flops += 2.0 * M * N * K;
    bytes += 4.0 * ((double)M * K + (double)K * N + (double)M * N * (e.R ? 2 : 1));
  }
  int pair_mode = pick_pair_mode(gs, n, tile_mode);
  for (int i = 0; i < n; ++i) if ((gs[i].emit.hi || gs[i].ksplit > 1) && pair_mode <= 2) pair_mode = 0;      // (the one-tile-per-cluster kernels do not write the pair output)
  if (pair_mode) {
    const int64_t slots = persistent_grid(148) / 2;
    int np = n;
    if (pair_mode == 4) { choose_widths(&g, n, (int)slots); np = cut_widths(&g, n, (int)slots); }
    else for (int i = 0; i < n; ++i) set_tiles(&g.pr[i], pair_mode == 2 ? 256 : 128);
    PMB_SMEM_OPT_IN((PairCfg<true, 256>::SMEM_BYTES), gemm_bf16_pair_kernel<true, 256>);
    PMB_SMEM_OPT_IN((PairCfg<true, 128>::SMEM_BYTES), gemm_bf16_pair_kernel<true, 128>);
    int64_t clusters = 0;
    for (int i = 0, of = 0; i < np; ++i) {
      Problem& q = g.pr[i];
      if (i > 0 && q.n_begin == 0) ++of;                     // (the product that the problem is of)
      const PairGemm& e = gs[of];
      // B boxes of the pair kernels are half a tile tall (K-major tiles); MN-major boxes stay 64 columns wide
      const int half = q.p.bn / 2;
      if (e.tb) { PMB_TRY(make_map(&q.mB, e.B.hi, e.K, e.N, e.B.ld, TBK, half)); PMB_TRY(make_map(&q.mBlo, e.B.lo, e.K, e.N, e.B.ld, TBK, half)); }
      clusters += q.tiles;
    }
    if (pair_mode >= 3) {
      ProfScope prof(st, "gemm_bf16x2", flops, bytes);
      const unsigned grid = 2u * (unsigned)(clusters < slots ? clusters : slots);
      set_lead(&g, np, (int)(grid / 2));
      if (pair_mode == 4) {
        PMB_SMEM_OPT_IN((PairPCfg<true, 256>::SMEM_BYTES), gemm_bf16_pairp_kernel<true, 256>);
        PMB_TRY(launch_pdl(st, gemm_bf16_pairp_kernel<true, 256>, grid, (PairPCfg<true, 256>::THREADS), PairPCfg<true, 256>::SMEM_BYTES, g, (int)clusters));
      } else {
        PMB_SMEM_OPT_IN((PairPCfg<true, 128>::SMEM_BYTES), gemm_bf16_pairp_kernel<true, 128>);
        PMB_TRY(launch_pdl(st, gemm_bf16_pairp_kernel<true, 128>, grid, (PairPCfg<true, 128>::THREADS), PairPCfg<true, 128>::SMEM_BYTES, g, (int)clusters));
      }
      return PMB_OK;
    }
    ProfScope prof(st, pair_mode == 2 ? "gemm_bf16x2_pair256" : "gemm_bf16x2_pair128", flops, bytes);
    if (pair_mode == 2) gemm_bf16_pair_kernel<true, 256><<<(unsigned)(2 * clusters), NTHREADS, PairCfg<true, 256>::SMEM_BYTES, st>>>(g);
    else gemm_bf16_pair_kernel<true, 128><<<(unsigned)(2 * clusters), NTHREADS, PairCfg<true, 128>::SMEM_BYTES, st>>>(g);
    PMB_LAUNCHED();
    return PMB_OK;
  }
  ProfScope prof(st, "gemm_bf16x2", flops, bytes);
  {
    unsigned long long t0 = 0;
    unsigned long long* sc = sched_counter(st, total, &t0);
    PMB_TRY(launch_pdl(st, gemm_bf16_kernel<true>, dim3((unsigned)(persistent_grid(total))), NTHREADS, Cfg<true>::SMEM_BYTES, g, (int)total, sc, t0));
  }
  return PMB_OK;
}

pmb_status gemm_pairs(cudaStream_t st, int ta, int tb, int64_t M, int64_t N, int64_t K, const Pair16& A, const Pair16& B,
                      float* C, int64_t ldc, const float* R, int tile_mode) {
  PairGemm e{ta, tb, M, N, K, A, B, C, ldc, R};
  return gemm_pairs_group(st, &e, 1, tile_mode);
}

// Library-owned scratch for the pairs of callers that hand in fp32 operands (one per device).
// pmb_gemm_reserve_scratch() sizes it up front for callers that must not allocate later.
// A block that has been handed out is never freed or moved: kernels already enqueued, and CUDA graphs that
// captured a call, keep using its address.  When a larger product arrives a new, larger block is allocated
// beside the old ones (the old ones stay until the process ends); there is no device-wide synchronisation.
static void* g_scratch[PMB_MAX_DEVICES] = {nullptr};
static size_t g_scratch_bytes[PMB_MAX_DEVICES] = {0};
static std::mutex g_scratch_mu;

pmb_status gemm_scratch(size_t bytes, void** out, cudaStream_t user_stream, bool check_capture) {
  int dev = 0;
  PMB_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= PMB_MAX_DEVICES) return fail(PMB_ERR_UNSUPPORTED, "device ordinal %d out of range", dev);
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  if (g_scratch_bytes[dev] < bytes) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (check_capture && cudaStreamIsCapturing(user_stream, &cap) == cudaSuccess && cap != cudaStreamCaptureStatusNone)
      return fail(PMB_ERR_WORKSPACE, "gemm: the pair scratch would have to grow during stream capture; call pmb_gemm_reserve_scratch(%zu) first", bytes);
    size_t want = align_up(bytes + bytes / 4, (size_t)1 << 20);
    void* fresh = nullptr;
    PMB_CUDA(cudaMalloc(&fresh, want));
    g_scratch[dev] = fresh;          // the previous block is deliberately kept alive
    g_scratch_bytes[dev] = want;
  }
  *out = g_scratch[dev];
  return PMB_OK;
}

// fp32 operands: one elementwise pass each into the scratch (rows compacted to a pitch that is a multiple of 8),
// then gemm_pairs.
pmb_status gemm_f32_via_bf16x2(cudaStream_t st, int ta, int tb, int64_t M, int64_t N, int64_t K, const float* A, int64_t lda,
                               const float* B, int64_t ldb, float* C, int64_t ldc, const float* R, int tile_mode) {
  const int64_t a_rows = ta ? K : M, a_cols = ta ? M : K, b_rows = tb ? N : K, b_cols = tb ? K : N;
  const int64_t a_ld = (int64_t)align_up((size_t)a_cols, 8), b_ld = (int64_t)align_up((size_t)b_cols, 8);
  const size_t a_el = align_up((size_t)a_rows * a_ld, 64), b_el = align_up((size_t)b_rows * b_ld, 64);
  void* scratch = nullptr;
  PMB_TRY(gemm_scratch((2 * a_el + 2 * b_el) * 2 + 1024, &scratch, st, true));
  uint16_t* a_hi = static_cast<uint16_t*>(scratch);
  uint16_t* a_lo = a_hi + a_el;
  uint16_t* b_hi = a_lo + a_el;
  uint16_t* b_lo = b_hi + b_el;
  PMB_TRY(split_pair16(st, A, a_rows, a_cols, lda, a_hi, a_lo, a_ld));
  PMB_TRY(split_pair16(st, B, b_rows, b_cols, ldb, b_hi, b_lo, b_ld));
  return gemm_pairs(st, ta, tb, M, N, K, Pair16{a_hi, a_lo, a_ld}, Pair16{b_hi, b_lo, b_ld}, C, ldc, R, tile_mode);
}

}  // namespace pmb

extern "C" pmb_status pmb_gemm_reserve_scratch(size_t bytes) {
  void* p = nullptr;
  return pmb::gemm_scratch(bytes, &p, nullptr, false);
}

extern "C" pmb_status pmb_gemm_bf16(void* stream, int32_t trans_a, int32_t trans_b, int64_t M, int64_t N, int64_t K,
                                    const uint16_t* d_A, int64_t lda, const uint16_t* d_B, int64_t ldb,
                                    void* d_C, int64_t ldc, const void* d_R, int32_t out_bf16) {
  using namespace pmb;
  if (!d_A || !d_B || !d_C) return fail(PMB_ERR_ARG, "gemm_bf16: NULL operand");
  if (lda < (trans_a ? M : K) || ldb < (trans_b ? K : N) || ldc < N) return fail(PMB_ERR_SHAPE, "gemm_bf16: leading dimension smaller than the row length");
  return gemm_bf16(static_cast<cudaStream_t>(stream), trans_a != 0, trans_b != 0, M, N, K, d_A, lda, d_B, ldb, d_C, ldc, d_R, out_bf16 != 0);
}

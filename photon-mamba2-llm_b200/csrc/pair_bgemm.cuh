// Batched tile contraction on tcgen05 with operands that are already bf16 in HBM: plain bf16 (NS = 1) or the
// (hi, lo) pair of an fp32 tensor (NS = 2: lo*hi + hi*lo + hi*hi per k-step), specialised by an Op functor.
//
//   OUT[batch](m, n) = sum over segments s, k:  A_s[m,k] * B_s[k,n]
//
// Each CTA owns one 128 x BN output tile of one batch entry.  Operand tiles arrive by TMA (rank-3 bf16 tensor maps:
// contiguous axis, row axis, head/group axis; 128-byte swizzle) into a ring and go to the tensor core as they land:
// nothing rescales or splits a tile in shared memory (the producers of the operands wrote the scaled pairs).  One lane
// issues the MMAs into a TMEM accumulator that lives across all segments; eight warps then drain TMEM and hand
// 32-column row pieces to Op::store.  Operand majorness may differ per segment.  All mbarrier waits are bounded;
// expiry raises *status and the CTA leaves through the common exit.
//
// Op interface (device side; BN and NS are static constexpr):
//   int  Mdim, Ndim                                  output extents per batch entry
//   bool init(int batch, int m0, int n0)             false: tile not needed
//   int  nseg()
//   void seg(int s, int m0, int n0, int& kt0, int& kt1, int& amap, int& bmap, int& a_mn, int& b_mn)
//        k tiles [kt0, kt1) of 64; which of the 4 logical tensor maps feed A and B (map 2i = hi, 2i+1 = lo); majorness
//   void a_coord(int s, int kt, int m0, int& c0, int& c1, int& c2)   TMA coordinates of the A tile
//   void b_coord(int s, int kt, int n0, int& c0, int& c1, int& c2)   (K-major: (k, row, z); MN-major: (mn, k, z))
//   void store(int m, int nb, const float (&v)[32])  row m, columns nb..nb+31 (caller-checked m < Mdim)
#pragma once
#include "tc_common.cuh"

namespace pmb {
namespace pbg {

using namespace tcx;

constexpr int BM = 128, BK = 64, NEW_WARPS = 8, NEW = NEW_WARPS * 32, NTHREADS = 64 + NEW;

struct MapSet { CUtensorMap m[8]; };   // logical map i: m[2i] = hi (or the plain tensor), m[2i+1] = lo

template <int BN, int NS>
struct Geometry {
  static constexpr int A_BYTES = BM * 128;            // 128 rows x 64 bf16
  static constexpr int B_BYTES = BN * 128;
  static constexpr int PART = A_BYTES + B_BYTES;      // the hi (or lo) tiles of one stage
  static constexpr int STAGE_BYTES = NS * PART;
  // two stages, so that two CTAs share an SM: the problems are short chains that leave the SM idle between dependent steps
  static constexpr int STAGES = 2, CTAS_PER_SM = 2;
  static_assert(STAGES * STAGE_BYTES <= 100 * 1024, "two CTAs per SM");
  static constexpr int RING_BYTES = STAGES * STAGE_BYTES;
  static constexpr int SMEM_BASE = RING_BYTES + 1024 /*alignment slack*/ + 256 /*barriers*/;
};

template <class Op>
__global__ void __launch_bounds__(NTHREADS, Geometry<Op::BN, Op::NS>::CTAS_PER_SM)
pair_bgemm_kernel(const __grid_constant__ MapSet maps, Op op, unsigned int* __restrict__ status) {
  constexpr int BN = Op::BN, NS = Op::NS;
  using G = Geometry<BN, NS>;
  constexpr int STAGES = G::STAGES;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t tiles = (raw + 1023u) & ~1023u;
  uint8_t* tiles_ptr = smem_raw + (tiles - raw);
  const uint32_t bars = tiles + G::RING_BYTES;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
  const uint32_t accum_bar = bars + 8u * (2 * STAGES);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(tiles_ptr + G::RING_BYTES + 8 * (2 * STAGES + 1));
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = (int)blockIdx.y * BM, n0 = blockIdx.x * BN;
  if (!op.init((int)blockIdx.z, m0, n0)) return;   // uniform per CTA
  const int nseg = op.nseg();

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
    mbar_init(accum_bar, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  constexpr int TMEM_COLS = BN < 32 ? 32 : BN;
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_acc = *tmem_slot;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int it = 0;
      bool stop = false;
      for (int sg = 0; sg < nseg && !stop; ++sg) {
        int kt0, kt1, amap, bmap, a_mn, b_mn;
        op.seg(sg, m0, n0, kt0, kt1, amap, bmap, a_mn, b_mn);
        for (int kt = kt0; kt < kt1; ++kt, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(empty_bar(s), ph ^ 1u)) { atomicOr(status, 1u); *abort_flag = 1; stop = true; break; }
          if (*abort_flag) { stop = true; break; }
          mbar_expect_tx(full_bar(s), G::STAGE_BYTES);
          int a0, a1, a2, b0, b1, b2;
          op.a_coord(sg, kt, m0, a0, a1, a2);
          op.b_coord(sg, kt, n0, b0, b1, b2);
#pragma unroll
          for (int sp = 0; sp < NS; ++sp) {
            const uint32_t a_dst = tiles + s * G::STAGE_BYTES + sp * G::PART, b_dst = a_dst + G::A_BYTES;
            if (!a_mn) {
              tma_load_3d(a_dst, &maps.m[2 * amap + sp], a0, a1, a2, full_bar(s));
            } else {
#pragma unroll
              for (int j = 0; j < BM / 64; ++j) tma_load_3d(a_dst + j * (BK * 128), &maps.m[2 * amap + sp], a0 + 64 * j, a1, a2, full_bar(s));
            }
            if (!b_mn) {
              tma_load_3d(b_dst, &maps.m[2 * bmap + sp], b0, b1, b2, full_bar(s));
            } else {
#pragma unroll
              for (int j = 0; j < (BN + 63) / 64; ++j) tma_load_3d(b_dst + j * (BK * 128), &maps.m[2 * bmap + sp], b0 + 64 * j, b1, b2, full_bar(s));
            }
          }
        }
      }
      if (*abort_flag) {
        // give copies already in flight a bounded chance to land before the CTA exits
        for (int k = (it > STAGES ? it - STAGES : 0); k < it; ++k) mbar_wait(full_bar(k % STAGES), (k / STAGES) & 1);
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (the whole warp waits, one elected lane issues) ----------------
    auto wait_all = [&](uint32_t bar, uint32_t parity, unsigned int code) -> bool {
      const bool got = __all_sync(0xffffffffu, mbar_wait(bar, parity));
      if (!got && lane == 0) { atomicOr(status, code); *abort_flag = 1; }
      return got && !__any_sync(0xffffffffu, *abort_flag != 0);
    };
    {
      int it = 0;
      bool stop = false;
      const uint32_t d_hi = desc_hi(1024, 2);
      for (int sg = 0; sg < nseg && !stop; ++sg) {
        int kt0, kt1, amap, bmap, a_mn, b_mn;
        op.seg(sg, m0, n0, kt0, kt1, amap, bmap, a_mn, b_mn);
        const uint32_t idesc = idesc_bf16(a_mn, b_mn, BM, BN);
        // K-major: 128-byte rows, 8-row groups 1024 B apart, a k-step (16) advances 32 B.
        // MN-major: 64-wide blocks BK*128 B apart, 8-k-row groups 1024 B apart, a k-step advances 2048 B.
        const uint32_t a_lbo = a_mn ? BK * 128 : 16, b_lbo = b_mn ? BK * 128 : 16;
        const uint32_t a_step = (a_mn ? 2048u : 32u) >> 4, b_step = (b_mn ? 2048u : 32u) >> 4;
        constexpr uint32_t LO = G::PART >> 4;
        for (int kt = kt0; kt < kt1; ++kt, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!wait_all(full_bar(s), ph, 2u)) { stop = true; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a_s = tiles + s * G::STAGE_BYTES;
          const uint32_t al0 = desc_lo(a_s, a_lbo), bl0 = desc_lo(a_s + G::A_BYTES, b_lbo);
          if (elect_one()) {
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            const uint32_t al = al0 + k * a_step, bl = bl0 + k * b_step;
            const bool first = it == 0 && k == 0;
            if (NS == 2) {
              mma_f16_h(tmem_acc, al + LO, d_hi, bl, d_hi, idesc, first ? 0u : 1u);
              mma_f16_h(tmem_acc, al, d_hi, bl + LO, d_hi, idesc, 1u);
              mma_f16_h(tmem_acc, al, d_hi, bl, d_hi, idesc, 1u);
            } else {
              mma_f16_h(tmem_acc, al, d_hi, bl, d_hi, idesc, first ? 0u : 1u);
            }
          }
          umma_commit(empty_bar(s));
          }
          __syncwarp();
        }
      }
      if (elect_one()) umma_commit(accum_bar);
      __syncwarp();
    }
  } else {
    // ---------------- epilogue warps ----------------
    const int lane_base = (warp & 3) * 32;       // the TMEM lane quarter this warp may read
    const int grp = (warp - 2) >> 2;             // two warps share a quarter: they take alternate 32-column chunks
    const int m = m0 + lane_base + lane;
    const bool acc_ok = __all_sync(0xffffffffu, mbar_wait_idle(accum_bar, 0));
    if (!acc_ok && lane == 0) { atomicOr(status, 8u); *abort_flag = 1; }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const bool aborted = __any_sync(0xffffffffu, *abort_flag != 0);
    if (acc_ok && !aborted) {
#pragma unroll 1
      for (int c0 = grp * 32; c0 < BN; c0 += 64) {
        uint32_t r[32];
        tmem_ld32(tmem_acc + ((uint32_t)lane_base << 16) + (uint32_t)c0, r);
        if (m < op.Mdim && n0 + c0 < op.Ndim) {
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
          op.store(m, n0 + c0, v);
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_acc), "r"(TMEM_COLS) : "memory");
  }
}

template <class Op>
static pmb_status launch(cudaStream_t st, const MapSet& maps, const Op& op, int batches, unsigned int* status) {
  using G = Geometry<Op::BN, Op::NS>;
  PMB_SMEM_OPT_IN(G::SMEM_BASE, pair_bgemm_kernel<Op>);
  const dim3 grid((unsigned)cdiv(op.Ndim, Op::BN), (unsigned)cdiv(op.Mdim, BM), (unsigned)batches);
  pair_bgemm_kernel<Op><<<grid, NTHREADS, G::SMEM_BASE, st>>>(maps, op, status);
  PMB_LAUNCHED();
  return PMB_OK;
}

}  // namespace pbg
}  // namespace pmb

// spmm24.cu — C += A24 * B for the exact-2:4 blocks, on the structured-sparse
// tensor cores (tcgen05.mma.sp, kind::f16: M = 128 rows, N = 128 columns,
// K = 32 with A stored as 128 x 16 kept values plus 2-bit indices).
//
// The reference multiplies its 2:4 blocks with the warp-level mma.sp
// m16n8k32, one 16-row block row per warp (src/cuda_hgemm/src/mma/mmaOBTS_large.cu:19-254).
// tcgen05.mma.sp needs M = 64 or 128 rows of A, so a unit here is a group of
// 8 block rows (128 rows) times one 32-column window of B (the layout is in
// spmm24.h). It runs after the dense kernel, which writes every row of C from
// the other blocks, and adds its products into C.
//
// Roles (512 threads), one CTA per SM, groups taken round-robin from a list
// sorted by decreasing work:
//   warp 0        MMA issuer (one lane); owns TMEM (two 128-column
//                 accumulators, then the metadata column of each A-tile
//                 slot, 64 columns apart: the MMA's metadata address is
//                 kept on a 64-column boundary).
//   warp 1        stage copies: the compact unit data (values, metadata).
//   warp 2        B copies: one 8 KB tile (32 rows of B x 128 columns,
//                 64-byte swizzle) per unit, a batch of two at a time.
//   warps 4..7    epilogue: tcgen05.ld of the accumulator (lane = row) and
//                 C[row, :] += it, rows through the row map; C[row, :] = it
//                 where every block is on this path and no dense kernel ran.
//   warps 8..15   converters, two sets of four: each thread owns one of the 128
//                 rows of a unit, writes its 16 kept values into the zero-filled
//                 A tile in shared memory (32-byte swizzle) and its 32-bit
//                 metadata word into the unit's TMEM column (tcgen05.st).
// Units go from the converters to the MMA issuer in batches of two (half the
// A-tile slots each), with one wait, one fence and one arrival per batch; the
// sets take every other batch, and a batch's B tiles share a barrier. What
// bounds the kernel is the latency of the converters' work (330 cycles a unit)
// and of that hand-off, not the tensor cores; groups with more than an average CTA's units are therefore cut into
// parts over several CTAs (8192 x 8192, 12 % of the blocks, N = 128, 64 groups
// on 152 SMs, the whole step: 135 us without parts and batches, 68 with them, 61
// with the second set of converters and every launch a programmatic dependent of
// the one before, 53 without the dense kernel's pass, 44 with one wait and one
// release of B a batch instead of a unit).
// Waits are bounded like the dense kernel's; an expired wait aborts the CTA
// after its copies and MMAs in flight have landed.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "spmm24.h"
#include "spmm_tc.h"
#include "tc_ptx.cuh"

namespace smat {
namespace dev {

enum : int {
  ERR24_STAGE = 501,
  ERR24_B = 502,
  ERR24_CONV = 503,
  ERR24_MMA = 504,
  ERR24_EPI = 505,
  ERR24_DRAIN = 506
};

struct Sp24Cfg {
  static constexpr int NS = 4;                                   // stage slots
  static constexpr uint32_t STAGE_MAX =
      kSp24StageUnits * sizeof(Sp24Unit) + kSp24StageBlocks * kSp24BlockBytes;
  static constexpr uint32_t STAGE_SLOT = (STAGE_MAX + 1023) / 1024 * 1024;
  static constexpr int NT = 4;                                   // A tile slots (and metadata columns)
  static constexpr int NB = 2;                                   // batches of slots
  static constexpr int UB = NT / NB;                             // units per batch, at most
  static constexpr uint32_t ATILE = 128 * 32;                    // 128 rows x 16 kept values
  static constexpr int NBT = 6;                                  // slots of a batch's B tiles (8 KB copies from L2)
  static constexpr uint32_t BTILE = 128 * 64;                    // 128 columns x 32 k
  static constexpr uint32_t OFF_A = NS * STAGE_SLOT;
  static constexpr uint32_t OFF_B = OFF_A + NT * ATILE;
  static constexpr uint32_t RING = OFF_B + NBT * UB * BTILE;
  static constexpr uint32_t NBARS = 2 * NS + 2 * NB + 2 * NBT + 4 + 1;
  static constexpr uint32_t SMEM_BYTES = 1024 + RING + 8 * NBARS + 8 + 8;
  static constexpr uint32_t META_COL0 = 256;                     // metadata column of A slot t: META_COL0 + 64 t
  static constexpr uint32_t META_STRIDE = 64;
  static constexpr uint32_t TMEM_COLS = 512;                     // 2 x 128 accumulator + NT metadata
  static constexpr int THREADS = 512;
  static_assert(STAGE_MAX % 16 == 0, "stage bytes");
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");
  static_assert(META_COL0 + META_STRIDE * (NT - 1) < TMEM_COLS, "metadata columns inside the allocation");
  static_assert(UB == kSp24Batch, "stages hold whole batches");
};

__device__ __forceinline__ bool w24(uint32_t bar, uint32_t parity, volatile int* abort, int* err, int where,
                                    uint64_t lim) {
  return mbar_poll(bar, parity) || mbar_wait(bar, parity, abort, err, where, lim);
}

// For a whole warp: every lane polls, the vote makes the outcome uniform.
__device__ __forceinline__ bool w24_warp(uint32_t bar, uint32_t parity, volatile int* abort, int* err, int where,
                                         uint64_t lim) {
  return __all_sync(0xffffffffu, w24(bar, parity, abort, err, where, lim));
}

__device__ __noinline__ void drain24(uint32_t bar, uint32_t parity, int* err, uint64_t lim) {
  const uint64_t t0 = globaltimer();
  while (!mbar_try_wait(bar, parity))
    if (globaltimer() - t0 > lim) {
      atomicCAS(err, 0, ERR24_DRAIN);
      return;
    }
}

// 64-byte-swizzle K-major descriptor (rows of 64 bytes, 8-row groups 512 bytes apart).
__device__ __forceinline__ uint64_t desc_kmajor_sw64(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(1) << 16;
  d |= static_cast<uint64_t>(512 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(4) << 61;  // 64-byte swizzle
  return d;
}

__device__ __forceinline__ void umma_sp_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t tmem_meta,
                                            uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %5, 0;\n"
      " tcgen05.mma.sp.cta_group::1.kind::f16 [%0], %1, %2, [%3], %4, p;\n}" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(tmem_meta), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void tmem_st_x1(uint32_t taddr, uint32_t v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(taddr), "r"(v) : "memory");
}

__global__ void __launch_bounds__(Sp24Cfg::THREADS, 1) spmm24_kernel(const __grid_constant__ Sp24Args args) {
  using C = Sp24Cfg;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint64_t* s_full = reinterpret_cast<uint64_t*>(smem + C::RING);
  uint64_t* s_free = s_full + C::NS;
  uint64_t* a_ready = s_free + C::NS;
  uint64_t* a_free = a_ready + C::NB;
  uint64_t* b_full = a_free + C::NB;
  uint64_t* b_free = b_full + C::NBT;
  uint64_t* accfull = b_free + C::NBT;
  uint64_t* accempty = accfull + 2;
  uint64_t* drainbar = accempty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drainbar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint64_t lim = args.wait_ns ? args.wait_ns : kWaitTimeoutNs;
  int* err = args.err;

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::NS; i++) {
      mbar_init(smem_u32(&s_full[i]), 1);
      mbar_init(smem_u32(&s_free[i]), 4 * C::NB);
    }
    for (int i = 0; i < C::NB; i++) {
      mbar_init(smem_u32(&a_ready[i]), 4);
      mbar_init(smem_u32(&a_free[i]), 1);
    }
    for (int i = 0; i < C::NBT; i++) {
      mbar_init(smem_u32(&b_full[i]), 1);
      mbar_init(smem_u32(&b_free[i]), 1);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(smem_u32(&accfull[i]), 1);
      mbar_init(smem_u32(&accempty[i]), 4);
    }
    mbar_init(smem_u32(drainbar), 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(tmem_slot), C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t smem0 = smem_u32(smem);
  const int G = (int)gridDim.x;
  grid_release();  // the kernel that sums split groups may be set up

  if (warp == 1) {
    // ---------------------------------------------------------- stage copies
    if (elect_one()) {
      uint32_t sc = 0;
      bool ok = true;
      for (int gi = blockIdx.x; gi < args.n_groups && ok; gi += G) {
        const Sp24Group g = args.groups[gi];
        for (int nt = 0; nt < args.n_tiles && ok; ++nt)
          for (int st = 0; st < g.nstages; ++st, ++sc) {
            const uint32_t slot = sc % C::NS;
            if (sc == (uint32_t)C::NS) grid_wait();  // slots are freed behind it
            if (sc >= (uint32_t)C::NS &&
                !w24(smem_u32(&s_free[slot]), ((sc - C::NS) / C::NS) & 1, abort_flag, err, ERR24_STAGE, lim)) {
              ok = false;
              break;
            }
            const Sp24Stage s = args.stages[g.stage0 + st];
            const uint32_t fb = smem_u32(&s_full[slot]);
            mbar_arrive_expect_tx(fb, (uint32_t)s.bytes);
            bulk_load(smem0 + slot * C::STAGE_SLOT, args.stream + s.off, (uint32_t)s.bytes, fb);
          }
      }
      if (!ok) {
        const uint32_t lo = sc > (uint32_t)C::NS ? sc - C::NS : 0;
        for (uint32_t k = lo; k < sc; ++k) drain24(smem_u32(&s_full[k % C::NS]), (k / C::NS) & 1, err, lim);
      }
    }
  } else if (warp == 2) {
    // -------------------------------------------------------------- B copies
    // The whole warp, a batch of units at a time (a lane each); the windows of
    // 32 units are read together and ahead.
    const uint64_t pol = make_l2_policy_evict_last();
    uint32_t u = 0;
    bool ok = true;
    grid_wait();  // the windows, made by the launches before this one
    for (int gi = blockIdx.x; gi < args.n_groups && ok; gi += G) {
      const Sp24Group g = args.groups[gi];
      for (int nt = 0; nt < args.n_tiles && ok; ++nt) {
        int ahead = lane < g.nunits ? __ldg(args.unit_window + g.unit0 + lane) : 0;
        for (int i0 = 0; i0 < g.nunits && ok; i0 += 32) {
          const int mine = ahead;
          if (i0 + 32 + lane < g.nunits) ahead = __ldg(args.unit_window + g.unit0 + i0 + 32 + lane);
          const int cnt = min(32, g.nunits - i0);
          for (int i = 0; i < cnt; i += C::UB, ++u) {
            const uint32_t x = u % C::NBT;
            if (u >= (uint32_t)C::NBT &&
                !w24_warp(smem_u32(&b_free[x]), ((u - C::NBT) / C::NBT) & 1, abort_flag, err, ERR24_B, lim)) {
              ok = false;
              break;
            }
            const int n = min(C::UB, cnt - i);
            const int w = __shfl_sync(0xffffffffu, mine, (i + lane) & 31);
            const uint32_t fb = smem_u32(&b_full[x]);
            mbar_arrive_expect_tx_if(fb, (uint32_t)n * C::BTILE, lane == 0);
            __syncwarp();
            bulk_load_hint_if(smem0 + C::OFF_B + (x * C::UB + (lane & (C::UB - 1))) * C::BTILE,
                              args.bpack64 + ((int64_t)nt * args.kw + w) * C::BTILE, C::BTILE, fb, pol, lane < n);
          }
        }
      }
    }
    if (!ok && lane == 0) {
      const uint32_t lo = u > (uint32_t)C::NBT ? u - C::NBT : 0;
      for (uint32_t k = lo; k < u; ++k) drain24(smem_u32(&b_full[k % C::NBT]), (k / C::NBT) & 1, err, lim);
    }
  } else if (warp == 0) {
    // ----------------------------------------------------------------- MMAs
    if (elect_one()) {
      uint32_t k = 0, bc = 0;
      bool ok = true, issued = false;
      grid_wait();  // the limit of its waits is not for the launches before
      for (int gi = blockIdx.x; gi < args.n_groups && ok; gi += G) {
        const Sp24Group g = args.groups[gi];
        for (int nt = 0; nt < args.n_tiles && ok; ++nt, ++k) {
          const uint32_t buf = k & 1;
          if (!w24(smem_u32(&accempty[buf]), (k >> 1) & 1, abort_flag, err, ERR24_MMA, lim)) {
            ok = false;
            break;
          }
          tc_fence_after();
          for (int i = 0; i < g.nunits && ok; ++bc) {
            const uint32_t bt = bc % C::NB, x = bc % C::NBT;
            if (!w24(smem_u32(&a_ready[bt]), (bc / C::NB) & 1, abort_flag, err, ERR24_MMA, lim) ||
                !w24(smem_u32(&b_full[x]), (bc / C::NBT) & 1, abort_flag, err, ERR24_MMA, lim)) {
              ok = false;
              break;
            }
            tc_fence_after();
            const uint64_t ad = desc_kmajor_sw32(smem0 + C::OFF_A + bt * C::UB * C::ATILE);
            const uint64_t bd = desc_kmajor_sw64(smem0 + C::OFF_B + x * C::UB * C::BTILE);
#pragma unroll
            for (int j = 0; j < C::UB; ++j)
              if (i + j < g.nunits)
                umma_sp_f16(tmem + buf * 128, ad + ((j * C::ATILE) >> 4), bd + ((j * C::BTILE) >> 4),
                            tmem + C::META_COL0 + C::META_STRIDE * (bt * C::UB + j), args.idesc | ((128u >> 3) << 17),
                            i + j > 0 ? 1u : 0u);
            i += C::UB;
            issued = true;
            umma_commit(smem_u32(&b_free[x]));
            umma_commit(smem_u32(&a_free[bt]));
          }
          if (!ok) break;
          umma_commit(smem_u32(&accfull[buf]));
        }
      }
      if (!ok && issued) {
        umma_commit(smem_u32(drainbar));
        drain24(smem_u32(drainbar), 0, err, lim);
      }
    }
  } else if (warp >= 8) {
    // ------------------------------------------------------------ converters
    // Thread r (0..127) owns row r of every unit: block row j = r / 16 of the
    // group, row r % 16 of its blocks. It writes the row's 32 bytes of the A
    // tile (16 kept values: the window's first half, then its second; zeros
    // where the block row has no 2:4 block) in the 32-byte swizzle, and TMEM
    // lane r of the unit's metadata column. The sparse MMA reads metadata per
    // 16-row slab (here: one block row j): lane 16 j + 8 h + i holds the
    // 16-bit metadata of K-half h (the window's block h) for row i of the
    // slab in bits 0..15 and for row i + 8 in bits 16..31 (0x4444 for an
    // absent block: indices 0 and 1 of zero values).
    const int q = (warp - 8) & 3;
    const uint32_t set = (uint32_t)(warp - 8) >> 2;
    const int r = q * 32 + lane;
    const int j = r >> 4, rr = r & 15;
    uint32_t bc = 0, sc = 0;
    bool ok = true, behind = false;
    // what the first batches and stages need is there without the launches before;
    // the rest comes when MMAs have freed their slots
    auto wait_before = [&](bool first) {
      if (!first && !behind) grid_wait();
      behind |= !first;
    };
    for (int gi = blockIdx.x; gi < args.n_groups && ok; gi += G) {
      const Sp24Group g = args.groups[gi];
      for (int nt = 0; nt < args.n_tiles && ok; ++nt)
        for (int st = 0; st < g.nstages && ok; ++st, ++sc) {
          const uint32_t slot = sc % C::NS;
          wait_before(sc < (uint32_t)C::NS);
          if (!w24_warp(smem_u32(&s_full[slot]), (sc / C::NS) & 1, abort_flag, err, ERR24_CONV, lim)) {
            ok = false;
            break;
          }
          const int nunits = args.stages[g.stage0 + st].nunits;
          const int nblk = args.stages[g.stage0 + st].nblk;
          const uint8_t* sp = smem + slot * C::STAGE_SLOT;
          const Sp24Unit* units = reinterpret_cast<const Sp24Unit*>(sp);
          const uint8_t* vals = sp + nunits * sizeof(Sp24Unit);
          const uint8_t* metas = vals + (size_t)nblk * 256;
          for (int i0 = 0; i0 < nunits; i0 += C::UB, ++bc) {
            const uint32_t bt = bc % C::NB;
            if (bt != set) continue;  // the other set's batch
            const int n = min(C::UB, nunits - i0);
            wait_before(bc < (uint32_t)C::NB);
            if (bc >= (uint32_t)C::NB &&
                !w24_warp(smem_u32(&a_free[bt]), ((bc - C::NB) / C::NB) & 1, abort_flag, err, ERR24_CONV, lim)) {
              ok = false;
              break;
            }
#pragma unroll
            for (int y = 0; y < C::UB; ++y) {
              if (y >= n) break;
              const uint32_t t = bt * C::UB + (uint32_t)y;
              const uint32_t mask = units[i0 + y].mask;
              const uint32_t first = units[i0 + y].first;
              uint8_t* arow = smem + C::OFF_A + t * C::ATILE + r * 32;
#pragma unroll
              for (int h = 0; h < 2; ++h) {
                const uint32_t bit = 2u * j + h;
                uint4 v = make_uint4(0, 0, 0, 0);
                if ((mask >> bit) & 1u) {
                  const uint32_t blk = first + __popc(mask & ((1u << bit) - 1u));
                  v = *reinterpret_cast<const uint4*>(vals + (size_t)blk * 256 + rr * 16);
                }
                *reinterpret_cast<uint4*>(arow + ((h ^ ((r >> 2) & 1)) << 4)) = v;
              }
              uint32_t word = 0x44444444u;
              const uint32_t mh = (r >> 3) & 1u, mi = r & 7u;  // K-half and slab row of this lane
              const uint32_t bit = 2u * j + mh;
              if ((mask >> bit) & 1u) {
                const uint32_t blk = first + __popc(mask & ((1u << bit) - 1u));
                const uint16_t* mp = reinterpret_cast<const uint16_t*>(metas + (size_t)blk * 32);
                word = (uint32_t)mp[mi] | ((uint32_t)mp[mi + 8] << 16);
              }
              __syncwarp();
              tmem_st_x1(tmem + ((uint32_t)(q * 32) << 16) + C::META_COL0 + C::META_STRIDE * t, word);
            }
            __syncwarp();
            tmem_st_wait();
            fence_proxy_async_smem();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&a_ready[bt]));
          }
          __syncwarp();
          if (lane == 0 && ok) mbar_arrive(smem_u32(&s_free[slot]));
        }
    }
  } else if (warp >= 4) {
    // -------------------------------------------------------------- epilogue
    const int q = warp - 4;
    const int r = q * 32 + lane;
    if (lane == 0) {
      mbar_arrive(smem_u32(&accempty[0]));
      mbar_arrive(smem_u32(&accempty[1]));
    }
    uint32_t k = 0;
    bool ok = true;
    grid_wait();  // C of the dense kernel; the slabs of the call before
    for (int gi = blockIdx.x; gi < args.n_groups && ok; gi += G) {
      const Sp24Group g = args.groups[gi];
      const int64_t prow = (int64_t)g.group * 128 + r;
      const bool has = (g.row_mask >> (r >> 4)) & 1u;
      const bool mine = has || (args.whole_c && g.group * kSp24GroupRows + (r >> 4) < args.n_brows);
      const int crow = mine ? args.row_map[prow] : -1;
      for (int nt = 0; nt < args.n_tiles; ++nt, ++k) {
        const uint32_t buf = k & 1;
        if (!w24_warp(smem_u32(&accfull[buf]), (k >> 1) & 1, abort_flag, err, ERR24_EPI, lim)) {
          ok = false;
          break;
        }
        tc_fence_after();
#pragma unroll 1
        for (int c = 0; c < 128; c += 32) {
          float v[32];
          __syncwarp();
          tmem_ld_x32(tmem + ((uint32_t)(q * 32) << 16) + buf * 128 + c, v);
          if (g.slab >= 0) {
            float4* sp = reinterpret_cast<float4*>(args.slabs + (((int64_t)g.slab * args.n_tiles + nt) * 128 + r) * 128 + c);
#pragma unroll
            for (int m = 0; m < 8; ++m) __stcg(sp + m, make_float4(v[4 * m], v[4 * m + 1], v[4 * m + 2], v[4 * m + 3]));
          } else if (crow >= 0) {
            const int n0 = nt * 128 + c;
            if (!has) {
#pragma unroll
              for (int m = 0; m < 32; ++m) v[m] = 0.0f;
            }
            if (args.c_f16) {
              __half* cp = reinterpret_cast<__half*>(args.C) + (int64_t)crow * args.ldc + n0;
#pragma unroll
              for (int m = 0; m < 32; ++m)
                if (n0 + m < args.N) cp[m] = __float2half_rn(args.whole_c ? v[m] : __half2float(cp[m]) + v[m]);
            } else {
              float* cp = reinterpret_cast<float*>(args.C) + (int64_t)crow * args.ldc + n0;
#pragma unroll
              for (int m = 0; m < 32; ++m)
                if (n0 + m < args.N) cp[m] = args.whole_c ? v[m] : cp[m] + v[m];
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&accempty[buf]));
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, C::TMEM_COLS);
  }
}

// The split groups' parts, added in order and then into C: a block per 16 rows
// of a group, a thread per column.
// What is the handle's own is looked up before the wait for the parts (the step
// of 8192 x 8192, 12 % of the blocks: 44.4 us with the lookups behind it, 43.5).
__global__ void __launch_bounds__(128) sum24_kernel(const __grid_constant__ Sp24Args args) {
  const int u = (int)blockIdx.x / args.n_tiles, nt = (int)blockIdx.x % args.n_tiles;
  const Sp24Group g = args.split[u];
  const int j = (int)blockIdx.y;  // block row of the group
  const int n = nt * 128 + (int)threadIdx.x;
  const bool has = (g.row_mask >> j) & 1u;
  const bool mine = n < args.N && (has || (args.whole_c && g.group * kSp24GroupRows + j < args.n_brows));
  int4 rows[4] = {};
  if (mine) {
    const int4* const row4 = reinterpret_cast<const int4*>(args.row_map + (int64_t)g.group * 128 + 16 * j);
#pragma unroll
    for (int m = 0; m < 4; ++m) rows[m] = __ldg(row4 + m);
  }
  grid_wait();
  if (!mine) return;
  const float* src = args.slabs + (((int64_t)g.slab * args.n_tiles + nt) * 128 + 16 * j) * 128 + threadIdx.x;
  const int64_t step = (int64_t)args.n_tiles * 128 * 128;
  float acc[16];
#pragma unroll
  for (int m = 0; m < 16; ++m) acc[m] = 0.0f;
  for (int p = 0; has && p < g.nparts; ++p, src += step) {
    float t[16];
#pragma unroll
    for (int m = 0; m < 16; ++m) t[m] = __ldcg(src + m * 128);
#pragma unroll
    for (int m = 0; m < 16; ++m) acc[m] += t[m];
  }
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    const int4 r4 = rows[m / 4];
    const int row = m % 4 == 0 ? r4.x : (m % 4 == 1 ? r4.y : (m % 4 == 2 ? r4.z : r4.w));
    if (row < 0) continue;
    const int64_t off = (int64_t)row * args.ldc + n;
    if (args.c_f16) {
      __half* cp = reinterpret_cast<__half*>(args.C) + off;
      *cp = __float2half_rn(args.whole_c ? acc[m] : __half2float(*cp) + acc[m]);
    } else {
      float* cp = reinterpret_cast<float*>(args.C) + off;
      *cp = args.whole_c ? acc[m] : *cp + acc[m];
    }
  }
}

}  // namespace dev

cudaError_t sp24_launch(const Sp24Args& args, int grid, bool behind, cudaStream_t stream) {
  static std::atomic<uint64_t> done{0};
  int d = 0;
  if (cudaGetDevice(&d) != cudaSuccess) return cudaErrorInvalidDevice;
  const uint64_t bit = d < 64 ? (1ull << d) : 0;
  if (!bit || !(done.load() & bit)) {
    const cudaError_t e = cudaFuncSetAttribute(dev::spmm24_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               dev::Sp24Cfg::SMEM_BYTES);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return e;
    }
    done.fetch_or(bit);
  }
  void* params[] = {const_cast<Sp24Args*>(&args)};
  const cudaError_t e = launch_kernel(reinterpret_cast<const void*>(dev::spmm24_kernel), dim3((unsigned)grid),
                                      dim3(dev::Sp24Cfg::THREADS), dev::Sp24Cfg::SMEM_BYTES, stream, behind, params);
  if (e != cudaSuccess || args.n_split == 0) return e;
  return launch_kernel(reinterpret_cast<const void*>(dev::sum24_kernel),
                       dim3((unsigned)(args.n_split * args.n_tiles), kSp24GroupRows), dim3(128), 0, stream, true, params);
}

}  // namespace smat

// spmm_tc.cu — block-sparse x dense SpMM on sm_103a tensor cores.
//
// The reference computes each 16 x 8 tile of C with one warp and mma.sync,
// re-reading every A block ceil(N/8) times (src/cuda_hgemm/src/mma/mmaOBT.cu:18-158).
// Here one CTA owns a PANEL of R consecutive block rows and a 128*NSUB-wide
// column tile of C, and computes the transposed product
//
//     C[rows of block row r, n-tile]^T  +=  B[col : col+16, n-tile]^T * A_blk^T
//
// with tcgen05.mma (M = 128 dense columns of B, N = bh rows of the block,
// K = 16 = bw), accumulating in FP32 in tensor memory: R*NSUB accumulators of
// 128 lanes x bh columns per buffer, double buffered.
//
// Blocks of a panel are visited in order of their block column, so that the
// B tile of a column is loaded once and used by every block row of the panel
// that has a block there. Blocks with few nonzero columns are taken apart
// (bcsr.cpp: build_plan): sixteen nonzero columns of a block row, from
// whichever of its blocks, make one GATHERED block, whose B tile holds the
// sixteen rows of B they need. The A blocks are stored on the device in
// exactly the visiting order, already in the shared-memory layout the MMA
// reads (32-byte swizzle). The pipeline moves STAGES: one stage carries a
// number of A blocks, the packed B tiles they need and the stage's MMA list
// (precomputed on the host, stored before the blocks so that one copy brings
// both), so the hand-off between the copies and the tensor cores is one
// full/empty barrier pair per stage.
//
// Roles (576 threads, FP8 768):
//   warps 12..17    copy warps, in pairs that own whole stages: bulk copies for
//                   the list, the A blocks and the B tiles, 16-byte copies
//                   through the load path for the rows of gathered tiles.
//   warps 0..3      MMA issuers, one elected lane each, one per quarter of the
//                   panel's block rows (one thread issues at most one
//                   tcgen05.mma per 64-75 cycles, the tensor pipe takes one of
//                   this width every 39); warp 0 also owns TMEM.
//   warps 4..11     epilogue, two per TMEM lane quadrant: tcgen05.ld -> row
//                   scatter through row_map -> FP32 or FP16 stores of C
//                   (coalesced along N).
//
// Consecutive block rows with a block at the same column form one MMA
// (N = bh * run length), so dense panels need far fewer instructions.
//
// What bounds it (GB300; time of the whole step with the packing of B):
//   R-MAT, 2^16 rows, 816K blocks, N = 128: 256 us at first; 216 with waits
//     that branch on the barrier's own predicate, elected issue and no barrier
//     among the copy warps; 148 with gathered blocks (615K -> 284K MMAs, 1.6 ->
//     1.0 GB into shared memory); 115 with the drain as a loop, (item, column
//     tile) units and the roles above; 109 with the parts of split panels added
//     by a kernel of its own and the launches overlapping; 103 with A prefetched
//     into L2. The turn of a stage slot (copy issue, landing, MMAs) sets the
//     pace: 36 bytes a cycle into an SM of the 70 it can take, 44 % of the narrow
//     MMAs that the tensor pipe could issue.
//   64^3 stencil, N = 256: 358 -> 170 us, 62 of them packing the FP32 B at 6.5
//     TB/s; the kernel moves 450 MB of DRAM data in 108.
//   plain graph, 2^15 rows, 600K entries, N = 256: 231 -> 52 us.
//
// Every wait is bounded (see tc_ptx.cuh); on a timeout the kernel raises the
// CTA's abort flag, records the site in the global error word, lets the
// producers wait for their own copies in flight and the MMA threads for
// their own MMAs, frees TMEM and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>

#include "convert.h"
#include "spmm_tc.h"
#include "tc_ptx.cuh"

namespace smat {
namespace dev {

enum : int { KIND_PLAIN = 0, KIND_SPLIT = 1, KIND_FP8 = 2 };


// Error sites recorded in the global error word.
enum : int {
  ERR_PROD_A = 102,
  ERR_MMA_ACC = 201,
  ERR_MMA_A = 202,
  ERR_MMA_B = 203,
  ERR_MMA_STALL = 205,  // the test stall (SpmmArgs::stall_stage)
  ERR_EPI = 301,
  ERR_CONV = 302,
  ERR_DRAIN = 401,
  ERR_ITEM_TAKE = 103,  // the copy warps waited for a free item-ring slot
  ERR_ITEM_MMA = 204,   // an MMA warp waited for its next item
  ERR_ITEM_EPI = 303,
  ERR_ITEM_CONV = 304
};

// Entries of the CTA's ring of work items (the copy warps take items from
// the launch's counter and run up to a few items ahead of the other roles).
constexpr int kItemRing = 8;
// Units of a CTA that it takes note of, so that it can come back to those whose
// columns of B hold infinite or NaN values.
constexpr int kNotedUnits = 512;

template <int BH, int R, int NSUB, int KIND>
struct Cfg {
  static constexpr int BN = 128 * NSUB;                   // C columns per tile
  static constexpr int NOPS = (KIND == KIND_SPLIT) ? 2 : 1;
  // plan class (stage shape): 256-column B tiles (NSUB 2) halve the tiles per stage
  static constexpr int CLS = KIND == KIND_SPLIT ? 1 : (KIND == KIND_FP8 ? 2 : (NSUB == 2 ? 3 : 0));
  static constexpr int SB = stage_rows(CLS) / BH;         // A blocks per stage (at most)
  static constexpr int ST = stage_tiles(CLS);             // B tiles per stage (at most)
  static constexpr uint32_t ABLK = BH * 32;               // bytes of one A block (one operand)
  static constexpr uint32_t HALF = 2048 * NOPS;           // bytes of 64 columns of a B tile (hi, then lo)
  static constexpr uint32_t SUB = 2 * HALF;               // bytes of a 128-column subtile
  static constexpr uint32_t TILEB = SUB * NSUB;           // bytes of one B tile slot
  static constexpr bool FP8 = KIND == KIND_FP8;
  // stage: [header] [A blocks hi | lo] [B tiles]; the header and the blocks
  // land with one copy. The FP8 form lands [header | e4m3 blocks | scales],
  // which the converter warps turn into the FP16 A blocks after it.
  static constexpr uint32_t HDR = kStageHdrBytes;
  static constexpr uint32_t OFF_A = FP8 ? (HDR + SB * 256 + fp8_scale_bytes(SB) + 64 * ST + 255) / 256 * 256 : HDR;
  static constexpr uint32_t OFF_B = (OFF_A + SB * ABLK * NOPS + 1023) / 1024 * 1024;
  static constexpr uint32_t STAGE = (OFF_B + ST * TILEB + 1023) / 1024 * 1024;
  static constexpr uint32_t SMEM_AVAIL = 227 * 1024 - 14336;  // minus alignment slack, barriers and row tables
  static constexpr int NS_FIT = (int)(SMEM_AVAIL / STAGE);
  static constexpr int NS = NS_FIT < 2 ? 2 : (NS_FIT > 8 ? 8 : NS_FIT);  // stages
  static constexpr uint32_t SUB_COLS = R * BH;            // TMEM columns of one 128-column subtile
  static constexpr uint32_t ACC_COLS = NSUB * SUB_COLS;   // TMEM columns per buffer
  static constexpr uint32_t TMEM_COLS = 2 * ACC_COLS;
  static constexpr int NMMA = kMmaWarps;                  // MMA-issuing warps
  static constexpr int NEPI = 8;                          // epilogue warps: two per TMEM lane quadrant
  static constexpr int NPROD = FP8 ? 4 : 6;               // copy warps, in pairs (3 stages in flight)
  static constexpr int NCONV = FP8 ? 8 : 0;               // FP8 converter warps, two sets of four
  static constexpr uint32_t SMEM_BARS = 8 * (2 * NS + 4 + NMMA + (FP8 ? 2 * NS : 0) + 2 * kItemRing + 1);
  static constexpr int GLIST = (ST + 1) / 2 * 16 * 4;     // bytes of a copy warp's rows of gathered tiles
  // then the TMEM address, the abort flag, the ring of work items, the
  // epilogue warps' row tables, the copy warps' gather lists and the notes of units
  static constexpr uint32_t SMEM_BYTES = 1024 + NS * STAGE + SMEM_BARS + 24 + kItemRing * sizeof(WorkItem) +
                                         NEPI * (R * BH / 2) * 4 + NPROD * GLIST + kNotedUnits * 4 +
                                         (kNotedUnits / 32 + 1) * 4;
  static constexpr int THREADS = 32 * (4 + NEPI + NPROD + NCONV);  // MMA, epilogue, copy, converter warps
  static_assert(TMEM_COLS >= 32 && TMEM_COLS <= 512 && (TMEM_COLS & (TMEM_COLS - 1)) == 0,
                "TMEM allocation must be a power of two in [32, 512]");
  static_assert(BH == 16 || BH == 32, "block height");
  static_assert(NSUB == 1 || (NSUB == 2 && KIND == KIND_PLAIN), "256-column tiles: plain form only");
  static_assert(R <= 32, "slot field is 5 bits");
  static_assert(SB <= kMaxStageBlocks, "position field is 5 bits");
  static_assert(stage_hdr_max(SB) <= (int)HDR, "stage header");
  // a stage tile of NSUB 128-column subtiles is NSUB copies (packed B is
  // [128-column tile][k-block]: the subtiles are not adjacent)
  static_assert(ST * NSUB <= 32 && ST <= 16 && ST <= kMaxStageTiles, "a lane per copy, four per gathered tile");
  static_assert((ST + 1) / 2 * NSUB < 32, "lane 31 is free for the A region");
  static_assert(NS_FIT >= 2, "two stages must fit");
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory per CTA");
  static_assert(!FP8 || (BH == 16 && NSUB == 1), "FP8 form: 16 x 16 blocks, 128-column tiles");
};

// Longest wait for a warp's own copies after an abort.
constexpr uint64_t kDrainNs = 20000000ull;

// Wait used only while draining after an abort: bounded, ignores the flag.
__device__ __noinline__ bool mbar_wait_drain(uint32_t bar, uint32_t parity, int* err, uint64_t lim) {
  const uint64_t t0 = globaltimer();
  while (!mbar_try_wait(bar, parity)) {
    if (globaltimer() - t0 > lim) {
      atomicCAS(err, 0, ERR_DRAIN);
      return false;
    }
  }
  return true;
}

// Bounded wait: a tight poll first, then the timed one.
__device__ __forceinline__ bool wait_phase(uint32_t bar, uint32_t parity, volatile int* abort, int* err,
                                           int where, uint64_t lim) {
  return mbar_poll(bar, parity) || mbar_wait(bar, parity, abort, err, where, lim);
}

__device__ __forceinline__ bool wait_phase_sleepy(uint32_t bar, uint32_t parity, volatile int* abort, int* err,
                                                  int where, uint64_t lim) {
  return mbar_try_wait(bar, parity) || mbar_wait_sleepy(bar, parity, abort, err, where, lim);
}

// Item k of the CTA from the item ring, for a role that one lane runs alone:
// waits for it, reads it and frees the ring slot. panel = -1: no more work.
// Returns false when the CTA aborted.
__device__ __forceinline__ bool take_item_one(uint64_t* itemfull, uint64_t* itemempty, const WorkItem* ring,
                                              uint32_t k, volatile int* abort, int* err, int where, uint64_t lim,
                                              WorkItem& wi) {
  const uint32_t r = k % kItemRing;
  if (!wait_phase(smem_u32(&itemfull[r]), (k / kItemRing) & 1, abort, err, where, lim)) return false;
  wi = ring[r];
  mbar_arrive(smem_u32(&itemempty[r]));
  return true;
}

// The same for a whole warp: every lane waits and reads, the vote makes the
// warp's decision uniform, and one lane frees the slot.
__device__ __forceinline__ bool take_item_warp(uint64_t* itemfull, uint64_t* itemempty, const WorkItem* ring,
                                               uint32_t k, int lane, volatile int* abort, int* err, int where,
                                               uint64_t lim, bool sleepy, WorkItem& wi) {
  const uint32_t r = k % kItemRing, bar = smem_u32(&itemfull[r]), par = (k / kItemRing) & 1;
  const bool got = sleepy ? wait_phase_sleepy(bar, par, abort, err, where, lim)
                          : wait_phase(bar, par, abort, err, where, lim);
  if (!__all_sync(0xffffffffu, got)) return false;
  wi = ring[r];
  __syncwarp();
  if (lane == 0) mbar_arrive(smem_u32(&itemempty[r]));
  return true;
}

// Unit `pos` of the launch; panel -1 past the last one.
__device__ __forceinline__ WorkItem unit_at(const SpmmArgs& args, int pos) {
  WorkItem w;
  w.panel = -1;
  if (pos < args.n_items) {
    if (args.probs) {
      w = args.items[pos];
    } else {  // one problem: every item once per column tile
      const uint32_t it = (uint32_t)pos / (uint32_t)args.one.n_tiles;
      w = args.items[it];
      w.nt = pos - (int)(it * (uint32_t)args.one.n_tiles);
    }
  }
  return w;
}

// Infinite and NaN values of B. A block's stored zeros count: zero times such
// a value is NaN in every row of the block. The columns that gathering left
// out (all zero in the block) are looked up here, for a launch whose packed B
// says that it holds such values: which of the columns `open` of n0 .. n0 + 63 of C
// (n0 a multiple of 64; all of them below N) are NaN in the rows of the plan slot
// whose all-zero columns are poison[q0 .. q1). For a whole warp.
//
// What bounds it: latency, two loads behind each other for 128 entries. An entry (16
// rows of B) is looked at only for columns that its packing unit holds such a
// value in and that are not known yet, so that few are: a lane per entry and the
// unit's two words of columns, then a lane per 16 bytes of the rows. (One infinity
// in B, R-MAT of 2^16 rows and 1M entries, N = 128: 140 us a call, 50 without; a
// thread per column that read every zero column's value took 17,400.)
__device__ __forceinline__ uint64_t poisoned64(const ProblemDesc& P, int nops, int q0, int q1, int n0, uint64_t open,
                                               int lane) {
  const uint32_t E = P.b_bf16 ? 0x7f80u : 0x7c00u;
  const uint64_t* const cols = reinterpret_cast<const uint64_t*>(P.bcols) + (int64_t)(n0 >> 6) * pack_units_k(P.K);
  const int r = lane >> 3, c = lane & 7;  // rows r, r + 4, .. of an entry, columns n0 + 8 c ..
  const uint8_t* const tile = P.bpack + (int64_t)(n0 >> 7) * P.bp_kbs * (4096 * nops) + ((n0 >> 6) & 1) * (2048 * nops);
  uint64_t bad = 0;
  for (int q = q0 + lane; q - lane < q1 && open != 0; q += 32 * 4) {
    int kbs[4];
    uint64_t in[4], any = 0;
#pragma unroll
    for (int x = 0; x < 4; ++x) kbs[x] = q + 32 * x < q1 ? __ldg(&P.poison[q + 32 * x].x) : -1;
#pragma unroll
    for (int x = 0; x < 4; ++x) in[x] = kbs[x] >= 0 ? __ldcg(cols + kbs[x] / kPackUnitBlocks) : 0ull;
#pragma unroll
    for (int x = 0; x < 4; ++x) any |= in[x];
    if (!__any_sync(0xffffffffu, (any & open) != 0)) continue;
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      for (uint32_t m = __ballot_sync(0xffffffffu, (in[x] & open) != 0); m != 0; m &= m - 1) {
        const int src = __ffs((int)m) - 1;
        if ((__shfl_sync(0xffffffffu, in[x], src) & open) == 0) continue;
        const int kb = __shfl_sync(0xffffffffu, kbs[x], src);
        const uint32_t mask = (uint32_t)__ldg(&P.poison[q - lane + 32 * x + src].y);
        const uint8_t* const p = tile + (int64_t)kb * (4096 * nops);
        uint32_t b = 0;  // bit i: column n0 + 8 c + i
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int k = r + 4 * x;
          if (((mask >> k) & 1u) == 0) continue;
          const uint4 v = __ldcg(reinterpret_cast<const uint4*>(p + k * 128 + ((c ^ (k & 7)) << 4)));
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int z = 0; z < 4; ++z)
            b |= ((w[z] & E) == E ? 1u : 0u) << (2 * z) | (((w[z] >> 16) & E) == E ? 2u : 0u) << (2 * z);
        }
        b <<= 8 * (c & 3);
        const uint32_t lo = __reduce_or_sync(0xffffffffu, c < 4 ? b : 0u);
        const uint32_t hi = __reduce_or_sync(0xffffffffu, c < 4 ? 0u : b);
        bad |= (lo | (uint64_t)hi << 32) & open;
        open &= ~bad;
      }
    }
  }
  return bad;
}

__device__ __noinline__ uint64_t poisoned64_call(const ProblemDesc& P, int nops, int q0, int q1, int n0, uint64_t open,
                                               int lane) {
  return poisoned64(P, nops, q0, q1, n0, open, lane);
}

// The columns n0 .. n0 + 63 below N, of which `part` (a mask) is wanted.
__device__ __forceinline__ uint64_t columns64(int n0, int N, uint64_t part) {
  return N - n0 >= 64 ? part : (N > n0 ? part & ((1ull << (N - n0)) - 1) : 0ull);
}

// The same for column n alone, by one thread, one load behind the other: in the
// drain, for units beyond those that a CTA takes note of. (The search above called
// there, or given to two more warps, took 1-8 % of the time of calls with finite B;
// at the kernel's end it is inlined for the same reason.)
__device__ __noinline__ bool poisoned1(const ProblemDesc& P, int nops, int q0, int q1, int64_t n) {
  const uint32_t E = P.b_bf16 ? 0x7f80u : 0x7c00u;
  const uint8_t* base =
      P.bpack + (n >> 7) * P.bp_kbs * (4096 * nops) + ((n >> 6) & 1) * (2048 * nops) + (n & 7) * 2;
  const uint32_t* const cols = P.bcols + (n >> 6) * pack_units_k(P.K) * 2 + ((n >> 5) & 1);
  const uint32_t c = (uint32_t)(n >> 3) & 7u;
  for (int q = q0; q < q1; ++q) {
    const int2 e = P.poison[q];
    if (((cols[e.x / kPackUnitBlocks * 2] >> (n & 31)) & 1u) == 0) continue;
    for (uint32_t m = (uint32_t)e.y; m != 0; m &= m - 1) {
      const uint32_t k = (uint32_t)__ffs((int)m) - 1;
      const uint32_t v = *reinterpret_cast<const uint16_t*>(base + (int64_t)e.x * (4096 * nops) + k * 128 +
                                                            ((c ^ (k & 7)) << 4));
      if ((v & E) == E) return true;
    }
  }
  return false;
}

// Whether the packed B of a column tile holds infinite or NaN values, for a whole
// warp, looked up once per problem and column tile.
struct OddTiles {
  int prob = -1;                // problem that known and val are about
  uint64_t known = 0, val = 0;  // a bit per column tile below 64
  __device__ __forceinline__ bool look(const ProblemDesc& P, int nsub, int p, int nt, int lane) {
    if (p != prob) {
      prob = p;
      known = val = 0;
    }
    const uint64_t bit = nt < 64 ? 1ull << nt : 0ull;
    if (known & bit) return (val & bit) != 0;
    const int64_t fs = pack_flag_stride(P.K);
    const int h0 = nt * (2 * nsub), h1 = min(h0 + 2 * nsub, (P.N + 63) >> 6);
    const uint4* fl = reinterpret_cast<const uint4*>(P.bflags + (int64_t)h0 * fs);
    uint32_t any = 0;
#pragma unroll 4
    for (int64_t x = lane; x < (h1 - h0) * fs / 16; x += 32) {
      const uint4 f = __ldcg(fl + x);
      any |= f.x | f.y | f.z | f.w;
    }
    const bool odd = __any_sync(0xffffffffu, any != 0);
    known |= bit;
    if (odd) val |= bit;
    return odd;
  }
};

// NaN into what gathering left out of a plan slot's rows (`bh` of them) of C,
// columns n0 .. n0 + 63, when finite values are stored there.
__device__ __forceinline__ void poison_slot(const ProblemDesc& P, int nops, int slot, int bh, int n0, uint64_t part,
                                            int lane) {
  const int q0 = __ldg(P.poison_ptr + slot), q1 = __ldg(P.poison_ptr + slot + 1);
  part = columns64(n0, P.N, part);
  const uint64_t bad = q0 < q1 && part != 0 ? poisoned64(P, nops, q0, q1, n0, part, lane) : 0ull;
  if (bad == 0) return;
  const int32_t* const rows = P.row_map + (int64_t)slot * bh;
  for (int m = 0; m < bh; ++m) {
    const int row = __ldg(rows + m);
    for (int n = lane; n < 64; n += 32) {
      if (row < 0 || ((bad >> n) & 1ull) == 0) continue;
      const int64_t at = (int64_t)row * P.ldc + n0 + n;
      if (P.c_f16) static_cast<__half*>(P.C)[at] = __float2half_rn(__int_as_float(0x7fffffff));
      else static_cast<float*>(P.C)[at] = __int_as_float(0x7fffffff);
    }
  }
  __syncwarp();
}

// The same for the units whose bits are set in `odd` (units[k]: the CTA's k-th
// unit), when all of the CTA's units are stored. The CTA's warps share the slots and
// 64-column pieces of a unit.
__device__ __forceinline__ void poison_units(const SpmmArgs& args, const int* units, const uint32_t* odd, int nops,
                                             int bh, int R, int nsub, int warp, int nwarps, int lane) {
  for (int k = 0; k < kNotedUnits; ++k) {
    if (((odd[k >> 5] >> (k & 31)) & 1u) == 0) continue;
    const WorkItem w = unit_at(args, units[k]);
    const ProblemDesc& P = args.probs ? args.probs[w.prob] : args.one;
    for (int t = warp; t < 2 * nsub * R; t += nwarps)
      poison_slot(P, nops, w.panel * R + t % R, bh, w.nt * 128 * nsub + t / R * 64, ~0ull, lane);
  }
}

// For an epilogue warp of the FP8 form, behind a unit's drain: its half of the slots
// and its 32 columns.
__device__ __noinline__ void poison_half(const ProblemDesc& P, int s0, int nslots, int n0, uint64_t part, int lane) {
  for (int s = s0; s < s0 + nslots; ++s) poison_slot(P, 1, s, 16, n0, part, lane);
}

// Bounded wait for a whole warp: lane 0 polls, the warp learns the outcome
// by shuffle and leaves converged (lanes that each polled would leave the
// loop on different iterations and could run the code after it diverged).
// The __syncwarp puts the other lanes behind what lane 0 acquired; a shuffle
// orders no memory.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, int lane, volatile int* abort, int* err,
                                          int where, bool sleepy, uint64_t lim) {
  int got = 1;
  if (lane == 0)
    got = (sleepy ? wait_phase_sleepy(bar, parity, abort, err, where, lim)
                  : wait_phase(bar, parity, abort, err, where, lim))
              ? 1
              : 0;
  __syncwarp();
  return __shfl_sync(0xffffffffu, got, 0) != 0;
}

// Stores a column of 16 rows of C: v[m] to row rows[m] (in shared memory, the
// same for every lane; -1: none) of rows `ldb` bytes apart, base = the
// column's first element. `full`: no row is missing, and nothing is tested per
// row.
template <typename T>
__device__ __forceinline__ T c_value(float v);
template <>
__device__ __forceinline__ float c_value<float>(float v) {
  return v;
}
template <>
__device__ __forceinline__ __half c_value<__half>(float v) {
  return __float2half_rn(v);
}
template <typename T>
__device__ __forceinline__ void store_rows16(uint8_t* base, int64_t ldb, const int* rows, bool full, const float* v) {
  if (full) {
#pragma unroll
    for (int m = 0; m < 16; m += 4) {
      const int4 r = *reinterpret_cast<const int4*>(rows + m);
      __stcs(reinterpret_cast<T*>(base + r.x * ldb), c_value<T>(v[m]));
      __stcs(reinterpret_cast<T*>(base + r.y * ldb), c_value<T>(v[m + 1]));
      __stcs(reinterpret_cast<T*>(base + r.z * ldb), c_value<T>(v[m + 2]));
      __stcs(reinterpret_cast<T*>(base + r.w * ldb), c_value<T>(v[m + 3]));
    }
  } else {
#pragma unroll
    for (int m = 0; m < 16; ++m)
      if (rows[m] >= 0) __stcs(reinterpret_cast<T*>(base + rows[m] * ldb), c_value<T>(v[m]));
  }
}

// Units with at most this many stages: the CTA's next unit is taken when the
// copies of one begin.
constexpr int kShortUnit = 24;

// Unit `k` of the CTA into the item ring (one thread): the launch's unit
// blockIdx.x first, then the next one nobody has taken; panel -1 at the end.
__device__ __forceinline__ void put_unit(const SpmmArgs& args, uint32_t k, uint64_t* itemfull, uint64_t* itemempty,
                                         WorkItem* ring, int* units, volatile int* abort, int* err, uint64_t lim) {
  const uint32_t r = k % kItemRing;
  if (!wait_phase(smem_u32(&itemempty[r]), ((k / kItemRing) & 1) ^ 1, abort, err, ERR_ITEM_TAKE, lim)) return;
  const int pos = k == 0 ? (int)blockIdx.x : (int)gridDim.x + atomicAdd(args.next_item, 1);
  if (k < (uint32_t)kNotedUnits) units[k] = pos;
  ring[r] = unit_at(args, pos);
  mbar_arrive(smem_u32(&itemfull[r]));
}

// A stage record as its copy warp holds it: the counts in every lane, its bulk
// tile's k-block in each lane, and (after load_rows) a 16-byte piece of the
// rows of B of the warp's gathered tiles (every other one, from hf).
struct StageView {
  int4 r1;  // nblk | ntiles, hdr_bytes | ngath, g0, aoff256: as loaded (unpacking them would wait for the load)
  int kb;
  int4 rows0;
  __device__ __forceinline__ int nblk() const { return r1.x & 0xffff; }
  __device__ __forceinline__ int ntiles() const { return r1.x >> 16; }
  __device__ __forceinline__ int ngath() const { return r1.y >> 16; }
};
__device__ __forceinline__ void load_stage(StageView& v, const StageRec* recs, int i, int n, int tile) {
  v.r1 = make_int4(0, 0, 0, 0);
  v.kb = 0;
  if (i >= 0 && i < n) {
    const StageRec* rp = recs + i;
    v.r1 = __ldg(reinterpret_cast<const int4*>(rp) + 1);
    v.kb = __ldg(rp->kb + min(tile, kMaxStageTiles - 1));
  }
}
__device__ __forceinline__ void load_rows(StageView& v, const int32_t* gcol, int hf, int lane) {
  const int t = (lane >> 2) * 2 + hf;  // four pieces per tile
  if (t < v.ngath()) v.rows0 = __ldg(reinterpret_cast<const int4*>(gcol + ((int64_t)v.r1.z + t) * 16) + (lane & 3));
}

// A gathered tile: row r of the tile from B's row at list[...] (its place in
// the packed column tile, in 128-byte rows; -1: zeros). A lane moves 16-byte
// chunks: 8 lanes bring the 128 bytes of 64 columns of a row, undoing the
// swizzle of the source row (its low three bits) and applying that of row r &
// 7. The list holds the four rows of a lane side by side (rows q, q + 4, q + 8,
// q + 12 for lanes 8 q .. 8 q + 7), so one load brings them.
template <int NOPS>
__device__ __forceinline__ void gather_tile(uint32_t dst, const uint8_t* b, const int* list, int nh, int lane) {
  const int c = lane & 7, q = lane >> 3;
  const int4 k4 = reinterpret_cast<const int4*>(list)[q];
  const int k[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
  for (int rr = 0; rr < 4; ++rr) {
    const uint32_t n = k[rr] < 0 ? 0u : 16u;
    const int kk = max(k[rr], 0);
    const uint8_t* src = b + (int64_t)kk * 128 + ((c ^ (kk & 7)) << 4);
    // row r = 4 rr + q: its swizzle is 4 (rr & 1) + q
    const uint32_t d = dst + (rr * 4 + q) * 128 + ((c ^ ((rr & 1) * 4 + q)) << 4);
#pragma unroll
    for (int o = 0; o < NOPS; ++o) cp_async16(d + o * 2048, src + o * 2048, n);
    if (nh > 1) {
#pragma unroll
      for (int o = 0; o < NOPS; ++o)
        cp_async16(d + 2048 * NOPS + o * 2048, src + 2048 * NOPS + o * 2048, n);
    }
  }
}

// Warp roles: 0..3 MMA issuers (0 also owns TMEM), 4..11 epilogue (two per TMEM
// lane quadrant), then NPROD copy warps, then (FP8) the converter warps.
template <int BH, int R, int NSUB, int KIND>
__global__ void __launch_bounds__(Cfg<BH, R, NSUB, KIND>::THREADS, 1)
    spmm_tc_kernel(const __grid_constant__ SpmmArgs args) {
  using C = Cfg<BH, R, NSUB, KIND>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::NS * C::STAGE);
  uint64_t* full = bars;
  uint64_t* empty = full + C::NS;
  uint64_t* accfull = empty + C::NS;
  uint64_t* accempty = accfull + 2;
  uint64_t* drainbar = accempty + 2;
  uint64_t* conv = drainbar + C::NMMA;  // FP8: the stage's A blocks are converted
  // FP8: the stage's A copy landed (the converters start on it while the B
  // tiles are still landing on full[])
  uint64_t* afull = conv + (C::FP8 ? C::NS : 0);
  uint64_t* itemfull = afull + (C::FP8 ? C::NS : 0);  // [kItemRing] an item index is in the ring
  uint64_t* itemempty = itemfull + kItemRing;        // [kItemRing] every role has read it
  uint64_t* stallbar = itemempty + kItemRing;        // nothing arrives here (test stall)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(stallbar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // [kItemRing] work items (panel -1: no more work), 16-byte aligned
  WorkItem* item_ring = reinterpret_cast<WorkItem*>((reinterpret_cast<uintptr_t>(tmem_slot + 2) + 15) &
                                                    ~static_cast<uintptr_t>(15));
  int* row_tab = reinterpret_cast<int*>(item_ring + kItemRing);  // [NEPI][R * BH / 2] C rows, a table per epilogue warp
  int* glists = row_tab + C::NEPI * (R * BH / 2);                    // [NPROD][GLIST / 4] rows of B of gathered tiles
  int* units = glists + C::NPROD * (C::GLIST / 4);                   // [kNotedUnits] the CTA's first units
  // [kNotedUnits / 32 + 1] a bit per unit: to come back to; then whether any bit is set
  volatile uint32_t* odd_units = reinterpret_cast<uint32_t*>(units + kNotedUnits);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);  // uniform for the compiler
  const int lane = threadIdx.x & 31;
  const uint64_t lim = args.wait_ns ? args.wait_ns : kWaitTimeoutNs;
  // stage slots in use (the pipeline depth): all that fit, or fewer when the
  // launch asks
  const uint32_t nsr = (args.depth >= 2 && args.depth < C::NS) ? (uint32_t)args.depth : (uint32_t)C::NS;

  if (threadIdx.x == 0) {
    for (int i = 0; i < C::NS; i++) {
      // the stage's two copy warps: 32 arrivals each (+ their bulk copies'
      // bytes), for a lane's gathered rows count when they land
      mbar_init(smem_u32(&full[i]), 64);
      mbar_init(smem_u32(&empty[i]), C::NMMA);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(smem_u32(&accfull[i]), C::NMMA);
      mbar_init(smem_u32(&accempty[i]), C::NEPI);
    }
    for (int i = 0; i < C::NMMA; i++) mbar_init(smem_u32(&drainbar[i]), 1);
    if (C::FP8)
      for (int i = 0; i < C::NS; i++) {
        mbar_init(smem_u32(&conv[i]), C::NCONV / 2);
        mbar_init(smem_u32(&afull[i]), 1);
      }
    for (int i = 0; i < kItemRing; i++) {
      mbar_init(smem_u32(&itemfull[i]), 1);
      mbar_init(smem_u32(&itemempty[i]), C::NMMA + C::NEPI + C::NCONV + C::NPROD);  // one lane of every warp
    }
    mbar_init(smem_u32(stallbar), 1);
    *abort_flag = 0;
    for (int i = 0; i <= kNotedUnits / 32; i++) odd_units[i] = 0;
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
  grid_release();  // the kernel that sums split panels may be set up
  // What the launch before this one makes (the packed B and its flags, the
  // zero next-unit counter, a C nobody reads any more) is first used by the
  // copy warps and the epilogue, which wait for it there; the plan and A's
  // stream are the handle's own, so the first unit's lookups overlap the
  // packing of B. The other roles wait for it too, before their first bounded
  // wait: a limit is for this kernel's work, not for the launch before it.

  int* err = args.err;
  const uint32_t smem0 = smem_u32(smem);

  if (C::FP8 && warp >= 4 + C::NEPI + C::NPROD) {
    // ------------------------------------------------------ FP8 converters
    // Each stage's e4m3 blocks and FP32 scales land in the staging area;
    // a set of four warps writes them to the stage's A area as FP16 (value times
    // its block's scale, one rounding) in the 32-byte-swizzled layout the
    // MMA reads, make the writes visible to the tensor core's async proxy,
    // and release the stage to the MMA warps (conv barrier). One set of four
    // warps took 1,750 cycles a stage, more than half of them in the fence, and
    // set the pace; two sets take every other slot (48^3 stencil, N = 256: 115 us
    // a call with one set, 106 with two, 101 with stages of 9 tiles, four in
    // flight, instead of 12). A slot always goes to the same set: a set that met
    // a slot every other time only could take the phase before last for its own.
    const int ct = (threadIdx.x - 32 * (4 + C::NEPI + C::NPROD)) & 127;
    const uint32_t set = (uint32_t)(warp - 4 - C::NEPI - C::NPROD) >> 2;
    uint32_t ci = 0;
    bool ok = true;
    grid_wait();
    for (uint32_t kk = 0; ok; ++kk) {
      WorkItem wi;
      if (!take_item_warp(itemfull, itemempty, item_ring, kk, lane, abort_flag, err, ERR_ITEM_CONV, lim, false, wi)) {
        ok = false;
        break;
      }
      if (wi.panel < 0) break;
      {
        for (int c = wi.s0; c < wi.s1; ++c, ++ci) {
          const uint32_t s = ci % nsr;
          if ((s & 1) != set) continue;
          if (!warp_wait(smem_u32(&afull[s]), (ci / nsr) & 1, lane, abort_flag, err, ERR_CONV, false, lim)) {
            ok = false;
            break;
          }
          uint8_t* stp = smem + s * C::STAGE;
          const int nblk = *reinterpret_cast<const uint16_t*>(stp + 8);
          const uint8_t* stg = stp + C::HDR;
          const float* scl = reinterpret_cast<const float*>(stg + nblk * 256);
          // gathered blocks: a scale per column, after the blocks' scales
          const uint32_t gmask = *reinterpret_cast<const uint32_t*>(stp + 12);
          const float4* gscl = reinterpret_cast<const float4*>(stg + nblk * 256 + fp8_scale_bytes(nblk));
          // a thread widens whole 16-value rows; its rows are loaded first, so
          // that the loads overlap (FP8 stencil 192 against 209 us with one
          // 8-value piece loaded, widened and stored at a time)
          constexpr int XN = (C::SB * 16 + 127) / 128;
          uint4 raw[XN];
          float sc[XN];
#pragma unroll
          for (int q = 0; q < XN; ++q) {
            const int b = (ct >> 4) + 8 * q;  // block; the row is ct & 15
            if (b < nblk) {
              raw[q] = *reinterpret_cast<const uint4*>(stg + b * 256 + (ct & 15) * 16);
              sc[q] = scl[b];
            }
          }
#pragma unroll
          for (int q = 0; q < XN; ++q) {
            const int b = (ct >> 4) + 8 * q, r = ct & 15;
            if (b >= nblk) break;
            const uint32_t in[4] = {raw[q].x, raw[q].y, raw[q].z, raw[q].w};
            const bool gat = (gmask >> b) & 1u;
            const float4* gs = gscl + 4 * __popc(gmask & ((1u << b) - 1));
            uint32_t w[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float4 s4 = gat ? gs[i] : make_float4(sc[q], sc[q], sc[q], sc[q]);
              const float2 f0 = __half22float2(e4m3x2_to_half2((uint16_t)(in[i] & 0xffffu)));
              const float2 f1 = __half22float2(e4m3x2_to_half2((uint16_t)(in[i] >> 16)));
              const __half2 o0 = __floats2half2_rn(f0.x * s4.x, f0.y * s4.y);
              const __half2 o1 = __floats2half2_rn(f1.x * s4.z, f1.y * s4.w);
              w[2 * i] = *reinterpret_cast<const uint32_t*>(&o0);
              w[2 * i + 1] = *reinterpret_cast<const uint32_t*>(&o1);
            }
            uint4* dst = reinterpret_cast<uint4*>(stp + C::OFF_A + b * 512 + r * 32);
            const int sw = (r >> 2) & 1;
            dst[sw] = make_uint4(w[0], w[1], w[2], w[3]);
            dst[sw ^ 1] = make_uint4(w[4], w[5], w[6], w[7]);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&conv[s]));
        }
      }
    }
  } else if (warp >= 4 + C::NEPI) {
    // ---------------------------------------------------------------- copies
    // Stage number c (counted over the CTA's whole run) belongs to pair c mod
    // np of copy warps, which bring all of it: a bulk copy for the A region
    // (header and blocks) and one per 128-column subtile of the B tiles, issued
    // by the lanes side by side (about 55 cycles each; two warps reach the SM's
    // 74-78 bytes a cycle), and the rows of the gathered tiles with 16-byte
    // copies through the load path. The warps of a pair take every other tile;
    // as many pairs are at work as stages are in flight (FP8: two). (Eight that each
    // brought two of every stage's tiles spent 940 cycles a stage on waits,
    // shuffles and arrivals.) A stage's record is read two of the pair's stages
    // ahead, its rows of B one.
    //
    // np must not exceed the stages in flight: the wait for a slot tells its
    // phase by parity, so a warp may not come to it before the use before last
    // has been consumed, and its own last stage, c - np, shows only that stage
    // c - np - nsr has.
    const int pw = warp - 4 - C::NEPI;
    const uint64_t pol_a = make_l2_policy_evict_first();  // A streams through L2 once
    const uint64_t pol_b = make_l2_policy_evict_last();   // B tiles are re-read by many CTAs
    const int hf = pw & 1;
    int* const glist = glists + pw * (C::GLIST / 4);
    uint32_t ci = 0;           // the item's first stage
    const uint32_t pair = (uint32_t)pw >> 1, np = min((uint32_t)C::NPROD / 2, nsr);
    const bool active = pair < np;  // the others only pass the units on
    uint32_t my_c = pair, slot_s = pair, phase_s = 1u;  // the warp's next stage, its slot and phase
    bool ok = true, mine = false;
    uint32_t last_mine = 0;    // last stage this warp copied into (for the drain)
    uint32_t taken = 0;        // units put in the ring
    for (uint32_t kk = 0; ok; ++kk) {
      // The CTA's next unit: the first copy warp takes it from the launch's
      // list (the CTA's own index first, then the shared counter) and puts it
      // in the item ring once every role has read the entry it replaces.
      if (pw == 0 && taken == kk) {
        if (elect_one()) put_unit(args, taken, itemfull, itemempty, item_ring, units, abort_flag, err, lim);
        __syncwarp();
        ++taken;
      }
      WorkItem wi;
      if (!take_item_warp(itemfull, itemempty, item_ring, kk, lane, abort_flag, err, ERR_ITEM_TAKE, lim, false, wi)) {
        ok = false;
        break;
      }
      if (wi.panel < 0) {
        if (kk == 0) grid_wait();
        break;
      }
      const ProblemDesc& P = args.probs ? args.probs[wi.prob] : args.one;
      // fields used after shared-memory stores, held in registers (the stores
      // could alias P for the compiler and force a reload each time)
      const StageRec* const p_stages = P.stages + wi.s0;
      const uint8_t* const p_aval = P.aval;
      const int32_t* const p_gcol = P.gcol;
      const int64_t sub_bytes = P.bp_kbs * (int64_t)C::SUB;
      // the packed tiles of this unit ([128-column tile][k-block]); a half
      // without a column below N is not copied (its rows of the accumulators
      // are never stored)
      const uint8_t* const p_b = P.bpack + (int64_t)wi.nt * NSUB * sub_bytes;
      const int left = P.N - wi.nt * C::BN;
      // this lane's bulk copy: subtile sub of the stage's tile bt
      const int bt = (lane / NSUB) * 2 + hf, sub = lane % NSUB;
      const uint32_t bbytes = (uint32_t)max(0, min(2, (left - sub * 128 + 63) >> 6)) * C::HALF;
      const uint8_t* const lane_b = p_b + sub * sub_bytes;
      uint32_t tile_bytes = 0;  // bulk bytes of one tile
#pragma unroll
      for (int j = 0; j < NSUB; ++j)
        tile_bytes += (uint32_t)max(0, min(2, (left - j * 128 + 63) >> 6)) * C::HALF;
      const int nst = active ? wi.s1 - wi.s0 : 0;
      int i = active ? (int)(my_c - ci) : 0;  // the warp's next stage of the unit (>= 0)
      StageView cur, nxt;
      load_stage(cur, p_stages, i, nst, bt);
      load_stage(nxt, p_stages, i + (int)np, nst, bt);
      load_rows(cur, p_gcol, hf, lane);
      if (kk == 0) grid_wait();
      // a short unit: take the next one now, so that its copies follow
      // without a wait (a long one would be taken from a CTA that is free
      // earlier)
      if (pw == 0 && wi.s1 - wi.s0 <= kShortUnit) {
        if (elect_one()) put_unit(args, taken, itemfull, itemempty, item_ring, units, abort_flag, err, lim);
        __syncwarp();
        ++taken;
      }
      for (; i < nst; i += (int)np) {
        const int nblk = cur.nblk(), ngath = cur.ngath(), na = cur.ntiles() - ngath;
        const int ng = (ngath + 1 - hf) / 2;  // gathered tiles of this warp
        const int nb = (na + 1 - hf) / 2;                                     // and bulk ones
        const int kb = cur.kb, aoff = cur.r1.w;
        const uint32_t abytes = (uint32_t)stage_a_bytes(C::CLS, BH, nblk, ngath);
        if (lane < ng * 4) reinterpret_cast<int4*>(glist)[lane] = cur.rows0;  // for every lane to look up
        cur = nxt;
        load_rows(cur, p_gcol, hf, lane);
        load_stage(nxt, p_stages, i + 2 * (int)np, nst, bt);
        const bool good = wait_phase(smem_u32(&empty[slot_s]), phase_s, abort_flag, err, ERR_PROD_A, lim);
        if (!__all_sync(0xffffffffu, good)) {
          ok = false;
          break;
        }
        __syncwarp();  // the gather list is read by other lanes than those that wrote it; a vote orders no memory
        const uint32_t st = smem0 + slot_s * C::STAGE;
        const uint32_t fb = smem_u32(&full[slot_s]);
        // One bulk copy per lane: the warp's B tiles on the stage's barrier, and
        // on lane 31 (the pair's second warp, which has the smaller half) the
        // A region, which has a barrier of its own in the FP8 form, for the
        // converters wait for it alone
        const bool la = hf && lane == 31;
        const uint32_t fa = C::FP8 ? smem_u32(&afull[slot_s]) : fb;
        const uint32_t bytes = (uint32_t)nb * tile_bytes + (!C::FP8 && hf ? abytes : 0u);
        mbar_expect_tx_if(fb, bytes, lane == 0 && bytes != 0);
        if (C::FP8) mbar_arrive_expect_tx_if(fa, abytes, lane == 0 && hf);
        bulk_load_hint_if(la ? st : st + C::OFF_B + (bt * NSUB + sub) * C::SUB,
                          la ? p_aval + (int64_t)aoff * 256 : lane_b + (int64_t)kb * C::SUB, la ? abytes : bbytes,
                          la ? fa : fb, la ? pol_a : pol_b, la || (bt < na && bbytes != 0));
#pragma unroll 1
        for (int g = 0; g < ng; ++g) {
#pragma unroll
          for (int j = 0; j < NSUB; ++j) {
            const int nh = min(2, (left - j * 128 + 63) >> 6);
            if (nh > 0)
              gather_tile<C::NOPS>(st + C::OFF_B + ((na + 2 * g + hf) * NSUB + j) * C::SUB, p_b + j * sub_bytes,
                                   glist + g * 16, nh, lane);
          }
        }
        cp_async_arrive(fb);
        __syncwarp();
        if (!C::FP8) {
          // The A region of the pair's next stage on its way from HBM into L2,
          // a line per lane: the stage's copy then waits for L2 alone (R-MAT,
          // 2^16 rows: 109 us a call without, 104 with; with bulk prefetches
          // 106). Not for FP8, whose regions are half as large: 117.6 without,
          // 121 with.
          const int abytes_next = cur.nblk() ? stage_a_bytes(C::CLS, BH, cur.nblk(), cur.ngath()) : 0;
          const uint8_t* const a_next = p_aval + (int64_t)cur.r1.w * 256;
          for (int x = (lane + 32 * hf) * 128; x < abytes_next; x += 64 * 128) prefetch_l2(a_next + x);
        }
        last_mine = my_c;
        mine = true;
        my_c += np;
        slot_s += np;
        if (slot_s >= nsr) {  // np <= nsr: at most one turn of the ring
          slot_s -= nsr;
          phase_s ^= 1u;
        }
      }
      ci += (uint32_t)(wi.s1 - wi.s0);
    }
    if (!ok) cp_async_wait_all();
    if (!ok && lane == 0 && mine) {
      // wait for this warp's own copies still in flight: they can only be in
      // its stages among the last NS
      const uint64_t dl = lim < kDrainNs ? lim : kDrainNs;
      for (uint32_t k = last_mine + 1 > nsr ? last_mine + 1 - nsr : 0; k <= last_mine; ++k) {
        if (k % np != pair) continue;
        mbar_wait_drain(smem_u32(&full[k % nsr]), (k / nsr) & 1, err, dl);
        if (C::FP8) mbar_wait_drain(smem_u32(&afull[k % nsr]), (k / nsr) & 1, err, dl);
      }
    }
  } else if (warp < C::NMMA) {
    if (elect_one()) {
      // ----------------------------------------------------------- MMA issuers
      // Issuer w runs the MMA groups of its quarter of the panel's block rows,
      // from the list the copy brought in with the stage, and releases every
      // stage once. One thread issues a tcgen05.mma only every 64-75 cycles;
      // four keep the tensor pipe near its rate for these narrow MMAs.
      uint32_t ci = 0, k = 0, slot_s = 0, phase_s = 0;
      bool ok = true, issued = false;
      const uint32_t stall = (blockIdx.x == 0 && warp == 0) ? (uint32_t)args.stall_stage : 0u;
      grid_wait();
      for (uint32_t kk = 0; ok; ++kk) {
        WorkItem wi;
        if (!take_item_one(itemfull, itemempty, item_ring, kk, abort_flag, err, ERR_ITEM_MMA, lim, wi)) {
          ok = false;
          break;
        }
        if (wi.panel < 0) break;
        const ProblemDesc& P = args.probs ? args.probs[wi.prob] : args.one;
        const uint32_t idesc0 = P.idesc;  // without the N field
        const int nstages = wi.s1 - wi.s0;
        {
          const uint32_t buf = k & 1;
          const uint32_t dbase = tmem + buf * C::ACC_COLS;
          // use u = k / 2 of this buffer waits for phase u of accempty: the
          // epilogue's initial zeroing (u = 0), then each drain-and-zero
          if (!wait_phase(smem_u32(&accempty[buf]), (k >> 1) & 1, abort_flag, err, ERR_MMA_ACC, lim)) {
            ok = false;
            break;
          }
          tc_fence_after();
          for (int c = 0; c < nstages; ++c, ++ci) {
            const uint32_t s = slot_s;  // == ci % nsr, kept incrementally
            if (stall != 0u && ci + 1 == stall) {
              // test stall: nothing arrives on this barrier, so the wait runs
              // into its limit (half of the others', so that it is the one
              // that reports) and the CTA aborts
              ok = wait_phase(smem_u32(stallbar), 0, abort_flag, err, ERR_MMA_STALL, lim / 2);
              if (!ok) break;
            }
            // the stage's copies landed (complete_tx); the MMA reads shared
            // memory through the async proxy, so no tcgen05 fence is needed
            // (FP8: the converted A blocks, then the B tiles)
            if (!wait_phase(smem_u32(C::FP8 ? &conv[s] : &full[s]), phase_s, abort_flag, err, ERR_MMA_A, lim) ||
                (C::FP8 && !wait_phase(smem_u32(&full[s]), phase_s, abort_flag, err, ERR_MMA_B, lim))) {
              ok = false;
              break;
            }
            const uint8_t* stp = smem + s * C::STAGE;
            // (first, count) of each warp, block and tile counts, gathered blocks
            const uint4 hd = *reinterpret_cast<const uint4*>(stp);
            if (hd.w != 0) fence_proxy_async_smem();  // gathered rows were written through the generic proxy
            const uint32_t wl = ((warp & 2 ? hd.y : hd.x) >> (16 * (warp & 1))) & 0xffffu;
            const uint32_t first = wl & 0xffu, cnt = wl >> 8;
            const uint32_t* ent = reinterpret_cast<const uint32_t*>(stp + kStageHdrFixed) + first;
            // lo blocks follow the stage's nblk hi blocks (split form)
            const uint32_t lo_off = KIND == KIND_SPLIT ? (hd.z & 0xffffu) * C::ABLK : 0;
            // descriptors of operands inside the stage = stage descriptor + offset / 16
            const uint64_t sdesc = desc_kmajor_sw32(smem0 + s * C::STAGE + C::OFF_A);
            const uint64_t bdesc = desc_mnmajor_sw128(smem0 + s * C::STAGE + C::OFF_B, C::HALF);
            for (uint32_t e = 0; e < cnt; ++e) {
              const uint32_t m = ent[e];
              const uint32_t pos = m & 31u, tile = (m >> 5) & 15u, slot = (m >> 9) & 31u;
              const uint32_t len = ((m >> 14) & 15u) + 1u, acc = (m >> 18) & 1u;
              const uint32_t idesc = idesc0 | (((len * BH) >> 3) << 17);
              const uint64_t a_hi = sdesc + ((pos * C::ABLK) >> 4);
              const uint64_t b_hi0 = bdesc + ((tile * C::TILEB) >> 4);
#pragma unroll
              for (int j = 0; j < NSUB; ++j) {
                const uint32_t dcol = dbase + j * C::SUB_COLS + slot * BH;
                const uint64_t b_hi = b_hi0 + ((j * C::SUB) >> 4);
                umma_f16(dcol, b_hi, a_hi, idesc, acc);
                if (KIND == KIND_SPLIT) {
                  const uint64_t a_lo = a_hi + (lo_off >> 4);
                  const uint64_t b_lo = b_hi + (2048 >> 4);
                  umma_f16(dcol, b_hi, a_lo, idesc, 1);
                  umma_f16(dcol, b_lo, a_hi, idesc, 1);
                }
              }
              issued = true;
            }
            umma_commit(smem_u32(&empty[s]));
            if (++slot_s == nsr) {
              slot_s = 0;
              phase_s ^= 1u;
            }
          }
          if (!ok) break;
          umma_commit(smem_u32(&accfull[buf]));
          ++k;
        }
      }
      if (!ok && issued) {
        const uint32_t db = smem_u32(&drainbar[warp]);
        umma_commit(db);
        mbar_wait_drain(db, 0, err, lim);
      }
    }
  } else if (warp >= 4) {
    // -------------------------------------------------------------- epilogue
    // Eight warps drain a unit together, while the MMAs of the next one fill
    // the other accumulator buffer: warp (q, h) takes TMEM lane quadrant q (C
    // columns q*32 .. q*32+31 of each 128-column subtile) of half h of the
    // slots, and writes zeros back: the accumulators are all zero whenever the
    // MMA warps receive a buffer, so a part that starts in the middle of a panel
    // accumulates onto zero. The next unit's rows are on their way meanwhile.
    // (A set of four warps per buffer took 18,000 cycles for a unit of the 64^3
    // stencil, with the MMAs' 10,000 before them in the same buffer, and the
    // lookups, one row load behind the other, 10,000 more: 177 us a call against
    // 170.)
    const uint32_t q = warp & 3, h = (uint32_t)(warp - 4) >> 2;
    const uint32_t lane_base = tmem + ((q * 32u) << 16);
    for (uint32_t c = h * C::ACC_COLS; c < (h + 1) * C::ACC_COLS; c += 16) tmem_st_x16_zero(lane_base + c);
    tmem_st_wait();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(smem_u32(&accempty[0]));
      mbar_arrive(smem_u32(&accempty[1]));
    }
    constexpr int SLAB = R * BH * C::BN;  // floats per slab
    constexpr int PW = (R % kMmaWarps == 0) ? R / kMmaWarps : 0;  // slots per issuing warp
    // A drain step takes 16 TMEM columns (a 16-row slot, half a 32-row one) with
    // one load. The steps are a loop: unrolled, the drain was about 16,000
    // instructions a pass, and fetching them set the kernel's pace (64^3 stencil,
    // N = 256: 235 us with every copy and MMA in place, 190 us with none).
    constexpr int STEP = 16, HALF_ROWS = R * BH / 2, NROW = HALF_ROWS / 32;
    static_assert(HALF_ROWS % 32 == 0, "a lane per row");
    int* const rows = row_tab + (warp - 4) * HALF_ROWS;  // this warp's table of its half's C rows
    bool ok = true;
    OddTiles odds;
    // what the drain of a unit looks up: its half's C rows and the slot masks
    int row[NROW];
    uint32_t slot_mask = 0, ext_mask = 0;
    bool more = true;  // not the end of the work
    auto look_up = [&](uint32_t kk) {
      const uint32_t bar = smem_u32(&itemfull[kk % kItemRing]);
      ok = __all_sync(0xffffffffu, wait_phase_sleepy(bar, (kk / kItemRing) & 1, abort_flag, err, ERR_ITEM_EPI, lim));
      if (!ok) return;
      const WorkItem* const it = item_ring + kk % kItemRing;
      const int panel = it->panel;
      more = panel >= 0;
      if (!more) return;
      const ProblemDesc& P = args.probs ? args.probs[it->prob] : args.one;
      const int32_t* const rm = P.row_map + (int64_t)panel * R * BH + h * HALF_ROWS + lane;
#pragma unroll
      for (int x = 0; x < NROW; ++x) row[x] = __ldg(rm + x * 32);
      slot_mask = __ldg(&P.panels[panel].slot_mask);
      // a hub row cut over the issuing warps has its parts in slots s, s + PW,
      // s + 2 PW, ...; the parts after the first are added into it here
      ext_mask = __ldg(&P.panels[panel].ext_mask);
    };
    look_up(0);
    for (uint32_t kk = 0; ok && more; ++kk) {
      const WorkItem wi = item_ring[kk % kItemRing];
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&itemempty[kk % kItemRing]));
      const uint32_t buf = kk & 1, dbase = lane_base + buf * C::ACC_COLS;
      const ProblemDesc& P = args.probs ? args.probs[wi.prob] : args.one;
      // fields used between the stores to C, held in registers (the stores
      // could alias P for the compiler and force reloads of every field)
      const int p_N = P.N, p_f16 = P.c_f16, n_tiles = P.n_tiles;
      const int64_t p_ldc = P.ldc;
      void* const p_C = P.C;
      const int panel = wi.panel, nt = wi.nt;
      const bool split = wi.split >= 0;
      const int elt = p_f16 ? 2 : 4;
      const int64_t ldb = p_ldc * elt;
      // bit x of `full`: the half's rows 16 x .. 16 x + 15 are all there
      uint32_t full = 0;
#pragma unroll
      for (int x = 0; x < NROW; ++x) {
        rows[x * 32 + lane] = row[x];
        const uint32_t there = __ballot_sync(0xffffffffu, row[x] >= 0);
        full |= ((there & 0xffffu) == 0xffffu ? 1u : 0u) << (2 * x);
        full |= ((there >> 16) == 0xffffu ? 1u : 0u) << (2 * x + 1);
      }
      const uint32_t slots = slot_mask, exts = ext_mask;
      if (kk == 0) grid_wait();  // the warp's first unit
      const int32_t* const p_pois = P.poison_ptr;
      // Does the packed B of these columns hold infinite or NaN values? Then the CTA
      // comes back to the unit at its end (FP8: the warp does so behind the drain,
      // 48^3 stencil 100 us a call that way and 103 the other, 101 before).
      bool odd = p_pois != nullptr && !split && odds.look(P, NSUB, wi.prob, nt, lane);
      if (!C::FP8 && odd && kk < (uint32_t)kNotedUnits) {
        if (warp == 4 && lane == 0) {
          odd_units[kk >> 5] |= 1u << (kk & 31);
          odd_units[kNotedUnits / 32] = 1;
        }
        odd = false;
      }
      __syncwarp();
      if (!warp_wait(smem_u32(&accfull[buf]), (kk >> 1) & 1, lane, abort_flag, err, ERR_EPI, true, lim)) {
        ok = false;
        break;
      }
      tc_fence_after();
      // slab of (part, column tile): (first slab of the panel + part) * n_tiles + nt
      float* const slab = split ? P.slabs + ((size_t)(wi.slab + wi.part) * n_tiles + nt) * SLAB : nullptr;
      look_up(kk + 1);
      if (!ok) break;
#pragma unroll 1
      for (int j = 0; j < NSUB; ++j) {
        const int nl = j * 128 + (int)q * 32 + lane;  // column inside the tile
        const int n = nt * C::BN + nl;
        uint8_t* const col = static_cast<uint8_t*>(p_C) + (int64_t)n * elt;
#pragma unroll 1
        for (int x = 0; x < HALF_ROWS; x += STEP) {
          const int r0 = (int)h * HALF_ROWS + x;      // row of the panel
          const int sl = r0 / BH, off = r0 % BH;      // slot, row inside it
          if ((exts >> sl) & 1u) continue;            // its first part's warp adds it and writes the zeros
          float v[STEP];
          const uint32_t ta = dbase + j * C::SUB_COLS + r0;
          __syncwarp();  // lanes past N skipped the stores: together again for the aligned loads
          // an empty slot reads zeros: slots are zeroed after every drain and
          // no MMA writes an empty one
          if ((slots >> sl) & 1u) {
            tmem_ld_x16(ta, v);
            tmem_st_x16_zero(ta);
          } else {
#pragma unroll
            for (int m = 0; m < STEP; ++m) v[m] = 0.0f;
          }
          __syncwarp();
          if constexpr (PW > 0) {
#pragma unroll 1
            for (int t = sl + PW; t < R && ((exts >> t) & 1u); t += PW) {
              if (((slots >> t) & 1u) == 0) continue;
              float u[16];
              const uint32_t tb = dbase + j * C::SUB_COLS + t * BH + off;
              tmem_ld_x16(tb, u);
              tmem_st_x16_zero(tb);
#pragma unroll
              for (int m = 0; m < 16; ++m) v[m] += u[m];
            }
          }
          if (split) {
            if (((slots >> sl) & 1u) == 0) continue;  // taken as zeros
            float* const dst = slab + (size_t)r0 * C::BN + nl;
#pragma unroll
            for (int m = 0; m < 16; ++m) __stcg(dst + (size_t)m * C::BN, v[m]);
          } else {
            if (!C::FP8 && odd) {
              const int q0 = p_pois[panel * R + sl], q1 = p_pois[panel * R + sl + 1];
              if (q0 < q1 && n < p_N && poisoned1(P, C::NOPS, q0, q1, n)) {
#pragma unroll
                for (int m = 0; m < 16; ++m) v[m] = __int_as_float(0x7fffffff);
              }
            }
            const bool fl = (full >> (x / 16)) & 1u;
            if (n < p_N) {
              if (p_f16) store_rows16<__half>(col, ldb, rows + x, fl, v);
              else store_rows16<float>(col, ldb, rows + x, fl, v);
            }
          }
        }
      }
      __syncwarp();
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&accempty[buf]));
      if (C::FP8 && odd)
        poison_half(P, panel * R + (int)h * (R / 2), R / 2, nt * C::BN + (int)(q >> 1) * 64, 0xffffffffull << (32 * (q & 1)),
                    lane);
    }
  }

  // lane 0 of the MMA and copy warps ran their roles alone: reconverge
  // every warp before the CTA-wide barrier
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, C::TMEM_COLS);
  }
  if (!C::FP8 && odd_units[kNotedUnits / 32] != 0 && *abort_flag == 0)
    poison_units(args, units, const_cast<const uint32_t*>(odd_units), C::NOPS, BH, R, NSUB, warp, C::THREADS / 32, lane);
}

// C of the split panels: block (unit, 16 plan rows) adds the parts' slab rows
// in part order, a thread per column. What bounds it: latency of its one or
// two rounds of loads; the slabs (96 parts of 128 KB at most per problem and
// column tile) are in L2. Adding them at the end of the SpMM kernel, by the
// part that came last, took 15-20 us of one SM's time on the R-MAT workload
// and on 24 grouped matrices while the other SMs were done.
__global__ void __launch_bounds__(256) sum_parts_kernel(const __grid_constant__ SumArgs a) {
  grid_wait();
  const int u = (int)blockIdx.x, r0 = (int)blockIdx.y * 16;
  WorkItem w;
  if (a.probs) {
    w = a.splits[u];
  } else {
    w = a.splits[u / a.one.n_tiles];
    w.nt = u % a.one.n_tiles;
  }
  const ProblemDesc& P = a.probs ? a.probs[w.prob] : a.one;
  const int sl = r0 / a.bh, bn = 128 * a.nsub;
  const uint32_t slot_mask = P.panels[w.panel].slot_mask, ext_mask = P.panels[w.panel].ext_mask;
  if ((ext_mask >> sl) & 1u) return;  // added into its first part's rows
  const int n = w.nt * bn + (int)threadIdx.x;
  float acc[16];
#pragma unroll
  for (int m = 0; m < 16; ++m) acc[m] = 0.0f;
  if ((slot_mask >> sl) & 1u) {
    const size_t step = (size_t)P.n_tiles * (a.R * a.bh * bn);
    const float* src = P.slabs + ((size_t)w.slab * P.n_tiles + w.nt) * (a.R * a.bh * bn) + (size_t)r0 * bn + threadIdx.x;
    int p = 0;
    for (; p + 2 <= w.nparts; p += 2, src += 2 * step) {
      float t[32];
#pragma unroll
      for (int m = 0; m < 16; ++m) {
        t[m] = __ldcg(src + (size_t)m * bn);
        t[16 + m] = __ldcg(src + step + (size_t)m * bn);
      }
#pragma unroll
      for (int m = 0; m < 16; ++m) acc[m] = (acc[m] + t[m]) + t[16 + m];
    }
    if (p < w.nparts) {
#pragma unroll
      for (int m = 0; m < 16; ++m) acc[m] += __ldcg(src + (size_t)m * bn);
    }
  }
  if (P.poison_ptr != nullptr) {
    const int q0 = P.poison_ptr[w.panel * a.R + sl], q1 = P.poison_ptr[w.panel * a.R + sl + 1];
    if (q0 < q1) {
      const int64_t fs = pack_flag_stride(P.K);
      const int h0 = w.nt * (2 * a.nsub), h1 = min(h0 + 2 * a.nsub, (P.N + 63) >> 6);
      const uint4* fl = reinterpret_cast<const uint4*>(P.bflags + (int64_t)h0 * fs);
      uint32_t any = 0;
      for (int64_t x = threadIdx.x; x < (h1 - h0) * fs / 16; x += blockDim.x) {
        const uint4 f = __ldcg(fl + x);
        any |= f.x | f.y | f.z | f.w;
      }
      const int lane = (int)threadIdx.x & 31, n64 = n & ~63;
      const uint64_t part = columns64(n64, P.N, 0xffffffffull << (n & 32));
      if (__syncthreads_or((int)any) && part != 0 &&
          ((poisoned64_call(P, a.nops, q0, q1, n64, part, lane) >> (n & 63)) & 1ull)) {
#pragma unroll
        for (int m = 0; m < 16; ++m) acc[m] = __int_as_float(0x7fffffff);
      }
    }
  }
  if (n >= P.N) return;
  const int32_t* rows = P.row_map + (int64_t)w.panel * a.R * a.bh + r0;
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    const int row = __ldg(rows + m);
    if (row < 0) continue;
    const int64_t off = (int64_t)row * P.ldc + n;
    if (P.c_f16)
      __stcs(reinterpret_cast<__half*>(P.C) + off, __float2half_rn(acc[m]));
    else
      __stcs(reinterpret_cast<float*>(P.C) + off, acc[m]);
  }
}

// Raises the variant's dynamic shared memory limit once per device (a
// launch inside a stream capture then makes no other CUDA call).
template <int BH, int R, int NSUB, int KIND>
static cudaError_t prepare_one() {
  using C = Cfg<BH, R, NSUB, KIND>;
  static std::atomic<uint64_t> done{0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return cudaErrorInvalidDevice;
  const uint64_t bit = dev < 64 ? (1ull << dev) : 0;
  if (bit && (done.load() & bit)) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(spmm_tc_kernel<BH, R, NSUB, KIND>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES);
  if (e != cudaSuccess) {
    cudaGetLastError();  // do not leave the error for the next call to find
    return e;
  }
  done.fetch_or(bit);
  return cudaSuccess;
}

template <int BH, int R, int NSUB, int KIND>
static cudaError_t launch_one(const SpmmArgs& args, int grid, bool behind, cudaStream_t stream) {
  using C = Cfg<BH, R, NSUB, KIND>;
  auto kfn = spmm_tc_kernel<BH, R, NSUB, KIND>;
  cudaError_t e = prepare_one<BH, R, NSUB, KIND>();
  if (e != cudaSuccess) return e;
  void* params[] = {const_cast<SpmmArgs*>(&args)};
  return launch_kernel(reinterpret_cast<const void*>(kfn), dim3((unsigned)grid), dim3(C::THREADS), C::SMEM_BYTES, stream,
                       behind, params);
}

// Co-resident CTAs per SM: limited by TMEM (512 columns per SM) and by what
// the occupancy calculator reports for the shared memory and registers.
template <int BH, int R, int NSUB, int KIND>
static int ctas_per_sm_one() {
  using C = Cfg<BH, R, NSUB, KIND>;
  auto kfn = spmm_tc_kernel<BH, R, NSUB, KIND>;
  int by_tmem = 512 / C::TMEM_COLS;
  int occ = 1;
  if (prepare_one<BH, R, NSUB, KIND>() != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kfn, C::THREADS, C::SMEM_BYTES) != cudaSuccess) {
    cudaGetLastError();
    occ = 1;
  }
  int n = by_tmem < occ ? by_tmem : occ;
  return n < 1 ? 1 : n;
}

}  // namespace dev

cudaError_t launch_kernel(const void* fn, dim3 grid, dim3 block, size_t smem, cudaStream_t stream, bool behind,
                          void** args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = behind ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelExC(&cfg, fn, args);
  const cudaError_t last = cudaGetLastError();  // do not leave the error for the next call to find
  return e != cudaSuccess ? e : last;
}

cudaError_t tc_sum_parts(const SumArgs& args, cudaStream_t stream) {
  if (args.n_units == 0) return cudaSuccess;
  void* params[] = {const_cast<SumArgs*>(&args)};
  return launch_kernel(reinterpret_cast<const void*>(dev::sum_parts_kernel),
                       dim3((unsigned)args.n_units, (unsigned)(args.R * args.bh / 16)), dim3((unsigned)(128 * args.nsub)), 0,
                       stream, true, params);
}

#define SMAT_TC_VARIANTS(X) \
  X(16, 4, 1, 0)            \
  X(16, 8, 1, 0)            \
  X(16, 16, 1, 0)           \
  X(16, 4, 2, 0)            \
  X(16, 8, 2, 0)            \
  X(32, 4, 1, 0)            \
  X(32, 8, 1, 0)            \
  X(16, 4, 1, 1)            \
  X(16, 8, 1, 1)            \
  X(16, 16, 1, 1)           \
  X(32, 4, 1, 1)            \
  X(32, 8, 1, 1)            \
  X(16, 4, 1, 2)            \
  X(16, 8, 1, 2)            \
  X(16, 16, 1, 2)

bool tc_variant_supported(int bh, int R, int nsub, int kind) {
#define SMAT_TC_MATCH(BH, R_, NS, K) \
  if (bh == BH && R == R_ && nsub == NS && kind == K) return true;
  SMAT_TC_VARIANTS(SMAT_TC_MATCH)
#undef SMAT_TC_MATCH
  return false;
}

int tc_ctas_per_sm(int bh, int R, int nsub, int kind) {
#define SMAT_TC_OCC(BH, R_, NS, K) \
  if (bh == BH && R == R_ && nsub == NS && kind == K) return dev::ctas_per_sm_one<BH, R_, NS, K>();
  SMAT_TC_VARIANTS(SMAT_TC_OCC)
#undef SMAT_TC_OCC
  return 1;
}

cudaError_t tc_launch(int bh, int R, int nsub, int kind, const SpmmArgs& args, int grid, bool behind,
                      cudaStream_t stream) {
#define SMAT_TC_LAUNCH(BH, R_, NS, K)                             \
  if (bh == BH && R == R_ && nsub == NS && kind == K) \
    return dev::launch_one<BH, R_, NS, K>(args, grid, behind, stream);
  SMAT_TC_VARIANTS(SMAT_TC_LAUNCH)
#undef SMAT_TC_LAUNCH
  return cudaErrorInvalidValue;
}

}  // namespace smat

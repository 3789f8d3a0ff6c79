// spmm_tc.h — launch interface of the tensor-core SpMM kernels and the
// layout of their device work plan.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace smat {

// A pipeline STAGE carries up to stage_rows(cls) / bh A blocks of one panel
// (in the order the kernel consumes them), up to stage_tiles(cls) packed B
// tiles those blocks need, and the stage's MMA list. There are four stage
// shapes ("plan classes"), each the largest that still leaves three stages
// (FP8: four, for one more role between copies and MMAs) in flight in shared
// memory: class 0 for the FP16 and BF16 forms (28
// blocks of 16 rows and 14 B tiles: 14 KB of A and 56 KB of B), class 1
// for the split form, whose stages hold hi and lo copies of everything (14
// blocks and 7 tiles: the same bytes), class 2 for the FP8 form, whose
// stages also stage the e4m3 blocks before conversion (20 blocks, 9
// tiles), class 3 for the FP16 and BF16 forms with 256-column B tiles (N >
// 128 in one pass over A: 14 blocks and 7 tiles of 8 KB).
constexpr int kPlanClasses = 4;
constexpr int kMaxStageTiles = 16;   // StageRec::kb capacity (a copy warp issues at most two copies)
constexpr int kMaxStageBlocks = 31;  // the entry's position field has 5 bits
__host__ __device__ constexpr int stage_rows(int cls) { return cls == 0 ? 448 : (cls == 2 ? 320 : 224); }
__host__ __device__ constexpr int stage_tiles(int cls) { return cls == 0 ? 14 : (cls == 2 ? 9 : 7); }
constexpr int kMmaWarps = 4;      // MMA-issuing warps; each owns a quarter of a panel's TMEM slots
constexpr int kMinCutBlocks = 16; // a block row is cut over the issuing warps only from this many blocks
constexpr int kMaxGroupN = 256;   // widest tcgen05.mma N (kind::f16, M = 128)

// Per-panel record (8 x int32).
struct PanelInfo {
  int32_t stage_off;   // first stage of the panel
  int32_t nstages;     // stages of the panel
  int32_t nblk;        // blocks in the panel
  int32_t nucol;       // distinct block columns of the panel
  uint32_t slot_mask;  // bit s set: slot s of the panel has at least one block
  uint32_t ext_mask;   // bit s set: slot s holds a later part of the row in slot s - R / kMmaWarps
  int32_t pad1, pad2;
};

// Per-stage record (96 bytes), read by the copy warps. In the device A
// stream of a form (ABLK = bh * 32 bytes per block and operand, NOPS = 2 for
// the split form, else 1) a stage occupies
//     [header, kStageHdrBytes][nblk * ABLK blocks (hi)][nblk * ABLK blocks (lo, split form only)]
// and in the FP8 stream (16 x 16 blocks)
//     [header, kStageHdrBytes][nblk * 256 e4m3 blocks][nblk FP32 scales, padded to 16 bytes]
//     [16 FP32 scales per gathered block (its columns come from several blocks)]
// starting at byte aoff256 * 256 (the stages of the FP8 stream are padded to
// that), so the header is always at the stage's start and the MMA threads
// need no word that says where.
// Padded bytes of the FP32 scales of n FP8 blocks.
__host__ __device__ constexpr int fp8_scale_bytes(int n) { return (4 * n + 15) / 16 * 16; }
// Bytes of a stage of nblk blocks, ngath of them gathered, in the A stream of
// plan class cls.
constexpr int kStageHdrBytes = 256;  // a header's room in the A stream and in shared memory
__host__ __device__ constexpr int stage_a_bytes(int cls, int bh, int nblk, int ngath) {
  return kStageHdrBytes +
         (cls == 2 ? nblk * 256 + fp8_scale_bytes(nblk) + 64 * ngath : nblk * bh * 32 * (cls == 1 ? 2 : 1));
}
struct StageRec {
  int64_t blk_off;     // blocks before this stage (plan order)
  int64_t hdr_off;     // header bytes before this stage (Plan::headers)
  int16_t nblk;        // A blocks in the stage
  int16_t ntiles;      // B tiles of the stage, 1..stage_tiles
  int16_t hdr_bytes;   // bytes of this stage's header (multiple of 16)
  int16_t ngath;       // gathered blocks; their tiles come last
  int32_t g0;          // the first of them (they are consecutive)
  int32_t aoff256;     // start of the stage in the A stream, in units of 256 bytes
  int32_t kb[kMaxStageTiles];  // k-block (column / 16) of each tile; -(g + 1): rows of B of gathered block g
};


// Stage header (little-endian), kStageHdrFixed bytes then one 32-bit entry
// per MMA group, grouped by issuing warp:
//   uint16 warp_list[4]   bits 0-7 first entry of warp w, bits 8-15 its entry count
//   uint16 nblk, ntiles
//   uint32 gathered       bit q set: block q of the stage is gathered
//   uint32 entry[...]
// A group is a run of consecutive block rows ("slots") with a block at the
// same block column, the same accumulate flag and the same owner; it is one
// tcgen05.mma with N = bh * len (its accumulators are adjacent in TMEM and
// its A blocks adjacent in the stage). Entry bits:
//   0-4 position of the first A block in the stage, 5-8 B tile in the stage,
//   9-13 first slot, 14-17 len - 1, 18 accumulate (else overwrite).
constexpr int kStageHdrFixed = 16;
constexpr uint32_t kEntAccBit = 1u << 18;
// Largest header of a stage with sb blocks (one entry per block at most).
__host__ __device__ constexpr int stage_hdr_max(int sb) { return kStageHdrFixed + 4 * sb; }

// A unit of work of one CTA: stages [s0, s1) of a panel. A panel whose
// stages are split over several items ("parts", for load balance) has a
// split index: its parts write partial sums to workspace slabs, and a second
// kernel (tc_sum_parts) adds the slabs and writes C.
static_assert(sizeof(StageRec) == 96, "the kernel reads 16-byte pieces");

struct alignas(16) WorkItem {
  int32_t panel;
  int32_t s0, s1;      // stage range, relative to the panel's first stage
  int32_t split;       // -1: the whole panel; else index of the split panel
  int32_t part;        // part number within the split panel
  int32_t nparts;      // parts of the split panel
  int32_t slab;        // first slab of the split panel (one per part and column tile)
  int32_t prob;        // problem of a grouped launch (0 for a single SpMM)
  int32_t nt = 0;      // column tile (grouped launches; else set when the item is taken)
  int32_t pad[3] = {};
};

// Everything the kernel needs about one SpMM problem.
struct ProblemDesc {
  const uint8_t* bpack;      // B in 4 KB tiles [128-column tile][k-block] (pack_b), 8 KB in the split form
  const uint8_t* bflags;     // a byte per packing unit: holds infinite or NaN values
  const uint32_t* bcols;     // a bit per packing unit and column: the same
  const int32_t* gcol;       // [16 g + x]: rows of B of gathered block g (gather_list), or -1
  const int32_t* poison_ptr; // [panels * R + 1] per plan slot: its range of `poison`; null without gathering
  const int2* poison;        // k-block and mask of its all-zero columns, per gathered block
  int64_t bp_kbs;            // k-blocks per 128-column tile in bpack ([column tile][k-block])
  const uint8_t* aval;       // A stream of the form (see StageRec)
  const PanelInfo* panels;
  const StageRec* stages;
  const int32_t* row_map;    // [panels * R * bh] plan row -> C row, or -1
  void* C;
  int64_t ldc;
  float* slabs;              // partial sums of split panels: [slab][R * bh rows][BN] FP32
  int32_t N;
  int32_t n_tiles;
  int32_t c_f16;
  uint32_t idesc;            // instruction descriptor without the N field
  int32_t K;
  int32_t b_bf16;            // packed B is BF16 (else FP16)
};

// Kernel arguments (one __grid_constant__ parameter). A single SpMM passes
// its problem by value (one); a grouped launch passes a device array
// (probs, indexed by WorkItem::prob).
// A launch: its problems and work items, by decreasing estimated cost and
// with the stage range counted from the plan's first stage. A unit of work is
// an item and a column tile (one problem: unit u is item u / n_tiles, tile u %
// n_tiles; a grouped launch lists every unit). CTA b takes unit b, then unit
// grid + atomicAdd(next_item, 1), ... until all n_items units are done:
// whichever CTA is free first takes the largest one left (the counter is zero
// at launch).
// wait_ns bounds every device-side wait (0: 4 s); stall_stage k > 0 makes
// the first MMA-issuing thread of CTA 0 wait, before its k-th stage, on a
// barrier nothing arrives at (a test of the bounded-wait error path);
// depth >= 2 caps the stage slots in flight (the pipeline depth; 0: all
// that fit in shared memory).
struct SpmmArgs {
  ProblemDesc one;
  const ProblemDesc* probs;
  int32_t* next_item;        // zero at launch
  const WorkItem* items;
  int* err;
  int32_t n_items;
  int32_t stall_stage;
  uint64_t wait_ns;
  int32_t depth;
  int32_t pad_;
};

// Kernel kinds: 0 plain (FP16 or BF16 A and B), 1 split hi+lo BF16, 2 FP8 A
// (e4m3 + per-block scale, converted to FP16 in shared memory).
enum : int { TC_KIND_PLAIN = 0, TC_KIND_SPLIT = 1, TC_KIND_FP8 = 2 };
bool tc_variant_supported(int bh, int R, int nsub, int kind);
int tc_ctas_per_sm(int bh, int R, int nsub, int kind);
// `behind`: launched right behind the kernel before it in the stream, which is
// one of this library's; its set-up then overlaps that kernel's end.
cudaError_t tc_launch(int bh, int R, int nsub, int kind, const SpmmArgs& args, int grid, bool behind,
                      cudaStream_t stream);

// C of the split panels from their parts' slabs. splits: one item per split
// panel (panel, nparts, slab, prob), and per column tile in a grouped launch;
// n_units of them, counted as in SpmmArgs. Launched behind the kernel that
// wrote the slabs.
struct SumArgs {
  ProblemDesc one;
  const ProblemDesc* probs;
  const WorkItem* splits;
  int32_t n_units;
  int32_t bh, R, nsub, nops;
};
cudaError_t tc_sum_parts(const SumArgs& args, cudaStream_t stream);

// Launches kernel `fn` behind the one before it in the stream (programmatic
// dependent launch) or after it.
cudaError_t launch_kernel(const void* fn, dim3 grid, dim3 block, size_t smem, cudaStream_t stream, bool behind,
                          void** args);

}  // namespace smat

// smat_internal.h — shared declarations of libsmat's host side.
#pragma once

#include <atomic>
#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

#include "smat.h"
#include "spmm24.h"
#include "spmm_tc.h"

namespace smat {

// Thread-local last-error text behind smat_last_error().
void set_error(const std::string& msg);
smat_status fail(smat_status st, const std::string& msg);

// CUDA device ordinal a handle was built on (api.cu).
int bcsr_device(const smat_bcsr* A);

// A CUDA driver API function by name, looked up through the runtime
// (cudaGetDriverEntryPointByVersion), or nullptr. libsmat does not link
// libcuda, so that it loads (and its host-only entry points run) on machines
// without a GPU driver.
void* driver_fn(const char* name);

// ------------------------------------------------------------------ reorder
struct ReorderResult {
  std::vector<int64_t> grouping;
  std::vector<int64_t> perm;
  int64_t comparisons = 0;
  int64_t merges = 0;
};

// Distances of a chunk of Keeper candidates on a device: init() takes every
// row's block-column runs once; fill() writes, for rows j0 .. j1 - 1, the
// Jaccard distance (JaccardDistanceGroup, blocking.cpp:904-975) of the
// row's runs to the given pattern runs at group size g into out[j - j0]
// (every row, grouped or not: the caller reads the ones it compares).
struct KeeperDevice {
  virtual ~KeeperDevice() {}
  virtual bool init(const std::vector<int64_t>& runs, const std::vector<int64_t>& run_ptr) = 0;
  virtual bool fill(const int64_t* pattern, int64_t np, int64_t g, int64_t j0, int64_t j1, float* out) = 0;
  virtual const char* error() const = 0;
};
// A KeeperDevice on CUDA device `device` (reorder_gpu.cu); nullptr if the
// device cannot be used.
KeeperDevice* make_keeper_device(int device);

// Keeper grouping (blocking.cpp:431-547), bit-exact: the seed loop on the
// host; candidate distances on the host's cores, or on `dev` when given.
// Returns false when the device failed (its error() says why).
bool keeper_grouping(int64_t rows, const int64_t* rowptr, const int32_t* cols, float tau, int64_t col_block,
                     int64_t max_row_block, std::vector<int64_t>& grouping, int64_t& comparisons, int64_t& merges,
                     KeeperDevice* dev);
inline void keeper_grouping_host(int64_t rows, const int64_t* rowptr, const int32_t* cols, float tau,
                                 int64_t col_block, int64_t max_row_block, std::vector<int64_t>& grouping,
                                 int64_t& comparisons, int64_t& merges) {
  keeper_grouping(rows, rowptr, cols, tau, col_block, max_row_block, grouping, comparisons, merges, nullptr);
}
// get_permutation / get_fixed_size_grouping (utilities.cpp:8-20, 45-54).
std::vector<int64_t> permutation_of(const std::vector<int64_t>& grouping);
std::vector<int64_t> fixed_size_grouping(const std::vector<int64_t>& grouping, int64_t row_block);

// ------------------------------------------------------------------ BCSR
// Host-side BCSR structure (bh x bw blocks), bit-identical to csrToBcsr.
struct HostBcsr {
  int64_t rows = 0, cols = 0;        // logical
  int64_t rows_p = 0, cols_p = 0;    // padded
  int32_t bh = 16, bw = 16;
  int64_t nnz = 0;
  std::vector<int32_t> rowptr;       // nbr + 1
  std::vector<int32_t> colidx;       // nnzb, column start
  std::vector<float> val;            // nnzb * bh * bw (exact source values, FP32)
  std::vector<uint16_t> val_f16;     // same, as the FP16 the reference stores
  std::vector<int32_t> row_map;      // rows_p: BCSR row -> original row (or -1)
  std::vector<uint8_t> is24;         // per block: exactly 2:4 (values as FP16)
  std::vector<uint32_t> colmask;     // per block: bit c set where column c holds a nonzero
  std::vector<int32_t> kperm;        // permuted column -> original column (empty: none)
  int64_t nnzb() const { return (int64_t)colidx.size(); }
  int64_t nbr() const { return rows_p / bh; }
};

smat_status build_host_bcsr(const smat_csr& A, int32_t bh, int32_t bw, const int64_t* row_perm,
                            HostBcsr& out);

// HostBcsr from an existing BCSR (16 x 16 or 16 x 32 blocks, values FP16
// row-major per block, column starts), e.g. the arrays of the reference's
// SparseMatrix; 16 x 32 blocks are split into two 16 x 16 blocks.
smat_status build_host_bcsr_from_blocks(int64_t rows, int64_t cols, int32_t bh, int32_t bw, int64_t nnzb,
                                        const int32_t* row_ptr, const int32_t* col_idx, const uint16_t* vals,
                                        HostBcsr& out);

// Columns of a gathered block that hold no nonzero: a stored zero times an
// infinite or NaN value of B is NaN, so these columns still count for such B.
struct Poison {
  int32_t kb;    // k-block
  int32_t mask;  // bit c: column 16 kb + c
};

// Work plan of the tensor-core SpMM. Panels of `R` block rows; the blocks of
// a panel are ordered by block column (then block row) and cut into stages
// of at most stage_rows(cls) / bh blocks and stage_tiles(cls) block columns
// (cls: the plan class, spmm_tc.h). Each stage
// has a record (StageRec) and a header with its MMA list (spmm_tc.h).
struct Plan {
  int32_t R = 8;
  int32_t n_panels = 0;
  std::vector<PanelInfo> panels;
  std::vector<StageRec> stages;
  std::vector<int32_t> stream_blk;   // BCSR block index at each stream position
  std::vector<uint8_t> headers;      // stage headers, concatenated (StageRec::hdr_off)
  // C row of each plan row: inside a panel the block rows take TMEM slots in
  // an order that gives the MMA-issuing warps equal shares of the blocks
  std::vector<int32_t> row_map;
  int64_t n_groups = 0;              // MMA instructions per pass over A
  int64_t n_tiles = 0;               // B tile loads per pass over A
  size_t a_bytes = 0;                // bytes of the A stream
  // gathered blocks (stream_blk and StageRec::kb: -(g + 1)): sixteen nonzero
  // columns of one block row, from whichever of its blocks, side by side;
  // their B tile holds the sixteen rows of B they need
  std::vector<int64_t> gsrc;         // [16 g + q]: BCSR block * 16 + its column, or -1 (zeros)
  std::vector<int32_t> gcol;         // [16 g + q]: row of B, or -1
  // per plan slot (panel * R + slot; the head slot of a cut row): the all-zero
  // columns of its gathered blocks
  std::vector<int32_t> poison_ptr;   // [panels * R + 1], empty without gathering
  std::vector<Poison> poison;
};

// skip (optional): blocks with skip[k] != 0 are left out of the plan (the
// exact-2:4 blocks that the structured-sparse path computes). gather: blocks
// with few nonzero columns are taken apart and their columns gathered.
smat_status build_plan(const HostBcsr& b, int32_t R, int32_t cls, Plan& plan,
                       const std::vector<uint8_t>* skip = nullptr, bool gather = false);

// The device's copy of Plan::gcol for a form with nops operands: columns 4 rr +
// q of a block at place 4 q + rr, and instead of row k of B its place in the
// packed column tile, in 128-byte rows (the copy warps then neither shuffle nor
// divide).
std::vector<int32_t> gather_list(const Plan& pl, int nops);

// ------------------------------------------------------------------ 2:4 path
// The structured-sparse path's units, stages and groups (spmm24.h) and the
// compressed stream, for the blocks with take[k] != 0 (16 x 16 blocks, all
// exactly 2:4); fmt 0: FP16 values, 1: BF16.
struct Sp24Host {
  std::vector<uint8_t> stream;
  std::vector<Sp24Stage> stages;
  std::vector<Sp24Group> groups;     // heaviest first
  std::vector<int32_t> unit_window;
  int64_t n_blocks = 0, n_units = 0;
};
smat_status build_sp24(const HostBcsr& b, const std::vector<uint8_t>& take, int fmt, Sp24Host& out);
// The work list of `workers` CTAs: groups with more than the average share of
// units are cut at stage boundaries into parts (heaviest first; `split` gets
// the first part of each cut group, n_slabs their number of parts).
void split_sp24(const Sp24Host& sp, int32_t workers, std::vector<Sp24Group>& items, std::vector<Sp24Group>& split,
                int32_t& n_slabs);
// Blocks routed to the 2:4 path: exactly 2:4 (is24), in a unit (8 block
// rows x one 32-column window) holding at least min_unit such blocks.
void route_sp24(const HostBcsr& b, int min_unit, std::vector<uint8_t>& take);

// The reference's per-block sparsity label (csrToBcsr, matrix.h:679-711), per
// BCSR block: 1 = "2:4" (the default), 2 = dense once a row of the block has
// three consecutive columns (file order) ending at column % 4 in {2, 3}.
smat_status block_info_ref(const smat_csr& A, const int64_t* perm, const HostBcsr& b, std::vector<int8_t>& info);

// FP8 form: per block (BCSR order) the e4m3 codes of value / scale and one
// FP32 scale, chosen among candidates mapping the block's largest magnitude
// to 448 ... 224 to minimise the block's squared quantisation error.
smat_status quantize_fp8(const HostBcsr& b, std::vector<uint8_t>& q, std::vector<float>& scale);

// Work items of one launch shape: panels whose cost exceeds max_item_frac
// of the per-worker average are split into parts (stage ranges) of about
// that size. `order` lists the items by decreasing estimated cost: the CTAs
// of a launch take them in that order, each the next one when it is done
// with its last (the first from its own index). n_split = split panels,
// n_slabs = their parts (one partial-sum slab per part and column tile).
void build_work_items(const Plan& pl, int32_t bh, int32_t workers, double max_item_frac,
                      std::vector<WorkItem>& items, std::vector<int32_t>& order, int32_t& n_split,
                      int32_t& n_slabs);


// ------------------------------------------------------------------ handle
// Work list of one launch shape (NSUB).
struct Sched {
  int workers = 1;      // CTAs the device holds at once
  int32_t n_items = 0;
  WorkItem* d_items = nullptr;  // by decreasing estimated cost, absolute stage ranges
  WorkItem* d_whole = nullptr;  // the same without split panels (null when there are none)
  int32_t n_whole = 0;
  WorkItem* d_splits = nullptr;  // the split panels, an item each (n_split)
  int32_t n_split = 0;  // panels split into parts
  int32_t n_slabs = 0;  // parts of split panels
};

// A plan class's plan and its device copies and work lists.
struct PlanDev {
  Plan plan;
  bool built = false;
  PanelInfo* d_panels = nullptr;
  StageRec* d_stages = nullptr;
  int32_t* d_row_map = nullptr;
  int32_t* d_gcol = nullptr;        // gathered blocks' rows of B (null: none)
  int32_t* d_poison_ptr = nullptr;  // null: no gathering
  Poison* d_poison = nullptr;
  Sched sched[3];  // by NSUB (1, 2)
};

struct SmatBcsrBody {
  int device = 0;
  HostBcsr host;
  int32_t R = 16;  // block rows per panel
  PlanDev pc[kPlanClasses];
  uint32_t forms = 0;
  int use24 = 0;
  int64_t n_24 = 0;
  // 2:4 path (use24 and 16 x 16 blocks): the groups, stages and unit windows
  // (shared by the forms) and one compressed stream per form (FP16, BF16)
  int sp24_on = 0;
  int sp24_all = 0;  // no block is left to the dense plan of the FP16 / BF16 forms
  int32_t sp24_ngroups = 0;
  int32_t sp24_nitems = 0, sp24_nsplit = 0, sp24_nslabs = 0;  // the list with split groups
  Sp24Group* d_sp24_items = nullptr;
  Sp24Group* d_sp24_split = nullptr;
  int64_t sp24_units = 0;
  Sp24Stage* d_sp24_stages = nullptr;
  Sp24Group* d_sp24_groups = nullptr;
  int32_t* d_sp24_unit_window = nullptr;
  uint8_t* d_sp24_stream[2] = {nullptr, nullptr};
  int32_t* d_bcsr_row_map = nullptr;  // [rows_padded] BCSR row -> C row
  int num_sms = 0;
  int32_t* d_kperm = nullptr;  // column permutation for the B gather (or null)
  // A stream per form (F16, BF16, -, SPLIT): per stage the pre-swizzled
  // blocks in consumption order (hi, then lo for the split form) and the
  // stage header
  uint8_t* d_aval[4] = {nullptr, nullptr, nullptr, nullptr};
  // the same for the 256-column plan (class 3): FP16, BF16
  uint8_t* d_aval_wide[2] = {nullptr, nullptr};
  int32_t depth = 0;                 // pipeline stages in flight (0: all that fit)
  // FP8 form, BCSR block order: e4m3 codes and per-block scales (for export)
  std::vector<uint8_t> fp8_q;
  std::vector<float> fp8_scale;
  int* d_err = nullptr;
  uint64_t wait_ns = 0;              // device-side wait limit (0: the kernels' default)
  std::atomic<int32_t> stall{0};     // testing hook: one-shot stall stage of the next launch
  // smat_spmm_host staging
  std::mutex mu;
  void* d_bstage = nullptr;
  size_t bstage_bytes = 0;
  void* d_cstage = nullptr;
  size_t cstage_bytes = 0;
  void* d_ws = nullptr;
  size_t ws_bytes = 0;
};


}  // namespace smat (the handle type is declared in the global namespace by smat.h)

struct smat_bcsr : smat::SmatBcsrBody {};

namespace smat {

// Kernel kind of an arithmetic form, its plan class, and the N-tile width
// (128 * nsub) used for N.
int kind_of(int32_t form);
inline int plan_class(int32_t form, int nsub = 1) {
  return form == SMAT_FORM_SPLIT_BF16 ? 1 : (form == SMAT_FORM_FP8 ? 2 : (nsub == 2 ? 3 : 0));
}
inline int plan_class_of_kind(int kind, int nsub = 1) {
  return kind == TC_KIND_SPLIT ? 1 : (kind == TC_KIND_FP8 ? 2 : (nsub == 2 ? 3 : 0));
}
// Block rows per panel when the caller leaves it to the library: 256 rows
// (16 blocks of 16 rows, 8 of 32: two TMEM accumulator buffers of 256 columns)
// where that makes at least four panels per SM, else 128. Tall panels share
// more tiles of B, short ones balance better and have half the rows to drain
// at the end (256 against 128 rows, GB300: 64^3 stencil, 6.7 tall panels per
// SM, 184 against 192 us; R-MAT 2^16, 1.7, 112 against 113; split stencil, 2.5,
// 79 against 74; plain graph 2^15, 0.8, 64 against 60; 24 grouped matrices 53
// against 47; a ragged block matrix, 0.1, 31 against 24). Panels costing more
// than kDefaultSplitFrac of the average CTA load are split into parts; finer
// parts cost more than they balance (304 slabs in place of 96: R-MAT 126 us,
// the graph 83).
inline int default_panel_rows(int bh, int64_t nbr, int num_sms) {
  const bool tall = nbr * bh >= (int64_t)1024 * num_sms;
  return (tall ? 256 : 128) / bh;
}
constexpr double kDefaultSplitFrac = 0.5;
int pick_nsub(const smat_bcsr* h, int64_t N, int kind);

// Workspace layout of one SpMM: [packed B (x2 for the split form)]
// [the 2:4 path's copy of B, when the handle uses it for this form]
// [the launch's next-unit counter, 256 bytes]
// [per part of a split panel and column tile: an R*bh x BN FP32 slab]
// [per part of a split 2:4 group and column tile: a 128 x 128 FP32 slab]
// [a byte per packing unit of B, then two words: whether and in which columns it
// holds infinite or NaN values].
struct WsLayout {
  size_t counters = 0, slabs = 0, flags = 0, total = 0;
  size_t b64 = 0;  // the 2:4 path's copy of B (0: none)
  size_t slabs24 = 0;  // the 2:4 path's partial sums
};
WsLayout ws_layout(const smat_bcsr* A, int32_t form, int64_t N, bool whole = false);

// The 2:4 path of a handle for a form: whether it takes blocks of that form,
// the bytes of its partial sums, and its launch arguments for the B windows at
// `b64` (pack_b_sw64); without slabs no group is cut into parts. err, wait_ns and
// whole_c are the caller's to set.
bool uses_sp24(const smat_bcsr* A, int32_t form);
size_t sp24_slab_bytes(const smat_bcsr* A, int64_t N);
void fill_sp24(const smat_bcsr* A, int32_t form, const uint8_t* b64, float* slabs, int64_t N, void* C, int32_t c_dtype,
               int64_t ldc, Sp24Args& a);

// smat_spmm; `whole`: with no panel split over CTAs, so that the workspace
// needs no partial sums.
smat_status spmm_impl(const smat_bcsr* A, int32_t form, const void* B, int32_t b_dtype, int32_t b_layout, int64_t ldb,
                      void* C, int32_t c_dtype, int64_t ldc, int64_t N, void* workspace, size_t workspace_bytes,
                      void* stream, bool whole);

// Whether a call's scratch fits the static scratch, and with whole panels
// only (spmm_static.cu).
bool static_scratch_fits(const smat_bcsr* A, int32_t form, int64_t N, bool* whole);

// The kernel's view of one SpMM: A's device plan and stream for the form,
// the packed B and scratch at `ws` (laid out as wl), C.
void fill_problem(const smat_bcsr* A, int32_t form, const void* ws, int64_t N, void* C, int32_t c_dtype,
                  int64_t ldc, int nsub, const WsLayout& wl, ProblemDesc& P);

// The same over several problems (WorkItem::prob = index into plans); the
// split decisions use the total over all problems; n_split / n_slabs per
// problem.
void build_work_items_multi(const std::vector<const Plan*>& plans, const std::vector<int32_t>& bhs, int32_t workers,
                            double max_item_frac, std::vector<WorkItem>& items, std::vector<int32_t>& order,
                            std::vector<int32_t>& n_split, std::vector<int32_t>& n_slabs);

// ------------------------------------------------------------------ autotuner
// Key of the tuning cache: block-density statistics of a matrix (blocks per
// block row and blocks per B tile of a 16-row panel, log2-bucketed), the
// N-tile count and the kernel kind.
struct TuneKey {
  int32_t bh = 16, bpr_bucket = 0, reuse_bucket = 0, ntile_bucket = 0, kind = 0;
  bool operator<(const TuneKey& o) const {
    if (bh != o.bh) return bh < o.bh;
    if (bpr_bucket != o.bpr_bucket) return bpr_bucket < o.bpr_bucket;
    if (reuse_bucket != o.reuse_bucket) return reuse_bucket < o.reuse_bucket;
    if (ntile_bucket != o.ntile_bucket) return ntile_bucket < o.ntile_bucket;
    return kind < o.kind;
  }
};
struct TuneVal {
  int32_t panel_rows = 16;
  float split_frac = 1.0f;
  int32_t n_tile_cols = 128;
  int32_t depth = 0;
  double ms = 0.0;
};
bool tune_key_of(const HostBcsr& b, int kind, int64_t N, TuneKey& key);
bool tune_lookup(const TuneKey& key, TuneVal& val);
void tune_store(const TuneKey& key, const TuneVal& val);

// The device's list: the items in `order`, their stage ranges counted from
// the plan's first stage (a role then reads one 48-byte item, not an index,
// an item and the panel's record one after the other).
// n_tiles (grouped launches): column tiles per problem, each a unit of its own.
std::vector<WorkItem> device_items(const std::vector<const Plan*>& plans, const std::vector<WorkItem>& items,
                                   const std::vector<int32_t>& order, const std::vector<int32_t>* n_tiles = nullptr);

// One item per split panel (its first part's), and column tile when n_tiles is
// given: what sum_parts goes over.
std::vector<WorkItem> split_items(const std::vector<WorkItem>& items, const std::vector<int32_t>* n_tiles = nullptr);

// Item indices by decreasing cost (ties by index).
void order_items(const std::vector<double>& item_cost, std::vector<int32_t>& order);

}  // namespace smat

// Host-side execution plan for the GPU numeric phase of SPR.
//
// Built once per symbolic structure (MSPAR/MTREES/MSIFA as produced by the
// SPR host pipeline, src/SPR/sprtrs.f + sprsmb.f + sprpmp.f) and cached by the
// C-ABI layer.  It turns SPR's postordered supernode list into
//   * elimination-tree levels (all fronts of a level are independent),
//   * relative-index maps child -> parent (the integer merge of SPRF12,
//     src/SPR/sprfc1.f:716-790, done once instead of per factorisation),
//   * per-parent contribution lists (which child update column lands on which
//     parent column), so extend-add is a deterministic, atomic-free gather,
//   * a device arena layout for fronts / update matrices (first-fit reuse:
//     a child's buffer is released once its parent level is assembled),
//   * the batched task lists of the panel steps of the large fronts.
#pragma once
#include <cstdint>
#include <vector>

namespace sprb {

constexpr int kSmallMaxF = 176;     // fronts up to this order: one CTA, shared memory
constexpr int kNB = 64;             // panel width of the blocked LDL' for large fronts
constexpr int kTRSMRows = 64;       // rows per CTA in the panel (TRSM) kernel
constexpr int kTile = 64;           // Schur-update tile of small updates (rows x cols)
#ifndef SPR_TILE_BIG
#define SPR_TILE_BIG 64
#endif
constexpr int kTileBig = SPR_TILE_BIG;   // Schur-update tile of large updates
constexpr int kTileTiny = 32;            // the autotuner's alternative tile for the small updates
constexpr int kSuperPanel = 512;    // trailing updates are applied per 512 columns (K = 512)
constexpr int kAsmChunk = 256;      // rows per warp pass in the large-front assembly

// A job is one front's share of one batched launch.  Tasks inside a job are
// decoded on the device (binary search over `task0`, then closed-form
// arithmetic), so the plan stays O(fronts x steps) instead of O(tiles).
//   assembly / write-back : one task per column in [c0, c_end)
//   panel (TRSM)          : task 0 = diagonal-block CTA, then row blocks of
//                           kTRSMRows rows starting at c0 (= k_hi)
//   Schur update          : lower-triangle tiles (Launch::tile) of rows
//                           [c0, r_end) x columns [c0, c_end), contraction
//                           over [k_lo, k_hi)
// Blocked right-looking LDL' of the S fully-summed columns with two levels:
// 64-wide panels (diagonal block + TRSM) whose updates stay inside their
// kSuperPanel-wide super-panel, one K = kSuperPanel trailing update per
// super-panel for the remaining fully-summed columns, and one K=S update of
// the (F-S) block.
struct Job {
    int32_t node;
    int32_t c0, c_end, r_end;
    int32_t k_lo, k_hi;
    int64_t task0;                   // first task of this job within its launch
    int64_t slab = 0;                // tensor-core updates: first row of the job's operand slabs
    // integer-digit updates: where the job's row scales and the job's flag
    // (negative pivots, or left out) are, and the slabs' padded rows
    int64_t aux = 0, aux_job = 0;
    int32_t np = 0;
};

struct Launch {                      // a contiguous range of Plan::jobs
    int64_t job_begin = 0, job_count = 0, ntasks = 0;
    int32_t tile = kTile;            // Schur-update launches: tile size of the decode
    int64_t map_begin = -1;          // task -> job map of this launch in Plan::task_map
    int32_t alt = -1;                // a kTile update launch: the same jobs in kTileTiny tiles (Plan::alt)
};

// A tensor-core Schur-update launch: the split of the panel into FP32 hi/lo
// operand slabs, then the 128x128-tile update (one task per lower tile).
constexpr int kTcTile = 128;
constexpr int kTcBK = 32;
struct TcLaunch {
    Launch split;                    // one task per 32 rows x 32 columns of each job's panel
    Launch gemm;                     // one task per lower 128x128 tile of each job's block
};

// An FP64 Schur-update launch on the integer tensor cores: the split of the
// panel into digit slabs, then the update of 128x64 lower tiles; for the
// trailing updates the same slabs serve the next super-panel's columns (gemm)
// and the ones beyond it (far).  The digit sums are exact in 32 bits for
// K <= kI8MaxK (7 products of at most 2^14 in the last level).
constexpr int kI8TileM = 128, kI8TileN = 64;
constexpr int kI8BK = 128;
constexpr int kI8Digits = 7;
constexpr int kI8MaxK = 16384;
constexpr int kI8MinRows = 1024;
constexpr int kI8MinK = 128;
// Fronts whose update is too small for that (fewer than kI8MinRows rows or
// kI8MinK columns) stay on the FP64 kernel: rest and far_rest.  A small front
// has few 128-row tiles, half of them on the diagonal.  Factor ms with the line at
// 256/128, 512/256, 1024/128, 1024/384 and with none: 512 boxes of 3^3 to 12^3
// 30.5, 30.2, 30.4, 30.4, 31.8 (no integer update at all: 30.6); 24^3 14.93, 14.92,
// 14.82, 14.98, 15.07; 32^3 35.2, 35.3, 34.9, 35.8, 35.0.
struct I8Launch {
    Launch split, gemm, far;
    std::vector<Launch> rest, far_rest;
    double flops = 0.0;              // algorithmic flops of gemm and far
};

struct LevelPlan {
    std::vector<int32_t> small_nodes;        // fronts done by the fused one-CTA kernel
    std::vector<int32_t> large_nodes;        // fronts done by the blocked path (assembly, write-back)
    std::vector<int32_t> elim_nodes;         // of those, the ones eliminated (not retained)
    int32_t small_maxF = 0;
    // small fronts in size classes (F <= 64, 96, 128, 176), one launch each so
    // that the smaller fronts get the shared memory (and occupancy) they need:
    // {first index into small_nodes, count, largest F, largest trapezoid of L}
    struct SmallClass {
        int32_t begin, count, maxF, maxL;
    };
    std::vector<SmallClass> small_classes;
    Launch assemble;                          // large fronts: extend-add into dense fronts
    // per panel step: the panel's diagonal block and TRSM; inside a super-panel
    // the launch of the TRSM also updates the next panel's columns (by this panel
    // and the one before) and does the next diagonal block
    std::vector<Launch> panel;
    // per step that ends a super-panel: the next super-panel's columns (one launch per tile size)
    std::vector<std::vector<Launch>> update;
    // per panel step inside a super-panel: the update of the columns after the
    // next two panels (look-ahead stream, beside the next step)
    std::vector<std::vector<Launch>> ahead;
    // mixed precision: a super-panel's K = kSuperPanel update of the next super-panel's
    // columns (the update[st] jobs of a step that ends a super-panel) as a
    // split + tensor-core pair, and its algorithmic flops
    std::vector<std::vector<TcLaunch>> next_tc;
    std::vector<double> next_flops;
    std::vector<Launch> outer;                // update block, K = S (one launch per tile size)
    Launch writeback;                         // S columns -> LNZ
    // per panel step: the columns of the super-panels that end at that step
    // (their last panel's TRSM is done), for writing LNZ early
    std::vector<Launch> wb_sp;
    // solves, rows [S, F) of the eliminated large fronts: forward one task per
    // kFwdRows x kFwdCols tile, back one per kRectRows x kRectCols tile
    Launch rect, rect_back;
    Launch rect_rows;                         // forward, fronts of several column tiles: one task per row
    bool retained_large = false;              // the level has a retained large front
    // triangle of the solves as one dataflow launch: tasks (node, 64-row
    // block) of the level's eliminated large fronts, block-major, in
    // Plan::tri_tasks[tri_begin .. tri_begin + tri_count)
    int64_t tri_begin = 0, tri_count = 0;
    // trailing update columns beyond the next super-panel (side stream)
    std::vector<std::vector<Launch>> far;
    std::vector<std::vector<TcLaunch>> far_tc;
    std::vector<double> far_flops;            // algorithmic flops of each step's far launches
    double outer_flops = 0.0;                 // and of the K = S update
    // FP64 on the integer tensor cores: per panel step that ends a super-panel
    // the trailing update, and the K = S update (one entry per kI8MaxK columns)
    std::vector<I8Launch> trail_i8, outer_i8;
    std::vector<TcLaunch> outer_tc;                 // mixed precision: the K = S update
};

constexpr int kFwdRows = 64, kFwdCols = 256;   // tile of the forward rectangle launches
constexpr int kFwdNarrow = 64;                 // up to this S a tile has 256 rows and all S columns
constexpr int fwd_rows(int s) { return s <= kFwdNarrow ? 256 : kFwdRows; }
constexpr int kRectCols = 64, kRectRows = 256; // tile of the back rectangle launches

struct Plan {
    // sizes
    int64_t neq = 0, nsuper = 0, nzerol = 0, nofsub = 0, maxsup = 0, mfront = 0;
    // per supernode (postorder index js = 0..nsuper-1)
    std::vector<int32_t> fst, S, F, parent, level;
    std::vector<int64_t> lnz_off, lindx_off;
    std::vector<int32_t> child_ptr, child;   // children in SIBL order
    std::vector<int32_t> rows;               // LINDX (0-based rows), concatenated like LINDX
    // partial factorisation (MSPAR(57) > 0): the retained supernodes
    // (SUPSUP > 0, src/SPR/sprtrs.f:1142-1204) are assembled but not
    // eliminated (sprfc1.f:587) and skipped by the solves (sprfs1.f:371)
    std::vector<uint8_t> retained;
    bool any_retained = false;
    // update-row -> parent-row maps, one per non-root supernode with F > S
    std::vector<int64_t> rel_off;            // per node, offset into rel
    std::vector<int32_t> rel;
    // contribution CSR: for parent p, column j: entries [cptr[rbase[p]+j], cptr[rbase[p]+j+1])
    std::vector<int64_t> rbase;              // per node, prefix of F
    std::vector<int64_t> cptr;
    std::vector<int32_t> cchild, ct;         // (child, child update column)
    // device arena (units of doubles)
    std::vector<int64_t> buf_off;            // per node: start of its buffer
    std::vector<int32_t> buf_ld;             // leading dimension of the front / update buffer
    std::vector<int64_t> upd_off;            // per node: where its update matrix (F-S)^2 starts
    int64_t arena_doubles = 0;
    // inverses of the unit-lower diagonal blocks of the large fronts: block st
    // of node js is the column-major kNB x kNB matrix at linv_off[js] + st*kNB*kNB
    std::vector<int64_t> linv_off;
    int64_t linv_doubles = 0;
    // rectangle partial sums (one per right-hand side and entry): back, node js
    // uses rect_off[js] .. + nrc*S, forward fwd_off[js] .. + ncc*(F-S) entries of a
    // scratch of rect_entries / fwd_entries (max over levels)
    std::vector<int64_t> rect_off;
    int64_t rect_entries = 0;
    std::vector<int64_t> fwd_off;
    int64_t fwd_entries = 0;
    // the solves' triangle tasks (pairs node, 64-row block) of every level
    std::vector<int32_t> tri_tasks;
    bool any_large = false;
    // levels and tasks
    std::vector<LevelPlan> levels;
    std::vector<Job> jobs;
    // for every launch: the job (relative to Launch::job_begin) of each task,
    // so a CTA finds its job with one load instead of a binary search
    std::vector<int32_t> task_map;
    std::vector<Launch> alt;                 // kTileTiny versions of the small-tile update launches
    // statistics (the reference's own counters are recomputed for reporting)
    double factor_flops = 0.0;               // = RINFO(3) formula, src/SPR/sprtrs.f:1961-1969
    double solve_flops = 0.0;                // = RINFO(4) formula, src/SPR/sprtrs.f:1976-1980
    double gemm_flops = 0.0;                 // algorithmic flops of the Schur-update launches
    double tc_flops = 0.0;                   // of those, the updates the mixed mode runs on tensor cores
    int64_t slab_rows = 0;                   // largest operand-slab need of one tensor-core launch (128-byte rows)
    int64_t slab_rows_far = 0;               // the same for the side-stream launches
    int64_t i8_rows = 0, i8_scales = 0;      // largest digit slab (128-byte rows) and scale array of an integer launch
    double small_flops = 0.0;                // factor flops done by the fused small-front kernel
};

// Builds the plan from the SPR control arrays.  Returns 0 on success or a
// negative code when the structure is inconsistent (mirrors IERR=-2 checks).
int build_plan(const int64_t* mspar, const int64_t* mtrees, const int64_t* msifa, Plan& plan);

// Size in doubles of a node's device buffer (update matrix or dense front).
int64_t buffer_doubles(const Plan& P, int64_t js);
// Self-check of the arena layout and the index maps: counts buffers outside
// the arena plus relative-index / contribution-list entries out of range or
// not used exactly once (oob), and overlaps between buffers that are live at
// the same level.
void check_plan(const Plan& P, int64_t& oob, int64_t& overlaps);
// Schur-update coverage: every column c of every large front must receive
// exactly the K ranges that tile [0, 64 floor(c / 64)) for c < S (earlier
// panels; a column's own panel is eliminated by the diagonal block and TRSM)
// and [0, S) for c >= S (nothing for a retained front),
// once, across the update, far and K = S launches.  Counts the columns that
// do not, for the FP64 launch lists (fp64) and the tensor-core lists in the
// mixed mode's use (tc: FP64 panel-chain updates + tensor-core far and K = S).
void check_coverage(const Plan& P, int64_t& fp64, int64_t& tc);
// Happens-before check of the factorisation's launch schedule on its four streams
// (small fronts, panels, look-ahead and far updates, K = S update, write-back), of
// the fronts' memory over the levels and of the integer updates' digit slab: the number of
// ordering violations, 0 for a race-free schedule.  tc: the far and K = S
// updates on the tensor-core path; int_min: launches of at least this many flops as
// integer-digit updates (infinity: none).  skip leaves out joins, or puts a split before
// the join of the far launch that still reads the slab (self-tests: must report
// violations where there is such a launch, see SchedCounts).
enum SchedSkip { kSkipFar = 1, kSkipAhead = 2, kSkipSlab = 4, kSkipWriteback = 8, kSkipSmall = 16 };
struct SchedCounts {
    int64_t slab_shared = 0;         // splits that take the slab of a far launch on the side stream
    int64_t reused = 0;              // fronts whose memory a later front takes
    int64_t small_beside = 0;        // levels with small fronts on other streams
};
int64_t check_schedule(const Plan& P, bool tc, double int_min, int skip, SchedCounts* counts = nullptr);
// Self-check of the solves' plan: every eliminated large front of a level has
// each of its 64-row triangle blocks as one task of that level's dataflow
// launch, after the task of the block above it (the forward sweep takes them
// in list order, the back sweep in reverse), with its own equations (the
// fronts' solved rows disjoint and inside NEQ); each front with F > S has one
// rectangle job per sweep and, with several column tiles, one forward-rows
// job, of the right sizes, and the partial-sum ranges of a level's fronts (rect_off, fwd_off) are
// disjoint and inside their scratch.  Returns the number of violations.
// plant: 0 checks P as built; 1 swaps the first two blocks of a front in a
// copy, 2 moves one front's forward partials onto another's in a copy (a
// self-test: both must report violations where such fronts exist).
int64_t check_solve_plan(const Plan& P, int plant, int64_t* tasks = nullptr);

}  // namespace sprb

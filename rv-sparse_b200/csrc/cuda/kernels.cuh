// Internal interface between the plan (plan.cu) and the kernel files.
#pragma once

#include <cstddef>
#include <cstdint>
#include <utility>
#include <vector>
#include <cuda_runtime.h>

#include "stripe_rule.cuh"

struct rvsp_mlp;

namespace rvsp {

// Device pointer of a model's parameters (model.cu).
const float *mlp_device_params(const rvsp_mlp *m);

// Row classes.  A row is classed twice: for the symbolic pass by the upper
// bound ub = min(ops_i, b_cols) on its output nnz, and for the numeric pass
// by its exact output nnz m_i.  The same table serves both.
//
//   EMPTY   no products
//   M<K>    at most K (4, 8, 16) A nonzeros and at most kMergeMaxOps
//           products, in a matrix of at least kMergeMinRows rows: one thread
//           merges the row's K sorted B rows, taking the smallest head
//           column each step; equal heads are added in A-nonzero order, and
//           columns come out sorted with no scratch
//   W<T>    one warp, shared-memory hash table of T slots (bound <= T/2)
//   B8192   one 256-thread block, hash table of 8192 slots (bound <= 4096)
//   DENSE   one 512-thread block, dense accumulator over all of B's columns
//   STRIPE8, STRIPE  the B8192 and DENSE rows of a product whose B suits
//           column stripes: a warp per run of stripes (k_stripe.cu), where that
//           pays (stripe_rule.cuh); reported as the classes they come from
enum RowClass : int {
  kEmpty_ = 0,
  kM4,
  kM8,
  kM16,
  kW64,
  kW128,
  kW256,
  kW512,
  kW1024,
  kW2048,
  kB8192,
  kDense,
  kStripe8,
  kStripe,
  kNumClasses
};

// A thread merges serially, so the longest row of a launch is its time.  On
// R-MAT matrices (short A rows that select hub B rows) a bound of 2048 kept
// a few blocks busy for milliseconds after the rest were done: one product at
// n = 2^16 17.6 ms against 13.7 (512), 13.1 (256) and 13.1 (128, 64), a
// repeat at 2^15 6.4 ms against 3.1, 2.9, 2.6 and 2.6.  Mesh rows (25
// products) stay far below any of them.
constexpr int kMergeMaxOps = 128;
// Nonzeros in consecutive columns of A select neighbouring rows of B, whose
// columns, in a mesh's matrix, are mostly the same: the hash pass inserts each
// of few columns many times, while the merge takes them together.  Where a
// quarter of the nonzeros (of the rows that the shift probe samples) are like
// that, the symbolic pass merges rows of up to twice the products.  80^3 grid,
// 13 points with 3% of the entries dropped (159 products, 70 outputs a row):
// product 1516 -> 1316 us; 400,000 uniform rows of 12 would take 1963 us instead
// of 1778.  (By its own nonzeros, row by row, a band of 15 in 60 columns took
// 1162 instead of 1045: some rows of a warp in each pass.  In the numeric pass
// a repeat would lose what the product gains: 1316 -> 1141, 515 -> 556.  Where
// shift classes take most rows, the few that are left, a thread each, would
// hold the others up: 127x90x113 27-point stencil 1469 -> 1504.)
constexpr int kMergeNearOps = 256;
constexpr int kMergeMaxNnz = 16;
constexpr int kMergeThreads = 128;
// The merge classes put one row on one thread; below this many rows the GPU
// would sit mostly idle, so smaller matrices use the warp-per-row classes.
constexpr int32_t kMergeMinRows = 32768;
constexpr int kWarpHashMinLog2 = 6;    // W64
constexpr int kWarpHashMaxLog2 = 11;   // W2048
constexpr int kBlockHashLog2 = 13;     // B8192
constexpr int kBlockHashThreads = 256;
constexpr int kDenseThreads = 512;
constexpr int kWarpsPerBlock = 4;      // warp-per-row kernels
// Dense rows keep their column bitmap in shared memory up to this many
// columns (48 Ki words = 192 KiB), else in global scratch.
constexpr int64_t kSmemBitmapMaxCols = 48 * 1024 * 32;
// rowstats hands rows with more A nonzeros than this to a warp-per-row pass.
constexpr int kLongRowNnz = 64;

// merge_ok: the matrix has at least kMergeMinRows rows; merge_ops: the most
// products of a merge row.
__host__ __device__ inline int classify_row(int32_t nnz_a, int64_t ops, int64_t bound,
                                            bool merge_ok, int merge_ops = kMergeMaxOps) {
  if (ops <= 0) return kEmpty_;
  if (merge_ok && nnz_a <= kMergeMaxNnz && ops <= merge_ops)
    return nnz_a <= 4 ? kM4 : nnz_a <= 8 ? kM8 : kM16;
  const int64_t need = 2 * bound;
  for (int l = kWarpHashMinLog2; l <= kWarpHashMaxLog2; ++l)
    if (need <= (int64_t(1) << l)) return kW64 + (l - kWarpHashMinLog2);
  if (bound <= (int64_t(1) << (kBlockHashLog2 - 1))) return kB8192;
  return kDense;
}

inline int class_log2(int cls) { return kWarpHashMinLog2 + (cls - kW64); }
inline bool is_merge_class(int cls) { return cls == kM4 || cls == kM8 || cls == kM16; }

// Pointers of one product.  A's columns index B's rows.
struct Operands {
  int32_t a_rows;
  int32_t b_cols;
  const int32_t *a_rp;
  const int32_t *a_col;
  const float *a_val;
  const int32_t *b_rp;
  const int32_t *b_col;
  const float *b_val;
  // Rows may take the merge classes (set by the plan from its merge policy
  // and the row count; see classify_row).
  bool merge_ok;
  // When >= 0: A's entry count and B's row count, which bound every index
  // the row statistics read, so they run safely on structure whose device
  // check has not finished yet (rvsp_cuda_symbolic_checked).
  int32_t a_nnz = -1;
  int32_t b_rows = -1;
  // B8192 and DENSE rows take the STRIPE classes.
  bool stripes = false;
};

__host__ __device__ inline int with_stripes(int cls, bool stripes) {
  return !stripes || cls < kB8192 ? cls : cls == kB8192 ? kStripe8 : kStripe;
}

// The device-side verdict of CSR checks queued earlier on the same stream:
// n words at w, each ~0ull when its structure passed.  A pass given a guard
// that failed returns without reading the structure or writing anything, so
// it can be queued before the verdict reaches the host.  n == 0: no check.
struct CheckGuard {
  const unsigned long long *w = nullptr;
  int n = 0;
#ifdef __CUDACC__
  __device__ __forceinline__ bool failed() const {
    for (int i = 0; i < n; ++i)
      if (w[i] != ~0ull) return true;
    return false;
  }
#endif
};

// Merge policies of a plan: automatic (merge classes when the matrix has at
// least kMergeMinRows rows), never, or whenever a row is eligible.
enum MergePolicy : int { kMergeAuto = 0, kMergeNever = 1, kMergeAlways = 2 };

inline bool merge_allowed(int policy, int32_t a_rows) {
  return policy == kMergeAlways || (policy == kMergeAuto && a_rows >= kMergeMinRows);
}

// Where the fused (learned) pass writes each row: a slot of fo.cap[row]
// entries at fo.off[row] in the slab (the c_col / c_val pointers of the fill
// kernels).  The kernel writes the row's nnz to fo.counts[row], or -1 and
// appends the row to ovf_rows when it needs more than its capacity.
struct FusedOut {
  const int64_t *off;
  const int32_t *cap;
  int32_t *counts;
  int32_t *ovf_rows;
  int32_t *ovf_count;
};

// ---- k_rowstats.cu ---------------------------------------------------------
// ops[i] = sum of B row lengths over A row i; cls[i] = symbolic class of the
// row; class_count[c] += rows per class; counts[i] = 0 for empty rows.  *heavy (zeroed
// by the caller): the STRIPE rows.  near (may be null): *near != 0 merges rows of
// up to kMergeNearOps products.
void launch_rowstats(const Operands &op, int64_t *ops, uint8_t *cls,
                     int32_t *counts, int32_t *class_count, int32_t *long_rows,
                     int32_t *long_count, int32_t max_long, HeavyRows *heavy,
                     const int32_t *near, cudaStream_t s);
void launch_rowstats_long(const Operands &op, const int32_t *long_rows,
                          const int32_t *long_count, int64_t *ops, uint8_t *cls,
                          int32_t *counts, int32_t *class_count, HeavyRows *heavy,
                          int num_sms, cudaStream_t s);
// off[c] = exclusive prefix of count over the non-empty classes.
void launch_class_offsets(const int32_t *count, int32_t *off, cudaStream_t s);
// rows_by_class[class_off[c] + r] = i for every non-empty row i of class c.
void launch_scatter_rows(int32_t n, const uint8_t *cls, const int32_t *class_off,
                         int32_t *class_fill, int32_t *rows_by_class,
                         cudaStream_t s);

// ---- k_scan.cu -------------------------------------------------------------
// row_ptr = exclusive scan of counts (n + 1 entries), *total = sum (int64).
// Also classes every row for the numeric pass (cls, class_count); rows with
// skip[row] >= 0 (the shift-class members) are classed empty.  With hslot,
// rows that the stripe count took (hslot[row] >= 0) are classed STRIPE8 or
// STRIPE: those of more than 1024 outputs, or all of them (hslot_all).  With a
// guard that failed, nothing is written but the tile partials.
size_t scan_partials_bytes(int32_t n);
void launch_scan_and_class(int32_t n, const int32_t *counts, const int64_t *ops,
                           const int32_t *a_rp, int32_t *row_ptr,
                           int64_t *partials, int64_t *total, uint8_t *cls,
                           int32_t *class_count, bool merge_ok, cudaStream_t s,
                           CheckGuard guard = CheckGuard(), const int32_t *skip = nullptr,
                           const int32_t *hslot = nullptr, bool hslot_all = false);

// out[i] = sum of in[0..i) as int64 (n entries), *total = sum of all.
void launch_scan_i64(int32_t n, const int32_t *in, int64_t *out, int64_t *partials,
                     int64_t *total, cudaStream_t s);

// ---- k_fused.cu ------------------------------------------------------------
// Copies every row that fits its slab slot (0 <= counts[row] <= cap[row]) from
// there to C at row_ptr[row]; values too when with_values.  big: scratch of
// a_rows + 1 words (count and list of the rows copied by whole blocks).
void launch_compact(int32_t a_rows, const int32_t *counts, const int32_t *cap,
                    const int64_t *off, const int32_t *row_ptr, const int32_t *slab_col,
                    const float *slab_val, int32_t *c_col, float *c_val,
                    bool with_values, int32_t *big, int num_sms, cudaStream_t s);
// Puts the n listed rows (null: rows 0 .. n - 1) on the overflow list.
void launch_list_overflow(const int32_t *rows, int32_t n, const FusedOut &fo, cudaStream_t s);
// Classes the rows of a list (symbolic: by ub = min(ops, b_cols); numeric: by
// exact nnz counts[row]); cls_out[j] for list entry j; class_count += rows.
void launch_list_classify(const int32_t *list, int32_t n, const int64_t *ops,
                          const int32_t *a_rp, const int32_t *counts, int32_t b_cols,
                          bool numeric, uint8_t *cls_out, int32_t *class_count,
                          cudaStream_t s);
// out[off[c] + r] = list[j] for the entries j of class c (any order).
void launch_scatter_list(const int32_t *list, int32_t n, const uint8_t *cls,
                         const int32_t *class_off, int32_t *class_fill, int32_t *out,
                         cudaStream_t s);
// Order-independent 64-bit fingerprint of n floats added into *h.
void launch_values_hash(const float *v, int64_t n, unsigned long long salt,
                        unsigned long long *h, cudaStream_t s);

// ---- k_merge.cu ------------------------------------------------------------
// Thread-per-row K-way merge for the M<K> classes: counts (symbolic) or
// values and sorted columns (numeric).
void launch_merge_symbolic(int cls, const Operands &op, const int32_t *rows,
                           int32_t nrows, int32_t *counts, cudaStream_t s);
// The symbolic pass of every M4, M8 and M16 row, with no row lists and no
// host-side class counts: one launch per merge class over all a_rows rows,
// each thread skipping rows whose cls is another class.  Three launches.
void launch_merge_symbolic_all(const Operands &op, const uint8_t *cls, int32_t a_rows,
                               int32_t *counts, CheckGuard guard, cudaStream_t s);
void launch_merge_numeric(int cls, const Operands &op, const int32_t *rows,
                          int32_t nrows, const int32_t *c_rp, int32_t *c_col,
                          float *c_val, bool fill, int32_t *status,
                          const FusedOut *fo, cudaStream_t s);

// ---- k_symbolic.cu ---------------------------------------------------------
// W1024 / W2048 rows: counted first in a 512-slot table with bounded probes;
// rows that do not fit go to retry[] (count at *retry_n, zeroed by the
// caller, room for nrows) and are counted at their class size.
bool symbolic_optimistic_class(int cls);
void launch_symbolic_optimistic(int cls, const Operands &op, const int32_t *rows,
                                int32_t nrows, int32_t *counts, int32_t *retry,
                                int32_t *retry_n, int32_t *status, int num_sms,
                                cudaStream_t s);
// counts[row] = nnz of output row, for the rows of one class.
void launch_symbolic_class(int cls, const Operands &op, const int32_t *rows,
                           int32_t nrows, int32_t *counts, uint32_t *gbitmap,
                           int32_t gbitmap_slots, int32_t *status, int num_sms,
                           cudaStream_t s);

// ---- k_heavy.cu ------------------------------------------------------------
// B8192 and DENSE rows when B has at most kHeavyMaxCols columns: block per
// row, shared-memory column bitmap, accumulation at output positions.
constexpr int32_t kHeavyMaxCols = 1 << 20;
bool heavy_fits(int32_t b_cols);
void launch_heavy_symbolic(const Operands &op, const int32_t *rows, int32_t nrows,
                           int32_t *counts, int num_sms, cudaStream_t s);
// fill: write C's sorted columns too (fo: the fused pass's slab slots, with
// overflow when a row needs more than its capacity); else reuse C's columns.
void launch_heavy_numeric(const Operands &op, const int32_t *rows, int32_t nrows,
                          const int32_t *c_rp, int32_t *c_col, float *c_val, bool fill,
                          int32_t *status, const FusedOut *fo, int num_sms,
                          cudaStream_t s);

// ---- k_stripe.cu -------------------------------------------------------------
// STRIPE rows, for B of 1025 .. kStripeMaxCols columns whose table of stripe
// starts stays within 256 MB (else off: the block-per-row kernels).
constexpr int32_t kStripeMaxCols = 1 << 17;
constexpr int kMaxStripes = 96;
struct StripeShape {
  bool on = false;
  int32_t words = 0;   // 32-column words of B's columns
  int32_t ns_max = 0;  // stripes at most
};
__host__ __device__ inline int32_t stripe_groups(int32_t words) { return (words + 31) >> 5; }
StripeShape stripe_shape(int32_t b_rows, int32_t b_cols);
// Stripes of B: hist of words entries, bound of ns_max + 1, share of ns_max,
// ptr of b_rows * (ns_max + 1).
void launch_stripe_table(const StripeShape &g, int32_t b_rows, const int32_t *b_rp,
                         const int32_t *b_col, int32_t *hist, int32_t *bound, float *share,
                         int32_t *ptr, int num_sms, cudaStream_t s);
// counts[row] of the listed rows; hslot[row] = the row's place in the list,
// which indexes its bitmap (words) in bits, its outputs before each 32 words of
// it (stripe_groups) in gpre and before each stripe (ns_max + 1) in soff.
// Scratch: stripe_tasks(nrows) tasks, three words cnt, nrows words done.
size_t stripe_tasks(int32_t nrows);
void launch_stripe_count(const StripeShape &g, const Operands &op, const int32_t *rows,
                         int32_t nrows, const int64_t *ops, const int32_t *bound, int2 *tasks,
                         int32_t *cnt, int32_t *done, int32_t *counts, int32_t *hslot,
                         uint32_t *bits, int32_t *gpre, int32_t *soff, int num_sms,
                         cudaStream_t s);
// The work items of counted rows: items of cap = nrows * ns_max, cnt of two.
void launch_stripe_items(const StripeShape &g, const int32_t *rows, int32_t nrows,
                         const int64_t *ops, const int32_t *hslot, const int32_t *soff,
                         const int32_t *bound, const float *share, int4 *items, int64_t cap,
                         int32_t *cnt, cudaStream_t s);
// Fill: C's columns of counted rows, from their bitmaps.
void launch_stripe_columns(const StripeShape &g, const int32_t *rows, int32_t nrows,
                           const int32_t *hslot, const uint32_t *bits, const int32_t *gpre,
                           const int32_t *soff, const int32_t *c_rp, int32_t *c_col,
                           int32_t *status, cudaStream_t s);
// C's values of the items' rows (columns in C; verify: not written by this
// plan just now, so they are compared with the bitmaps).  nrows: the rows the
// items cover; a row whose length in c_rp is not counts[row] is reported and
// left alone.
void launch_stripe_values(const StripeShape &g, const Operands &op, int32_t nrows,
                          const int4 *items, int64_t cap, const int32_t *cnt, int32_t *head,
                          const int32_t *bound, const float *share, const int32_t *ptr,
                          const int32_t *hslot, const uint32_t *bits, const int32_t *gpre,
                          const int32_t *counts, const int32_t *c_rp, const int32_t *c_col,
                          float *c_val, bool verify, int32_t *status, int num_sms,
                          cudaStream_t s);

// ---- k_reuse.cu ------------------------------------------------------------
// Reuse map of the W<T> classes: per product, its position in C's row.
bool map_class(int cls);
// mops[row] = ops[row] for the listed rows (the caller zeroes mops);
// *too_long |= 1 when a row has more than INT32_MAX / 2 products.
void launch_map_ops(const int32_t *rows, int32_t nrows, const int64_t *ops, int32_t *mops,
                    int32_t *too_long, cudaStream_t s);
// map[moff[row] + t] = position in C's row of the row's t-th product;
// key[row] (when key is not null) = fingerprint of the row's map, 0 when the
// row met a missing column.
void launch_map_build(int cls, const Operands &op, const int32_t *rows, int32_t nrows,
                      const int32_t *c_rp, const int32_t *c_col, const int64_t *moff,
                      uint16_t *map, unsigned long long *key, int32_t *status,
                      cudaStream_t s);
// Sharing of identical maps: insert every listed row's key into the table
// (tkey zeroed, trow filled with 0x7f bytes, mask + 1 a power of two at least
// twice the rows inserted over all calls); then resolve, which points
// moff[row] at the map of the smallest row c with an identical map, sets
// canon[row] = c (row itself when no other row shares its map, -1 for a row
// without a fingerprint), adds 1 to share_count[c] (zeroed by the caller)
// and the rows so redirected to *shared_rows.
void launch_map_dedup_insert(const int32_t *rows, int32_t nrows,
                             const unsigned long long *key, unsigned long long *tkey,
                             int32_t *trow, unsigned long long mask, cudaStream_t s);
void launch_map_dedup_resolve(const int32_t *rows, int32_t nrows,
                              const unsigned long long *key,
                              const unsigned long long *tkey, const int32_t *trow,
                              unsigned long long mask, const int32_t *c_rp,
                              const int32_t *mops, int64_t *moff, const uint16_t *map,
                              int32_t *shared_rows, int32_t *canon, int32_t *share_count,
                              cudaStream_t s);
// Values of the listed rows of class cls from the map (structure in C).
void launch_map_numeric(int cls, const Operands &op, const int64_t *ops, const int32_t *rows,
                        int32_t nrows, const int32_t *c_rp, float *c_val,
                        const int64_t *moff, const uint16_t *map, int32_t *status,
                        cudaStream_t s);

// ---- k_pattern.cu ----------------------------------------------------------
// Term tables of the rows that share a reuse map (see k_pattern.cu).
// Select: canonical rows shared by at least min_share rows (itself included)
// whose row fits a table get pat_of[row] = id (pat_of filled with -1 by the
// caller), pat_canon[id], pat_cap[id] records; *npat counts them;
// maxima[0] / maxima[1] (zeroed by the caller) receive the largest products
// (rounded up to 32) and C row of the tables.
void launch_pat_select(const int32_t *rows, int32_t nrows, const int32_t *canon,
                       const int32_t *share_count, int32_t min_share, const int32_t *a_rp,
                       const int32_t *c_rp, const int32_t *mops, int32_t *pat_of,
                       int32_t *pat_canon, int32_t *pat_cap, int32_t *npat, int32_t *maxima,
                       cudaStream_t s);
// The most records one table can take.
int64_t pat_max_records();
// Build: the npat tables at rec + pat_off[id]; psteps[id] = steps, or -1.
void launch_pat_build(int32_t npat, const int32_t *pat_canon, const int32_t *a_rp,
                      const int32_t *a_col, const int32_t *b_rp, const int32_t *c_rp,
                      const int64_t *moff, const uint16_t *map, const int64_t *pat_off,
                      const int32_t *pat_cap, uint32_t *rec, int32_t *psteps,
                      cudaStream_t s);
// Split a class's rows into table rows (pat_rows / pat_ids, appended at
// *pat_n; pid_of_row[row] = id when pid_of_row is not null) and the rest
// (res_rows, appended at *res_n).
void launch_pat_split(const int32_t *rows, int32_t nrows, const int32_t *canon,
                      const int32_t *pat_of, const int32_t *psteps, const int32_t *a_rp,
                      const int32_t *a_col, const int32_t *b_rp, int32_t *pat_rows,
                      int32_t *pat_ids, int32_t *pat_n, int32_t *res_rows, int32_t *res_n,
                      int32_t *pid_of_row, cudaStream_t s);
// Values of the n table rows (structure in C); max_ops / max_out: the
// maxima the select step found.
void launch_pat_numeric(const Operands &op, const int64_t *ops, const int32_t *pat_rows,
                        const int32_t *pat_ids, int32_t n, const int32_t *c_rp, float *c_val,
                        const int64_t *pat_off, const int32_t *psteps, const uint32_t *rec,
                        int32_t max_ops, int32_t max_out, cudaStream_t s);

// ---- k_tile.cu -------------------------------------------------------------
// Row tiles of the table rows (see k_tile.cu).  Warps per block of the tile
// kernel; uint16 entries per pattern in
// the tile tables (tab has npat * tile_tab_stride() entries).
constexpr int kTileKernelWarps = 2;
// A nonzeros staged together by a pattern kernel (k_jit.cu): runs of at most
// this many.
constexpr int kJitMaxGroup = 8;
int32_t tile_tab_stride();
// Per pattern: its table, B row lengths (lens[id * 32 + j]), column offsets of
// its canonical row (offs[id * 32 + j]) and desc[id] = (na, m, ops, 0), or
// na = -1 when the pattern is not tiled; *b_nnz = B's entries.
void launch_tile_tab(int32_t npat, const int32_t *pat_canon, const int32_t *psteps,
                     const int32_t *a_rp, const int32_t *a_col, const int32_t *b_rp,
                     const int32_t *c_rp, const int64_t *moff, const uint16_t *map,
                     int32_t b_rows, uint16_t *tab, uint16_t *lens, int32_t *offs, int4 *desc,
                     int32_t *b_nnz, cudaStream_t s);
// Tiles of the n rows (pid_of_row: pattern of each table row, -1 for the
// others; shifted: a pattern's rows are its canonical row moved), one per
// chunk of 32 rows: tiles[chunk] = (first row, lane mask, pattern or -1, 0);
// the table rows no tile takes go to lo_rows / lo_ids.  counts[0] tiles, [1]
// leftovers, [2..4] the stage floats, A segment entries and C row the tile
// kernel must hold; per pattern its tiles, its longest A segment and its union
// spans (32 * kJitMaxGroup; see k_tile.cu).  counts, pcount, pseg and spans are zeroed by the caller.
void launch_tile_build(int32_t n, bool shifted, const int32_t *pid_of_row, const int4 *desc,
                       const uint16_t *lens, const int32_t *offs, const int32_t *a_rp,
                       const int32_t *a_col, const int32_t *b_rp, const int32_t *c_rp,
                       int4 *tiles, int32_t *pcount, int32_t *pseg, int32_t *spans,
                       int32_t *lo_rows, int32_t *lo_ids, int32_t *counts, int num_sms,
                       cudaStream_t s);
// rows / ids (count at *count, zeroed by the caller): every row with
// pid_of_row[row] >= 0 and its pattern.
void launch_tile_list(int32_t n, const int32_t *pid_of_row, int32_t *rows, int32_t *ids,
                      int32_t *count, cudaStream_t s);
// Shared memory one warp of the tile kernel needs for those maxima.
size_t tile_smem_per_warp(int32_t stage_need, int32_t a_seg, int32_t max_out,
                          int32_t *acc_rows, int32_t *work_floats, int32_t *stage_cap);
// Values of the tiled rows (structure in C).
void launch_tile_numeric(const Operands &op, int32_t b_nnz, const int4 *tiles, int32_t ntiles,
                         const int4 *desc, const uint16_t *lens, const uint16_t *tab,
                         const int32_t *c_rp, float *c_val, int32_t stage_need, int32_t a_seg,
                         int32_t max_out, cudaStream_t s);

// ---- k_persist.cu ----------------------------------------------------------
// One persistent launch for the numeric-only pass of the merge and map rows
// of a plan (see k_persist.cu): the rows of each class cut into items of
// per_item rows, numbered from item0; segments heaviest class first.
constexpr int kPersistThreads = 256;
struct PersistSeg {
  const int32_t *rows;  // the class's row list (nullptr: rows 0.. in order)
  int32_t cls, count, per_item, item0;
};
struct PersistPlan {
  PersistSeg seg[kNumClasses];
  int32_t nseg = 0, n_items = 0;
};
// Classes the persistent kernel takes (merge and map classes).
bool persist_class(int cls);
// head: one int the launch clears first; max_map_out: the largest C row of
// the map classes in the plan (their accumulators).
void launch_persist_numeric(const Operands &op, const int64_t *ops, const PersistPlan &pp,
                            int32_t *head, const int32_t *c_rp, float *c_val,
                            const int64_t *moff, const uint16_t *map, int32_t *status,
                            int32_t max_map_out, int blocks_per_sm, int num_sms,
                            cudaStream_t s);

// ---- k_jit.cu --------------------------------------------------------------
// One pattern for a compiled kernel (see k_jit.cu): na A nonzeros, B row
// lengths len[j], slot[t] = output position of flattened product t, m
// outputs, groups = [first, end) runs of A nonzeros whose B values are
// staged by one copy.
struct JitRequest {
  int na = 0, m = 0;
  int len[32] = {};
  std::vector<int> slot;
  std::vector<std::pair<int, int>> groups;
  void *kernel = nullptr;  // out: nullptr when NVRTC is missing or the compile failed
};
// Compiles the requests' kernels (side by side; cached for the process);
// returns how many compiled.
int jit_pattern_kernels(std::vector<JitRequest> &reqs);
void jit_stats(int32_t *compiles, double *ms);
// The groups of a pattern from its union spans (launch_tile_build): runs of
// A nonzeros grown while the next one adds less than half its own span and
// the union stays within max_span floats.  *stage_need = the largest union.
std::vector<std::pair<int, int>> jit_groups(int na, const int *len, const int32_t *span,
                                            int32_t max_span, int32_t *stage_need);
// out[*n] = the tiles whose pattern has no compiled kernel (desc[pid].w == 0;
// *n zeroed by the caller).
void launch_table_tiles(const int4 *tiles, int32_t nchunks, const int4 *desc, int4 *out,
                        int32_t *n, cudaStream_t s);
// Words of one tile record of a pattern kernel (na A nonzeros, ngroups
// staging groups).
int32_t jit_record_words(int na, int ngroups);
// The compiled patterns of a tile set: pattern pid of na A nonzeros, group[j]
// the staging group of A nonzero j (of ng; kNoGroup outside them), its records
// (rw words a tile) and the tiles' A ranges.
constexpr int kJitMaxPatterns = 12;
constexpr uint8_t kNoGroup = 255;
struct TileProgram {
  int32_t *prog;
  int2 *arange;
  int32_t pid, na, ng, rw;
  uint8_t group[32];
};
struct TilePrograms {
  TileProgram p[kJitMaxPatterns];
  int32_t n = 0;
};
// Their tile records (see k_jit.cu), in row order, from the tiles of
// launch_tile_build (whose last words it uses); sets desc[pid].w = 1, which
// makes the table kernel skip their tiles.  rank: tile_rank_words(nchunks).
size_t tile_rank_words(int32_t nchunks);
void launch_tile_records(int4 *tiles, int32_t nchunks, bool shifted, const TilePrograms &P,
                         int32_t *rank, const uint16_t *lens, const int32_t *offs,
                         const int32_t *a_rp, const int32_t *a_col, const int32_t *b_rp,
                         int4 *desc, cudaStream_t s);
// Shared memory of one warp of a pattern kernel, in floats: two tile buffers
// (record + A values) of *abuf_floats and two B stage buffers of *stage_cap
// (the largest B range `need` plus widening; room for 16 output rows).
void jit_layout(int32_t rw, int32_t seg_max, int32_t need, int32_t m, int32_t *stage_cap,
                int32_t *abuf_floats, int32_t *work_floats);
// Blocks of a persistent pattern kernel launch: the tiles' pairs, at most
// what fits the SMs at once.
int jit_grid(void *kernel, int32_t ntiles, int32_t work_floats, int32_t m, int num_sms);
// One launch of a pattern kernel over its tile records (head: one device
// word for the launch's tile queue, zeroed here; status: kDevWaitTimeout
// when a bounded wait ran out).
cudaError_t launch_pattern_kernel(void *kernel, const Operands &op, const int32_t *prog,
                                  const int2 *arange, int32_t ntiles, const int32_t *c_rp,
                                  float *c_val, int32_t stage_cap, int32_t abuf_floats,
                                  int32_t work_floats, int grid, int32_t *head,
                                  int32_t *status, cudaStream_t s);

// ---- k_shift.cu ------------------------------------------------------------
// Shift classes (see k_shift.cu).  Every pass but the probe is gated by the
// device flag *on, which the probe's decision sets, so the plan queues them
// without a host round trip.
int32_t shift_max_ops();
int32_t shift_samples();
// Keys and product counts of up to shift_samples() rows spread over A (keys:
// twice that many words) and the decision *on (1: at least half of them
// share their key and they average at least min_mean_ops products).
void launch_shift_decide(const Operands &op, unsigned long long *keys, int32_t min_mean_ops,
                         int32_t *on, CheckGuard guard, cudaStream_t s);
// bcls[b_rows], rcls[a_rows]: the class (smallest verified translate) of
// every B row and row; bkey / rkey / tkey / trow scratch, tcap a power of two
// >= 2 max(a_rows, b_rows).
void launch_shift_classes(const int32_t *on, const Operands &op, int32_t b_rows,
                          const int64_t *ops, unsigned long long *bkey,
                          unsigned long long *rkey, unsigned long long *tkey, int32_t *trow,
                          size_t tcap, int32_t *bcls, int32_t *rcls, cudaStream_t s);
// Patterns (classes of at least min_share rows whose canonical row has at
// most 512 outputs): pat_of[row] / pat_canon / pat_cap / pat_m (-1: dropped)
// / *npat (zeroed by the caller); members: pid_of_row[row] = their pattern
// (else -1; all -1 when *on is 0), cls[row] = empty, *members += count;
// class_count = the census of cls afterwards.
void launch_shift_patterns(const int32_t *on, const Operands &op, const int32_t *rcls,
                           int32_t *share, int32_t min_share, const int64_t *ops,
                           int32_t *pat_of, int32_t *pat_canon, int32_t *pat_cap,
                           int32_t *pat_m, int32_t *npat, int32_t cap_pat,
                           int32_t *pid_of_row, uint8_t *cls, int32_t *members,
                           int32_t *class_count, int num_sms, cudaStream_t s);
// counts[member] = counts[its canonical row].
void launch_shift_copy_counts(const int32_t *on, int32_t n, const int32_t *pid_of_row,
                              const int32_t *rcls, int32_t *counts, cudaStream_t s);
// Member rows' columns: the canonical row's moved by the row distance.
void launch_shift_fill(int32_t n, const int32_t *pid_of_row, const int32_t *rcls,
                       const int32_t *c_rp, int32_t *c_col, cudaStream_t s);
// Maps of the canonical rows (moff[canonical] = id * shift_max_ops()).
void launch_shift_canon_map(int32_t npat, const int32_t *pat_canon, const Operands &op,
                            const int32_t *c_rp, const int32_t *c_col, int64_t *moff,
                            uint16_t *map, cudaStream_t s);
// out[0] = largest products (rounded up to 32), out[1] = largest C row over
// the patterns with pat_m >= 0 (out zeroed by the caller).
void launch_pat_maxima(int32_t npat, const int32_t *pat_canon, const int32_t *pat_m,
                       const int64_t *ops, int32_t *out, cudaStream_t s);

// ---- k_check.cu ------------------------------------------------------------
// *result (initialised to ~0ull) receives min over bad rows of
// ((row + 1) << 8 | code); row -1 means row_ptr[0] != 0.  long_rows: scratch
// of 1 + check_long_rows_cap(rows, nnz) ints, long_rows[0] zeroed by the
// caller (the count of rows over 256 entries, listed after it).
int32_t check_long_rows_cap(int32_t rows, int32_t nnz);
void launch_csr_check(int32_t rows, int32_t cols, const int32_t *row_ptr,
                      const int32_t *col_idx, int32_t nnz,
                      unsigned long long *result, int32_t *long_rows,
                      cudaStream_t s);

// ---- k_numeric.cu ----------------------------------------------------------
// Values (and, when fill, sorted columns) of the rows of one class.  With
// fo, the fused pass: rows go to their slab slots (c_col / c_val = slab),
// c_rp is unused and fill is implied.
void launch_numeric_class(int cls, const Operands &op, const int64_t *ops,
                          const int32_t *rows, int32_t nrows,
                          const int32_t *c_rp, int32_t *c_col, float *c_val,
                          bool fill, float *dense_acc, uint32_t *dense_bits,
                          int32_t dense_slots, int32_t *status, int num_sms,
                          cudaStream_t s, const FusedOut *fo = nullptr);
// Global scratch one dense numeric slot needs (accumulator + bitmap if the
// bitmap does not fit shared memory), 256-byte aligned.
size_t dense_slot_acc_bytes(int32_t b_cols);
size_t dense_slot_bits_bytes(int32_t b_cols);

// ---- k_mlp.cu ----------------------------------------------------------------
// Parameter layout of the 8 -> 32 -> 32 -> 2 row-binning MLP (floats):
// W1[32][8] b1[32] W2[32][32] b2[32] W3[2][32] b3[2] (trained), then the
// per-feature standardisation mean[8] and 1/sd[8] (set, not trained).
constexpr int kMlpIn = 8, kMlpHidden = 32, kMlpOut = 2;
constexpr int kW1 = 0;
constexpr int kB1 = kW1 + kMlpHidden * kMlpIn;
constexpr int kW2 = kB1 + kMlpHidden;
constexpr int kB2 = kW2 + kMlpHidden * kMlpHidden;
constexpr int kW3 = kB2 + kMlpHidden;
constexpr int kB3 = kW3 + kMlpOut * kMlpHidden;
constexpr int kMlpTrained = kB3 + kMlpOut;  // 1410
constexpr int kMu = kMlpTrained;
constexpr int kInvSd = kMu + kMlpIn;
constexpr int kMlpParams = kInvSd + kMlpIn;  // 1426
constexpr int kMlpParamsPad = (kMlpParams + 3) & ~3;

void launch_features(const Operands &op, float b_mean_len, float *feat,
                     int64_t *ops, int num_sms, cudaStream_t s);
// pred[row] = (y0, y1); ops (optional) = per-row op counts.
void launch_predict(const Operands &op, float b_mean_len, const float *params,
                    float2 *pred, int64_t *ops, int num_sms, cudaStream_t s);
// Learned binning for the fused pass: ops, class and slab capacity per row
// (counts[row] = 0 for empty rows) and rows per class.  The B8192 and DENSE
// rows are STRIPE rows without a slab slot where stripes pay (with op.stripes,
// or always; *heavy, zeroed by the caller, holds them).
void launch_learned_plan(const Operands &op, float b_mean_len, const float *params,
                         float scale, bool merge_ok, int64_t *ops, uint8_t *cls,
                         int32_t *cap, int32_t *counts, int32_t *class_count,
                         HeavyRows *heavy, int32_t b_rows, bool always, bool repeats,
                         int num_sms, cudaStream_t s);
// grad (kMlpTrained floats, accumulated) and *loss_sum (accumulated) of the
// mean loss over n_total samples, for samples [0, n).
void launch_mlp_grad(const float *params, const float *feat, const float *target,
                     int32_t n, int32_t n_total, float *grad, float *loss_sum,
                     cudaStream_t s);
void launch_mlp_adam(float *params, const float *grad, float *m, float *v, float lr,
                     float b1, float b2, float eps, int step, cudaStream_t s);

}  // namespace rvsp

// The plan: device-resident analysis state of one product and the C-ABI
// entry points of rvsp_cuda.h that drive the kernel phases.
//
// Flow of rvsp_cuda_symbolic (the GPU form of rvsp_symbolic_count,
// rvsp_symbolic.c:13-86):
//   rowstats -> [host: symbolic class sizes] -> scatter rows by class ->
//   symbolic kernel per class -> scan + numeric classes ->
//   [host: total, numeric class sizes, status] -> scatter rows by class.
// Two host round trips, both for sizes the host must know (grid shapes and
// nnz(C), which the API returns).  rvsp_cuda_numeric then launches one kernel
// per non-empty numeric class with no host round trip.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>
#include <new>
#include <utility>
#include <vector>

#include "device_common.cuh"
#include "kernels.cuh"
#include "rvsp_cuda.h"

using namespace rvsp;

namespace {

template <class T>
struct DevArray {
  T *p = nullptr;
  size_t cap = 0;
  cudaError_t reserve(size_t n) {
    if (n <= cap && p) return cudaSuccess;
    release();
    if (n == 0) n = 1;
    cudaError_t e = cudaMalloc(reinterpret_cast<void **>(&p), n * sizeof(T));
    if (e != cudaSuccess) {
      p = nullptr;
      return e;
    }
    cap = n;
    return cudaSuccess;
  }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
  }
};

// Page-locked host memory, grown on demand and kept: the tile builds'
// transfers go through it (a copy from or to pageable memory is staged and
// synchronous, tens of microseconds each).
struct HostArray {
  char *p = nullptr;
  size_t cap = 0;
  cudaError_t reserve(size_t n) {
    if (n <= cap && p) return cudaSuccess;
    release();
    if (cudaMallocHost(reinterpret_cast<void **>(&p), n ? n : 1) != cudaSuccess) {
      p = nullptr;
      return cudaErrorMemoryAllocation;
    }
    cap = n;
    return cudaSuccess;
  }
  void release() {
    if (p) cudaFreeHost(p);
    p = nullptr;
    cap = 0;
  }
};

rvsp_status_t map_cuda(cudaError_t e) {
  switch (e) {
    case cudaSuccess: return RVSP_SUCCESS;
    case cudaErrorMemoryAllocation: return RVSP_ERROR_ALLOCATION_FAILED;
    case cudaErrorNoDevice:
    case cudaErrorInsufficientDriver:
    case cudaErrorNoKernelImageForDevice:
    case cudaErrorInvalidDevice: return RVSP_ERROR_UNSUPPORTED_BACKEND;
    default: return RVSP_ERROR_DEVICE;
  }
}

// misc int32 words
constexpr int kSymCount = 0;
constexpr int kSymOff = kNumClasses;
constexpr int kSymFill = 2 * kNumClasses;
constexpr int kNumCount = 3 * kNumClasses;
constexpr int kNumOff = 4 * kNumClasses;
constexpr int kNumFill = 5 * kNumClasses;
constexpr int kStatus = 6 * kNumClasses;
constexpr int kLongCount = 6 * kNumClasses + 1;
constexpr int kRetryCount = 6 * kNumClasses + 2;  // two: W1024, W2048 retry lists
constexpr int kShiftMembers = 6 * kNumClasses + 4;  // shift-class member rows
constexpr int kShiftNpat = 6 * kNumClasses + 5;     // shift-class pattern candidates
constexpr int kHeavy = 6 * kNumClasses + 6;  // a HeavyRows
constexpr int kMiscWords = kHeavy + sizeof(HeavyRows) / sizeof(int32_t);
static_assert(kHeavy % 2 == 0, "aligned for 64 bits");
// Stripes for the heavy rows: where they pay, never, always, where they pay for
// numeric-only repeats.
constexpr int kStripesAuto = 0, kStripesNever = 1, kStripesAlways = 2, kStripesRepeats = 3;
// A map shared by at least this many rows gets a term table.
constexpr int32_t kPatMinShare = 16;
constexpr int kPatCountWords = 4 + kNumClasses;

}  // namespace

namespace rvsp {
// Row tiles over one set of term-table patterns (k_tile.cu): per pattern its
// tile table, B row lengths and shape; per row its pattern (pid, -1 for rows
// outside the set); the tiles, one entry per chunk of 32 rows; the pattern
// rows left to the warp-per-row table kernel (lo_rows / lo_ids); for the shift
// classes also every pattern row (all_rows / all_ids, for calls with tiles off;
// listed before the build's wait, so that they are there for every later call,
// on any stream and under capture).
struct JitPattern {
  void *kernel = nullptr;
  DevArray<int32_t> prog;  // tile records (k_jit.cu)
  DevArray<int2> arange;   // per tile its A range
  DevArray<int32_t> head;  // the launch's tile queue
  int32_t n = 0, m = 0, stage_cap = 0, abuf_floats = 0, work_floats = 0;
  int grid = 0;
  void release() {
    prog.release();
    arange.release();
    head.release();
  }
};
struct TileBuild {
  std::vector<JitPattern> jit;   // patterns with their own kernel (k_jit.cu)
  std::vector<JitPattern> pool;  // device arrays of earlier builds, for reuse
  HostArray staging;             // host side of the build's read-back
  int ready = 0;
  int32_t n_tiles = 0, n_lo = 0, stage = 0, aseg = 0, max_out = 0, b_nnz = 0;
  // counts, then per pattern its tiles, its longest A segment and its union
  // spans: one array, zeroed and read back whole
  DevArray<int32_t> counts;
  DevArray<uint16_t> tab, lens;
  DevArray<int32_t> offs, rank;
  DevArray<int4> desc, tiles;
  DevArray<int4> table;  // the tiles left to the table kernel
  int32_t n_table = 0;
  DevArray<int32_t> pid, lo_rows, lo_ids, all_rows, all_ids;
  void release() {
    tab.release();
    lens.release();
    offs.release();
    rank.release();
    desc.release();
    tiles.release();
    table.release();
    n_table = 0;
    pid.release();
    lo_rows.release();
    lo_ids.release();
    counts.release();
    all_rows.release();
    all_ids.release();
    for (auto &j : jit) j.release();
    for (auto &j : pool) j.release();
    jit.clear();
    pool.clear();
    staging.release();
    ready = 0;
  }
};
}  // namespace rvsp

// Memory of the stripe rows of one analysis.  A square product of 2^17 columns
// with every row a stripe row takes 2.5 GiB (18.8 KB a row, of which 16 are its
// bitmap); at 1025 columns a row takes 0.8 KB (0.7 of them items and offsets).
constexpr size_t kStripeBytesMax = size_t(3) << 30;

struct rvsp_cuda_plan {
  int device = 0;
  int num_sms = 148;

  int analysed = 0;
  int merge_policy = kMergeAuto;
  int32_t a_rows = 0, b_rows = 0, b_cols = 0;
  int64_t c_nnz = 0;

  DevArray<int64_t> ops;
  DevArray<uint8_t> cls;
  // Numeric classes from the scan queued before the class census (plain
  // symbolic with merge classes); swapped into cls when that scan is final.
  DevArray<uint8_t> cls_spec;
  DevArray<int32_t> counts;
  DevArray<int32_t> rows_sym, rows_num, long_rows;
  DevArray<int32_t> misc;
  DevArray<int64_t> partials, total;
  DevArray<uint32_t> sym_bits;
  DevArray<unsigned long long> check;
  DevArray<int32_t> check_long;  // count + list of the long rows the check met
  DevArray<int32_t> check_long_b;  // the same for B in rvsp_cuda_symbolic_checked
  int32_t sym_bits_slots = 0;

  int32_t *h_misc = nullptr;  // pinned, kMiscWords
  int64_t *h_total = nullptr;  // pinned
  unsigned long long *h_check = nullptr;  // pinned

  int32_t sym_count[kNumClasses] = {};
  int32_t num_count[kNumClasses] = {};
  int32_t num_off[kNumClasses] = {};
  int32_t dense_slots = 0;
  size_t numeric_ws = 0;
  int num_whole = -1;  // numeric class holding every row (no row list), or -1

  // Learned (fused) analysis: per-row capacity and slab slot, the slab with
  // every non-overflowed row's sorted columns and values, the overflow rows
  // grouped by numeric class, and the fingerprint of the values used.
  int learned = 0;
  DevArray<int32_t> cap;
  DevArray<int64_t> slab_off;
  DevArray<int32_t> slab_col;
  DevArray<float> slab_val;
  DevArray<int32_t> ovf_rows, ovf_sorted;
  DevArray<int32_t> big_rows;  // count + list of the rows compacted by whole blocks
  DevArray<uint8_t> ovf_cls;
  DevArray<char> fused_ws;
  DevArray<unsigned long long> vhash;
  unsigned long long *h_vhash = nullptr;  // pinned, 2 words
  unsigned long long est_hash = 0;
  int32_t n_ovf = 0;
  int32_t a_nnz = 0, b_nnz = 0;
  int32_t ovf_num_count[kNumClasses] = {};
  int32_t ovf_num_off[kNumClasses] = {};
  int64_t slab_total = 0;

  // Reuse map of the W<T> rows (k_reuse.cu), built for one C column array
  // (rmap_col) of the current analysis; rmap_state 0 = not tried, 1 = built,
  // -1 = not used (no W rows, over the memory budget, or a row too long).
  DevArray<uint16_t> rmap;
  DevArray<int64_t> rmap_off;
  DevArray<int32_t> rmap_ops;
  // Sharing of identical maps: per-row fingerprints, the table they meet in,
  // and a counter of the rows that read another row's map.
  DevArray<unsigned long long> rmap_key, rmap_tkey;
  DevArray<int32_t> rmap_trow, rmap_shared, rmap_canon, rmap_share_count;
  // Term tables of the shared maps (k_pattern.cu): per table its records,
  // offset and steps; the rows that use one (pat_rows, pat_ids) and, per W
  // class, the rows that keep the map (res_rows at res_off[c], res_count[c]).
  int pat_ready = 0;
  int32_t n_pat = 0, n_pat_rows = 0;
  int32_t res_off[kNumClasses] = {};
  int32_t res_count[kNumClasses] = {};
  DevArray<int32_t> pat_of, pat_canon, pat_cap, pat_steps, pat_rows, pat_ids, res_rows;
  // [0] tables, [1] table rows, [2 + c] map rows of class c, then the
  // tables' largest products and C row
  DevArray<int32_t> pat_counts;
  int32_t pat_max_ops = 0, pat_max_out = 0;
  DevArray<int64_t> pat_off;
  DevArray<uint32_t> pat_rec;
  // Row tiles of the table rows of shared maps (k_tile.cu).
  int tiles_enabled = 1;
  int pattern_kernels = 1;  // compile kernels for the largest patterns (k_jit.cu)
  TileBuild rt;
  // Shift classes (k_shift.cu): rows that are translates of a canonical row.
  // The probe sets the device flag sh_on; shift_active when the current
  // analysis has member rows (pattern in st.pid).  Their patterns' term
  // tables (sh_*) and row tiles (st) are built from the canonical rows' maps
  // on the first numeric call (shift_tables 1, or -1 when that failed).
  // Persistent numeric-only pass (k_persist.cu): merge rows per item (0: off)
  // and blocks per SM.
  int32_t persist_merge_rows = 0, persist_blocks = 2;
  DevArray<int32_t> persist_head;
  int shift_enabled = 1;
  int shift_active = 0;
  int shift_tables = 0;
  int32_t shift_members = 0, shift_npat = 0, shift_cap_pat = 0;
  int32_t sh_max_ops = 0, sh_max_out = 0;
  DevArray<int32_t> sh_on, sh_trow, sh_bcls, sh_rcls, sh_share, sh_pat_of, sh_pat_canon,
      sh_pat_cap, sh_pat_m, sh_steps, sh_counts;
  DevArray<unsigned long long> sh_probe, sh_bkey, sh_rkey, sh_tkey;
  DevArray<int64_t> sh_moff, sh_pat_off;
  DevArray<uint16_t> sh_map;
  DevArray<uint32_t> sh_rec;
  TileBuild st;
  // Stripe rows (k_stripe.cu): B's stripes, and of the rows counted by the
  // current analysis (sp_ready) their bitmaps, their outputs before each
  // stripe, their slot by row, and the value items of the numeric STRIPE rows.
  StripeShape sp;
  int sp_ready = 0;
  size_t stripe_max = kStripeBytesMax;  // bytes
  int32_t stripe_policy = kStripesAuto;
  int64_t sp_cap = 0;
  DevArray<int32_t> sp_hist, sp_bound, sp_ptr, sp_gpre, sp_soff, sp_hslot, sp_done;
  DevArray<int32_t> sp_cnt;  // items from the front, from the back, queue head
  DevArray<float> sp_share;
  DevArray<uint32_t> sp_bits;
  DevArray<int4> sp_items;
  const int32_t *rmap_col = nullptr;
  int rmap_state = 0;
  int64_t rmap_entries = 0;

  // Side streams of the numeric-only pass (created on first use; state 0
  // untried, 1 ready, -1 unavailable).
  static constexpr int kSide = 6;
  cudaStream_t side[kSide] = {};
  cudaEvent_t fork_ev = nullptr, join_ev[kSide] = {};
  int side_state = 0;

  bool profiling = false;
  struct Pending {
    cudaEvent_t a, b;
    int phase;
    int launches;
  };
  std::vector<Pending> pending;
  std::vector<cudaEvent_t> pool;
  double ms[RVSP_PHASE_COUNT] = {};
  int64_t launches[RVSP_PHASE_COUNT] = {};

  cudaEvent_t take_event() {
    if (!pool.empty()) {
      cudaEvent_t e = pool.back();
      pool.pop_back();
      return e;
    }
    cudaEvent_t e = nullptr;
    cudaEventCreate(&e);
    return e;
  }
};

namespace {

struct PhaseScope {
  rvsp_cuda_plan *pl;
  cudaStream_t s;
  int phase;
  int launches = 0;
  cudaEvent_t a = nullptr;
  PhaseScope(rvsp_cuda_plan *p, cudaStream_t st, int ph) : pl(p), s(st), phase(ph) {
    if (pl->profiling) {
      a = pl->take_event();
      cudaEventRecord(a, s);
    }
  }
  ~PhaseScope() {
    if (pl->profiling && a) {
      cudaEvent_t b = pl->take_event();
      cudaEventRecord(b, s);
      pl->pending.push_back({a, b, phase, launches});
    }
  }
};

void resolve_pending(rvsp_cuda_plan *pl) {
  for (auto &q : pl->pending) {
    float t = 0.0f;
    if (cudaEventSynchronize(q.b) == cudaSuccess &&
        cudaEventElapsedTime(&t, q.a, q.b) == cudaSuccess) {
      pl->ms[q.phase] += t;
    }
    pl->launches[q.phase] += q.launches;
    pl->pool.push_back(q.a);
    pl->pool.push_back(q.b);
  }
  pl->pending.clear();
}

// Side streams are made one by one, when one is first handed out (at the
// highest stream priority, on the plan's device, never while `s` is being
// captured): all six at the first use added 0.3 ms to a plan's first product.
bool may_make_streams(const rvsp_cuda_plan *p, cudaStream_t s) {
  int dev = -1;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaGetDevice(&dev) == cudaSuccess && dev == p->device &&
      cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone)
    return true;
  cudaGetLastError();
  return false;
}

bool side_streams(rvsp_cuda_plan *p, cudaStream_t s) {
  if (p->side_state == 0 && may_make_streams(p, s)) {
    p->side_state =
        cudaEventCreateWithFlags(&p->fork_ev, cudaEventDisableTiming) == cudaSuccess ? 1 : -1;
    if (p->side_state < 0) cudaGetLastError();
  }
  return p->side_state == 1;
}

bool side_stream(rvsp_cuda_plan *p, int i, cudaStream_t s) {
  if (p->side[i]) return true;
  if (p->side_state != 1 || !may_make_streams(p, s)) return false;
  int least = 0, greatest = 0;
  cudaStream_t made = nullptr;
  if (cudaDeviceGetStreamPriorityRange(&least, &greatest) == cudaSuccess &&
      (p->join_ev[i] ||
       cudaEventCreateWithFlags(&p->join_ev[i], cudaEventDisableTiming) == cudaSuccess) &&
      cudaStreamCreateWithPriority(&made, cudaStreamNonBlocking, greatest) == cudaSuccess) {
    p->side[i] = made;
    return true;
  }
  cudaGetLastError();
  return false;
}

// Streams of one pass whose row groups are independent: the numeric pass's
// (pattern kernels, table tiles, leftover rows, class kernels) write disjoint
// rows of C and only read A, B and the plan's tables, the symbolic pass's
// write disjoint counts.  All but the largest go to the side streams, forked
// from the caller's stream and joined back into it: the small launches, each
// bound by the latency of a few long rows, run beside the large one and
// beside each other instead of after one another.  main() is the caller's
// stream; next() hands out the side streams in turn (without side streams,
// the caller's stream); a side stream that is not handed out is not waited
// for.
struct Lanes {
  rvsp_cuda_plan *pl;
  cudaStream_t s;
  bool forked = false;
  bool used[rvsp_cuda_plan::kSide] = {};    // has work to join
  bool behind[rvsp_cuda_plan::kSide] = {};  // waits for the last fork
  int turn = 0;
  Lanes(rvsp_cuda_plan *p, cudaStream_t st, bool want) : pl(p), s(st) {
    forked = want && side_streams(p, st) && cudaEventRecord(p->fork_ev, st) == cudaSuccess;
  }
  cudaStream_t main() const { return s; }
  cudaStream_t next() {
    if (!forked) return s;
    const int i = turn;
    turn = (turn + 1) % rvsp_cuda_plan::kSide;
    if (!side_stream(pl, i, s)) return s;
    if (!behind[i]) {
      if (cudaStreamWaitEvent(pl->side[i], pl->fork_ev, 0) != cudaSuccess) return s;
      behind[i] = used[i] = true;
    }
    return pl->side[i];
  }
  // What next() hands out from here on also comes after the work queued on
  // the caller's stream so far; work already on a side stream stays there.
  void refork() {
    if (!forked) return;
    if (cudaEventRecord(pl->fork_ev, s) != cudaSuccess) return join();
    for (bool &b : behind) b = false;
  }
  void join() {
    if (!forked) return;
    for (int i = 0; i < rvsp_cuda_plan::kSide; ++i) {
      if (!used[i]) continue;
      cudaEventRecord(pl->join_ev[i], pl->side[i]);
      cudaStreamWaitEvent(s, pl->join_ev[i], 0);
      used[i] = behind[i] = false;
    }
    forked = false;
  }
  ~Lanes() { join(); }
};

HeavyRows *heavy_rows(int32_t *misc) { return reinterpret_cast<HeavyRows *>(misc + kHeavy); }

// Whether a census has rows in several classes that launch of their own.
bool several_classes(const int32_t *count) {
  int n = count[kStripe8] + count[kStripe] > 0;
  for (int c = kEmpty_ + 1; c < kStripe8; ++c) n += count[c] > 0;
  return n > 1;
}

rvsp_status_t device_status_to_rvsp(int32_t st) {
  return st == kDevOk ? RVSP_SUCCESS : RVSP_ERROR_DEVICE;
}

// The class that holds every non-empty row, when there is exactly one and
// its kernel may also see the empty rows (merge kernels handle them; the
// others are used only when there are none).  Its rows then need no list.
int whole_matrix_class(const int32_t *count, int32_t a_rows) {
  int found = -1;
  for (int c = kEmpty_ + 1; c < kNumClasses; ++c) {
    if (count[c] <= 0) continue;
    if (found >= 0) return -1;
    found = c;
  }
  if (found < 0 || count[found] + count[kEmpty_] != a_rows) return -1;
  const bool merge = found == kM4 || found == kM8 || found == kM16;
  return (count[kEmpty_] == 0 || merge) ? found : -1;
}

// The STRIPE8 and STRIPE rows of one census: their lists lie one after the
// other; one that holds every row needs none.
struct RowList {
  const int32_t *rows;
  int32_t n;
};
RowList stripe_rows(const int32_t *count, const int32_t *off, int whole, const int32_t *list) {
  return {whole >= kStripe8 ? nullptr : list + off[kStripe8], count[kStripe8] + count[kStripe]};
}

// After the final scan (class counts of the numeric pass in h_misc): host
// offsets, the row lists (unless one class holds every row) and the dense
// workspace the numeric pass will need.
void finish_numeric_bins(rvsp_cuda_plan *p, int32_t a_rows, int32_t b_cols,
                         cudaStream_t s) {
  int32_t *misc = p->misc.p;
  int32_t off = 0;
  for (int c = 0; c < kNumClasses; ++c) {
    p->num_count[c] = p->h_misc[kNumCount + c];
    p->num_off[c] = off;
    if (c != kEmpty_) off += p->num_count[c];
  }
  p->num_whole = p->shift_active ? -1 : whole_matrix_class(p->num_count, a_rows);
  if (p->num_whole < 0) {
    PhaseScope ph(p, s, RVSP_PHASE_SCAN);
    launch_class_offsets(misc + kNumCount, misc + kNumOff, s);
    launch_scatter_rows(a_rows, p->cls.p, misc + kNumOff, misc + kNumFill,
                        p->rows_num.p, s);
    ph.launches = 2;
  }
  const RowList sr = stripe_rows(p->num_count, p->num_off, p->num_whole, p->rows_num.p);
  if (p->sp_ready && sr.n > 0) {
    PhaseScope ph(p, s, RVSP_PHASE_SCAN);
    launch_stripe_items(p->sp, sr.rows, sr.n, p->ops.p, p->sp_hslot.p, p->sp_soff.p,
                        p->sp_bound.p, p->sp_share.p, p->sp_items.p, p->sp_cap, p->sp_cnt.p, s);
    ph.launches = 1;
  }
  if (p->num_count[kDense] > 0) {
    p->dense_slots = p->num_count[kDense] < p->num_sms ? p->num_count[kDense] : p->num_sms;
    p->numeric_ws = size_t(p->dense_slots) *
                    (dense_slot_acc_bytes(b_cols) + dense_slot_bits_bytes(b_cols));
  } else {
    p->dense_slots = 0;
    p->numeric_ws = 0;
  }
}

// The exact counts of the nrows STRIPE rows listed at rows (null: every row),
// with what their columns and values need later.  Sets sp_ready; it stays 0,
// and nothing was counted, when all of that would take more than stripe_max
// bytes or, where it has to grow, a quarter of the free memory.
cudaError_t count_stripe_rows(rvsp_cuda_plan *p, const Operands &op, int32_t b_rows,
                              const int32_t *rows, int32_t nrows, cudaStream_t s) {
  const StripeShape &g = p->sp;
  const size_t n = static_cast<size_t>(nrows), stops = static_cast<size_t>(g.ns_max) + 1;
  const size_t words = static_cast<size_t>(g.words);
  p->sp_cap = int64_t(nrows) * g.ns_max;
  auto each = [&](auto f) {
    f(p->sp_bits, n * words);
    f(p->sp_gpre, n * size_t(stripe_groups(g.words)));
    f(p->sp_soff, n * stops);
    f(p->sp_items, std::max(size_t(p->sp_cap), stripe_tasks(nrows)));
    f(p->sp_done, n);
    f(p->sp_hslot, size_t(op.a_rows));
    f(p->sp_hist, words);
    f(p->sp_bound, stops);
    f(p->sp_share, stops);
    f(p->sp_cnt, size_t(3));
    f(p->sp_ptr, size_t(b_rows) * stops);
  };
  size_t need = 0, grow = 0;
  each([&](auto &a, size_t count) {
    const size_t bytes = count * sizeof(*a.p);
    need += bytes;
    if (count > a.cap) grow += bytes;
  });
  if (need > p->stripe_max) return cudaSuccess;
  if (grow > 0) {
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) return cudaGetLastError();
    if (grow > free_b / 4) return cudaSuccess;
  }
  bool room = true;
  each([&](auto &a, size_t count) { room = room && a.reserve(count) == cudaSuccess; });
  if (!room) {  // the rows take the block-per-row kernels, which get the memory back
    cudaGetLastError();
    each([](auto &a, size_t) { a.release(); });
    return cudaSuccess;
  }
  launch_stripe_table(g, b_rows, op.b_rp, op.b_col, p->sp_hist.p, p->sp_bound.p, p->sp_share.p,
                      p->sp_ptr.p, p->num_sms, s);
  cudaMemsetAsync(p->sp_hslot.p, 0xff, size_t(op.a_rows) * sizeof(int32_t), s);
  // (the items' memory is free until the numeric bins are known)
  launch_stripe_count(g, op, rows, nrows, p->ops.p, p->sp_bound.p,
                      reinterpret_cast<int2 *>(p->sp_items.p), p->sp_cnt.p, p->sp_done.p,
                      p->counts.p, p->sp_hslot.p, p->sp_bits.p, p->sp_gpre.p, p->sp_soff.p,
                      p->num_sms, s);
  p->sp_ready = 1;
  return cudaGetLastError();
}

// Reserves (and zeroes when grown) the global bitmaps dense symbolic rows use
// when B is too wide for a shared-memory bitmap; returns the slot count.
cudaError_t ensure_sym_bits(rvsp_cuda_plan *p, int32_t dense_rows, int32_t b_cols,
                            cudaStream_t s, int32_t *slots_out) {
  *slots_out = 0;
  const size_t bits_bytes = dense_slot_bits_bytes(b_cols);
  if (dense_rows <= 0 || bits_bytes == 0) return cudaSuccess;
  const int32_t slots = dense_rows < p->num_sms ? dense_rows : p->num_sms;
  const size_t words = bits_bytes / sizeof(uint32_t) * size_t(slots);
  if (words > p->sym_bits.cap) {
    cudaError_t e = p->sym_bits.reserve(words);
    if (e != cudaSuccess) return e;
    cudaMemsetAsync(p->sym_bits.p, 0, words * sizeof(uint32_t), s);
  }
  p->sym_bits_slots = slots;
  *slots_out = slots;
  return cudaSuccess;
}

unsigned long long values_fingerprint_launch(rvsp_cuda_plan *p, const float *a_val,
                                             int64_t a_n, const float *b_val, int64_t b_n,
                                             cudaStream_t s) {
  cudaMemsetAsync(p->vhash.p, 0, sizeof(unsigned long long), s);
  launch_values_hash(a_val, a_n, 0x41ull, p->vhash.p, s);
  launch_values_hash(b_val, b_n, 0x42ull << 40, p->vhash.p, s);
  cudaMemcpyAsync(p->h_vhash, p->vhash.p, sizeof(unsigned long long),
                  cudaMemcpyDeviceToHost, s);
  return 0;
}

}  // namespace

extern "C" {

rvsp_status_t rvsp_cuda_plan_create(rvsp_cuda_plan_t *plan) {
  if (!plan) return RVSP_ERROR_NULL_POINTER;
  *plan = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) {
    cudaGetLastError();
    return RVSP_ERROR_UNSUPPORTED_BACKEND;
  }
  int dev = 0, major = 0, minor = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return RVSP_ERROR_UNSUPPORTED_BACKEND;
  cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev);
  cudaDeviceGetAttribute(&minor, cudaDevAttrComputeCapabilityMinor, dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (major != 10 || minor != 0) return RVSP_ERROR_UNSUPPORTED_BACKEND;
  rvsp_cuda_plan *p = new (std::nothrow) rvsp_cuda_plan();
  if (!p) return RVSP_ERROR_ALLOCATION_FAILED;
  p->device = dev;
  p->num_sms = sms > 0 ? sms : 148;
  cudaError_t e = p->misc.reserve(kMiscWords);
  if (e == cudaSuccess) e = p->total.reserve(1);
  if (e == cudaSuccess) e = p->check.reserve(2);
  if (e == cudaSuccess) e = cudaMallocHost(reinterpret_cast<void **>(&p->h_misc), kMiscWords * sizeof(int32_t));
  if (e == cudaSuccess) e = cudaMallocHost(reinterpret_cast<void **>(&p->h_total), sizeof(int64_t));
  if (e == cudaSuccess) e = cudaMallocHost(reinterpret_cast<void **>(&p->h_check), 2 * sizeof(unsigned long long));
  if (e == cudaSuccess) e = cudaMallocHost(reinterpret_cast<void **>(&p->h_vhash), 2 * sizeof(unsigned long long));
  if (e == cudaSuccess) e = p->vhash.reserve(2);
  if (e == cudaSuccess) e = cudaMemset(p->misc.p, 0, kMiscWords * sizeof(int32_t));
  if (e != cudaSuccess) {
    rvsp_cuda_plan_destroy(p);
    return map_cuda(e);
  }
  *plan = p;
  return RVSP_SUCCESS;
}

void rvsp_cuda_plan_destroy(rvsp_cuda_plan_t p) {
  if (!p) return;
  resolve_pending(p);
  for (cudaEvent_t e : p->pool) cudaEventDestroy(e);
  for (int i = 0; i < rvsp_cuda_plan::kSide; ++i) {
    if (p->side[i]) cudaStreamDestroy(p->side[i]);
    if (p->join_ev[i]) cudaEventDestroy(p->join_ev[i]);
  }
  if (p->fork_ev) cudaEventDestroy(p->fork_ev);
  p->rmap.release();
  p->rmap_off.release();
  p->rmap_ops.release();
  p->rmap_key.release();
  p->rmap_tkey.release();
  p->rmap_trow.release();
  p->rmap_shared.release();
  p->rmap_canon.release();
  p->rmap_share_count.release();
  p->pat_of.release();
  p->pat_canon.release();
  p->pat_cap.release();
  p->pat_steps.release();
  p->pat_rows.release();
  p->pat_ids.release();
  p->res_rows.release();
  p->pat_counts.release();
  p->pat_off.release();
  p->pat_rec.release();
  p->rt.release();
  p->st.release();
  p->persist_head.release();
  for (auto *a : {&p->sh_on, &p->sh_trow, &p->sh_bcls, &p->sh_rcls, &p->sh_share,
                  &p->sh_pat_of, &p->sh_pat_canon, &p->sh_pat_cap, &p->sh_pat_m,
                  &p->sh_steps, &p->sh_counts})
    a->release();
  for (auto *a : {&p->sh_probe, &p->sh_bkey, &p->sh_rkey, &p->sh_tkey}) a->release();
  p->sh_moff.release();
  p->sh_pat_off.release();
  p->sh_map.release();
  p->sh_rec.release();
  for (auto *a : {&p->sp_hist, &p->sp_bound, &p->sp_ptr, &p->sp_gpre, &p->sp_soff, &p->sp_hslot,
                  &p->sp_done, &p->sp_cnt})
    a->release();
  p->sp_share.release();
  p->sp_bits.release();
  p->sp_items.release();
  p->ops.release();
  p->cls.release();
  p->cls_spec.release();
  p->counts.release();
  p->rows_sym.release();
  p->rows_num.release();
  p->long_rows.release();
  p->misc.release();
  p->partials.release();
  p->total.release();
  p->sym_bits.release();
  p->check.release();
  p->check_long.release();
  p->check_long_b.release();
  p->cap.release();
  p->slab_off.release();
  p->slab_col.release();
  p->slab_val.release();
  p->ovf_rows.release();
  p->ovf_sorted.release();
  p->ovf_cls.release();
  p->fused_ws.release();
  p->vhash.release();
  if (p->h_misc) cudaFreeHost(p->h_misc);
  if (p->h_total) cudaFreeHost(p->h_total);
  if (p->h_check) cudaFreeHost(p->h_check);
  if (p->h_vhash) cudaFreeHost(p->h_vhash);
  delete p;
}

namespace {

// Matrices of at least this many rows run the shift-class probe.
// The shift analysis runs by default (setting 1) on matrices of at least
// kShiftMinRows rows whose sampled rows average kShiftMinMeanOps products;
// setting 2 runs it on any matrix whose rows are translates.
constexpr int32_t kShiftMinRows = 32768;
constexpr int32_t kShiftMinMeanOps = 64;
int32_t shift_bar(const rvsp_cuda_plan *p) { return p->shift_enabled == 2 ? 0 : kShiftMinMeanOps; }
bool shift_size_ok(const rvsp_cuda_plan *p, int32_t a_rows) {
  return p->shift_enabled == 2 ? a_rows >= 64 : a_rows >= kShiftMinRows;
}

// Scratch of the shift-class analysis (k_shift.cu).  The key table is a
// power of two of at least twice the rows; a larger one kept from before is
// used whole.
cudaError_t reserve_shift(rvsp_cuda_plan *p, int32_t a_rows, int32_t b_rows) {
  const size_t n = static_cast<size_t>(a_rows), nb = static_cast<size_t>(b_rows);
  size_t tcap = 64;
  while (tcap < 2 * (n > nb ? n : nb)) tcap <<= 1;
  p->shift_cap_pat = static_cast<int32_t>(n / kPatMinShare + 1);
  const size_t cp = static_cast<size_t>(p->shift_cap_pat);
  cudaError_t e = p->sh_on.reserve(2);
  if (e == cudaSuccess) e = p->sh_probe.reserve(2 * size_t(shift_samples()));
  if (e == cudaSuccess) e = p->sh_bkey.reserve(nb);
  if (e == cudaSuccess) e = p->sh_rkey.reserve(n);
  if (e == cudaSuccess) e = p->sh_tkey.reserve(tcap);
  if (e == cudaSuccess) e = p->sh_trow.reserve(p->sh_tkey.cap);
  if (e == cudaSuccess) e = p->sh_bcls.reserve(nb);
  if (e == cudaSuccess) e = p->sh_rcls.reserve(n);
  if (e == cudaSuccess) e = p->sh_share.reserve(n);
  if (e == cudaSuccess) e = p->sh_pat_of.reserve(n);
  if (e == cudaSuccess) e = p->st.pid.reserve(n);
  if (e == cudaSuccess) e = p->sh_pat_canon.reserve(cp);
  if (e == cudaSuccess) e = p->sh_pat_cap.reserve(cp);
  if (e == cudaSuccess) e = p->sh_pat_m.reserve(cp);
  return e;
}

// The structure checks rvsp_cuda_symbolic_checked folds into the symbolic
// pass: A always, B unless it is A.
struct PreCheck {
  int32_t a_cols, a_nnz, b_nnz;
  bool check_b;
};

rvsp_status_t symbolic_impl(rvsp_cuda_plan_t p, cudaStream_t s, int32_t a_rows,
                            int32_t b_rows, int32_t b_cols, const int32_t *a_row_ptr,
                            const int32_t *a_col_idx, const int32_t *b_row_ptr,
                            const int32_t *b_col_idx, int32_t *c_row_ptr,
                            int64_t *c_nnz_out, const PreCheck *chk);
cudaError_t symbolic_rest(rvsp_cuda_plan *p, cudaStream_t s, const Operands &op,
                          int32_t a_rows, int32_t b_rows, int32_t b_cols,
                          const int32_t *a_row_ptr, int32_t *c_row_ptr,
                          const int32_t *sym_off, bool merge_done);

}  // namespace

rvsp_status_t rvsp_cuda_symbolic(rvsp_cuda_plan_t p, void *stream, int32_t a_rows,
                                 int32_t b_rows, int32_t b_cols,
                                 const int32_t *a_row_ptr,
                                 const int32_t *a_col_idx,
                                 const int32_t *b_row_ptr,
                                 const int32_t *b_col_idx, int32_t *c_row_ptr,
                                 int64_t *c_nnz_out) {
  if (!p || !a_row_ptr || !a_col_idx || !b_row_ptr || !b_col_idx || !c_row_ptr ||
      !c_nnz_out)
    return RVSP_ERROR_NULL_POINTER;
  if (a_rows <= 0 || b_rows <= 0 || b_cols <= 0) return RVSP_ERROR_INVALID_ARGUMENT;
  return symbolic_impl(p, static_cast<cudaStream_t>(stream), a_rows, b_rows, b_cols,
                       a_row_ptr, a_col_idx, b_row_ptr, b_col_idx, c_row_ptr, c_nnz_out,
                       nullptr);
}

rvsp_status_t rvsp_cuda_symbolic_checked(rvsp_cuda_plan_t p, void *stream, int32_t a_rows,
                                         int32_t a_cols, int32_t a_nnz, int32_t b_rows,
                                         int32_t b_cols, int32_t b_nnz,
                                         const int32_t *a_row_ptr, const int32_t *a_col_idx,
                                         const int32_t *b_row_ptr, const int32_t *b_col_idx,
                                         int check_b, int32_t *c_row_ptr,
                                         int64_t *c_nnz_out) {
  if (!p || !a_row_ptr || !a_col_idx || !b_row_ptr || !b_col_idx || !c_row_ptr ||
      !c_nnz_out)
    return RVSP_ERROR_NULL_POINTER;
  if (a_rows <= 0 || b_rows <= 0 || b_cols <= 0 || a_cols < 0 || a_nnz < 0 || b_nnz < 0)
    return RVSP_ERROR_INVALID_ARGUMENT;
  // A's columns index B's rows: a column the check lets through is < a_cols
  // = b_rows, so every pass after the verdict reads B's row pointers in
  // bounds (the row statistics bound it by b_rows as well).
  if (a_cols != b_rows) return RVSP_ERROR_INVALID_ARGUMENT;
  const PreCheck chk{a_cols, a_nnz, b_nnz, check_b != 0};
  return symbolic_impl(p, static_cast<cudaStream_t>(stream), a_rows, b_rows, b_cols,
                       a_row_ptr, a_col_idx, b_row_ptr, b_col_idx, c_row_ptr, c_nnz_out,
                       &chk);
}

namespace {

rvsp_status_t symbolic_impl(rvsp_cuda_plan_t p, cudaStream_t s, int32_t a_rows,
                            int32_t b_rows, int32_t b_cols, const int32_t *a_row_ptr,
                            const int32_t *a_col_idx, const int32_t *b_row_ptr,
                            const int32_t *b_col_idx, int32_t *c_row_ptr,
                            int64_t *c_nnz_out, const PreCheck *chk) {
  p->analysed = 0;
  p->rmap_state = 0;
  p->rmap_col = nullptr;
  p->sp = p->stripe_policy == kStripesNever ? StripeShape() : stripe_shape(b_rows, b_cols);
  p->sp_ready = 0;
  const size_t n = static_cast<size_t>(a_rows);

  cudaError_t e = p->ops.reserve(n);
  if (e == cudaSuccess) e = p->cls.reserve(n);
  if (e == cudaSuccess) e = p->counts.reserve(n);
  if (e == cudaSuccess) e = p->rows_sym.reserve(n);
  if (e == cudaSuccess) e = p->rows_num.reserve(n);
  if (e == cudaSuccess) e = p->long_rows.reserve(n);
  if (e == cudaSuccess) e = p->partials.reserve(scan_partials_bytes(a_rows) / sizeof(int64_t));
  if (e == cudaSuccess && merge_allowed(p->merge_policy, a_rows)) e = p->cls_spec.reserve(n);
  if (e == cudaSuccess && chk)
    e = p->check_long.reserve(1 + size_t(check_long_rows_cap(a_rows, chk->a_nnz)));
  if (e == cudaSuccess && chk && chk->check_b)
    e = p->check_long_b.reserve(1 + size_t(check_long_rows_cap(b_rows, chk->b_nnz)));
  if (e != cudaSuccess) return map_cuda(e);

  Operands op{a_rows, b_cols, a_row_ptr, a_col_idx, nullptr,
              b_row_ptr, b_col_idx, nullptr,
              merge_allowed(p->merge_policy, a_rows)};
  op.stripes = p->sp.on;
  if (chk) {
    // Checks of A (and B) run first; the row statistics after them are
    // bounded (they read nothing outside A's entries and B's row pointers),
    // and one host round trip brings back both the checks' verdicts and the
    // class sizes.  Nothing that depends on the structure runs before it.
    op.a_nnz = chk->a_nnz;
    op.b_rows = b_rows;
    cudaMemsetAsync(p->check.p, 0xff, 2 * sizeof(unsigned long long), s);
    cudaMemsetAsync(p->check_long.p, 0, sizeof(int32_t), s);
    if (chk->check_b) cudaMemsetAsync(p->check_long_b.p, 0, sizeof(int32_t), s);
    PhaseScope ph(p, s, RVSP_PHASE_CHECK);
    launch_csr_check(a_rows, chk->a_cols, a_row_ptr, a_col_idx, chk->a_nnz, p->check.p,
                     p->check_long.p, s);
    ph.launches = 2;
    if (chk->check_b) {
      launch_csr_check(b_rows, b_cols, b_row_ptr, b_col_idx, chk->b_nnz, p->check.p + 1,
                       p->check_long_b.p, s);
      ph.launches += 2;
    }
  }
  int32_t *misc = p->misc.p;
  cudaMemsetAsync(misc, 0, kMiscWords * sizeof(int32_t), s);
  CheckGuard guard;
  if (chk) {
    guard.w = p->check.p;
    guard.n = chk->check_b ? 2 : 1;
  }
  p->shift_active = 0;
  p->shift_tables = 0;
  p->shift_members = 0;
  p->shift_npat = 0;
  bool shift = p->shift_enabled && shift_size_ok(p, a_rows) &&
               reserve_shift(p, a_rows, b_rows) == cudaSuccess;
  if (!shift) cudaGetLastError();
  {
    PhaseScope ph(p, s, RVSP_PHASE_ROWSTATS);
    if (shift)
      launch_shift_decide(op, p->sh_probe.p, shift_bar(p), p->sh_on.p, guard, s);
    launch_rowstats(op, p->ops.p, p->cls.p, p->counts.p, misc + kSymCount,
                    p->long_rows.p, misc + kLongCount, a_rows, heavy_rows(misc),
                    shift ? p->sh_on.p + 1 : nullptr, s);
    launch_rowstats_long(op, p->long_rows.p, misc + kLongCount, p->ops.p, p->cls.p,
                         p->counts.p, misc + kSymCount, heavy_rows(misc), p->num_sms, s);
    ph.launches = 2;
    if (shift) {
      // Shift classes: the probe decides on the device and one small read
      // brings the decision to the host, so a matrix without them queues
      // none of the analysis's passes (each a full grid that would only
      // read the flag and return).  Member rows leave the symbolic classes
      // (census recounted).
      e = cudaMemcpyAsync(p->h_misc, p->sh_on.p, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) return map_cuda(e);
      shift = p->h_misc[0] != 0;
      ph.launches += 2;
    }
    if (shift) {
      launch_shift_classes(p->sh_on.p, op, b_rows, p->ops.p, p->sh_bkey.p, p->sh_rkey.p,
                           p->sh_tkey.p, p->sh_trow.p, p->sh_tkey.cap, p->sh_bcls.p,
                           p->sh_rcls.p, s);
      launch_shift_patterns(p->sh_on.p, op, p->sh_rcls.p, p->sh_share.p, kPatMinShare,
                            p->ops.p, p->sh_pat_of.p, p->sh_pat_canon.p, p->sh_pat_cap.p,
                            p->sh_pat_m.p, misc + kShiftNpat, p->shift_cap_pat, p->st.pid.p,
                            p->cls.p, misc + kShiftMembers, misc + kSymCount, p->num_sms, s);
      ph.launches += 18;
    }
  }
  const int32_t *skip = shift ? p->st.pid.p : nullptr;
  // Merge-class rows need no host-side census: their symbolic pass (one
  // launch for M4 and M8 and one for M16, over all rows, each skipping the rest)
  // and the scan are queued at once, behind the check verdict, so a product
  // whose rows are all merge rows takes one host round trip.  When other
  // classes turn up, their pass and the scan follow the census.  The early
  // scan writes its numeric classes to cls_spec: the census-driven pass
  // still needs the symbolic classes in cls.
  const bool spec = op.merge_ok;
  if (spec) {
    {
      PhaseScope ph(p, s, RVSP_PHASE_SYMBOLIC);
      launch_merge_symbolic_all(op, p->cls.p, a_rows, p->counts.p, guard, s);
      ph.launches = 2;
    }
    {
      PhaseScope ph(p, s, RVSP_PHASE_SCAN);
      if (shift)
        launch_shift_copy_counts(p->sh_on.p, a_rows, p->st.pid.p, p->sh_rcls.p, p->counts.p, s);
      launch_scan_and_class(a_rows, p->counts.p, p->ops.p, a_row_ptr, c_row_ptr,
                            p->partials.p, p->total.p, p->cls_spec.p, misc + kNumCount,
                            op.merge_ok, s, guard, skip);
      ph.launches = shift ? 4 : 3;
    }
    cudaMemcpyAsync(p->h_misc, misc, kMiscWords * sizeof(int32_t), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(p->h_total, p->total.p, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
  } else {
    cudaMemcpyAsync(p->h_misc, misc, kMiscWords * sizeof(int32_t), cudaMemcpyDeviceToHost, s);
  }
  if (chk)
    cudaMemcpyAsync(p->h_check, p->check.p, 2 * sizeof(unsigned long long),
                    cudaMemcpyDeviceToHost, s);
  e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return map_cuda(e);
  if (chk && (p->h_check[0] != ~0ull || (chk->check_b && p->h_check[1] != ~0ull)))
    return RVSP_ERROR_INVALID_CSR;  // not canonical: nothing ran on it
  if (shift) {
    p->shift_members = p->h_misc[kShiftMembers];
    p->shift_npat = p->h_misc[kShiftNpat] < p->shift_cap_pat ? p->h_misc[kShiftNpat]
                                                              : p->shift_cap_pat;
    p->shift_active = p->shift_members > 0;
  }
  int32_t sym_off[kNumClasses];
  int32_t off = 0;
  bool rest = !spec;  // classes left for the census-driven pass
  for (int c = 0; c < kNumClasses; ++c) {
    p->sym_count[c] = p->h_misc[kSymCount + c];
    sym_off[c] = off;
    if (c != kEmpty_) off += p->sym_count[c];
    if (c != kEmpty_ && !is_merge_class(c) && p->sym_count[c] > 0) rest = true;
  }
  if (rest) {
    e = symbolic_rest(p, s, op, a_rows, b_rows, b_cols, a_row_ptr, c_row_ptr, sym_off, spec);
    if (e != cudaSuccess) return map_cuda(e);
  } else {
    std::swap(p->cls, p->cls_spec);  // the early scan's numeric classes
  }
  if (p->h_misc[kStatus] != kDevOk) {
    cudaMemsetAsync(misc + kStatus, 0, sizeof(int32_t), s);
    return RVSP_ERROR_DEVICE;
  }
  const int64_t total = *p->h_total;
  if (total > INT32_MAX) return RVSP_ERROR_ALLOCATION_FAILED;

  finish_numeric_bins(p, a_rows, b_cols, s);
  e = cudaGetLastError();
  if (e != cudaSuccess) return map_cuda(e);

  p->learned = 0;
  p->a_rows = a_rows;
  p->b_rows = b_rows;
  p->b_cols = b_cols;
  p->c_nnz = total;
  p->analysed = 1;
  *c_nnz_out = total;
  return RVSP_SUCCESS;
}

// The symbolic pass of the rows the census found outside the merge classes
// (all rows when merge_done is false), then the scan again, and the host
// copy of the counters and the total (one more round trip).
cudaError_t symbolic_rest(rvsp_cuda_plan *p, cudaStream_t s, const Operands &op,
                          int32_t a_rows, int32_t b_rows, int32_t b_cols,
                          const int32_t *a_row_ptr, int32_t *c_row_ptr,
                          const int32_t *sym_off, bool merge_done) {
  int32_t *misc = p->misc.p;
  cudaError_t e = cudaSuccess;
  // Global bitmaps for dense symbolic rows when B is too wide for shared memory.
  const size_t bits_bytes = dense_slot_bits_bytes(b_cols);
  int32_t slots = 0;
  if (p->sym_count[kDense] > 0 && bits_bytes > 0) {
    slots = p->sym_count[kDense] < p->num_sms ? p->sym_count[kDense] : p->num_sms;
    const size_t words = bits_bytes / sizeof(uint32_t) * size_t(slots);
    if (words > p->sym_bits.cap) {
      e = p->sym_bits.reserve(words);
      if (e != cudaSuccess) return e;
      cudaMemsetAsync(p->sym_bits.p, 0, words * sizeof(uint32_t), s);
    }
    p->sym_bits_slots = slots;
  }
  {
    PhaseScope ph(p, s, RVSP_PHASE_SYMBOLIC);
    // W1024 / W2048 rows count optimistically in a small table first; their
    // retry lists live in long_rows (free once the row statistics are done),
    // W1024's from 0, W2048's after it.
    auto launch_class = [&](int c, const int32_t *rows, int32_t nrows, cudaStream_t cs) {
      if (symbolic_optimistic_class(c)) {
        const int32_t base = c == kW1024 ? 0 : p->sym_count[kW1024];
        launch_symbolic_optimistic(c, op, rows, nrows, p->counts.p, p->long_rows.p + base,
                                   misc + kRetryCount + (c == kW1024 ? 0 : 1),
                                   misc + kStatus, p->num_sms, cs);
        return 2;
      }
      launch_symbolic_class(c, op, rows, nrows, p->counts.p, p->sym_bits.p, slots,
                            misc + kStatus, p->num_sms, cs);
      return 1;
    };
    // whole >= 0 is never a merge class here when merge_done (a class
    // outside them is non-empty).
    const int whole = p->shift_active ? -1 : whole_matrix_class(p->sym_count, a_rows);
    if (whole < 0) {
      launch_class_offsets(misc + kSymCount, misc + kSymOff, s);
      launch_scatter_rows(a_rows, p->cls.p, misc + kSymOff, misc + kSymFill,
                          p->rows_sym.p, s);
      ph.launches = 2;
    }
    Lanes ln(p, s, several_classes(p->sym_count));
    for (int c = kEmpty_ + 1; c < kStripe8; ++c) {
      if (p->sym_count[c] <= 0 || (merge_done && is_merge_class(c))) continue;
      ph.launches += whole >= 0 ? launch_class(c, nullptr, a_rows, s)
                                : launch_class(c, p->rows_sym.p + sym_off[c], p->sym_count[c],
                                               ln.next());
    }
    const RowList sr = stripe_rows(p->sym_count, sym_off, whole, p->rows_sym.p);
    if (sr.n > 0) {
      if (p->stripe_policy == kStripesAlways ||
          stripes_pay(*heavy_rows(p->h_misc), b_rows, b_cols,
                      p->stripe_policy == kStripesRepeats))
        e = count_stripe_rows(p, op, b_rows, sr.rows, sr.n, s);
      if (e != cudaSuccess) return e;
      // else, or without room, they take the block kernels (either class)
      ph.launches += p->sp_ready ? 5 : launch_class(kStripe8, sr.rows, sr.n, s);
    }
  }
  if (merge_done)  // the first scan counted numeric classes already
    cudaMemsetAsync(misc + kNumCount, 0, kNumClasses * sizeof(int32_t), s);
  {
    PhaseScope ph(p, s, RVSP_PHASE_SCAN);
    const int32_t *skip = nullptr;
    if (p->shift_active) {
      launch_shift_copy_counts(p->sh_on.p, a_rows, p->st.pid.p, p->sh_rcls.p, p->counts.p, s);
      skip = p->st.pid.p;
    }
    launch_scan_and_class(a_rows, p->counts.p, p->ops.p, a_row_ptr, c_row_ptr,
                          p->partials.p,
                          p->total.p, p->cls.p, misc + kNumCount, op.merge_ok, s,
                          CheckGuard(), skip, p->sp_ready ? p->sp_hslot.p : nullptr);
    ph.launches = skip ? 4 : 3;
  }
  cudaMemcpyAsync(p->h_misc + kNumCount, misc + kNumCount,
                  (kMiscWords - kNumCount) * sizeof(int32_t), cudaMemcpyDeviceToHost, s);
  cudaMemcpyAsync(p->h_total, p->total.p, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
  return cudaStreamSynchronize(s);
}

}  // namespace

rvsp_status_t rvsp_cuda_learned_symbolic(
    rvsp_cuda_plan_t p, rvsp_mlp_t model, void *stream, int32_t a_rows, int32_t b_rows,
    int32_t b_cols, const int32_t *a_row_ptr, const int32_t *a_col_idx,
    const float *a_values, int32_t a_nnz, const int32_t *b_row_ptr,
    const int32_t *b_col_idx, const float *b_values, int32_t b_nnz,
    float capacity_scale, int32_t *c_row_ptr, int64_t *c_nnz_out) {
  if (!p || !model || !a_row_ptr || !a_col_idx || !a_values || !b_row_ptr ||
      !b_col_idx || !b_values || !c_row_ptr || !c_nnz_out)
    return RVSP_ERROR_NULL_POINTER;
  if (a_rows <= 0 || b_rows <= 0 || b_cols <= 0 || a_nnz < 0 || b_nnz < 0 ||
      !(capacity_scale > 0.0f))
    return RVSP_ERROR_INVALID_ARGUMENT;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  p->analysed = 0;
  p->learned = 0;
  p->rmap_state = 0;
  p->rmap_col = nullptr;
  p->shift_active = 0;
  p->shift_tables = 0;
  p->shift_members = 0;
  if (p->shift_enabled && shift_size_ok(p, a_rows)) {
    // Rows that are translates of a few canonical rows need no prediction:
    // their structure comes from the canonical rows.  When the probe finds
    // them common, the analysis is the shift-class one (symbolic_impl).
    if (reserve_shift(p, a_rows, b_rows) == cudaSuccess) {
      const Operands pop{a_rows, b_cols, a_row_ptr, a_col_idx, nullptr,
                         b_row_ptr, b_col_idx, nullptr, false};
      launch_shift_decide(pop, p->sh_probe.p, shift_bar(p), p->sh_on.p, CheckGuard(), s);
      cudaError_t e = cudaMemcpyAsync(p->h_misc, p->sh_on.p, sizeof(int32_t),
                                      cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) return map_cuda(e);
      if (p->h_misc[0])
        return symbolic_impl(p, s, a_rows, b_rows, b_cols, a_row_ptr, a_col_idx, b_row_ptr,
                             b_col_idx, c_row_ptr, c_nnz_out, nullptr);
    } else {
      cudaGetLastError();
    }
  }
  const size_t n = static_cast<size_t>(a_rows);
  cudaError_t e = p->ops.reserve(n);
  if (e == cudaSuccess) e = p->cls.reserve(n);
  if (e == cudaSuccess) e = p->counts.reserve(n);
  if (e == cudaSuccess) e = p->rows_sym.reserve(n);
  if (e == cudaSuccess) e = p->rows_num.reserve(n);
  if (e == cudaSuccess) e = p->cap.reserve(n);
  if (e == cudaSuccess) e = p->slab_off.reserve(n);
  if (e == cudaSuccess) e = p->ovf_rows.reserve(n);
  if (e == cudaSuccess) e = p->big_rows.reserve(n + 1);
  if (e == cudaSuccess) e = p->partials.reserve(scan_partials_bytes(a_rows) / sizeof(int64_t));
  if (e != cudaSuccess) return map_cuda(e);

  Operands op{a_rows, b_cols, a_row_ptr, a_col_idx, a_values,
              b_row_ptr, b_col_idx, b_values,
              merge_allowed(p->merge_policy, a_rows)};
  p->sp = p->stripe_policy == kStripesNever ? StripeShape() : stripe_shape(b_rows, b_cols);
  p->sp_ready = 0;
  op.stripes = p->sp.on;
  int32_t *misc = p->misc.p;
  cudaMemsetAsync(misc, 0, kMiscWords * sizeof(int32_t), s);
  // 1. Predict every row's class and capacity; slab offsets = scan of capacities.
  {
    PhaseScope ph(p, s, RVSP_PHASE_PREDICT);
    const float b_mean = static_cast<float>(b_nnz) / static_cast<float>(b_rows);
    launch_learned_plan(op, b_mean, mlp_device_params(model), capacity_scale,
                        op.merge_ok, p->ops.p, p->cls.p, p->cap.p,
                        p->counts.p, misc + kSymCount, heavy_rows(misc), b_rows,
                        p->stripe_policy == kStripesAlways,
                        p->stripe_policy == kStripesRepeats, p->num_sms, s);
    launch_scan_i64(a_rows, p->cap.p, p->slab_off.p, p->partials.p, p->total.p, s);
    ph.launches = op.stripes ? 5 : 4;
  }
  cudaMemcpyAsync(p->h_misc, misc, kNumClasses * sizeof(int32_t), cudaMemcpyDeviceToHost, s);
  cudaMemcpyAsync(p->h_total, p->total.p, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
  e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return map_cuda(e);
  int32_t pred_off[kNumClasses];
  int32_t off = 0;
  for (int c = 0; c < kNumClasses; ++c) {
    p->sym_count[c] = p->h_misc[kSymCount + c];
    pred_off[c] = off;
    if (c != kEmpty_) off += p->sym_count[c];
  }
  p->slab_total = *p->h_total;
  e = p->slab_col.reserve(size_t(p->slab_total));
  if (e == cudaSuccess) e = p->slab_val.reserve(size_t(p->slab_total));
  if (e != cudaSuccess) return map_cuda(e);
  // Dense rows of the fused pass use a plan-owned dense workspace.
  int32_t fslots = 0;
  float *facc = nullptr;
  uint32_t *fbits = nullptr;
  if (p->sym_count[kDense] > 0) {
    fslots = p->sym_count[kDense] < p->num_sms ? p->sym_count[kDense] : p->num_sms;
    const size_t acc_b = dense_slot_acc_bytes(b_cols), bits_b = dense_slot_bits_bytes(b_cols);
    const size_t need = size_t(fslots) * (acc_b + bits_b);
    e = p->fused_ws.reserve(need);
    if (e != cudaSuccess) return map_cuda(e);
    cudaMemsetAsync(p->fused_ws.p, 0, need, s);
    facc = reinterpret_cast<float *>(p->fused_ws.p);
    fbits = reinterpret_cast<uint32_t *>(p->fused_ws.p + size_t(fslots) * acc_b);
  }

  // 2. The fused pass: every row into its slab slot, or onto the overflow list.
  const FusedOut fo{p->slab_off.p, p->cap.p, p->counts.p, p->ovf_rows.p,
                    misc + kLongCount};
  {
    PhaseScope ph(p, s, RVSP_PHASE_FUSED);
    const int whole = whole_matrix_class(p->sym_count, a_rows);
    if (whole < 0) {
      launch_class_offsets(misc + kSymCount, misc + kSymOff, s);
      launch_scatter_rows(a_rows, p->cls.p, misc + kSymOff, misc + kSymFill,
                          p->rows_sym.p, s);
      ph.launches = 2;
    }
    Lanes ln(p, s, several_classes(p->sym_count));
    for (int c = kEmpty_ + 1; c < kStripe8; ++c) {
      if (p->sym_count[c] <= 0) continue;
      const bool all = c == whole;
      launch_numeric_class(c, op, p->ops.p, all ? nullptr : p->rows_sym.p + pred_off[c],
                           all ? a_rows : p->sym_count[c], nullptr, p->slab_col.p,
                           p->slab_val.p, true, facc, fbits, fslots, misc + kStatus,
                           p->num_sms, ln.next(), &fo);
      ph.launches += 1;
    }
    const RowList sr = stripe_rows(p->sym_count, pred_off, whole, p->rows_sym.p);
    if (sr.n > 0) {
      // counted here, written at C by the compute (no slab slot); without
      // room for their bitmaps, the plain two-pass path takes them
      e = count_stripe_rows(p, op, b_rows, sr.rows, sr.n, s);
      if (e != cudaSuccess) return map_cuda(e);
      if (!p->sp_ready) launch_list_overflow(sr.rows, sr.n, fo, s);
      ph.launches += p->sp_ready ? 4 : 1;
    }
  }
  // 3. Optimistic scan (valid when nothing overflowed) and the fingerprint of
  //    the values the fused pass used.
  {
    PhaseScope ph(p, s, RVSP_PHASE_SCAN);
    launch_scan_and_class(a_rows, p->counts.p, p->ops.p, a_row_ptr, c_row_ptr,
                          p->partials.p, p->total.p, p->cls.p, misc + kNumCount,
                          op.merge_ok, s, CheckGuard(), nullptr,
                          p->sp_ready ? p->sp_hslot.p : nullptr, true);
    ph.launches = 3;
  }
  values_fingerprint_launch(p, a_values, a_nnz, b_values, b_nnz, s);
  cudaMemcpyAsync(p->h_misc + kNumCount, misc + kNumCount,
                  (kMiscWords - kNumCount) * sizeof(int32_t), cudaMemcpyDeviceToHost, s);
  cudaMemcpyAsync(p->h_total, p->total.p, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
  e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return map_cuda(e);
  if (p->h_misc[kStatus] != kDevOk) {
    cudaMemsetAsync(misc + kStatus, 0, sizeof(int32_t), s);
    return RVSP_ERROR_DEVICE;
  }
  p->est_hash = p->h_vhash[0];
  p->n_ovf = p->h_misc[kLongCount];

  // 4. Overflowed rows: the plain symbolic pass, then the scan again.
  if (p->n_ovf > 0) {
    e = p->ovf_cls.reserve(size_t(p->n_ovf));
    if (e == cudaSuccess) e = p->ovf_sorted.reserve(size_t(p->n_ovf));
    if (e != cudaSuccess) return map_cuda(e);
    cudaMemsetAsync(misc + kSymCount, 0, 3 * kNumClasses * sizeof(int32_t), s);
    launch_list_classify(p->ovf_rows.p, p->n_ovf, p->ops.p, a_row_ptr, p->counts.p, b_cols,
                         false, p->ovf_cls.p, misc + kSymCount, s);
    cudaMemcpyAsync(p->h_misc, misc, kNumClasses * sizeof(int32_t), cudaMemcpyDeviceToHost, s);
    e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return map_cuda(e);
    int32_t ocount[kNumClasses], ooff[kNumClasses];
    off = 0;
    for (int c = 0; c < kNumClasses; ++c) {
      ocount[c] = p->h_misc[kSymCount + c];
      ooff[c] = off;
      if (c != kEmpty_) off += ocount[c];
    }
    int32_t slots = 0;
    e = ensure_sym_bits(p, ocount[kDense], b_cols, s, &slots);
    if (e != cudaSuccess) return map_cuda(e);
    {
      PhaseScope ph(p, s, RVSP_PHASE_SYMBOLIC);
      launch_class_offsets(misc + kSymCount, misc + kSymOff, s);
      launch_scatter_list(p->ovf_rows.p, p->n_ovf, p->ovf_cls.p, misc + kSymOff,
                          misc + kSymFill, p->rows_sym.p, s);
      ph.launches = 3;
      for (int c = kEmpty_ + 1; c < kNumClasses; ++c) {
        if (ocount[c] <= 0) continue;
        launch_symbolic_class(c, op, p->rows_sym.p + ooff[c], ocount[c], p->counts.p,
                              p->sym_bits.p, slots, misc + kStatus, p->num_sms, s);
        ph.launches += 1;
      }
    }
    {
      PhaseScope ph(p, s, RVSP_PHASE_SCAN);
      cudaMemsetAsync(misc + kNumCount, 0, kNumClasses * sizeof(int32_t), s);
      launch_scan_and_class(a_rows, p->counts.p, p->ops.p, a_row_ptr, c_row_ptr,
                            p->partials.p, p->total.p, p->cls.p, misc + kNumCount,
                            op.merge_ok, s, CheckGuard(), nullptr,
                            p->sp_ready ? p->sp_hslot.p : nullptr, true);
      // The overflow rows by numeric class, for the first compute.
      cudaMemsetAsync(misc + kSymCount, 0, 3 * kNumClasses * sizeof(int32_t), s);
      launch_list_classify(p->ovf_rows.p, p->n_ovf, p->ops.p, a_row_ptr, p->counts.p,
                           b_cols, true, p->ovf_cls.p, misc + kSymCount, s);
      launch_class_offsets(misc + kSymCount, misc + kSymOff, s);
      launch_scatter_list(p->ovf_rows.p, p->n_ovf, p->ovf_cls.p, misc + kSymOff,
                          misc + kSymFill, p->ovf_sorted.p, s);
      ph.launches = 6;
    }
    cudaMemcpyAsync(p->h_misc, misc, kMiscWords * sizeof(int32_t), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(p->h_total, p->total.p, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
    e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return map_cuda(e);
    if (p->h_misc[kStatus] != kDevOk) {
      cudaMemsetAsync(misc + kStatus, 0, sizeof(int32_t), s);
      return RVSP_ERROR_DEVICE;
    }
    off = 0;
    for (int c = 0; c < kNumClasses; ++c) {
      p->ovf_num_count[c] = p->h_misc[kSymCount + c];
      p->ovf_num_off[c] = off;
      if (c != kEmpty_) off += p->ovf_num_count[c];
    }
  }
  const int64_t total = *p->h_total;
  if (total > INT32_MAX) return RVSP_ERROR_ALLOCATION_FAILED;
  finish_numeric_bins(p, a_rows, b_cols, s);
  e = cudaGetLastError();
  if (e != cudaSuccess) return map_cuda(e);
  p->learned = 1;
  p->a_nnz = a_nnz;
  p->b_nnz = b_nnz;
  p->a_rows = a_rows;
  p->b_rows = b_rows;
  p->b_cols = b_cols;
  p->c_nnz = total;
  p->analysed = 1;
  *c_nnz_out = total;
  return RVSP_SUCCESS;
}

rvsp_status_t rvsp_cuda_plan_set_merge_policy(rvsp_cuda_plan_t p, int32_t policy) {
  if (!p) return RVSP_ERROR_NULL_POINTER;
  if (policy < kMergeAuto || policy > kMergeAlways) return RVSP_ERROR_INVALID_ARGUMENT;
  p->merge_policy = policy;
  return RVSP_SUCCESS;
}

rvsp_status_t rvsp_cuda_plan_set_stripes(rvsp_cuda_plan_t p, int32_t policy) {
  if (!p) return RVSP_ERROR_NULL_POINTER;
  if (policy < kStripesAuto || policy > kStripesRepeats) return RVSP_ERROR_INVALID_ARGUMENT;
  p->stripe_policy = policy;
  return RVSP_SUCCESS;
}

rvsp_status_t rvsp_cuda_plan_set_stripe_memory(rvsp_cuda_plan_t p, size_t bytes) {
  if (!p) return RVSP_ERROR_NULL_POINTER;
  p->stripe_max = bytes;
  return RVSP_SUCCESS;
}

rvsp_status_t rvsp_cuda_plan_set_row_tiles(rvsp_cuda_plan_t p, int32_t enable) {
  if (!p) return RVSP_ERROR_NULL_POINTER;
  if (enable != 0 && enable != 1) return RVSP_ERROR_INVALID_ARGUMENT;
  if (enable && !p->tiles_enabled) {
    // tiles were never built for the current reuse map: build it again
    p->rmap_state = 0;
    p->rmap_col = nullptr;
  }
  p->tiles_enabled = enable;
  return RVSP_SUCCESS;
}

rvsp_status_t rvsp_cuda_plan_set_persistent(rvsp_cuda_plan_t p, int32_t merge_rows,
                                           int32_t blocks_per_sm) {
  if (!p) return RVSP_ERROR_NULL_POINTER;
  if (merge_rows < 0 || merge_rows > kPersistThreads || merge_rows % 32 != 0 ||
      blocks_per_sm < 1 || blocks_per_sm > 4)
    return RVSP_ERROR_INVALID_ARGUMENT;
  p->persist_merge_rows = merge_rows;
  p->persist_blocks = blocks_per_sm;
  return RVSP_SUCCESS;
}

rvsp_status_t rvsp_cuda_plan_set_pattern_kernels(rvsp_cuda_plan_t p, int32_t enable) {
  if (!p) return RVSP_ERROR_NULL_POINTER;
  if (enable != 0 && enable != 1) return RVSP_ERROR_INVALID_ARGUMENT;
  if (enable != p->pattern_kernels) {
    // the tiles are built with or without pattern kernels: rebuild them
    p->rmap_state = 0;
    p->rmap_col = nullptr;
    if (p->shift_tables == 1) p->shift_tables = 0;
  }
  p->pattern_kernels = enable;
  return RVSP_SUCCESS;
}

int32_t rvsp_cuda_plan_pattern_kernel_rows(rvsp_cuda_plan_t p) {
  if (!p || !p->tiles_enabled) return 0;
  int32_t n = 0;
  if (p->rmap_state == 1 && p->pat_ready && p->rt.ready)
    for (const auto &j : p->rt.jit) n += 32 * j.n;
  if (p->shift_active && p->shift_tables == 1 && p->st.ready)
    for (const auto &j : p->st.jit) n += 32 * j.n;
  return n;
}

void rvsp_cuda_pattern_kernel_stats(int32_t *compiles, double *compile_ms) {
  jit_stats(compiles, compile_ms);
}

rvsp_status_t rvsp_cuda_plan_set_shift_classes(rvsp_cuda_plan_t p, int32_t enable) {
  if (!p) return RVSP_ERROR_NULL_POINTER;
  if (enable < 0 || enable > 2) return RVSP_ERROR_INVALID_ARGUMENT;
  p->shift_enabled = enable;
  return RVSP_SUCCESS;
}

int32_t rvsp_cuda_plan_shift_rows(rvsp_cuda_plan_t p) {
  return (p && p->analysed && p->shift_active) ? p->shift_members : 0;
}

int32_t rvsp_cuda_plan_tiled_rows(rvsp_cuda_plan_t p) {
  if (!p || !p->tiles_enabled) return 0;
  int32_t n = 0;
  if (p->rmap_state == 1 && p->pat_ready && p->rt.ready) n += p->n_pat_rows - p->rt.n_lo;
  if (p->shift_active && p->shift_tables == 1 && p->st.ready)
    n += p->shift_members - p->st.n_lo;
  return n;
}

int32_t rvsp_cuda_plan_overflow_rows(rvsp_cuda_plan_t p) {
  return (p && p->analysed && p->learned) ? p->n_ovf : 0;
}

size_t rvsp_cuda_numeric_workspace_bytes(rvsp_cuda_plan_t p) {
  return (p && p->analysed) ? p->numeric_ws : 0;
}

namespace {

// The reuse map may take at most this much device memory (and a quarter of
// what is free).
constexpr size_t kReuseMapMaxBytes = size_t(24) << 30;

// The tile tables may take at most this much device memory.
constexpr size_t kTileTablesMaxBytes = size_t(256) << 20;
// Patterns with at least this many tiles (of 32 rows) get a compiled kernel,
// the kJitMaxPatterns largest of them, when their rows have at most
// kJitMaxOut outputs (one register each).
constexpr int32_t kJitMinTiles = 128;
constexpr int32_t kJitMaxOut = 160;
// Largest B range (floats) one stage buffer of a pattern kernel takes.
constexpr int32_t kJitMaxSpan = 4096;

constexpr int kTileCountWords = 8;  // tiles, leftovers, 3 maxima, b_nnz, table tiles, all rows
constexpr int kCountBnnz = 5, kCountTable = 6, kCountAll = 7;
constexpr size_t kSpanWords = size_t(32) * kJitMaxGroup;  // a pattern's union spans
// Patterns whose spans and tables are read back with the counts, before it is
// known which of them get a kernel (1 MB at most).
constexpr int32_t kReadAllPatterns = 256;

// Compiled kernels for the patterns that cover the most tiles, from what the
// tile builder measured (on the host): the staging groups are chosen from the
// union spans, the kernels compiled side by side (k_jit.cu; a structure seen
// before finds them compiled) and the tile records of all of them queued as
// one launch.  A pattern whose compile fails stays on the table kernel.  The
// device arrays of earlier builds are kept and reused.
void build_pattern_kernels(rvsp_cuda_plan *p, cudaStream_t s, const Operands &op, bool shifted,
                           const std::vector<int32_t> &order, const int32_t *pcount,
                           const int32_t *pseg, const int4 *desc, const uint16_t *lens,
                           const std::vector<const int32_t *> &spans,
                           const std::vector<const uint16_t *> &tabs, TileBuild &tb) {
  const size_t K = order.size();
  std::vector<JitRequest> reqs(K);
  std::vector<int32_t> need(K, 0);
  for (size_t k = 0; k < K; ++k) {
    const int4 d = desc[size_t(order[k])];
    if (d.x <= 0 || d.x > 32 || d.y <= 0 || d.y > kJitMaxOut) continue;
    JitRequest rq;
    rq.na = d.x;
    rq.m = d.y;
    int32_t off = 0;
    rq.slot.reserve(size_t(d.z));
    for (int j = 0; j < d.x; ++j) {
      rq.len[j] = lens[size_t(order[k]) * 32 + j];
      for (int e = 0; e < rq.len[j]; ++e) rq.slot.push_back(tabs[k][off + e] & 0x7fff);
      off += (rq.len[j] + 7) & ~7;
    }
    rq.groups = jit_groups(d.x, rq.len, spans[k], kJitMaxSpan, &need[k]);
    // (offsets into a group's B range are 16 bits)
    if (!rq.groups.empty() && need[k] > 0 && need[k] <= kJitMaxSpan) reqs[k] = std::move(rq);
  }
  jit_pattern_kernels(reqs);
  int dev_max = 0;
  cudaDeviceGetAttribute(&dev_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, p->device);
  TilePrograms P;
  for (size_t k = 0; k < K; ++k) {
    const JitRequest &rq = reqs[k];
    if (!rq.kernel) continue;
    const int32_t n = pcount[order[k]], rw = jit_record_words(rq.na, int(rq.groups.size()));
    // the arrays of an earlier build: the smallest whose tile capacity holds
    // this pattern's tiles, else the largest (so that a repeated analysis of
    // the same structure allocates nothing)
    JitPattern jp;
    if (!tb.pool.empty()) {
      size_t best = 0;
      for (size_t q = 1; q < tb.pool.size(); ++q) {
        const size_t c = tb.pool[q].arange.cap, bc = tb.pool[best].arange.cap;
        const bool f = c >= size_t(n), bf = bc >= size_t(n);
        if ((f && (!bf || c < bc)) || (!f && !bf && c > bc)) best = q;
      }
      jp = tb.pool[best];
      tb.pool.erase(tb.pool.begin() + static_cast<std::ptrdiff_t>(best));
    }
    jp.n = n;
    jp.m = rq.m;
    jit_layout(rw, pseg[order[k]], need[k], jp.m, &jp.stage_cap, &jp.abuf_floats,
               &jp.work_floats);
    // two warps must fit one block's shared memory
    if (n <= 0 || size_t(2) * size_t(jp.work_floats) * sizeof(float) > size_t(dev_max) ||
        jp.prog.reserve(size_t(n) * size_t(rw)) != cudaSuccess ||
        jp.arange.reserve(size_t(n)) != cudaSuccess || jp.head.reserve(1) != cudaSuccess) {
      cudaGetLastError();
      tb.pool.push_back(jp);
      continue;
    }
    jp.kernel = rq.kernel;
    jp.grid = jit_grid(jp.kernel, n, jp.work_floats, jp.m, p->num_sms);
    TileProgram &q = P.p[P.n++];
    q.prog = jp.prog.p;
    q.arange = jp.arange.p;
    q.pid = order[k];
    q.na = rq.na;
    q.ng = static_cast<int32_t>(rq.groups.size());
    q.rw = rw;
    std::fill(q.group, q.group + 32, kNoGroup);
    for (size_t g = 0; g < rq.groups.size(); ++g)
      std::fill(q.group + rq.groups[g].first, q.group + rq.groups[g].second,
                static_cast<uint8_t>(g));
    tb.jit.push_back(jp);
  }
  launch_tile_records(tb.tiles.p, static_cast<int32_t>((int64_t(p->a_rows) + 31) / 32), shifted, P,
                      tb.rank.p, tb.lens.p, tb.offs.p, op.a_rp, op.a_col, op.b_rp, tb.desc.p, s);
}

// Row tiles of a set of table patterns (k_tile.cu): the per-pattern tile
// tables (from each pattern's canonical row map: moff[row], map), then tiles
// over chunks of 32 consecutive rows of tb.pid (the pattern of each row, -1
// elsewhere, filled by the caller) and the leftover list; one read-back of
// what the builder counted, from which the compiled patterns are chosen and
// everything else is queued.  Leaves tb.ready 0 (every pattern row on the
// warp-per-row kernel) when nothing is tiled.  With `shifted` (the shift
// classes: each pattern's rows are its canonical row moved, and they have no
// other path) a failed allocation is an error.  Synchronizes `s`.
cudaError_t build_row_tiles(rvsp_cuda_plan *p, cudaStream_t s, const Operands &op,
                            const int32_t *c_rp, int32_t npat, const int32_t *pat_canon,
                            const int32_t *psteps, const int64_t *moff, const uint16_t *map,
                            TileBuild &tb, bool shifted = false) {
  tb.ready = 0;
  tb.n_lo = 0;
  tb.n_tiles = 0;
  tb.n_table = 0;
  for (auto &j : tb.jit) tb.pool.push_back(j);
  tb.jit.clear();
  const size_t n = static_cast<size_t>(p->a_rows), np = static_cast<size_t>(npat);
  const size_t stride = size_t(tile_tab_stride()), nchunks = (n + 31) / 32;
  // counts | tiles per pattern | A segment per pattern | spans per pattern
  const size_t words = kTileCountWords + np * (2 + kSpanWords);
  if (tb.tab.reserve(np * stride) != cudaSuccess || tb.lens.reserve(np * 32) != cudaSuccess ||
      tb.offs.reserve(np * 32) != cudaSuccess || tb.desc.reserve(np) != cudaSuccess ||
      tb.tiles.reserve(nchunks) != cudaSuccess || tb.table.reserve(nchunks) != cudaSuccess ||
      tb.rank.reserve(tile_rank_words(static_cast<int32_t>(nchunks))) != cudaSuccess ||
      tb.lo_rows.reserve(n) != cudaSuccess || tb.lo_ids.reserve(n) != cudaSuccess ||
      tb.counts.reserve(words) != cudaSuccess ||
      (shifted && (tb.all_rows.reserve(n) != cudaSuccess ||
                   tb.all_ids.reserve(n) != cudaSuccess))) {
    const cudaError_t err = cudaGetLastError();
    return shifted ? err : cudaSuccess;
  }
  // the read-back: the words above (spans only of few patterns), then desc,
  // lens and, of few patterns, the tables (16-byte aligned pieces)
  const bool all = npat <= kReadAllPatterns;
  auto up16 = [](size_t x) { return (x + 15) & ~size_t(15); };
  const size_t word_bytes = (all ? words : kTileCountWords + 2 * np) * sizeof(int32_t);
  const size_t o_desc = up16(word_bytes), o_lens = o_desc + up16(np * sizeof(int4));
  const size_t o_tabs = o_lens + up16(np * 32 * sizeof(uint16_t));
  const size_t tab_bytes = stride * sizeof(uint16_t);
  const size_t o_spans = o_tabs + up16((all ? np : size_t(kJitMaxPatterns)) * tab_bytes);
  const size_t total = o_spans + (all ? 0 : kJitMaxPatterns * kSpanWords * sizeof(int32_t));
  cudaError_t e = tb.staging.reserve(total);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return shifted ? e : cudaSuccess;
  }
  int32_t *const d_count = tb.counts.p + kTileCountWords, *const d_seg = d_count + np;
  int32_t *const d_spans = d_seg + np;
  cudaMemsetAsync(tb.counts.p, 0, words * sizeof(int32_t), s);
  if (shifted)
    launch_tile_list(p->a_rows, tb.pid.p, tb.all_rows.p, tb.all_ids.p, tb.counts.p + kCountAll,
                     s);
  launch_tile_tab(npat, pat_canon, psteps, op.a_rp, op.a_col, op.b_rp, c_rp, moff, map, p->b_rows,
                  tb.tab.p, tb.lens.p, tb.offs.p, tb.desc.p, tb.counts.p + kCountBnnz, s);
  launch_tile_build(p->a_rows, shifted, tb.pid.p, tb.desc.p, tb.lens.p, tb.offs.p, op.a_rp,
                    op.a_col, op.b_rp, c_rp, tb.tiles.p, d_count, d_seg, d_spans, tb.lo_rows.p,
                    tb.lo_ids.p, tb.counts.p, p->num_sms, s);
  char *const h = tb.staging.p;
  e = cudaMemcpyAsync(h, tb.counts.p, word_bytes, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(h + o_desc, tb.desc.p, np * sizeof(int4), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(h + o_lens, tb.lens.p, np * 32 * sizeof(uint16_t),
                        cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess && all && p->pattern_kernels)
    e = cudaMemcpyAsync(h + o_tabs, tb.tab.p, np * tab_bytes, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return e;
  const int32_t *const hc = reinterpret_cast<const int32_t *>(h);
  const int32_t *const pcount = hc + kTileCountWords;
  const int4 *const desc = reinterpret_cast<const int4 *>(h + o_desc);
  const uint16_t *const lens = reinterpret_cast<const uint16_t *>(h + o_lens);
  tb.n_lo = hc[1];
  if (hc[0] <= 0) return cudaSuccess;
  int32_t acc_rows = 0, work = 0, stage_cap = 0;
  const size_t per_warp = tile_smem_per_warp(hc[2], hc[3], hc[4], &acc_rows, &work, &stage_cap);
  int dev_max = 0;
  cudaDeviceGetAttribute(&dev_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, p->device);
  // (cannot happen: the tile limits keep one block under 140 KB)
  if (per_warp * kTileKernelWarps > size_t(dev_max))
    return shifted ? cudaErrorInvalidValue : cudaSuccess;
  tb.n_tiles = hc[0];
  tb.stage = hc[2];
  tb.aseg = hc[3];
  tb.max_out = hc[4];
  tb.b_nnz = hc[kCountBnnz];
  tb.ready = 1;
  tb.n_table = tb.n_tiles;
  if (p->pattern_kernels) {
    std::vector<int32_t> order;
    for (int32_t id = 0; id < npat; ++id)
      if (pcount[id] >= kJitMinTiles) order.push_back(id);
    std::sort(order.begin(), order.end(),
              [&](int32_t a, int32_t b) { return pcount[a] > pcount[b]; });
    if (order.size() > size_t(kJitMaxPatterns)) order.resize(size_t(kJitMaxPatterns));
    std::vector<const int32_t *> spans;
    std::vector<const uint16_t *> tabs;
    for (size_t k = 0; k < order.size(); ++k) {
      const size_t id = size_t(order[k]);
      if (all) {
        spans.push_back(pcount + 2 * np + id * kSpanWords);
        tabs.push_back(reinterpret_cast<const uint16_t *>(h + o_tabs) + id * stride);
        continue;
      }
      char *const ht = h + o_tabs + k * tab_bytes;
      char *const hs = h + o_spans + k * kSpanWords * sizeof(int32_t);
      tabs.push_back(reinterpret_cast<const uint16_t *>(ht));
      spans.push_back(reinterpret_cast<const int32_t *>(hs));
      e = cudaMemcpyAsync(ht, tb.tab.p + id * stride, tab_bytes, cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(hs, d_spans + id * kSpanWords, kSpanWords * sizeof(int32_t),
                            cudaMemcpyDeviceToHost, s);
      if (e != cudaSuccess) return e;
    }
    if (!all && !order.empty()) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return e;
    build_pattern_kernels(p, s, op, shifted, order, pcount, pcount + np, desc, lens, spans, tabs,
                          tb);
    for (const auto &j : tb.jit) tb.n_table -= j.n;
  }
  if (tb.n_table > 0)
    launch_table_tiles(tb.tiles.p, static_cast<int32_t>(nchunks), tb.desc.p, tb.table.p,
                       tb.counts.p + kCountTable, s);
  return cudaGetLastError();
}

// Builds the reuse map of the W<T> rows for the structure in c_col (written
// by an earlier fill).  Leaves rmap_state -1 when the map does not apply:
// no W rows, a row of more than INT32_MAX / 2 products, or over the memory
// budget.  Synchronizes s.
// Term tables for the maps that many rows share (k_pattern.cu), and the
// split of the W rows into table rows and map rows.  Leaves pat_ready 0 (all
// W rows on the map) when no map is shared widely enough or the tables would
// take more than an eighth of the map's bytes.  Synchronizes `s`.
cudaError_t build_term_tables(rvsp_cuda_plan *p, cudaStream_t s, const Operands &op,
                              const int32_t *c_rp, int64_t map_entries) {
  const size_t n = static_cast<size_t>(p->a_rows);
  cudaError_t e = p->pat_of.reserve(n);
  if (e == cudaSuccess) e = p->pat_canon.reserve(n);
  if (e == cudaSuccess) e = p->pat_cap.reserve(n);
  if (e == cudaSuccess) e = p->pat_counts.reserve(kPatCountWords);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return cudaSuccess;
  }
  cudaMemsetAsync(p->pat_of.p, 0xff, n * sizeof(int32_t), s);
  cudaMemsetAsync(p->pat_counts.p, 0, kPatCountWords * sizeof(int32_t), s);
  for (int c = kEmpty_ + 1; c < kNumClasses; ++c) {
    if (!map_class(c) || p->num_count[c] <= 0) continue;
    const bool whole = c == p->num_whole;
    launch_pat_select(whole ? nullptr : p->rows_num.p + p->num_off[c],
                      whole ? p->a_rows : p->num_count[c], p->rmap_canon.p,
                      p->rmap_share_count.p, kPatMinShare, op.a_rp, c_rp, p->rmap_ops.p,
                      p->pat_of.p, p->pat_canon.p, p->pat_cap.p, p->pat_counts.p,
                      p->pat_counts.p + 2 + kNumClasses, s);
  }
  int32_t npat = 0;
  e = cudaMemcpyAsync(&npat, p->pat_counts.p, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return e;
  if (npat <= 0) return cudaSuccess;
  e = p->pat_off.reserve(size_t(npat));
  if (e == cudaSuccess) e = p->pat_steps.reserve(size_t(npat));
  if (e != cudaSuccess) {
    cudaGetLastError();
    return cudaSuccess;
  }
  launch_scan_i64(npat, p->pat_cap.p, p->pat_off.p, p->partials.p, p->total.p, s);
  int64_t records = 0;
  e = cudaMemcpyAsync(&records, p->total.p, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return e;
  const int64_t budget = map_entries * int64_t(sizeof(uint16_t)) / 8;
  if (records <= 0 || records * int64_t(sizeof(uint32_t)) > budget) return cudaSuccess;
  if (p->pat_rec.reserve(size_t(records)) != cudaSuccess ||
      p->pat_rows.reserve(n) != cudaSuccess || p->pat_ids.reserve(n) != cudaSuccess ||
      p->res_rows.reserve(n) != cudaSuccess) {
    cudaGetLastError();
    return cudaSuccess;
  }
  launch_pat_build(npat, p->pat_canon.p, op.a_rp, op.a_col, op.b_rp, c_rp, p->rmap_off.p,
                   p->rmap.p, p->pat_off.p, p->pat_cap.p, p->pat_rec.p, p->pat_steps.p, s);
  // per-row pattern ids for the row tiles (skipped when they do not fit)
  const size_t tab_entries = size_t(npat) * size_t(tile_tab_stride());
  const bool tiles_fit = p->tiles_enabled &&
                         tab_entries * sizeof(uint16_t) <= kTileTablesMaxBytes &&
                         p->rt.pid.reserve(n) == cudaSuccess;
  if (!tiles_fit) cudaGetLastError();
  if (tiles_fit) cudaMemsetAsync(p->rt.pid.p, 0xff, n * sizeof(int32_t), s);
  int32_t off = 0;
  for (int c = kEmpty_ + 1; c < kNumClasses; ++c) {
    p->res_off[c] = off;
    if (!map_class(c) || p->num_count[c] <= 0) continue;
    const bool whole = c == p->num_whole;
    launch_pat_split(whole ? nullptr : p->rows_num.p + p->num_off[c],
                     whole ? p->a_rows : p->num_count[c], p->rmap_canon.p, p->pat_of.p,
                     p->pat_steps.p, op.a_rp, op.a_col, op.b_rp, p->pat_rows.p,
                     p->pat_ids.p, p->pat_counts.p + 1, p->res_rows.p + off,
                     p->pat_counts.p + 2 + c, tiles_fit ? p->rt.pid.p : nullptr, s);
    off += whole ? p->a_rows : p->num_count[c];
  }
  int32_t h[kPatCountWords] = {};
  e = cudaMemcpyAsync(h, p->pat_counts.p, sizeof(h), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return e;
  p->n_pat = npat;
  p->n_pat_rows = h[1];
  for (int c = 0; c < kNumClasses; ++c) p->res_count[c] = h[2 + c];
  p->pat_max_ops = h[2 + kNumClasses];
  p->pat_max_out = h[3 + kNumClasses];
  p->pat_ready = 1;
  p->rt.ready = 0;
  if (tiles_fit && p->n_pat_rows > 0) {
    e = build_row_tiles(p, s, op, c_rp, npat, p->pat_canon.p, p->pat_steps.p, p->rmap_off.p,
                        p->rmap.p, p->rt);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// Term tables and row tiles of the shift-class patterns, from the canonical
// rows' structure in C (c_rp, c_col): their maps (binary search in C's row),
// the warp-per-row tables (k_pattern.cu) and the row tiles of the member
// rows (k_tile.cu).  Every member row is then in a tile or on the leftover
// list.  Synchronizes `s`.
cudaError_t build_shift_tables(rvsp_cuda_plan *p, cudaStream_t s, const Operands &op,
                               const int32_t *c_rp, const int32_t *c_col) {
  p->shift_tables = -1;
  const int32_t npat = p->shift_npat;
  if (npat <= 0) return cudaErrorInvalidValue;
  const size_t n = static_cast<size_t>(p->a_rows);
  cudaError_t e = p->sh_moff.reserve(n);
  if (e == cudaSuccess) e = p->sh_map.reserve(size_t(npat) * size_t(shift_max_ops()));
  if (e == cudaSuccess) e = p->sh_pat_off.reserve(size_t(npat));
  if (e == cudaSuccess) e = p->sh_steps.reserve(size_t(npat));
  if (e == cudaSuccess) e = p->sh_counts.reserve(4);
  if (e != cudaSuccess) return e;
  launch_shift_canon_map(npat, p->sh_pat_canon.p, op, c_rp, c_col, p->sh_moff.p, p->sh_map.p,
                         s);
  launch_scan_i64(npat, p->sh_pat_cap.p, p->sh_pat_off.p, p->partials.p, p->total.p, s);
  cudaMemsetAsync(p->sh_counts.p, 0, 4 * sizeof(int32_t), s);
  launch_pat_maxima(npat, p->sh_pat_canon.p, p->sh_pat_m.p, p->ops.p, p->sh_counts.p, s);
  // The tables' records: few patterns take the most they can need, so that the
  // host need not ask (12 KB a pattern); many take the scan's total.
  int64_t records = int64_t(npat) * pat_max_records();
  int32_t *const maxima = p->h_misc;  // (read with the tile builder's counts)
  e = cudaMemcpyAsync(maxima, p->sh_counts.p, 4 * sizeof(int32_t), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess && npat > 4096) {
    e = cudaMemcpyAsync(p->h_total, p->total.p, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    records = *p->h_total;
  }
  if (e != cudaSuccess) return e;
  e = p->sh_rec.reserve(size_t(records > 0 ? records : 1));
  if (e != cudaSuccess) return e;
  launch_pat_build(npat, p->sh_pat_canon.p, op.a_rp, op.a_col, op.b_rp, c_rp, p->sh_moff.p,
                   p->sh_map.p, p->sh_pat_off.p, p->sh_pat_cap.p, p->sh_rec.p, p->sh_steps.p,
                   s);
  e = build_row_tiles(p, s, op, c_rp, npat, p->sh_pat_canon.p, p->sh_steps.p, p->sh_moff.p,
                      p->sh_map.p, p->st, true);
  if (e != cudaSuccess) return e;
  p->sh_max_ops = maxima[0];
  p->sh_max_out = maxima[1];
  p->shift_tables = 1;
  return cudaSuccess;
}

// The table kernel over the tiles of the patterns without a compiled kernel;
// returns the launches.
int launch_table_tile_kernel(const TileBuild &tb, const Operands &op, const int32_t *c_rp,
                             float *c_val, cudaStream_t s) {
  if (tb.n_table <= 0) return 0;
  launch_tile_numeric(op, tb.b_nnz, tb.table.p, tb.n_table, tb.desc.p, tb.lens.p, tb.tab.p, c_rp,
                      c_val, tb.stage, tb.aseg, tb.max_out, s);
  return 1;
}

// Pattern kernels of a tile set (k_jit.cu); returns the launches.  The
// first (the pattern with the most tiles, persistent over every SM) goes to
// the caller's stream, the others to the side streams in turn.  The caller
// launches the others (main = false) with its other small launches before
// the first (main = true), so that they reach the SMs before the persistent
// kernel fills them.
int launch_pattern_kernels(const TileBuild &tb, const Operands &op, const int32_t *c_rp,
                           float *c_val, int32_t *status, Lanes &ln, bool main) {
  int launches = 0;
  for (size_t i = main ? 0 : 1; i < (main ? std::min<size_t>(1, tb.jit.size()) : tb.jit.size());
       ++i) {
    const auto &j = tb.jit[i];
    launch_pattern_kernel(j.kernel, op, j.prog.p, j.arange.p, j.n, c_rp, c_val, j.stage_cap,
                          j.abuf_floats, j.work_floats, j.grid, j.head.p, status,
                          i == 0 ? ln.main() : ln.next());
    ++launches;
  }
  return launches;
}

// Values of the shift-class member rows (tables built): row tiles, then the
// members no tile took through the warp-per-row table kernel; every member
// through that kernel when tiles are off.
int launch_shift_numeric(rvsp_cuda_plan *p, Lanes &ln, const Operands &op,
                         const int32_t *c_rp, float *c_val) {
  int launches = 0;
  if (p->st.ready && p->tiles_enabled) {
    launches += launch_table_tile_kernel(p->st, op, c_rp, c_val, ln.next());
    if (p->st.n_lo > 0) {
      launch_pat_numeric(op, p->ops.p, p->st.lo_rows.p, p->st.lo_ids.p, p->st.n_lo, c_rp,
                         c_val, p->sh_pat_off.p, p->sh_steps.p, p->sh_rec.p, p->sh_max_ops,
                         p->sh_max_out, ln.next());
      ++launches;
    }
    launches += launch_pattern_kernels(p->st, op, c_rp, c_val, p->misc.p + kStatus, ln, false);
    launches += launch_pattern_kernels(p->st, op, c_rp, c_val, p->misc.p + kStatus, ln, true);
  } else {
    launch_pat_numeric(op, p->ops.p, p->st.all_rows.p, p->st.all_ids.p, p->shift_members,
                       c_rp, c_val, p->sh_pat_off.p, p->sh_steps.p, p->sh_rec.p,
                       p->sh_max_ops, p->sh_max_out, ln.main());
    ++launches;
  }
  return launches;
}

// The numeric STRIPE rows: columns first when they are to be filled, then
// the values; returns the launches.
int launch_stripe_rows(rvsp_cuda_plan *p, const Operands &op, const int32_t *c_rp,
                       int32_t *c_col, float *c_val, bool fill, cudaStream_t s) {
  const RowList sr = stripe_rows(p->num_count, p->num_off, p->num_whole, p->rows_num.p);
  if (!p->sp_ready || sr.n <= 0) return 0;
  int32_t *status = p->misc.p + kStatus;
  if (fill)
    launch_stripe_columns(p->sp, sr.rows, sr.n, p->sp_hslot.p, p->sp_bits.p, p->sp_gpre.p,
                          p->sp_soff.p, c_rp, c_col, status, s);
  launch_stripe_values(p->sp, op, sr.n, p->sp_items.p, p->sp_cap, p->sp_cnt.p,
                       p->sp_cnt.p + 2, p->sp_bound.p, p->sp_share.p, p->sp_ptr.p,
                       p->sp_hslot.p, p->sp_bits.p, p->sp_gpre.p, p->counts.p, c_rp, c_col,
                       c_val, !fill, status, p->num_sms, s);
  return fill ? 2 : 1;
}

cudaError_t build_reuse_map(rvsp_cuda_plan *p, cudaStream_t s, const Operands &op,
                            const int32_t *c_rp, const int32_t *c_col) {
  p->rmap_state = -1;
  p->rmap_col = nullptr;
  bool any = false;
  for (int c = kEmpty_ + 1; c < kNumClasses; ++c)
    any = any || (map_class(c) && p->num_count[c] > 0);
  if (!any) return cudaSuccess;
  const size_t n = static_cast<size_t>(p->a_rows);
  cudaError_t e = p->rmap_ops.reserve(n + 1);
  if (e == cudaSuccess) e = p->rmap_off.reserve(n);
  if (e != cudaSuccess) return e;
  cudaMemsetAsync(p->rmap_ops.p, 0, (n + 1) * sizeof(int32_t), s);
  for (int c = kEmpty_ + 1; c < kNumClasses; ++c) {
    if (!map_class(c) || p->num_count[c] <= 0) continue;
    const bool whole = c == p->num_whole;
    launch_map_ops(whole ? nullptr : p->rows_num.p + p->num_off[c],
                   whole ? p->a_rows : p->num_count[c], p->ops.p, p->rmap_ops.p,
                   p->rmap_ops.p + n, s);
  }
  launch_scan_i64(p->a_rows, p->rmap_ops.p, p->rmap_off.p, p->partials.p, p->total.p, s);
  int32_t too_long = 0;
  int64_t entries = 0;
  e = cudaMemcpyAsync(&entries, p->total.p, sizeof(int64_t), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(&too_long, p->rmap_ops.p + n, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return e;
  const size_t bytes = static_cast<size_t>(entries) * sizeof(uint16_t);
  if (too_long || entries <= 0 || bytes > kReuseMapMaxBytes) return cudaSuccess;
  // the free-memory bound only matters when the map must grow (a repeated
  // analysis of the same structure reuses its allocation without asking
  // the driver)
  if (static_cast<size_t>(entries) > p->rmap.cap) {
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) return cudaGetLastError();
    if (bytes > free_b / 4) return cudaSuccess;
  }
  if (p->rmap.reserve(static_cast<size_t>(entries)) != cudaSuccess) {
    cudaGetLastError();  // out of memory: keep the hash path
    return cudaSuccess;
  }
  // Fingerprints for sharing identical maps (skipped when the table does not
  // fit: every row then keeps its own map).
  int64_t map_rows = 0;
  for (int c = kEmpty_ + 1; c < kNumClasses; ++c)
    if (map_class(c) && p->num_count[c] > 0) map_rows += p->num_count[c];
  size_t tcap = 64;
  while (tcap < size_t(2 * map_rows)) tcap <<= 1;
  bool dedup = p->rmap_key.reserve(n) == cudaSuccess &&
               p->rmap_tkey.reserve(tcap) == cudaSuccess &&
               p->rmap_trow.reserve(tcap) == cudaSuccess &&
               p->rmap_shared.reserve(1) == cudaSuccess &&
               p->rmap_canon.reserve(n) == cudaSuccess &&
               p->rmap_share_count.reserve(n) == cudaSuccess;
  if (!dedup) {
    cudaGetLastError();
    if (p->rmap_shared.p) cudaMemsetAsync(p->rmap_shared.p, 0, sizeof(int32_t), s);
  }
  for (int c = kEmpty_ + 1; c < kNumClasses; ++c) {
    if (!map_class(c) || p->num_count[c] <= 0) continue;
    const bool whole = c == p->num_whole;
    launch_map_build(c, op, whole ? nullptr : p->rows_num.p + p->num_off[c],
                     whole ? p->a_rows : p->num_count[c], c_rp, c_col, p->rmap_off.p,
                     p->rmap.p, dedup ? p->rmap_key.p : nullptr, p->misc.p + kStatus, s);
  }
  if (dedup) {
    const unsigned long long mask = tcap - 1;
    cudaMemsetAsync(p->rmap_tkey.p, 0, tcap * sizeof(unsigned long long), s);
    cudaMemsetAsync(p->rmap_trow.p, 0x7f, tcap * sizeof(int32_t), s);
    cudaMemsetAsync(p->rmap_shared.p, 0, sizeof(int32_t), s);
    cudaMemsetAsync(p->rmap_share_count.p, 0, n * sizeof(int32_t), s);
    for (int pass = 0; pass < 2; ++pass) {
      for (int c = kEmpty_ + 1; c < kNumClasses; ++c) {
        if (!map_class(c) || p->num_count[c] <= 0) continue;
        const bool whole = c == p->num_whole;
        const int32_t *rows = whole ? nullptr : p->rows_num.p + p->num_off[c];
        const int32_t nrows = whole ? p->a_rows : p->num_count[c];
        if (pass == 0)
          launch_map_dedup_insert(rows, nrows, p->rmap_key.p, p->rmap_tkey.p,
                                  p->rmap_trow.p, mask, s);
        else
          launch_map_dedup_resolve(rows, nrows, p->rmap_key.p, p->rmap_tkey.p,
                                   p->rmap_trow.p, mask, c_rp, p->rmap_ops.p,
                                   p->rmap_off.p, p->rmap.p, p->rmap_shared.p,
                                   p->rmap_canon.p, p->rmap_share_count.p, s);
      }
    }
  }
  p->pat_ready = 0;
  if (dedup) {
    e = build_term_tables(p, s, op, c_rp, entries);
    if (e != cudaSuccess) return e;
  }
  p->rmap_state = 1;
  p->rmap_col = c_col;
  p->rmap_entries = entries;
  return cudaGetLastError();
}

}  // namespace

rvsp_status_t rvsp_cuda_plan_prepare_reuse(rvsp_cuda_plan_t p, void *stream,
                                           const int32_t *a_row_ptr, const int32_t *a_col_idx,
                                           const int32_t *b_row_ptr, const int32_t *b_col_idx,
                                           const int32_t *c_row_ptr, const int32_t *c_col_idx,
                                           int64_t *map_entries_out) {
  if (!p || !a_row_ptr || !a_col_idx || !b_row_ptr || !b_col_idx || !c_row_ptr ||
      !c_col_idx)
    return RVSP_ERROR_NULL_POINTER;
  if (!p->analysed) return RVSP_ERROR_INVALID_ARGUMENT;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const Operands op{p->a_rows, p->b_cols, a_row_ptr, a_col_idx, nullptr,
                    b_row_ptr, b_col_idx, nullptr,
                    merge_allowed(p->merge_policy, p->a_rows)};
  const cudaError_t e = build_reuse_map(p, s, op, c_row_ptr, c_col_idx);
  if (map_entries_out) *map_entries_out = p->rmap_state == 1 ? p->rmap_entries : 0;
  return map_cuda(e);
}

rvsp_status_t rvsp_cuda_plan_reuse_shared_rows(rvsp_cuda_plan_t p, void *stream,
                                               int32_t *shared_rows_out) {
  if (!p || !shared_rows_out) return RVSP_ERROR_NULL_POINTER;
  *shared_rows_out = 0;
  if (p->rmap_state != 1 || !p->rmap_shared.p) return RVSP_SUCCESS;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemcpyAsync(shared_rows_out, p->rmap_shared.p, sizeof(int32_t),
                                  cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  return map_cuda(e);
}

rvsp_status_t rvsp_cuda_numeric(rvsp_cuda_plan_t p, void *stream,
                                const int32_t *a_row_ptr, const int32_t *a_col_idx,
                                const float *a_values, const int32_t *b_row_ptr,
                                const int32_t *b_col_idx, const float *b_values,
                                const int32_t *c_row_ptr, int32_t *c_col_idx,
                                float *c_values, int fill, void *workspace,
                                size_t workspace_bytes) {
  if (!p || !a_row_ptr || !a_col_idx || !a_values || !b_row_ptr || !b_col_idx ||
      !b_values || !c_row_ptr || !c_col_idx || !c_values)
    return RVSP_ERROR_NULL_POINTER;
  if (!p->analysed) return RVSP_ERROR_INVALID_ARGUMENT;
  if (p->numeric_ws > 0 && (!workspace || workspace_bytes < p->numeric_ws))
    return workspace ? RVSP_ERROR_INVALID_ARGUMENT : RVSP_ERROR_NULL_POINTER;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const Operands op{p->a_rows, p->b_cols, a_row_ptr, a_col_idx, a_values,
                    b_row_ptr, b_col_idx, b_values,
                    merge_allowed(p->merge_policy, p->a_rows)};
  float *dense_acc = static_cast<float *>(workspace);
  uint32_t *dense_bits = nullptr;
  if (p->numeric_ws > 0) {
    // The dense accumulators (and global bitmaps) must start zeroed; every
    // row leaves what it touched zeroed again, but the caller owns this
    // memory between calls, so clear it each time.
    cudaMemsetAsync(workspace, 0, p->numeric_ws, s);
    dense_bits = reinterpret_cast<uint32_t *>(
        static_cast<char *>(workspace) +
        size_t(p->dense_slots) * dense_slot_acc_bytes(p->b_cols));
  }
  if (p->learned && fill) {
    // The fused pass already holds every non-overflowed row, sorted, with
    // its values: copy them; the overflowed rows take the plain fill.
    {
      PhaseScope ph(p, s, RVSP_PHASE_COMPACT);
      launch_compact(p->a_rows, p->counts.p, p->cap.p, p->slab_off.p, c_row_ptr,
                     p->slab_col.p, p->slab_val.p, c_col_idx, c_values, true,
                     p->big_rows.p, p->num_sms, s);
      ph.launches = 2 + launch_stripe_rows(p, op, c_row_ptr, c_col_idx, c_values, true, s);
      for (int c = kEmpty_ + 1; c < kNumClasses && p->n_ovf > 0; ++c) {
        if (p->ovf_num_count[c] <= 0) continue;
        launch_numeric_class(c, op, p->ops.p, p->ovf_sorted.p + p->ovf_num_off[c],
                             p->ovf_num_count[c], c_row_ptr, c_col_idx, c_values, true,
                             dense_acc, dense_bits, p->dense_slots, p->misc.p + kStatus,
                             p->num_sms, s);
        ph.launches += 1;
      }
    }
    // Those values are the ones A and B held at estimation; if they changed
    // since, recompute every value with the structure now in C.
    values_fingerprint_launch(p, a_values, p->a_nnz, b_values, p->b_nnz, s);
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return map_cuda(e);
    if (p->h_vhash[0] == p->est_hash) return map_cuda(cudaGetLastError());
    fill = 0;
  }
  if (fill == 0 && (p->rmap_state == 0 || (p->rmap_state == 1 && p->rmap_col != c_col_idx))) {
    // First numeric-only call on this structure: build the reuse map, unless
    // the stream is being captured (building synchronizes).
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone) {
      const cudaError_t e = build_reuse_map(p, s, op, c_row_ptr, c_col_idx);
      if (e != cudaSuccess) return map_cuda(e);
    }
  }
  const bool use_map = fill == 0 && p->rmap_state == 1 && p->rmap_col == c_col_idx;
  // numeric-only with every table in place: all row groups run side by side;
  // else the classes do (the members of shift classes follow, below)
  const bool all_lanes = use_map && (!p->shift_active || p->shift_tables == 1);
  Lanes ln(p, s, all_lanes || several_classes(p->num_count));
  bool rt_main = false;  // the largest shared-map pattern kernel, launched last
  {
    PhaseScope ph(p, s, RVSP_PHASE_NUMERIC);
    if (use_map && p->pat_ready && p->n_pat_rows > 0) {
      if (p->rt.ready && p->tiles_enabled) {
        ph.launches += launch_table_tile_kernel(p->rt, op, c_row_ptr, c_values, ln.next());
        ph.launches += launch_pattern_kernels(p->rt, op, c_row_ptr, c_values,
                                              p->misc.p + kStatus, ln, false);
        rt_main = true;
        if (p->rt.n_lo > 0) {
          launch_pat_numeric(op, p->ops.p, p->rt.lo_rows.p, p->rt.lo_ids.p, p->rt.n_lo,
                             c_row_ptr, c_values, p->pat_off.p, p->pat_steps.p, p->pat_rec.p,
                             p->pat_max_ops, p->pat_max_out, ln.next());
          ph.launches += 1;
        }
      } else {
        launch_pat_numeric(op, p->ops.p, p->pat_rows.p, p->pat_ids.p, p->n_pat_rows,
                           c_row_ptr, c_values, p->pat_off.p, p->pat_steps.p, p->pat_rec.p,
                           p->pat_max_ops, p->pat_max_out, ln.main());
        ph.launches += 1;
      }
    }
    // Persistent pass: the merge and map rows in one launch over a queue of
    // row bins, heaviest class first.
    const bool persist = use_map && p->persist_merge_rows > 0 &&
                         p->persist_head.reserve(1) == cudaSuccess;
    if (persist) {
      PersistPlan pp;
      int32_t max_out = 0;
      const int order[] = {kW2048, kW1024, kW512, kW256, kW128, kW64, kM16, kM8, kM4};
      for (int c : order) {
        if (p->num_count[c] <= 0) continue;
        const bool whole = c == p->num_whole;
        PersistSeg g;
        g.cls = c;
        if (map_class(c) && p->pat_ready) {
          g.rows = p->res_rows.p + p->res_off[c];
          g.count = p->res_count[c];
        } else {
          g.rows = whole ? nullptr : p->rows_num.p + p->num_off[c];
          g.count = whole ? p->a_rows : p->num_count[c];
        }
        if (g.count <= 0) continue;
        g.per_item = map_class(c) ? kPersistThreads / 32 : p->persist_merge_rows;
        g.item0 = pp.n_items;
        pp.seg[pp.nseg++] = g;
        pp.n_items += (g.count + g.per_item - 1) / g.per_item;
        if (map_class(c) && max_out == 0) max_out = 1 << (class_log2(c) - 1);
      }
      launch_persist_numeric(op, p->ops.p, pp, p->persist_head.p, c_row_ptr, c_values,
                             p->rmap_off.p, p->rmap.p, p->misc.p + kStatus, max_out,
                             p->persist_blocks, p->num_sms, ln.next());
      ph.launches += 2;
    } else {
      cudaGetLastError();
    }
    for (int c = kEmpty_ + 1; c < kStripe8; ++c) {
      if (p->num_count[c] <= 0) continue;
      if (persist && persist_class(c)) continue;
      const bool whole = c == p->num_whole;
      const int32_t *rows = whole ? nullptr : p->rows_num.p + p->num_off[c];
      const int32_t nrows = whole ? p->a_rows : p->num_count[c];
      if (use_map && map_class(c) && p->pat_ready) {
        if (p->res_count[c] > 0)
          launch_map_numeric(c, op, p->ops.p, p->res_rows.p + p->res_off[c],
                             p->res_count[c], c_row_ptr, c_values, p->rmap_off.p,
                             p->rmap.p, p->misc.p + kStatus, ln.next());
      } else if (use_map && map_class(c))
        launch_map_numeric(c, op, p->ops.p, rows, nrows, c_row_ptr, c_values,
                           p->rmap_off.p, p->rmap.p, p->misc.p + kStatus, ln.next());
      else
        launch_numeric_class(c, op, p->ops.p, rows, nrows, c_row_ptr, c_col_idx, c_values,
                             fill != 0, dense_acc, dense_bits, p->dense_slots,
                             p->misc.p + kStatus, p->num_sms, ln.next());
      ph.launches += 1;
    }
    // the stripe rows, usually the most work, last and on the caller's stream:
    // their persistent blocks fill the SMs
    ph.launches += launch_stripe_rows(p, op, c_row_ptr, c_col_idx, c_values, fill != 0, ln.main());
    if (rt_main)
      ph.launches += launch_pattern_kernels(p->rt, op, c_row_ptr, c_values, p->misc.p + kStatus,
                                            ln, true);
    if (!p->shift_active || !all_lanes) ln.join();
  }
  if (p->shift_active) {
    // Shift-class members: columns by translation of their canonical rows
    // (filled above), values from the canonical rows' term tables.
    // (the columns beside the table builds: nothing here reads them)
    Lanes members(p, s, !ln.forked);
    if (fill) {
      PhaseScope ph(p, s, RVSP_PHASE_NUMERIC);
      launch_shift_fill(p->a_rows, p->st.pid.p, p->sh_rcls.p, c_row_ptr, c_col_idx,
                        members.next());
      ph.launches = 1;
    }
    if (p->shift_tables == 0) {
      cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
      if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone)
        return RVSP_ERROR_INVALID_ARGUMENT;  // building synchronizes: not under capture
      const cudaError_t e = build_shift_tables(p, s, op, c_row_ptr, c_col_idx);
      if (e != cudaSuccess) return map_cuda(e);
    }
    if (p->shift_tables != 1) return RVSP_ERROR_DEVICE;
    PhaseScope ph(p, s, RVSP_PHASE_NUMERIC);
    members.refork();
    ph.launches =
        launch_shift_numeric(p, ln.forked ? ln : members, op, c_row_ptr, c_values);
    members.join();
    ln.join();
  }
  return map_cuda(cudaGetLastError());
}

rvsp_status_t rvsp_cuda_op_counts(rvsp_cuda_plan_t p, void *stream,
                                  int64_t *host_out, int32_t n) {
  if (!p || !host_out) return RVSP_ERROR_NULL_POINTER;
  if (!p->analysed) return RVSP_ERROR_INVALID_ARGUMENT;
  if (n < p->a_rows) return RVSP_ERROR_INVALID_ARGUMENT;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemcpyAsync(host_out, p->ops.p, size_t(p->a_rows) * sizeof(int64_t),
                                  cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  return map_cuda(e);
}

rvsp_status_t rvsp_cuda_plan_status(rvsp_cuda_plan_t p, void *stream) {
  if (!p) return RVSP_ERROR_NULL_POINTER;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int32_t st = 0;
  cudaError_t e = cudaMemcpyAsync(&st, p->misc.p + kStatus, sizeof(int32_t),
                                  cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return map_cuda(e);
  if (st != kDevOk) {
    cudaMemsetAsync(p->misc.p + kStatus, 0, sizeof(int32_t), s);
    cudaStreamSynchronize(s);
  }
  return device_status_to_rvsp(st);
}

rvsp_status_t rvsp_cuda_csr_check(rvsp_cuda_plan_t p, void *stream, int32_t rows,
                                  int32_t cols, const int32_t *row_ptr,
                                  const int32_t *col_idx, int32_t nnz,
                                  int32_t *code_out, int32_t *bad_row_out) {
  if (!p || !code_out || !bad_row_out) return RVSP_ERROR_NULL_POINTER;
  *code_out = 1;  // malformed row pointer
  *bad_row_out = -1;
  if (!row_ptr || rows < 0 || cols < 0 || nnz < 0) return RVSP_SUCCESS;
  if (nnz > 0 && !col_idx) return RVSP_SUCCESS;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t re = p->check_long.reserve(1 + size_t(check_long_rows_cap(rows, nnz)));
  if (re != cudaSuccess) return map_cuda(re);
  cudaMemsetAsync(p->check.p, 0xff, sizeof(unsigned long long), s);
  cudaMemsetAsync(p->check_long.p, 0, sizeof(int32_t), s);
  {
    PhaseScope ph(p, s, RVSP_PHASE_CHECK);
    launch_csr_check(rows, cols, row_ptr, col_idx, nnz, p->check.p, p->check_long.p, s);
    ph.launches = 2;
  }
  cudaMemcpyAsync(p->h_check, p->check.p, sizeof(unsigned long long),
                  cudaMemcpyDeviceToHost, s);
  cudaError_t e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return map_cuda(e);
  const unsigned long long r = *p->h_check;
  if (r == ~0ull) {
    *code_out = 0;
    *bad_row_out = -1;
  } else {
    *code_out = static_cast<int32_t>(r & 0xffu);
    *bad_row_out = static_cast<int32_t>(r >> 8) - 1;
  }
  return RVSP_SUCCESS;
}

rvsp_status_t rvsp_cuda_plan_set_profiling(rvsp_cuda_plan_t p, int enable) {
  if (!p) return RVSP_ERROR_NULL_POINTER;
  p->profiling = enable != 0;
  return RVSP_SUCCESS;
}

rvsp_status_t rvsp_cuda_plan_phase_times(rvsp_cuda_plan_t p, double *ms_out,
                                         int64_t *launches_out, int32_t n,
                                         int reset) {
  if (!p) return RVSP_ERROR_NULL_POINTER;
  resolve_pending(p);
  for (int i = 0; i < n && i < RVSP_PHASE_COUNT; ++i) {
    if (ms_out) ms_out[i] = p->ms[i];
    if (launches_out) launches_out[i] = p->launches[i];
  }
  if (reset) {
    for (int i = 0; i < RVSP_PHASE_COUNT; ++i) {
      p->ms[i] = 0.0;
      p->launches[i] = 0;
    }
  }
  return RVSP_SUCCESS;
}

rvsp_status_t rvsp_cuda_plan_class_counts(rvsp_cuda_plan_t p, int32_t *sym_out,
                                          int32_t *num_out, int32_t n) {
  if (!p) return RVSP_ERROR_NULL_POINTER;
  for (int i = 0; i < n; ++i) {
    // the stripe rows as the classes they come from
    const int from = i == kB8192 ? kStripe8 : i == kDense ? kStripe : -1;
    if (sym_out)
      sym_out[i] = i < kStripe8 ? p->sym_count[i] + (from >= 0 ? p->sym_count[from] : 0) : 0;
    if (num_out)
      num_out[i] = i < kStripe8 ? p->num_count[i] + (from >= 0 ? p->num_count[from] : 0) : 0;
  }
  return RVSP_SUCCESS;
}

}  // extern "C"

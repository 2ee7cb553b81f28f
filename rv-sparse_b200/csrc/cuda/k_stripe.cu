// Stripe rows: heavy rows (more than 1024 outputs possible) cut by columns, for
// B of at most kStripeMaxCols columns.
//
// A heavy row's cost is keeping the reference's order: every output sums its
// terms in ascending A-nonzero order.  A block that steps through the row one
// A nonzero at a time pays a barrier for each and leaves most threads idle on
// short B rows (k_heavy.cu).  Here the columns are cut into stripes and one
// warp takes all of a row's products in a run of stripes, in order, so no
// warp ever waits for another:
//
//   stripes   B's columns in runs of whole 32-column words, closed at equal
//             shares of B's entries (power-law columns: the first stripes
//             are narrow) and at the kStripeCols columns a warp's accumulator
//             holds; ptr[k][t] is where stripe t starts in B row k;
//   count     a block per row marks the row's columns in shared memory (no
//             order needed) and keeps their bitmap and the outputs before each
//             stripe;
//   items     (row, stripes [t0, t1)): as many stripes as hold about kItemOps
//             products and fit the accumulator by their columns or by the
//             row's outputs in them, so a hub row is many items and a row of a
//             few thousand products one or two; rows of many products are
//             drawn first;
//   values    persistent blocks of four warps draw items and cut each into four
//             runs of stripes of about equal products, a warp each over one
//             accumulator; a warp walks its products
//             in flattened order (ascending A nonzero, then column), up to 32
//             of one B row at a time, or 32 across short B rows with equal
//             columns in lane order, into an accumulator in shared memory: a
//             slot a column where the columns fit it (gathered at C's columns
//             at the end), else a slot an output, found by a population count
//             in the row's bitmap.
//
// Each output is the sum of its terms in ascending A-nonzero order from
// +0.0f, products and sums rounded separately (gustavson_core_f32.inc:31-62
// with accum_scalar_f32.c:20-71); the columns are the row's bitmap in order
// (rvsp_symbolic.c:91-137).
//
// A row of C that is not as long as the analysed one is reported and left as it
// is.  A C whose columns are not this product's is reported.  With a slot a column
// an accumulator word starts as kUntouched, a NaN pattern that no addition
// returns (results that are NaN are the canonical one), and the counts of
// first touches, of gathered words and of outputs must agree; with a slot an
// output, C's columns are compared with the bitmap.
//
// Bound: issue slots.  A product is a column, a value, a slot look-up, an add
// and its share of the walk, some 20 instructions for a lane; none of it waits
// for another warp.  R-MAT 2^16, 16 entries a row (402 M products), whole
// product on one B200, in ms: block-per-row kernels 13.1; a warp an item 7.2;
// four warps sharing one accumulator (runs of B entries four times longer),
// outputs ranked where columns do not fit, hub rows counted in parts 4.3; with
// items placed by one atomic a warp and slot checks folded into the bitmap
// word 3.5, of which the values take 1.8, the count 0.7, the columns 0.5.
// Numeric-only repeat at 2^15: 2.6 -> 0.92.  Measured and left: 5 warps (one
// reading ahead) 3.70 against 3.58, 6 to 9 blocks an SM by launch bounds 3.7
// to 4.4 (spills), accumulators of 2048 and 8192 slots, 8 or 2 steps in flight
// and items of 8 K to 128 K products each within 5%.  Which products take
// these kernels: stripe_rule.cuh.  B wider than kStripeMaxCols (2^17) keeps the
// block kernels: stripe_bounds_kernel is one block that holds four bitmap words
// a thread, 2^17 columns in all, and kMaxStripes (96) is what B of that width
// may need, 32 by shares and 64 by words.  (The count's shared memory would hold
// more: a row's bitmap and prefix take 17 KB at 2^17, 135 KB at 2^20.)
#include <climits>

#include "device_common.cuh"
#include "index.cuh"
#include "kernels.cuh"

namespace rvsp {

namespace {

constexpr int kAcc = kStripeAcc;     // accumulator slots of a block (16 KB)
constexpr int kStripeWords = 64;     // words (of 32 columns) a stripe spans at most
constexpr int kItemWords = 2048;     // bitmap words a block can hold for one item
constexpr int kStripeShares = 32;    // equal shares of B's entries
constexpr int kItemOps = kStripeItemOps;  // products an item aims at
constexpr int kTaskOps = 1 << 16;    // products of a part of a cut row (count)
constexpr int kSplitTasks = 1 << 15; // parts of cut rows at most
constexpr int kPtrThreads = 256;
constexpr int kItemRows = 64;        // rows a block of the item kernel
constexpr int kBigRowOps = 1 << 18;  // rows whose items are drawn first
constexpr size_t kStripeTableMax = size_t(256) << 20;

constexpr int kColumnWarps = 8;      // warps a row of the column kernel
constexpr int kCountThreads = 128;
constexpr int kCountWarps = kCountThreads / 32;
constexpr int kValueWarps = 4;       // warps a block of the value kernel
constexpr int kCountUnroll = 4;      // steps in flight a warp of the count kernel
constexpr int kUnroll = 4;           // 32-product batches in flight a warp
constexpr int kStepUnroll = 4;       // steps in flight a warp
constexpr int kStepLen = 8;          // mean entries a run from which steps pay
constexpr uint32_t kUntouched = 0xffffffffu;

// The values kernel's dynamic shared memory: the accumulator, a word a thread
// for products that have no slot, and, for each of
// item_words words of the bitmap, two half words with the outputs before them,
// and an empty word.
constexpr size_t value_bytes(int32_t item_words) {
  return size_t(kAcc + kValueWarps * 32) * 4 + size_t(item_words) * 8 + 16;
}

// ---- stripes of B -------------------------------------------------------------

__global__ void __launch_bounds__(512)
stripe_hist_kernel(const int32_t *__restrict__ b_rp, int32_t b_rows,
                   const int32_t *__restrict__ b_col, int32_t words,
                   int32_t *__restrict__ hist) {
  extern __shared__ int32_t s_hist[];
  for (int w = threadIdx.x; w < words; w += blockDim.x) s_hist[w] = 0;
  __syncthreads();
  const int32_t n = b_rp[b_rows];
  const int64_t stride = int64_t(gridDim.x) * blockDim.x;
  for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < n; e += stride)
    atomicAdd(&s_hist[__ldg(b_col + e) >> 5], 1);
  __syncthreads();
  for (int w = threadIdx.x; w < words; w += blockDim.x)
    if (s_hist[w]) atomicAdd(&hist[w], s_hist[w]);
}

// One block of 1024: bound[t] = first word of stripe t (words for t past the
// last), share[t] = its part of B's entries.
// words <= 4096: thread i owns words [4 i, 4 i + 4).
__global__ void __launch_bounds__(1024)
stripe_bounds_kernel(int32_t words, int32_t ns_max, const int32_t *__restrict__ hist,
                     int32_t *__restrict__ bound, float *__restrict__ share) {
  __shared__ int32_t s_warp[32], s_total;
  __shared__ int32_t s_bound[kMaxStripes + 1], s_mass[kMaxStripes + 1];
  const int lane = lane_id(), wid = threadIdx.x >> 5;
  auto block_scan = [&](int v) {  // exclusive; the sum goes to s_total
    const int incl = warp_incl_scan(v);
    if (lane == 31) s_warp[wid] = incl;
    __syncthreads();
    if (wid == 0) {
      const int x = s_warp[lane], xi = warp_incl_scan(x);
      s_warp[lane] = xi - x;
      if (lane == 31) s_total = xi;
    }
    __syncthreads();
    const int r = s_warp[wid] + incl - v;
    __syncthreads();
    return r;
  };
  int h[4], mine = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int w = threadIdx.x * 4 + i;
    h[i] = w < words ? hist[w] : 0;
    mine += h[i];
  }
  const int before = block_scan(mine);
  const int64_t total = s_total > 0 ? s_total : 1;
  // word w opens a stripe when its share index or its accumulator differs
  // from the word before
  bool open[4];
  int mass[4], opens = 0, run = before;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int w = threadIdx.x * 4 + i;
    // mass before word w and before word w - 1; the latter belongs to the
    // previous thread for i = 0, whose word's entries are read again
    const int prev = i ? h[i - 1] : (w > 0 && w < words ? hist[w - 1] : 0);
    mass[i] = run;
    open[i] = w < words &&
              (w % kStripeWords == 0 || run * int64_t(kStripeShares) / total !=
                                            (run - prev) * int64_t(kStripeShares) / total);
    opens += open[i];
    run += h[i];
  }
  int at = block_scan(opens);
  const int ns = s_total;
  for (int t = threadIdx.x; t <= kMaxStripes; t += blockDim.x) {
    s_bound[t] = words;
    s_mass[t] = static_cast<int32_t>(total);
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (open[i]) {
      s_bound[at] = threadIdx.x * 4 + i;
      s_mass[at] = mass[i];
      ++at;
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t <= ns_max; t += blockDim.x) {
    bound[t] = s_bound[t];
    if (t < ns_max)
      share[t] = t < ns ? float(s_mass[t + 1] - s_mass[t]) / float(total) : 0.0f;
  }
}

// Bound by the latency of the searches.
// ptr[k * (ns_max + 1) + t] = first entry of B row k in stripe t or after it
// (the row's end for t = ns_max).  A warp per row, a lane per stripe, each a
// binary search of the row: short rows cost a few cached loads, and a hub row
// of thousands of entries a dozen.
__global__ void __launch_bounds__(kPtrThreads)
stripe_ptr_kernel(int32_t b_rows, const int32_t *__restrict__ b_rp,
                  const int32_t *__restrict__ b_col, int32_t ns_max,
                  const int32_t *__restrict__ bound, int32_t *__restrict__ ptr) {
  __shared__ int32_t s_bound[kMaxStripes + 1];
  for (int t = threadIdx.x; t <= ns_max; t += blockDim.x) s_bound[t] = bound[t] << 5;
  __syncthreads();
  const int lane = lane_id();
  const int32_t step = (gridDim.x * blockDim.x) >> 5;
  for (int32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < b_rows; k += step) {
    const int32_t b0 = b_rp[k], b1 = b_rp[k + 1];
    for (int t = lane; t <= ns_max; t += 32) {
      const int32_t c = s_bound[t];
      int32_t lo = b0, hi = b1;
      while (lo < hi) {
        const int32_t mid = middle(lo, hi);  // (entries of all of B)
        if (__ldg(b_col + mid) < c) lo = mid + 1;
        else hi = mid;
      }
      ptr[int64_t(k) * (ns_max + 1) + t] = lo;
    }
  }
}

// ---- expanding products ---------------------------------------------------------

// Up to 32 runs of B entries, one per lane ([beg, beg + len), scaled by a),
// walked in order one of two ways.  Steps: up to 32 entries of one run at a
// time (distinct columns), for runs of kStepLen entries or more on average.
// Batches: 32 entries across runs at a time.  Either way the non-empty runs
// are compacted into shared memory, and the run that owns unit u (a step or
// an entry) is a population count over the mask of the runs that start in
// the 32 units around it.
struct Runs {
  int32_t excl;   // units before this lane's run
  int32_t total;  // units of the chunk (uniform)
  int started;    // non-empty runs that start before the units at hand (uniform)
  bool some;      // this lane's run is not empty
  bool steps;     // units are steps (uniform)
};

// seg[r] = (first entry, entries, a, units before) of the r-th non-empty run.
__device__ __forceinline__ Runs open_runs(int4 *seg, int32_t beg, int32_t len, float a) {
  Runs r;
  r.started = 0;
  r.some = len > 0;
  const unsigned some = __ballot_sync(kFull, r.some);
  const int32_t units = (len + 31) >> 5;
  int32_t incl = warp_incl_scan(len);
  const int32_t entries = __shfl_sync(kFull, incl, 31);
  r.steps = entries >= kStepLen * __popc(some);
  r.excl = incl - len;
  r.total = entries;
  if (r.steps) {
    incl = warp_incl_scan(units);
    r.excl = incl - units;
    r.total = __shfl_sync(kFull, incl, 31);
  }
  __syncwarp();  // the chunk before has been read
  if (r.some)
    seg[__popc(some & lanemask_lt())] = make_int4(beg, len, __float_as_int(a), r.excl);
  __syncwarp();
  return r;
}

// The run that owns unit u0 + lane (u0 advances by 32 a call); starts = the
// units among these 32 that open a run.
__device__ __forceinline__ int owner_of_unit(Runs &r, int32_t u0, unsigned &starts) {
  const int32_t d = r.excl - u0;
  starts = __reduce_or_sync(kFull, (r.some && d >= 0 && d < 32) ? 1u << d : 0u);
  const int own = r.started + __popc(starts & (lanemask_lt() * 2u + 1u)) - 1;
  r.started += __popc(starts);
  return own;
}

// Steps [u0, u0 + 32): step[i] = (first entry, entries, a) of step u0 + i, past
// the chunk's end the last run's first entry and no entries; returns how many
// there are.
__device__ __forceinline__ int open_steps(Runs &r, const int4 *seg, int4 *step, int32_t u0) {
  const int lane = lane_id();
  unsigned starts;
  const int own = owner_of_unit(r, u0, starts);
  const int32_t u = u0 + lane;
  int4 s = seg[own];
  if (u < r.total) {
    const int32_t skip = (u - s.w) << 5;
    s.x += skip;
    s.y = min(32, s.y - skip);
  } else {
    s.y = 0;
  }
  __syncwarp();  // the steps before have been read
  step[lane] = s;
  __syncwarp();
  return min(32, r.total - u0);
}

// The entry (and its run's a) of product u0 + lane.  solo: the batch's
// products come from one run (uniform).
__device__ __forceinline__ bool next_batch(Runs &r, const int4 *seg, int32_t u0, int32_t &entry,
                                           float &a, bool &solo) {
  unsigned starts;
  const int own = owner_of_unit(r, u0, starts);
  solo = (starts & ~1u) == 0u;
  const int32_t u = u0 + lane_id();
  const bool v = u < r.total;
  const int4 sg = seg[v ? own : 0];
  entry = sg.x + (u - sg.w);
  a = __int_as_float(sg.z);
  return v;
}

// ---- count ------------------------------------------------------------------------

// Tasks of the count: (r, part | parts << 16).  A row of more than kTaskOps
// products is cut into parts of its A nonzeros, so that a hub row does not
// keep one block long after the others are done; its bitmap in global memory
// is cleared here, and its tasks fill tasks[] from the front (cnt[0] of them,
// at most kSplitTasks; a row that finds no room stays whole).  Whole rows fill
// it from the back (cnt[1]).
__global__ void __launch_bounds__(128)
stripe_tasks_kernel(const int32_t *__restrict__ rows, int32_t nrows,
                    const int64_t *__restrict__ ops, int32_t words,
                    uint32_t *__restrict__ bits, int2 *__restrict__ tasks,
                    int32_t *__restrict__ cnt, int32_t *__restrict__ done) {
  __shared__ int32_t s_cut[128], s_n;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  const int32_t r = blockIdx.x * 128 + threadIdx.x;
  int parts = 0;
  if (r < nrows) {
    const int64_t o = ops[row_of(rows, r)];
    parts = max(1, static_cast<int>(min((o + kTaskOps - 1) / kTaskOps, int64_t(64))));
    if (parts > 1) {
      const int at = atomicAdd(&cnt[0], parts);
      if (at + parts > kSplitTasks) {
        for (int i = at; i < kSplitTasks; ++i) tasks[i] = make_int2(-1, 0);
        parts = 1;
      } else {
        for (int i = 0; i < parts; ++i) tasks[at + i] = make_int2(r, i | parts << 16);
        s_cut[atomicAdd(&s_n, 1)] = r;
        done[r] = 0;
      }
    }
  }
  const unsigned whole = __ballot_sync(kFull, parts == 1);
  int base = 0;
  if (lane_id() == 0 && whole) base = atomicAdd(&cnt[1], __popc(whole));
  base = __shfl_sync(kFull, base, 0);
  if (parts == 1)
    tasks[kSplitTasks + nrows - 1 - (base + __popc(whole & lanemask_lt()))] =
        make_int2(r, 1 << 16);
  __syncthreads();
  for (int i = 0; i < s_n; ++i)
    for (int w = threadIdx.x; w < words; w += 128) bits[int64_t(s_cut[i]) * words + w] = 0u;
}

// Bound by shared-memory atomics on a row's bitmap, read before they are set
// (a byte a column instead of a bit: 1.37 ms against 0.93 at 2^16 then, two
// blocks an SM).
// rows[r]: counts[row], hslot[row] = r, the row's bitmap at bits + r * words,
// the outputs before each 32 words of it at gpre + r * stripe_groups(words)
// and the outputs before stripe t at soff[r * (ns_max + 1) + t].  The parts of
// a cut row meet in its bitmap in global memory, and the last of them counts.
__global__ void __launch_bounds__(kCountThreads)
stripe_count_kernel(Operands op, const int32_t *__restrict__ rows, int32_t nrows,
                    int32_t words, int32_t ns_max, const int32_t *__restrict__ bound,
                    const int2 *__restrict__ tasks, const int32_t *__restrict__ cnt,
                    int32_t *__restrict__ done, int32_t *__restrict__ counts,
                    int32_t *__restrict__ hslot, uint32_t *__restrict__ bits_out,
                    int32_t *__restrict__ gpre, int32_t *__restrict__ soff,
                    int32_t *__restrict__ head) {
  extern __shared__ __align__(16) uint32_t s_mem[];
  const int32_t groups = stripe_groups(words);
  uint32_t *bits = s_mem;  // whole groups
  int32_t *pre = reinterpret_cast<int32_t *>(s_mem + 32 * groups);
  __shared__ int4 s_seg[kCountWarps][32], s_step[kCountWarps][32];
  __shared__ int32_t s_task, s_chunk, s_last;
  const int tid = threadIdx.x, lane = lane_id(), wid = tid >> 5;
  int4 *seg = s_seg[wid], *step = s_step[wid];
  auto mark = [&](int32_t col) {
    uint32_t *wp = bits + (col >> 5);
    const uint32_t bit = 1u << (col & 31);
    if (!(*reinterpret_cast<volatile uint32_t *>(wp) & bit)) atomicOr(wp, bit);
  };
  const int32_t n_cut = min(cnt[0], kSplitTasks), n_whole = cnt[1];
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      s_task = atomicAdd(head, 1);
      s_chunk = 0;
    }
    for (int w = tid; w < 32 * groups; w += kCountThreads) bits[w] = 0u;
    __syncthreads();
    const int32_t at = s_task;
    if (at >= n_cut + n_whole) return;
    const int2 task = tasks[at < n_cut ? at : kSplitTasks + nrows - 1 - (at - n_cut)];
    const int32_t r = task.x, part = task.y & 0xffff, parts = task.y >> 16;
    if (r < 0) continue;  // (a row that found no room for its parts)
    const int32_t row = row_of(rows, r);
    int32_t p0 = op.a_rp[row], p1 = op.a_rp[row + 1];
    if (parts > 1) {
      const int64_t n = p1 - p0;
      p1 = p0 + static_cast<int32_t>(n * (part + 1) / parts);
      p0 = p0 + static_cast<int32_t>(n * part / parts);
    }
    // A nonzeros a warp takes at a time: few enough that all warps get some
    const int32_t take = min(32, max(1, (p1 - p0) / (2 * kCountWarps)));
    for (;;) {
      int32_t c = 0;
      if (lane == 0) c = atomicAdd(&s_chunk, 1);
      c = __shfl_sync(kFull, c, 0);
      const int64_t p = p0 + int64_t(c) * take;
      if (p >= p1) break;
      int32_t beg = 0, len = 0;
      if (lane < take && p + lane < p1) {
        const int32_t k = __ldg(op.a_col + p + lane);
        beg = __ldg(op.b_rp + k);
        len = __ldg(op.b_rp + k + 1) - beg;
      }
      Runs run = open_runs(seg, beg, len, 0.0f);
      if (run.steps) {
        for (int32_t u0 = 0; u0 < run.total; u0 += 32) {
          const int n = open_steps(run, seg, step, u0);
          for (int i = 0; i < n; i += kCountUnroll) {
            int32_t col[kCountUnroll];
#pragma unroll
            for (int u = 0; u < kCountUnroll; ++u) {
              const int2 sg = *reinterpret_cast<const int2 *>(&step[i + u]);
              col[u] = lane < sg.y ? __ldg(op.b_col + sg.x + lane) : -1;
            }
#pragma unroll
            for (int u = 0; u < kCountUnroll; ++u)
              if (col[u] >= 0) mark(col[u]);
          }
        }
        continue;
      }
      for (int32_t t0 = 0; t0 < run.total; t0 += 32 * kUnroll) {
        int32_t col[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
          int32_t e;
          float a;
          bool solo;
          const bool v = next_batch(run, seg, t0 + 32 * u, e, a, solo);
          col[u] = v ? __ldg(op.b_col + e) : -1;
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u)
          if (col[u] >= 0) mark(col[u]);
      }
    }
    __syncthreads();
    uint32_t *own = bits_out + int64_t(r) * words;
    if (parts > 1) {
      for (int w = tid; w < words; w += kCountThreads)
        if (bits[w]) atomicOr(own + w, bits[w]);
      __threadfence();
      __syncthreads();
      if (tid == 0) s_last = atomicAdd(&done[r], 1) == parts - 1;
      __syncthreads();
      if (!s_last) continue;
      __threadfence();
      for (int w = tid; w < words; w += kCountThreads) bits[w] = __ldcg(own + w);
      __syncthreads();
    }
    // The bitmap out and the outputs of each group of 32 words, then their
    // prefix by the first warp.
    for (int32_t g = wid; g < groups; g += kCountWarps) {
      const int32_t w = (g << 5) + lane;
      const uint32_t x = bits[w];
      if (w < words && parts == 1) own[w] = x;
      const int c = warp_sum(__popc(x));
      if (lane == 0) pre[g] = c;
    }
    __syncthreads();
    if (wid == 0) {
      int base = 0;
      for (int32_t g0 = 0; g0 < groups; g0 += 32) {
        const int c = g0 + lane < groups ? pre[g0 + lane] : 0;
        const int incl = warp_incl_scan(c);
        if (g0 + lane < groups) {
          pre[g0 + lane] = base + incl - c;
          gpre[int64_t(r) * groups + g0 + lane] = base + incl - c;
        }
        base += __shfl_sync(kFull, incl, 31);
      }
      if (lane == 0) {
        pre[groups] = base;
        counts[row] = base;
        hslot[row] = r;
      }
    }
    __syncthreads();
    for (int t = tid; t <= ns_max; t += kCountThreads) {
      const int32_t b = bound[t];
      int o = pre[b >> 5];
      for (int32_t w = b & ~31; w < b; ++w) o += __popc(bits[w]);
      soff[int64_t(r) * (ns_max + 1) + t] = b < words ? o : pre[groups];
    }
  }
}

// ---- items ------------------------------------------------------------------------

// One thread per row: its runs of stripes, as long as they are fewer than the
// warps or hold about kItemOps products, and either their columns or, within kItemWords words,
// their outputs fit the accumulator.  Items of rows of at least kBigRowOps
// products fill items[] from the front (cnt[0]), the others from the back
// (cnt[1]).  item = (row, t0 | t1 << 16, outputs before, outputs).
__global__ void __launch_bounds__(kItemRows)
stripe_items_kernel(const int32_t *__restrict__ rows, int32_t nrows,
                    const int64_t *__restrict__ ops, const int32_t *__restrict__ hslot,
                    const int32_t *__restrict__ soff, int32_t ns_max,
                    const int32_t *__restrict__ bound, const float *__restrict__ share,
                    int4 *__restrict__ items, int64_t cap, int32_t *__restrict__ cnt) {
  __shared__ int32_t s_bound[kMaxStripes + 1], s_off[kItemRows][kMaxStripes + 1];
  __shared__ float s_share[kMaxStripes];
  for (int t = threadIdx.x; t <= ns_max; t += blockDim.x) {
    s_bound[t] = bound[t];
    if (t < ns_max) s_share[t] = share[t];
  }
  // the rows' outputs before each stripe, a warp a row (an odd row length in
  // shared memory: the threads then walk their rows without bank conflicts)
  const int32_t i0 = blockIdx.x * kItemRows;
  for (int r = threadIdx.x >> 5; r < kItemRows && i0 + r < nrows; r += kItemRows / 32) {
    const int64_t h = hslot[row_of(rows, i0 + r)];
    for (int t = lane_id(); t <= ns_max; t += 32) s_off[r][t] = soff[h * (ns_max + 1) + t];
  }
  __syncthreads();
  // (every thread stays for the warp's count; one past the rows has no stripes)
  const int32_t i = i0 + threadIdx.x;
  const bool live = i < nrows;
  const int32_t row = live ? row_of(rows, i) : 0;
  const int32_t *so = s_off[threadIdx.x];
  const float work = live ? static_cast<float>(ops[row]) : 0.0f;
  const bool big = work >= float(kBigRowOps);
  int64_t at = 0;
  for (int pass = 0; pass < 2; ++pass) {
    int n = 0;
    int32_t o = live ? so[0] : 0;
    for (int t0 = live ? 0 : ns_max; t0 < ns_max;) {
      const int32_t w0 = s_bound[t0];
      int t1 = t0 + 1;
      float part = s_share[t0];
      int32_t end = so[t1];
      while (t1 < ns_max &&
             (t1 - t0 < kValueWarps || work * (part + s_share[t1]) <= float(kItemOps))) {
        const int32_t nw = s_bound[t1 + 1] - w0, more = so[t1 + 1];
        if (nw > kAcc / 32 && (nw > kItemWords || more - o > kAcc)) break;
        part += s_share[t1];
        end = more;
        ++t1;
      }
      if (end > o) {
        if (pass) {
          const int64_t q = at + n;
          items[big ? q : cap - 1 - q] = make_int4(row, t0 | (t1 << 16), o, end - o);
        }
        ++n;
      }
      o = end;
      t0 = t1;
    }
    if (!pass) {
      // places for all of the warp's items of either kind by one atomic each
      const int mine = n;
      const int bigs = warp_incl_scan(big ? mine : 0), rest = warp_incl_scan(big ? 0 : mine);
      int base = 0, base_rest = 0;
      if (lane_id() == 31) {
        if (bigs) base = atomicAdd(&cnt[0], bigs);
        if (rest) base_rest = atomicAdd(&cnt[1], rest);
      }
      base = __shfl_sync(kFull, base, 31);
      base_rest = __shfl_sync(kFull, base_rest, 31);
      at = big ? base + bigs - mine : base_rest + rest - mine;
    }
  }
}

// ---- columns ----------------------------------------------------------------------

// Bound by issue slots (lanes walk bits of words of unequal population; 0.5 ms
// for R-MAT 2^16).
// 32 words at a time, a lane per word: each lane drops its set bits' columns
// into the warp's staging in order, and the warp copies them out together.
__global__ void __launch_bounds__(kColumnWarps * 32)
stripe_columns_kernel(const int32_t *__restrict__ rows, const int32_t *__restrict__ hslot,
                      const uint32_t *__restrict__ bits_in, const int32_t *__restrict__ gpre,
                      const int32_t *__restrict__ soff, int32_t ns_max, int32_t words,
                      const int32_t *__restrict__ c_rp, int32_t *__restrict__ c_col,
                      int32_t *__restrict__ status) {
  __shared__ int32_t s_stage[kColumnWarps][1024 + 32];
  const int lane = lane_id(), wid = threadIdx.x >> 5;
  const int32_t row = row_of(rows, blockIdx.x);
  const int64_t h = hslot[row];
  const uint32_t *bits = bits_in + h * words;
  const int32_t groups = stripe_groups(words);
  const int32_t c0 = c_rp[row], m = c_rp[row + 1] - c0;
  if (soff[h * (ns_max + 1) + ns_max] != m) {  // C's row pointers are not this analysis's
    if (threadIdx.x == 0) report(status, kDevCountMismatch);
    return;
  }
  int32_t *stage = s_stage[wid];
  for (int32_t g = wid; g < groups; g += kColumnWarps) {
    const int32_t w = (g << 5) + lane;
    uint32_t x = w < words ? __ldg(bits + w) : 0u;
    const int c = __popc(x), incl = warp_incl_scan(c);
    const int n = __shfl_sync(kFull, incl, 31);
    int at = incl - c;
    // (a pad word per 32: full words would all write one bank)
    while (x) {
      stage[at + (at >> 5)] = (w << 5) + __ffs(x) - 1;
      ++at;
      x &= x - 1u;
    }
    __syncwarp();
    int32_t *out = c_col + c0 + gpre[h * groups + g];
    for (int e = lane; e < n; e += 32) out[e] = stage[e + (e >> 5)];
    __syncwarp();
  }
}

// ---- values -----------------------------------------------------------------------

// acc[slot] += term; returns the slots this lane touched first (direct
// accumulators only).  Lanes without a product have a word of their own past
// the accumulator, so the code runs without predicates.  Solo: the lanes'
// slots are distinct (one B row).  Mixed: equal slots are added in lane order,
// which is A order.
template <bool kRank>
__device__ __forceinline__ float acc_value(uint32_t old, int &first) {
  if (kRank) return __uint_as_float(old);
  first = old == kUntouched;
  return first ? 0.0f : __uint_as_float(old);
}

template <bool kRank>
__device__ __forceinline__ int apply_solo(uint32_t *acc, int slot, float term) {
  int first = 0;
  acc[slot] = __float_as_uint(__fadd_rn(acc_value<kRank>(acc[slot], first), term));
  __syncwarp();
  return first;
}

template <bool kRank>
__device__ __forceinline__ int apply_mixed(uint32_t *acc, int slot, float term) {
  const int lane = lane_id();
  const unsigned peers = __match_any_sync(kFull, slot);
  const bool leader = (peers & lanemask_lt()) == 0u;
  unsigned rest = leader ? peers & ~(1u << lane) : 0u;  // the group's later lanes
  float a = 0.0f;
  int first = 0;
  if (leader) a = __fadd_rn(acc_value<kRank>(acc[slot], first), term);
  while (__any_sync(kFull, rest != 0u)) {
    const float t = __shfl_sync(kFull, term, rest ? __ffs(rest) - 1 : lane);
    if (rest) {
      a = __fadd_rn(a, t);
      rest &= rest - 1u;
    }
  }
  if (leader) acc[slot] = __float_as_uint(a);
  __syncwarp();
  return first;
}

// The block's accumulator, and for ranked items the row's bitmap over the
// item's columns: 16 columns in the low half of a word, the item's outputs
// before them in the high half.  Then the warp's walk.
struct WarpMem {
  uint32_t *acc;
  uint32_t *half;
  int4 *seg, *step;
};

struct Item {
  int32_t p0, p1;     // A entries of the row
  int32_t t0, t1;     // this warp's stripes
  int32_t c0, width;  // the item's columns
};

// The accumulator slot of column c0 + rel; missing turns non-zero when it has
// none (the slot is then any word of the block's).  A column outside a ranked
// item meets the empty word past its bitmap.
template <bool kRank>
__device__ __forceinline__ int32_t slot_of(const WarpMem &m, int32_t rel, int32_t width,
                                           uint32_t &missing) {
  if (!kRank) {
    const bool inside = static_cast<uint32_t>(rel) < static_cast<uint32_t>(width);
    missing |= inside ? 0u : 1u;
    return inside ? rel : kAcc;
  }
  const uint32_t x =
      m.half[min(static_cast<uint32_t>(rel) >> 4, static_cast<uint32_t>(width) >> 4)];
  const uint32_t bit = 1u << (rel & 15);
  missing |= bit & ~x;
  return static_cast<int32_t>((x >> 16) + __popc(x & (bit - 1u)));
}

// Applies the item's products; returns this lane's first touches.
template <bool kRank>
__device__ __forceinline__ int walk_item(const Operands &op, const Item &it, const WarpMem &m,
                                         const int32_t *__restrict__ ptr, int64_t stride,
                                         bool &bad) {
  const int lane = lane_id();
  int touched = 0;
  const int32_t spare = kAcc + static_cast<int32_t>(threadIdx.x);
  uint32_t missing = 0;  // non-zero once a column had no slot: B is not the analysed one
  // A's entries of the next chunk, and their stripe starts, are loaded while
  // this one is applied
  int64_t k_next = 0;
  float a = 0.0f, a_next = 0.0f;
  int32_t beg = 0, len = 0;
  auto load_k = [&](uint32_t q) {
    if (before(q, lane, it.p1)) {
      k_next = __ldg(op.a_col + q + lane) * stride;
      a_next = __ldg(op.a_val + q + lane);
    }
  };
  auto load_run = [&](uint32_t q) {  // of the entries load_k(q) read
    a = a_next;
    beg = len = 0;
    if (before(q, lane, it.p1)) {
      beg = __ldg(ptr + k_next + it.t0);
      len = __ldg(ptr + k_next + it.t1) - beg;
    }
  };
  uint32_t p = it.p0;  // (runs past p1, which may be 2^31 - 1)
  load_k(p);
  load_run(p);
  load_k(p + 32);
  while (before(p, 0, it.p1)) {
    Runs run = open_runs(m.seg, beg, len, a);
    p += 32;
    load_run(p);
    load_k(p + 32);
    if (run.steps) {
      for (int32_t u0 = 0; u0 < run.total; u0 += 32) {
        const int n = open_steps(run, m.seg, m.step, u0);
        // the next steps' entries are loaded while these are applied (lanes
        // past a step's entries read its first one and add to a spare word)
        int32_t col[kStepUnroll], len[kStepUnroll];
        float val[kStepUnroll], av[kStepUnroll];
        auto load = [&](int i) {
#pragma unroll
          for (int u = 0; u < kStepUnroll; ++u) {
            const int4 sg = m.step[i + u];
            const uint32_t e = sg.x + (lane < sg.y ? lane : 0);
            col[u] = __ldg(op.b_col + e);
            val[u] = __ldg(op.b_val + e);
            len[u] = sg.y;
            av[u] = __int_as_float(sg.z);
          }
        };
        load(0);
        for (int i = 0; i < n; i += kStepUnroll) {
          int32_t slot[kStepUnroll];
          float term[kStepUnroll];
#pragma unroll
          for (int u = 0; u < kStepUnroll; ++u) {
            term[u] = __fmul_rn(av[u], val[u]);
            slot[u] = slot_of<kRank>(m, col[u] - it.c0, it.width, missing);
            slot[u] = lane < len[u] ? slot[u] : spare;
          }
          if (i + kStepUnroll < n) load(i + kStepUnroll);
#pragma unroll
          for (int u = 0; u < kStepUnroll; ++u)
            touched += apply_solo<kRank>(m.acc, slot[u], term[u]);
        }
      }
      continue;
    }
    for (int32_t t = 0; t < run.total; t += 32 * kUnroll) {
      int32_t slot[kUnroll];
      float term[kUnroll];
      bool solo[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        int32_t e;
        float x;
        const bool v = next_batch(run, m.seg, t + 32 * u, e, x, solo[u]);
        slot[u] = INT_MAX;
        term[u] = 0.0f;
        if (v) {
          slot[u] = __ldg(op.b_col + e) - it.c0;
          term[u] = __fmul_rn(x, __ldg(op.b_val + e));
        }
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u)
        slot[u] = slot[u] != INT_MAX ? slot_of<kRank>(m, slot[u], it.width, missing) : spare;
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        if (t + 32 * u >= run.total) break;
        touched += solo[u] ? apply_solo<kRank>(m.acc, slot[u], term[u])
                           : apply_mixed<kRank>(m.acc, slot[u], term[u]);
      }
    }
  }
  bad |= missing != 0u;
  return touched;
}

// How many of cum[t0 .. t1) are below x (cum ascends); the warp together.
__device__ __forceinline__ int stripes_below(const float *cum, int t0, int t1, float x) {
  int n = 0;
  for (int t = t0; t < t1; t += 32)
    n += __popc(__ballot_sync(kFull, t + lane_id() < t1 && cum[t + lane_id()] < x));
  return n;
}

__global__ void __launch_bounds__(kValueWarps * 32)
stripe_values_kernel(Operands op, const int4 *__restrict__ items, int64_t cap,
                     const int32_t *__restrict__ cnt, int32_t *__restrict__ head,
                     int32_t ns_max, const int32_t *__restrict__ bound,
                     const float *__restrict__ share, const int32_t *__restrict__ ptr,
                     const int32_t *__restrict__ hslot,
                     const uint32_t *__restrict__ bits, const int32_t *__restrict__ gpre,
                     int32_t words, int32_t item_words, const int32_t *__restrict__ counts,
                     const int32_t *__restrict__ c_rp, const int32_t *__restrict__ c_col,
                     float *__restrict__ c_val, bool verify, int32_t *__restrict__ status) {
  extern __shared__ __align__(16) uint32_t s_mem[];
  __shared__ int4 s_seg[kValueWarps][32], s_step[kValueWarps][32];
  __shared__ int32_t s_next, s_touched, s_found;
  __shared__ float s_cum[kMaxStripes + 1];  // share of B's entries before a stripe
  const int tid = threadIdx.x, lane = lane_id(), wid = tid >> 5;
  constexpr int kThreads = kValueWarps * 32;
  WarpMem m;
  m.acc = s_mem;
  m.half = m.acc + kAcc + kThreads;
  m.seg = s_seg[wid];
  m.step = s_step[wid];
  fill_words(m.acc, kAcc, kUntouched, tid, kThreads);
  m.acc[kAcc + tid] = 0u;
  const int32_t n_front = cnt[0], n_items = n_front + cnt[1];
  const int64_t stride = ns_max + 1;
  const int32_t groups = stripe_groups(words);
  bool bad = false;
  if (tid == 0) {
    s_next = atomicAdd(head, 1);
    s_touched = s_found = 0;
    float sum = 0.0f;
    for (int t = 0; t < ns_max; ++t) {
      s_cum[t] = sum;
      sum += share[t];
    }
    s_cum[ns_max] = sum;
  }
  for (;;) {
    __syncthreads();
    const int32_t at = s_next;
    if (at >= n_items) break;
    const int4 q = items[at < n_front ? int64_t(at) : cap - 1 - (at - n_front)];
    const int32_t row = q.x, nout = q.w, before = q.z;
    if (c_rp[row + 1] - c_rp[row] != counts[row]) {  // (uniform)
      // C's row pointers are not this analysis's: the row stays as it is
      __syncthreads();  // s_next has been read
      if (tid == 0) {
        report(status, kDevCountMismatch);
        s_next = atomicAdd(head, 1);
      }
      continue;
    }
    const int32_t t0 = q.y & 0xffff, t1 = q.y >> 16;
    Item it;
    it.c0 = bound[t0] << 5;
    it.width = (bound[t1] << 5) - it.c0;
    it.p0 = op.a_rp[row];
    it.p1 = op.a_rp[row + 1];
    // this warp's stripes: about one share of the item's products, up to the
    // next warp's (each end is computed by two warps, so it is rounded once
    // and explicitly: no stripe may be taken twice or left out)
    const float first = s_cum[t0], part = (s_cum[t1] - first) * (1.0f / kValueWarps);
    auto cut = [&](int w) {
      return w == kValueWarps ? t1
                              : t0 + stripes_below(s_cum, t0, t1, __fmaf_rn(part, w, first));
    };
    it.t0 = cut(wid);
    it.t1 = cut(wid + 1);
    const int64_t out = int64_t(c_rp[row]) + before;
    const bool rank = it.width > kAcc;
    if (rank) {  // a slot an output: the bitmap, and zeroed slots
      const int64_t h = hslot[row];
      const int32_t w0 = it.c0 >> 5, w1 = w0 + (it.width >> 5);
      for (int32_t g = (w0 >> 5) + wid; (g << 5) < w1; g += kValueWarps) {
        const int32_t w = (g << 5) + lane;
        const uint32_t x = w < words ? __ldg(bits + h * words + w) : 0u;
        const int c = __popc(x), incl = warp_incl_scan(c);
        if (w >= w0 && w < w1) {
          const uint32_t o = __ldg(gpre + h * groups + g) + incl - c - before;
          const uint32_t lo = x & 0xffffu;
          *reinterpret_cast<uint2 *>(m.half + 2 * (w - w0)) =
              make_uint2(lo | o << 16, x >> 16 | (o + __popc(lo)) << 16);
        }
      }
      for (int32_t e = tid; e < nout; e += kThreads) m.acc[e] = 0u;
      if (tid == 0) m.half[it.width >> 4] = 0u;
    }
    __syncthreads();
    if (tid == 0) s_next = atomicAdd(head, 1);  // (read after the next barriers)
    if (it.t0 < it.t1) {
      if (rank) {
        walk_item<true>(op, it, m, ptr, stride, bad);
      } else {
        const int touched = warp_sum(walk_item<false>(op, it, m, ptr, stride, bad));
        if (lane == 0) atomicAdd(&s_touched, touched);
      }
    }
    __syncthreads();
    if (rank) {
      for (int32_t e = tid; e < nout; e += kThreads) {
        c_val[out + e] = __uint_as_float(m.acc[e]);
        m.acc[e] = kUntouched;
        if (verify) {
          uint32_t missing = 0;
          bad |= slot_of<true>(m, __ldg(c_col + out + e) - it.c0, it.width, missing) != e;
          bad |= missing != 0u;
        }
      }
      continue;
    }
    // a slot a column: the outputs at C's columns of these stripes, each word
    // back to untouched
    int found = 0;
    for (int32_t e0 = 0; e0 < nout; e0 += kThreads * kUnroll) {
      int32_t s[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int32_t e = e0 + kThreads * u + tid;
        s[u] = e < nout ? __ldg(c_col + out + e) - it.c0 : -1;
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        if (static_cast<uint32_t>(s[u]) < static_cast<uint32_t>(it.width)) {
          const uint32_t x = m.acc[s[u]];
          found += x != kUntouched;
          c_val[out + e0 + kThreads * u + tid] = __uint_as_float(x);
          m.acc[s[u]] = kUntouched;
        }
      }
    }
    found = warp_sum(found);
    if (lane == 0) atomicAdd(&s_found, found);
    __syncthreads();
    // every output met a product, every product an output
    const bool off = s_found != nout || s_touched != nout;
    __syncthreads();
    if (off) {
      bad = true;
      fill_words(m.acc, kAcc, kUntouched, tid, kThreads);
    }
    if (tid == 0) s_touched = s_found = 0;
  }
  if (bad) report(status, kDevKeyMissing);
}

}  // namespace

StripeShape stripe_shape(int32_t b_rows, int32_t b_cols) {
  StripeShape g;
  if (b_cols <= 1024 || b_cols > kStripeMaxCols) return g;
  g.words = (b_cols + 31) >> 5;
  g.ns_max = kStripeShares + (g.words + kStripeWords - 1) / kStripeWords;
  g.on = size_t(b_rows) * size_t(g.ns_max + 1) * sizeof(int32_t) <= kStripeTableMax;
  return g;
}

void launch_stripe_table(const StripeShape &g, int32_t b_rows, const int32_t *b_rp,
                         const int32_t *b_col, int32_t *hist, int32_t *bound, float *share,
                         int32_t *ptr, int num_sms, cudaStream_t s) {
  const size_t words = static_cast<size_t>(g.words);
  cudaMemsetAsync(hist, 0, words * sizeof(int32_t), s);
  stripe_hist_kernel<<<num_sms, 512, words * sizeof(int32_t), s>>>(b_rp, b_rows, b_col, g.words,
                                                                   hist);
  stripe_bounds_kernel<<<1, 1024, 0, s>>>(g.words, g.ns_max, hist, bound, share);
  int grid = num_sms * 8;
  const int need = (b_rows + kPtrThreads / 32 - 1) / (kPtrThreads / 32);
  if (grid > need) grid = need;
  stripe_ptr_kernel<<<grid, kPtrThreads, 0, s>>>(b_rows, b_rp, b_col, g.ns_max, bound, ptr);
}

size_t stripe_tasks(int32_t nrows) { return size_t(kSplitTasks) + size_t(nrows); }

void launch_stripe_count(const StripeShape &g, const Operands &op, const int32_t *rows,
                         int32_t nrows, const int64_t *ops, const int32_t *bound, int2 *tasks,
                         int32_t *cnt, int32_t *done, int32_t *counts, int32_t *hslot,
                         uint32_t *bits, int32_t *gpre, int32_t *soff, int num_sms,
                         cudaStream_t s) {
  if (nrows <= 0) return;
  const size_t smem = (size_t(stripe_groups(g.words)) * 33 + 1) * sizeof(uint32_t);
  int per_sm = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, stripe_count_kernel, kCountThreads,
                                                    smem) != cudaSuccess ||
      per_sm < 1)
    per_sm = 1;
  cudaMemsetAsync(cnt, 0, 3 * sizeof(int32_t), s);
  stripe_tasks_kernel<<<(nrows + 127) / 128, 128, 0, s>>>(rows, nrows, ops, g.words, bits, tasks,
                                                          cnt, done);
  const int64_t want = int64_t(num_sms) * per_sm, most = int64_t(stripe_tasks(nrows));
  stripe_count_kernel<<<static_cast<int>(most < want ? most : want), kCountThreads, smem, s>>>(
      op, rows, nrows, g.words, g.ns_max, bound, tasks, cnt, done, counts, hslot, bits, gpre,
      soff, cnt + 2);
}

void launch_stripe_items(const StripeShape &g, const int32_t *rows, int32_t nrows,
                         const int64_t *ops, const int32_t *hslot, const int32_t *soff,
                         const int32_t *bound, const float *share, int4 *items, int64_t cap,
                         int32_t *cnt, cudaStream_t s) {
  if (nrows <= 0) return;
  cudaMemsetAsync(cnt, 0, 2 * sizeof(int32_t), s);
  stripe_items_kernel<<<(nrows + kItemRows - 1) / kItemRows, kItemRows, 0, s>>>(
      rows, nrows, ops, hslot, soff, g.ns_max, bound, share, items, cap, cnt);
}

void launch_stripe_columns(const StripeShape &g, const int32_t *rows, int32_t nrows,
                           const int32_t *hslot, const uint32_t *bits, const int32_t *gpre,
                           const int32_t *soff, const int32_t *c_rp, int32_t *c_col,
                           int32_t *status, cudaStream_t s) {
  if (nrows <= 0) return;
  stripe_columns_kernel<<<nrows, kColumnWarps * 32, 0, s>>>(rows, hslot, bits, gpre, soff, g.ns_max,
                                                        g.words, c_rp, c_col, status);
}

void launch_stripe_values(const StripeShape &g, const Operands &op, int32_t nrows,
                          const int4 *items, int64_t cap, const int32_t *cnt, int32_t *head,
                          const int32_t *bound, const float *share, const int32_t *ptr,
                          const int32_t *hslot, const uint32_t *bits, const int32_t *gpre,
                          const int32_t *counts, const int32_t *c_rp, const int32_t *c_col,
                          float *c_val, bool verify, int32_t *status, int num_sms,
                          cudaStream_t s) {
  if (nrows <= 0) return;
  int32_t item_words = g.words < kItemWords ? g.words : kItemWords;
  item_words = (item_words + 7) & ~7;
  const size_t smem = value_bytes(item_words);
  cudaFuncSetAttribute(stripe_values_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       static_cast<int>(smem));
  int per_sm = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, stripe_values_kernel,
                                                    kValueWarps * 32, smem) != cudaSuccess ||
      per_sm < 1)
    per_sm = 1;
  cudaMemsetAsync(head, 0, sizeof(int32_t), s);
  stripe_values_kernel<<<num_sms * per_sm, kValueWarps * 32, smem, s>>>(
      op, items, cap, cnt, head, g.ns_max, bound, share, ptr, hslot, bits, gpre, g.words,
      item_words, counts, c_rp, c_col, c_val, verify, status);
}

}  // namespace rvsp

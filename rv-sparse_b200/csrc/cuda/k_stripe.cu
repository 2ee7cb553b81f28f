// Stripe rows: heavy rows (more than 1024 outputs possible) with enough
// products to be cut by columns, for B of at most kStripeMaxCols columns.
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
//   count     a block per row marks the row's columns in a shared-memory
//             bitmap (no order needed), keeps the bitmap and the outputs
//             before each stripe;
//   items     (row, stripes [t0, t1)): as many stripes as fit the accumulator
//             and about kItemOps products, so a hub row is many items and a
//             row of a few thousand products one per kStripeCols columns;
//             rows of many products are drawn first;
//   values    persistent warps draw items; per item a warp expands its
//             products 32 at a time in flattened order (ascending A nonzero,
//             then column) into a dense accumulator over the item's columns,
//             equal columns within the 32 in lane order, then gathers the
//             accumulator at C's columns.
//
// Each output is the sum of its terms in ascending A-nonzero order from
// +0.0f, products and sums rounded separately (gustavson_core_f32.inc:31-62
// with accum_scalar_f32.c:20-71); the columns are the row's bitmap in order
// (rvsp_symbolic.c:91-137).
//
// An accumulator word starts as kUntouched, a NaN pattern that no addition
// returns (results that are NaN are the canonical one), so a product whose
// column is not in C, or a column of C without a product, is seen: the counts
// of first touches and of outputs differ, or a gathered word is untouched.
#include <climits>

#include "device_common.cuh"
#include "kernels.cuh"

namespace rvsp {

namespace {

constexpr int kStripeCols = 4096;   // columns of a warp's accumulator (16 KB)
constexpr int kStripeWords = kStripeCols / 32;
constexpr int kStripeShares = 32;   // equal shares of B's entries
constexpr int kItemOps = 8192;      // products an item aims at
constexpr int kBigRowOps = 1 << 18; // rows whose items are drawn first
constexpr size_t kStripeTableMax = size_t(256) << 20;

constexpr int kCountThreads = 256;
constexpr int kCountWarps = kCountThreads / 32;
constexpr int kValueWarps = 2;      // warps a block of the value kernel
constexpr int kUnroll = 4;          // 32-product batches in flight a warp
constexpr uint32_t kUntouched = 0xffffffffu;

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
// last), share[t] = its part of B's entries, of_word[w] = the stripe of word w.
// words <= 4096: thread i owns words [4 i, 4 i + 4).
__global__ void __launch_bounds__(1024)
stripe_bounds_kernel(int32_t words, int32_t ns_max, const int32_t *__restrict__ hist,
                     int32_t *__restrict__ bound, float *__restrict__ share,
                     uint8_t *__restrict__ of_word) {
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
    const int w = threadIdx.x * 4 + i;
    if (open[i]) {
      s_bound[at] = w;
      s_mass[at] = mass[i];
      ++at;
    }
    if (w < words) of_word[w] = static_cast<uint8_t>(at - 1);
  }
  __syncthreads();
  for (int t = threadIdx.x; t <= ns_max; t += blockDim.x) {
    bound[t] = s_bound[t];
    if (t < ns_max)
      share[t] = t < ns ? float(s_mass[t + 1] - s_mass[t]) / float(total) : 0.0f;
  }
}

// ptr[k * (ns_max + 1) + t] = first entry of B row k in stripe t or after it
// (the row's end for t = ns_max).  A warp per row, its pointers gathered in
// shared memory and written together.
__global__ void __launch_bounds__(kCountThreads)
stripe_ptr_kernel(int32_t b_rows, const int32_t *__restrict__ b_rp,
                  const int32_t *__restrict__ b_col, int32_t words, int32_t ns_max,
                  const uint8_t *__restrict__ of_word, int32_t *__restrict__ ptr) {
  extern __shared__ uint8_t s_of[];
  __shared__ int32_t s_row[kCountWarps][kMaxStripes + 1];
  for (int w = threadIdx.x; w < words; w += blockDim.x) s_of[w] = of_word[w];
  __syncthreads();
  const int lane = lane_id();
  int32_t *buf = s_row[threadIdx.x >> 5];
  const int32_t step = (gridDim.x * blockDim.x) >> 5;
  for (int32_t k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < b_rows; k += step) {
    const int32_t b0 = b_rp[k], b1 = b_rp[k + 1];
    for (int t = lane; t <= ns_max; t += 32) buf[t] = b1;
    __syncwarp();
    for (int32_t e = b0 + lane; e < b1; e += 32) {
      const int s = s_of[__ldg(b_col + e) >> 5];
      const int p = e > b0 ? s_of[__ldg(b_col + e - 1) >> 5] : -1;
      for (int t = p + 1; t <= s; ++t) buf[t] = e;
    }
    __syncwarp();
    for (int t = lane; t <= ns_max; t += 32) ptr[int64_t(k) * (ns_max + 1) + t] = buf[t];
    __syncwarp();
  }
}

// ---- expanding products ---------------------------------------------------------

// Up to 32 runs of B entries, one per lane ([beg, beg + len), scaled by a),
// expanded in order.  The non-empty runs are compacted into shared memory;
// the run of flattened product t is then a population count over the mask of
// the runs that start in the 32 products around it.
struct Runs {
  int32_t excl;   // products before this lane's run
  int32_t len;
  int32_t total;  // products of the chunk (uniform)
  int started;    // non-empty runs that start before the next batch (uniform)
};

__device__ __forceinline__ Runs open_runs(int2 *seg, int32_t beg, int32_t len, float a) {
  Runs r;
  const int32_t incl = warp_incl_scan(len);
  r.excl = incl - len;
  r.len = len;
  r.total = __shfl_sync(kFull, incl, 31);
  r.started = 0;
  const unsigned some = __ballot_sync(kFull, len > 0);
  __syncwarp();  // the chunk before has been read
  if (len > 0) seg[__popc(some & lanemask_lt())] = make_int2(beg - r.excl, __float_as_int(a));
  __syncwarp();
  return r;
}

// The B entry (and run's a) of product t0 + lane; t0 advances by 32 a call.
// solo: the batch's products come from one run (uniform).
__device__ __forceinline__ bool next_batch(Runs &r, const int2 *seg, int32_t t0, int32_t &entry,
                                           float &a, bool &solo) {
  const int32_t d = r.excl - t0;
  const unsigned bit = (r.len > 0 && d >= 0 && d < 32) ? 1u << d : 0u;
  const unsigned starts = __reduce_or_sync(kFull, bit);
  const int own = r.started + __popc(starts & (lanemask_lt() * 2u + 1u)) - 1;
  r.started += __popc(starts);
  solo = (starts & ~1u) == 0u;
  const int32_t t = t0 + lane_id();
  const bool v = t < r.total;
  const int2 sg = seg[v ? own : 0];
  entry = sg.x + t;
  a = __int_as_float(sg.y);
  return v;
}

// ---- count ------------------------------------------------------------------------

// rows[r]: counts[row], hslot[row] = r, the row's bitmap at bits + r * words
// and the outputs before stripe t at soff[r * (ns_max + 1) + t].
__global__ void __launch_bounds__(kCountThreads)
stripe_count_kernel(Operands op, const int32_t *__restrict__ rows, int32_t nrows,
                    int32_t words, int32_t ns_max, const int32_t *__restrict__ bound,
                    int32_t *__restrict__ counts, int32_t *__restrict__ hslot,
                    uint32_t *__restrict__ bits_out, int32_t *__restrict__ soff,
                    int32_t *__restrict__ head) {
  extern __shared__ __align__(16) uint32_t s_mem[];
  uint32_t *bits = s_mem;
  int32_t *pre = reinterpret_cast<int32_t *>(s_mem + words);
  __shared__ int2 s_seg[kCountWarps][32];
  __shared__ int32_t s_row, s_chunk, s_sum[kCountWarps];
  const int tid = threadIdx.x, lane = lane_id(), wid = tid >> 5;
  int2 *seg = s_seg[wid];
  for (;;) {
    __syncthreads();
    if (tid == 0) {
      s_row = atomicAdd(head, 1);
      s_chunk = 0;
    }
    for (int w = tid; w < words; w += kCountThreads) bits[w] = 0u;
    __syncthreads();
    const int32_t r = s_row;
    if (r >= nrows) return;
    const int32_t row = row_of(rows, r);
    const int32_t p0 = op.a_rp[row], p1 = op.a_rp[row + 1];
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
        for (int u = 0; u < kUnroll; ++u) {
          if (col[u] >= 0) {
            uint32_t *wp = bits + (col[u] >> 5);
            const uint32_t bit = 1u << (col[u] & 31);
            if (!(*reinterpret_cast<volatile uint32_t *>(wp) & bit)) atomicOr(wp, bit);
          }
        }
      }
    }
    __syncthreads();
    // Prefix of the words' bit counts: warp i over its run of words.
    const int32_t per = ((words + kCountWarps - 1) / kCountWarps + 31) & ~31;
    const int32_t w0 = min(wid * per, words), w1 = min(w0 + per, words);
    int sum = 0;
    for (int32_t w = w0 + lane; w < w1; w += 32) sum += __popc(bits[w]);
    sum = warp_sum(sum);
    if (lane == 0) s_sum[wid] = sum;
    __syncthreads();
    int base = 0, total = 0;
#pragma unroll
    for (int i = 0; i < kCountWarps; ++i) {
      if (i < wid) base += s_sum[i];
      total += s_sum[i];
    }
    for (int32_t w = w0; w < w1; w += 32) {
      const uint32_t x = w + lane < w1 ? bits[w + lane] : 0u;
      const int c = __popc(x), incl = warp_incl_scan(c);
      if (w + lane < w1) {
        pre[w + lane] = base + incl - c;
        bits_out[int64_t(r) * words + w + lane] = x;
      }
      base += __shfl_sync(kFull, incl, 31);
    }
    __syncthreads();
    for (int t = tid; t <= ns_max; t += kCountThreads) {
      const int32_t b = bound[t];
      soff[int64_t(r) * (ns_max + 1) + t] = b < words ? pre[b] : total;
    }
    if (tid == 0) {
      counts[row] = total;
      hslot[row] = r;
    }
  }
}

// ---- items ------------------------------------------------------------------------

// One thread per row: its runs of stripes.  Items of rows of at least
// kBigRowOps products fill items[] from the front (cnt[0]), the others from
// the back (cnt[1]).  item = (row, t0 | t1 << 16, outputs before, outputs).
__global__ void __launch_bounds__(128)
stripe_items_kernel(const int32_t *__restrict__ rows, int32_t nrows,
                    const int64_t *__restrict__ ops, const int32_t *__restrict__ hslot,
                    const int32_t *__restrict__ soff, int32_t ns_max,
                    const int32_t *__restrict__ bound, const float *__restrict__ share,
                    int4 *__restrict__ items, int64_t cap, int32_t *__restrict__ cnt) {
  const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nrows) return;
  const int32_t row = row_of(rows, i);
  const int32_t *so = soff + int64_t(hslot[row]) * (ns_max + 1);
  const float work = static_cast<float>(ops[row]);
  const bool big = work >= float(kBigRowOps);
  int64_t at = 0;
  for (int pass = 0; pass < 2; ++pass) {
    int n = 0;
    for (int t0 = 0; t0 < ns_max;) {
      const int32_t w0 = bound[t0];
      int t1 = t0 + 1;
      float part = work * share[t0];
      while (t1 < ns_max && bound[t1 + 1] - w0 <= kStripeWords &&
             part + work * share[t1] <= float(kItemOps)) {
        part += work * share[t1];
        ++t1;
      }
      const int32_t o = so[t0], m = so[t1] - o;
      if (m > 0) {
        if (pass) {
          const int64_t q = at + n;
          items[big ? q : cap - 1 - q] = make_int4(row, t0 | (t1 << 16), o, m);
        }
        ++n;
      }
      t0 = t1;
    }
    if (!pass) at = atomicAdd(&cnt[big ? 0 : 1], n);
  }
}

// ---- columns ----------------------------------------------------------------------

__global__ void __launch_bounds__(kCountThreads)
stripe_columns_kernel(const int32_t *__restrict__ rows, const int32_t *__restrict__ hslot,
                      const uint32_t *__restrict__ bits_in, int32_t words,
                      const int32_t *__restrict__ c_rp, int32_t *__restrict__ c_col,
                      int32_t *__restrict__ status) {
  __shared__ int32_t s_sum[kCountWarps];
  const int lane = lane_id(), wid = threadIdx.x >> 5;
  const int32_t row = row_of(rows, blockIdx.x);
  const uint32_t *bits = bits_in + int64_t(hslot[row]) * words;
  const int32_t c0 = c_rp[row], m = c_rp[row + 1] - c0;
  const int32_t per = ((words + kCountWarps - 1) / kCountWarps + 31) & ~31;
  const int32_t w0 = min(wid * per, words), w1 = min(w0 + per, words);
  int sum = 0;
  for (int32_t w = w0 + lane; w < w1; w += 32) sum += __popc(__ldg(bits + w));
  sum = warp_sum(sum);
  if (lane == 0) s_sum[wid] = sum;
  __syncthreads();
  int base = 0, total = 0;
#pragma unroll
  for (int i = 0; i < kCountWarps; ++i) {
    if (i < wid) base += s_sum[i];
    total += s_sum[i];
  }
  if (total != m) {  // C's row pointers are not this analysis's
    if (threadIdx.x == 0) report(status, kDevCountMismatch);
    return;
  }
  int32_t *out = c_col + c0;
  for (int32_t w = w0; w < w1; w += 32) {
    const uint32_t x = w + lane < w1 ? __ldg(bits + w + lane) : 0u;
    const int c = __popc(x), incl = warp_incl_scan(c);
    unsigned some = __ballot_sync(kFull, x != 0u);
    while (some) {
      const int j = __ffs(some) - 1;
      some &= some - 1u;
      const uint32_t word = __shfl_sync(kFull, x, j);
      const int at = base + __shfl_sync(kFull, incl - c, j);
      if ((word >> lane) & 1u)
        out[at + __popc(word & lanemask_lt())] = ((w + j) << 5) + lane;
    }
    base += __shfl_sync(kFull, incl, 31);
  }
}

// ---- values -----------------------------------------------------------------------

// acc[slot] += term for the valid lanes, equal slots in lane order; returns
// the slots this lane touched first.
__device__ __forceinline__ int apply_batch(uint32_t *acc, bool v, int slot, float term,
                                           bool solo) {
  int first = 0;
  if (solo) {  // one B row: distinct columns
    if (v) {
      const uint32_t old = acc[slot];
      first = old == kUntouched;
      acc[slot] = __float_as_uint(__fadd_rn(first ? 0.0f : __uint_as_float(old), term));
    }
  } else {
    const int lane = lane_id();
    const unsigned peers = __match_any_sync(kFull, v ? slot : -1 - lane);
    unsigned rest = peers & ~lanemask_lt() & ~(1u << lane);  // the group's later lanes
    const bool leader = v && (peers & lanemask_lt()) == 0u;
    float a = 0.0f;
    if (leader) {
      const uint32_t old = acc[slot];
      first = old == kUntouched;
      a = __fadd_rn(first ? 0.0f : __uint_as_float(old), term);
    }
    if (!leader) rest = 0u;
    while (__any_sync(kFull, rest != 0u)) {
      const float t = __shfl_sync(kFull, term, rest ? __ffs(rest) - 1 : lane);
      if (rest) {
        a = __fadd_rn(a, t);
        rest &= rest - 1u;
      }
    }
    if (leader) acc[slot] = __float_as_uint(a);
  }
  __syncwarp();
  return first;
}

__global__ void __launch_bounds__(kValueWarps * 32)
stripe_values_kernel(Operands op, const int4 *__restrict__ items, int64_t cap,
                     const int32_t *__restrict__ cnt, int32_t *__restrict__ head,
                     int32_t ns_max, const int32_t *__restrict__ bound,
                     const int32_t *__restrict__ ptr, const int32_t *__restrict__ c_rp,
                     const int32_t *__restrict__ c_col, float *__restrict__ c_val,
                     int32_t *__restrict__ status) {
  extern __shared__ __align__(16) uint32_t s_acc[];
  __shared__ int2 s_seg[kValueWarps][32];
  const int lane = lane_id(), wid = threadIdx.x >> 5;
  uint32_t *acc = s_acc + wid * kStripeCols;
  int2 *seg = s_seg[wid];
  fill_words(acc, kStripeCols, kUntouched, lane, 32);
  __syncwarp();
  const int32_t n_front = cnt[0], n_items = n_front + cnt[1];
  const int64_t stride = ns_max + 1;
  bool bad = false;
  auto draw = [&]() {
    int32_t i = 0;
    if (lane == 0) i = atomicAdd(head, 1);
    return __shfl_sync(kFull, i, 0);
  };
  int32_t next = draw();
  while (next < n_items) {
    const int4 it = items[next < n_front ? int64_t(next) : cap - 1 - (next - n_front)];
    next = draw();  // (its answer is back by the end of this item)
    const int32_t row = it.x, t0 = it.y & 0xffff, t1 = it.y >> 16;
    const int32_t c0 = bound[t0] << 5;
    const int32_t width = (bound[t1] << 5) - c0;
    const int32_t p1 = op.a_rp[row + 1];
    int touched = 0;
    for (int32_t p = op.a_rp[row]; p < p1; p += 32) {
      int32_t beg = 0, len = 0;
      float a = 0.0f;
      if (p + lane < p1) {
        const int64_t k = __ldg(op.a_col + p + lane) * stride;
        a = __ldg(op.a_val + p + lane);
        beg = __ldg(ptr + k + t0);
        len = __ldg(ptr + k + t1) - beg;
      }
      Runs run = open_runs(seg, beg, len, a);
      for (int32_t t = 0; t < run.total; t += 32 * kUnroll) {
        int32_t slot[kUnroll];
        float term[kUnroll];
        bool solo[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
          int32_t e;
          float x;
          const bool v = next_batch(run, seg, t + 32 * u, e, x, solo[u]);
          slot[u] = -1;
          term[u] = 0.0f;
          if (v) {
            slot[u] = __ldg(op.b_col + e) - c0;
            term[u] = __fmul_rn(x, __ldg(op.b_val + e));
          }
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
          if (t + 32 * u >= run.total) break;
          // (outside the item's columns: B is not the analysed one)
          const bool in = static_cast<uint32_t>(slot[u]) < static_cast<uint32_t>(width);
          if (slot[u] != -1 && !in) bad = true;
          touched += apply_batch(acc, in, slot[u], term[u], solo[u]);
        }
      }
    }
    // the outputs: C's columns of these stripes, each word back to untouched
    const int64_t out = int64_t(c_rp[row]) + it.z;
    int found = 0;
    for (int32_t e0 = 0; e0 < it.w; e0 += 32 * kUnroll) {
      int32_t s[kUnroll];
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int32_t e = e0 + 32 * u + lane;
        s[u] = e < it.w ? __ldg(c_col + out + e) - c0 : -1;
      }
#pragma unroll
      for (int u = 0; u < kUnroll; ++u) {
        const int32_t e = e0 + 32 * u + lane;
        if (static_cast<uint32_t>(s[u]) < static_cast<uint32_t>(width)) {
          const uint32_t x = acc[s[u]];
          found += x != kUntouched;
          c_val[out + e] = __uint_as_float(x);
          acc[s[u]] = kUntouched;
        }
      }
    }
    __syncwarp();
    // every output met a product, every product an output
    if (warp_sum(found) != it.w || warp_sum(touched) != it.w) {
      bad = true;
      fill_words(acc, kStripeCols, kUntouched, lane, 32);
      __syncwarp();
    }
  }
  if (bad) report(status, kDevKeyMissing);
}

}  // namespace

StripeShape stripe_shape(int32_t b_rows, int32_t b_cols) {
  StripeShape g;
  if (b_cols <= 1024 || b_cols > kStripeMaxCols) return g;
  g.words = (b_cols + 31) >> 5;
  const int32_t accs = (g.words + kStripeWords - 1) / kStripeWords;
  g.ns_max = kStripeShares + accs;
  if (size_t(b_rows) * size_t(g.ns_max + 1) * sizeof(int32_t) > kStripeTableMax) return g;
  g.min_ops = 256 * int64_t(accs) > 2048 ? 256 * int64_t(accs) : 2048;
  return g;
}

void launch_stripe_table(const StripeShape &g, int32_t b_rows, const int32_t *b_rp,
                         const int32_t *b_col, int32_t *hist, int32_t *bound, float *share,
                         uint8_t *of_word, int32_t *ptr, int num_sms, cudaStream_t s) {
  const size_t words = static_cast<size_t>(g.words);
  cudaMemsetAsync(hist, 0, words * sizeof(int32_t), s);
  stripe_hist_kernel<<<num_sms, 512, words * sizeof(int32_t), s>>>(b_rp, b_rows, b_col, g.words,
                                                                   hist);
  stripe_bounds_kernel<<<1, 1024, 0, s>>>(g.words, g.ns_max, hist, bound, share, of_word);
  int grid = num_sms * 8;
  const int need = (b_rows + kCountWarps - 1) / kCountWarps;
  if (grid > need) grid = need;
  stripe_ptr_kernel<<<grid, kCountThreads, words, s>>>(b_rows, b_rp, b_col, g.words, g.ns_max,
                                                       of_word, ptr);
}

void launch_stripe_count(const StripeShape &g, const Operands &op, const int32_t *rows,
                         int32_t nrows, const int32_t *bound, int32_t *counts,
                         int32_t *hslot, uint32_t *bits, int32_t *soff, int32_t *head,
                         int num_sms, cudaStream_t s) {
  if (nrows <= 0) return;
  const size_t smem = size_t(g.words) * 2 * sizeof(uint32_t);
  int per_sm = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, stripe_count_kernel, kCountThreads,
                                                    smem) != cudaSuccess ||
      per_sm < 1)
    per_sm = 1;
  const int64_t want = int64_t(num_sms) * per_sm;
  const int grid = nrows < want ? nrows : static_cast<int>(want);
  cudaMemsetAsync(head, 0, sizeof(int32_t), s);
  stripe_count_kernel<<<grid, kCountThreads, smem, s>>>(op, rows, nrows, g.words, g.ns_max,
                                                        bound, counts, hslot, bits, soff, head);
}

void launch_stripe_items(const StripeShape &g, const int32_t *rows, int32_t nrows,
                         const int64_t *ops, const int32_t *hslot, const int32_t *soff,
                         const int32_t *bound, const float *share, int4 *items, int64_t cap,
                         int32_t *cnt, cudaStream_t s) {
  if (nrows <= 0) return;
  cudaMemsetAsync(cnt, 0, 2 * sizeof(int32_t), s);
  stripe_items_kernel<<<(nrows + 127) / 128, 128, 0, s>>>(rows, nrows, ops, hslot, soff,
                                                          g.ns_max, bound, share, items, cap,
                                                          cnt);
}

void launch_stripe_columns(const StripeShape &g, const int32_t *rows, int32_t nrows,
                           const int32_t *hslot, const uint32_t *bits, const int32_t *c_rp,
                           int32_t *c_col, int32_t *status, cudaStream_t s) {
  if (nrows <= 0) return;
  stripe_columns_kernel<<<nrows, kCountThreads, 0, s>>>(rows, hslot, bits, g.words, c_rp, c_col,
                                                        status);
}

void launch_stripe_values(const StripeShape &g, const Operands &op, int32_t nrows,
                          const int4 *items, int64_t cap, const int32_t *cnt, int32_t *head,
                          const int32_t *bound, const int32_t *ptr, const int32_t *c_rp,
                          const int32_t *c_col, float *c_val, int32_t *status, int num_sms,
                          cudaStream_t s) {
  if (nrows <= 0) return;
  const size_t smem = size_t(kValueWarps) * kStripeCols * sizeof(float);
  cudaFuncSetAttribute(stripe_values_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       static_cast<int>(smem));
  int per_sm = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, stripe_values_kernel,
                                                    kValueWarps * 32, smem) != cudaSuccess ||
      per_sm < 1)
    per_sm = 1;
  cudaMemsetAsync(head, 0, sizeof(int32_t), s);
  stripe_values_kernel<<<num_sms * per_sm, kValueWarps * 32, smem, s>>>(
      op, items, cap, cnt, head, g.ns_max, bound, ptr, c_rp, c_col, c_val, status);
}

}  // namespace rvsp

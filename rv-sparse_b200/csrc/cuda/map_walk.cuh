// The map walk of one row (k_reuse.cu), shared with the persistent numeric
// kernel (k_persist.cu): C's row values from the reuse map, one warp, into a
// shared-memory accumulator of at least the row's C length and a word a lane.
// Each output gets its terms in ascending A-nonzero order from +0.0f, rounded
// separately: stepping (one A nonzero at a time, lanes over its B row, whose
// positions are distinct) for all but the shortest B rows, flattened tiles with
// ordered_apply for those.  The walk waits on loads: the map and the values of
// kMapUnroll steps are loaded together before the first of them is applied.
// Repeat of a 48-product batch: 1.65 -> 1.42 ms; uniform rows of six to eight
// entries, stepped instead of tiled, 1.2 times as fast.
#pragma once

#include "device_common.cuh"
#include "kernels.cuh"

namespace rvsp {

constexpr int kMapSteppingMinAvgLen = 6;
constexpr int kMapUnroll = 4;

// Floats of a row's accumulator: its outputs, then a word a lane for lanes
// without a product.
__host__ __device__ constexpr int map_acc_floats(int outputs) {
  return ((outputs + 3) & ~3) + 32;
}

// seg: 32 entries of the warp's own shared memory; acc: map_acc_floats(cap),
// cap at least the row's outputs.
__device__ __forceinline__ void map_numeric_row(const Operands &op,
                                                const int64_t *__restrict__ ops, int32_t row,
                                                const int32_t *__restrict__ c_rp,
                                                float *__restrict__ c_val,
                                                const int64_t *__restrict__ moff,
                                                const uint16_t *__restrict__ map,
                                                int32_t *__restrict__ status, float *acc,
                                                int cap, int4 *seg, int lane) {
  const int32_t cs = c_rp[row];
  const int m = c_rp[row + 1] - cs;
  const uint16_t *mp = map + moff[row];
  const int32_t p0 = op.a_rp[row], p1 = op.a_rp[row + 1];
  const bool stepping =
      ops[row] >= static_cast<int64_t>(kMapSteppingMinAvgLen) * (p1 - p0);
  for (int e = lane; e < m; e += 32) acc[e] = 0.0f;
  const int spare = map_acc_floats(cap) - 32 + lane;
  acc[spare] = 0.0f;
  __syncwarp();
  bool bad = false;
  for (int32_t p = p0; p < p1; p += 32) {
    const AChunk c = load_chunk(op.a_col, op.a_val, op.b_rp, p + lane, p1, true);
    if (stepping) {
      seg[lane] = make_int4(c.bbeg, c.len, __float_as_int(c.a), c.incl - c.len);
      __syncwarp();
      const int cnt = min(32, p1 - p);
      for (int j = 0; j < cnt; j += kMapUnroll) {  // (past cnt: empty B rows)
        // (shared memory bounds the walk: each entry of seg is read once)
        int pos[kMapUnroll], len[kMapUnroll];
        float val[kMapUnroll], a[kMapUnroll];
#pragma unroll
        for (int u = 0; u < kMapUnroll; ++u) {
          const int4 s = seg[j + u];
          len[u] = s.y;
          a[u] = __int_as_float(s.z);
          pos[u] = spare;
          val[u] = 0.0f;
          if (lane < s.y) {
            pos[u] = __ldg(mp + s.w + lane);
            val[u] = __ldg(op.b_val + s.x + lane);
          }
        }
#pragma unroll
        for (int u = 0; u < kMapUnroll; ++u) {
          if (pos[u] >= m && pos[u] != spare) {  // C is not this product's
            bad = true;
            pos[u] = spare;
          }
          acc[pos[u]] = __fadd_rn(acc[pos[u]], __fmul_rn(a[u], val[u]));
          if (len[u] > 32) {
            const int4 s = seg[j + u];
            for (int e = 32 + lane; e < s.y; e += 32) {
              const int q = __ldg(mp + s.w + e);
              const float term = __fmul_rn(a[u], __ldg(op.b_val + s.x + e));
              if (q < m) acc[q] = __fadd_rn(acc[q], term);
              else bad = true;
            }
          }
          __syncwarp();
        }
      }
    } else {
      for (int t0 = 0; t0 < c.total; t0 += 32) {
        const int t = t0 + lane;
        bool v = t < c.total;
        const int j = warp_owner_of(c.incl, v ? t : 0);
        const int excl = __shfl_sync(kFull, c.incl - c.len, j);
        const int bbeg = __shfl_sync(kFull, c.bbeg, j);
        const float a = __shfl_sync(kFull, c.a, j);
        int pos = 0;
        float term = 0.0f;
        if (v) {
          pos = __ldg(mp + t);
          if (pos >= m) {
            bad = true;
            v = false;
          } else {
            term = __fmul_rn(a, __ldg(op.b_val + bbeg + (t - excl)));
          }
        }
        ordered_apply(acc, v, pos, term);
      }
    }
    mp += c.total;
  }
  __syncwarp();
  for (int e = lane; e < m; e += 32) c_val[cs + e] = acc[e];
  if (__any_sync(kFull, bad) && lane == 0) report(status, kDevKeyMissing);
}

}  // namespace rvsp

// When the stripe kernels (k_stripe.cu) pay for a product's heavy rows, the rows
// of more than 1024 possible outputs.
//
// The block-per-row kernels (k_heavy.cu) give every row a block of 16 warps at
// once, so a few rows take as long as the longest: some 45 us and 2.6 ns a
// product.  Stripes first take a histogram of B and the stripes' starts in
// every B row (20 us for 2000 rows of B, 90 for 100,000), and four warps an
// item that each read all of the row's A nonzeros, for every item of it.  So
// they pay in two ways, each measured both ways on one B200 with rows of 150 to
// 10,000 entries among light ones, B rows of 8 and of 30 entries, and on R-MAT
// graphs:
//
//   many rows   throughput: about 4.5 ps a product and 50 ps an A nonzero
//               against 16 ps a product, if that covers the fixed part, and
//               if the B rows are long enough beside the items a row is cut
//               into by its outputs.  1000 rows of 10,000 entries, B rows of 8,
//               in ms, blocks / stripes: 100,000 columns (16 items a row) 5.3 /
//               9.4, 10,000 columns (3 items) 2.1 / 1.7; R-MAT 2^11 (600 rows)
//               0.35 / 0.32, 2^12 0.83 / 0.42, 2^15 5.3 / 1.7.
//   long rows   the longest row is cut: one row of 90,000 products, B rows of 30,
//               0.70 / 0.52, of 300,000 1.41 / 0.70; of 80,000, B rows of 8,
//               0.54 / 0.64.
//
// A batch is made to be repeated: 48 products of 256 to 65536 rows repeat in 1.41
// ms with stripes and 1.56 without, though their starts alone (0.5 M rows of B)
// cost a product more than it gains.  Where neither holds: 100 rows of 1000
// entries, B rows of 8, 10,000 columns, product 0.22 / 0.33, repeat 0.07 / 0.11.
#pragma once

#include <cmath>
#include <cstdint>

namespace rvsp {

constexpr int kStripeAcc = 4096;        // accumulator slots of an item
constexpr int kStripeItemOps = 32768;   // products an item aims at
constexpr int kStripeManyRows = 256;    // rows that fill the SMs with blocks

// Over the heavy rows of a product: how many, their products and A nonzeros, and
// the products of the longest.
struct HeavyRows {
  unsigned long long rows, ops, nnz, most;
};

// The outputs of a row of ops products with columns at random.
__host__ __device__ inline float expected_outputs(float ops, float cols) {
  return cols * (1.0f - expf(-ops / cols));
}

// repeats: for numeric-only repeats, whose stripes are there.
__host__ __device__ inline bool stripes_pay(const HeavyRows &h, int32_t b_rows, int32_t b_cols,
                                            bool repeats = false) {
  if (h.rows == 0 || h.nnz == 0) return false;
  const float ops = static_cast<float>(h.ops), nnz = static_cast<float>(h.nnz);
  const float cols = static_cast<float>(b_cols), run = ops / nnz;
  const float outputs = expected_outputs(ops / static_cast<float>(h.rows), cols);
  const bool runs_long = outputs <= kStripeAcc || run * kStripeAcc >= 1.75f * outputs;
  const float gain = 11.5f * ops - 50.0f * nnz;  // ps
  const float fixed = repeats ? 6e6f : 12e6f + 350.0f * b_rows;
  if (h.rows >= kStripeManyRows && runs_long && gain >= fixed) return true;
  const float most = static_cast<float>(h.most);
  const bool cut =
      most >= 2.0f * kStripeItemOps || expected_outputs(most, cols) >= 2.0f * kStripeAcc;
  return run >= 16.0f && cut && most >= 16384.0f + 0.125f * cols;
}

}  // namespace rvsp

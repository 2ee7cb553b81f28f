// The entries of a Matrix Market text, parsed on the GPU, to canonical CSR.
//
// The tokens after the size line are numbered in file order; token g is field
// g % F of entry g / F (F = 2 for a pattern file, else 3), as fscanf's "%d %d
// %f" reads them while every conversion consumes its whole token
// (tools/src/mtx_to_csr_formatter.c:196-219 in the reference).  Two kernels
// over chunks of 4096 bytes: the first counts the tokens that start in each
// chunk, the second numbers them by the scan of those counts and converts.
//
// Values must be strtof's, bit for bit.  A decimal w * 10^e with w < 10^19 is
// converted in doubles with at most four roundings (w, and one per factor of
// up to 10^22, which a double holds exactly; digits after the 19th are left
// off), so the true value lies within d (1 -+ 2^-50); if both ends of the
// wider d (1 -+ 2^-49) round to the same float, rounding being monotone, so
// does the true value (the argument of Clinger's fast path, PLDI 1990).  Every
// token that this does not decide -- near a halfway point, infinite, signed or
// long indices, any other spelling -- is listed and converted by strtol /
// strtof on the host; a text with more than kMaxLeft of them, or with one that
// converts only in part, is left to the host parser, at once if a sample shows
// it.
//
// Bound: the copy of the text from pageable memory and the result's
// allocations.  For the 460,000 entries of a 512 x 300 grid's lower triangle
// the count takes 8.5 us, the conversion 21 us and canonical order 170 us of a
// 3.0 ms read, which took 13 ms while the host's cores parsed.
#include <cuda_runtime.h>

#include <cctype>
#include <cfloat>
#include <clocale>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "device_common.cuh"
#include "kernels.cuh"
#include "rvsp_cuda.h"
#include "scratch.cuh"

namespace rvsp {

namespace {

constexpr int kMtxThreads = 256;
constexpr int kMtxBytes = 16;                       // bytes a thread, one load
constexpr int kMtxChunk = kMtxThreads * kMtxBytes;  // 4096
constexpr int kMtxHalo = 64;      // read past the chunk for a token that starts in it
constexpr int kMtxMaxToken = 48;  // longer ones are left to the host
constexpr int kMaxLeft = 256;
constexpr int kMaxExp10 = 60;  // w * 10^e stays far inside the doubles' range
static_assert(kMtxMaxToken + 8 <= kMtxHalo, "a token's reads stay inside the halo");

struct LeftToken {
  int64_t index, pos;
};

#define RVSP_POW10                                                                    \
  {1e0,  1e1,  1e2,  1e3,  1e4,  1e5,  1e6,  1e7,  1e8,  1e9,  1e10, 1e11,             \
   1e12, 1e13, 1e14, 1e15, 1e16, 1e17, 1e18, 1e19, 1e20, 1e21, 1e22}
__device__ const double kPow10[23] = RVSP_POW10;

// (the parses of a token are for the host too, which tries a sample of them)
__host__ __device__ __forceinline__ double pow10_of(int k) {
#ifdef __CUDA_ARCH__
  return kPow10[k];
#else
  static const double pow10[23] = RVSP_POW10;
  return pow10[k];
#endif
}
#undef RVSP_POW10

// isspace in the "C" locale
__host__ __device__ __forceinline__ bool space(uint32_t c) { return c == 32 || c - 9u < 5u; }

// Bit i: byte i of x starts a token; before: the byte ahead of x is a space.
__device__ __forceinline__ uint32_t token_starts(uint4 x, bool before) {
  const uint32_t w[4] = {x.x, x.y, x.z, x.w};
  uint32_t sp = 0;
#pragma unroll
  for (int i = 0; i < kMtxBytes; ++i)
    sp |= (space((w[i >> 2] >> (8 * (i & 3))) & 0xffu) ? 1u : 0u) << i;
  return ~sp & ((sp << 1) | (before ? 1u : 0u)) & 0xffffu;
}

__device__ __forceinline__ uint32_t starts_at(const uint8_t *text, int64_t at) {
  const uint4 x = *reinterpret_cast<const uint4 *>(text + at);
  return token_starts(x, at == 0 || space(text[at - 1]));
}

__global__ void __launch_bounds__(kMtxThreads)
mtx_count_kernel(const uint8_t *__restrict__ text, int32_t *__restrict__ counts) {
  __shared__ int32_t s_n;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  int n = __popc(starts_at(text, int64_t(blockIdx.x) * kMtxChunk + threadIdx.x * kMtxBytes));
  n = __reduce_add_sync(kFull, n);
  if (lane_id() == 0) atomicAdd(&s_n, n);
  __syncthreads();
  if (threadIdx.x == 0) counts[blockIdx.x] = s_n;
}

// A 1-based index of at most nine digits.
__host__ __device__ __forceinline__ bool parse_index(const uint8_t *t, int32_t *out) {
  int32_t v = 0;
  int i = 0;
  while (i < 9 && uint32_t(t[i]) - '0' < 10u) v = v * 10 + (t[i++] - '0');
  *out = v - 1;
  return i > 0 && space(t[i]);
}

// (conversions, products and quotients round to nearest on both sides)
__host__ __device__ __forceinline__ bool parse_value(const uint8_t *t, float *out) {
  int i = 0;
  const bool neg = t[0] == '-';
  if (neg || t[0] == '+') i = 1;
  unsigned long long w = 0;
  int digits = 0, e10 = 0;  // of w: its significant digits and its exponent
  bool any = false, point = false, cut = false;
  for (; i < kMtxMaxToken; ++i) {
    const uint32_t d = uint32_t(t[i]) - '0';
    if (d < 10u) {
      any = true;
      if (digits < 19) {
        w = w * 10 + d;
        digits += w != 0;
        e10 -= point;
      } else {  // below 10^-18 of w, far inside the slack
        cut = true;
        e10 += !point;
      }
    } else if (t[i] == '.' && !point) {
      point = true;
    } else {
      break;
    }
  }
  if (!any || i == kMtxMaxToken) return false;
  if (t[i] == 'e' || t[i] == 'E') {
    ++i;
    const bool eneg = t[i] == '-';
    if (eneg || t[i] == '+') ++i;
    int e = 0, n = 0;
    while (n < 3 && uint32_t(t[i]) - '0' < 10u) {
      e = e * 10 + (t[i++] - '0');
      ++n;
    }
    if (n == 0) return false;
    e10 += eneg ? -e : e;
  }
  if (!space(t[i])) return false;
  float f;
  if (w == 0) {
    f = 0.0f;
  } else if (e10 == 0 && !cut) {
    f = static_cast<float>(w);
  } else {
    int n = e10 < 0 ? -e10 : e10;
    if (n > kMaxExp10) return false;
    double d = static_cast<double>(w);
    while (n > 0) {
      const int k = n < 22 ? n : 22;
      d = e10 < 0 ? d / pow10_of(k) : d * pow10_of(k);
      n -= k;
    }
    constexpr double kSlack = 1.0 / (1ull << 49);
    f = static_cast<float>(d * (1.0 - kSlack));
    if (f != static_cast<float>(d * (1.0 + kSlack)) || f > FLT_MAX) return false;
  }
  *out = neg ? -f : f;
  return true;
}

// Converts the tokens that start in the block's chunk.  The threads take the
// tokens of one field at a time: a warp's parses are alike and its stores
// run along one array.
template <int F>
__global__ void __launch_bounds__(kMtxThreads)
mtx_convert_kernel(const uint8_t *__restrict__ text, const int64_t *__restrict__ first,
                   int64_t limit, int32_t *__restrict__ row, int32_t *__restrict__ col,
                   float *__restrict__ val, unsigned long long *__restrict__ nleft,
                   LeftToken *__restrict__ left) {
  __shared__ __align__(16) uint8_t s_text[kMtxChunk + kMtxHalo];
  __shared__ uint16_t s_pos[kMtxChunk / 2];
  __shared__ int32_t s_warp[kMtxThreads / 32];
  const int64_t base = int64_t(blockIdx.x) * kMtxChunk;
  const int at = threadIdx.x * kMtxBytes;
  const uint4 x = *reinterpret_cast<const uint4 *>(text + base + at);
  *reinterpret_cast<uint4 *>(s_text + at) = x;
  if (threadIdx.x < kMtxHalo / kMtxBytes)
    *reinterpret_cast<uint4 *>(s_text + kMtxChunk + at) =
        *reinterpret_cast<const uint4 *>(text + base + kMtxChunk + at);
  const int64_t here = base + at;
  uint32_t starts = token_starts(x, here == 0 || space(text[here - 1]));
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  int incl = __popc(starts);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  int k = incl - __popc(starts), n = 0;
#pragma unroll
  for (int v = 0; v < kMtxThreads / 32; ++v) {
    if (v < warp) k += s_warp[v];
    n += s_warp[v];
  }
  for (; starts; starts &= starts - 1)
    s_pos[k++] = static_cast<uint16_t>(at + __ffs(starts) - 1);
  __syncthreads();
  const int64_t g0 = first[blockIdx.x];
  const int r0 = static_cast<int>(g0 % F);
#pragma unroll
  for (int f = 0; f < F; ++f) {
    const int k0 = f >= r0 ? f - r0 : f - r0 + F;
    const int64_t e0 = (g0 + k0) / F;
    for (int i = threadIdx.x; k0 + i * F < n; i += kMtxThreads) {
      const int64_t e = e0 + i;
      if (e >= limit) break;
      const int p = s_pos[k0 + i * F];
      bool ok;
      if (f < 2) {
        ok = parse_index(s_text + p, (f == 0 ? row : col) + e);
        if (F == 2 && f == 1) val[e] = 1.0f;
      } else {
        ok = parse_value(s_text + p, val + e);
      }
      if (!ok) {
        const unsigned long long q = atomicAdd(nleft, 1ull);
        if (q < kMaxLeft) left[q] = LeftToken{g0 + k0 + int64_t(i) * F, base + p};
      }
    }
  }
}

// Converts one listed token as the host parser does.  1: done; 0: nothing
// converts, the reading ends at its entry; -1: the host parser has to decide.
int convert_left(const char *text, size_t len, int64_t pos, bool index, int32_t *iv, float *fv) {
  char buf[128];
  size_t n = 0, i = static_cast<size_t>(pos);
  for (; i < len; ++i) {
    const unsigned char c = static_cast<unsigned char>(text[i]);
    const bool sp = c == 32 || (c >= 9 && c <= 13);
    if (sp != (std::isspace(c) != 0)) return -1;  // another locale's white space
    if (sp) break;
    if (n == sizeof(buf) - 1) return -1;
    buf[n++] = static_cast<char>(c);
  }
  buf[n] = '\0';
  char *stop = buf;
  if (index) *iv = static_cast<int32_t>(std::strtol(buf, &stop, 10)) - 1;
  else *fv = std::strtof(buf, &stop);
  if (stop == buf) return 0;
  return stop == buf + n ? 1 : -1;
}

// Whether the text is of a kind that the device does not decide (signed
// indices, values of 48 characters or more, infinities, exponents past 60), so
// that sending it would be in vain: in pieces of it, each from the start of a
// line, an eighth of the lines or more, and by their number surely more than
// kMaxLeft tokens in all, are undecided.  A line is taken for an entry; a text
// with other lines is at worst parsed on the side that takes longer.  Sent in
// vain, 10 MB of signed indices took 13.1 ms against 12.9, 7.6 MB of infinities
// 10.9 against 8.9, 0.1 MB of them 0.63 against 0.55; the sample takes 5 us.
bool mostly_undecided(const char *text, size_t len, int fields) {
  constexpr size_t kPiece = 256;
  const size_t pieces = len / 16384 < 2 ? 2 : len / 16384 > 8 ? 8 : len / 16384;
  const uint8_t *t = reinterpret_cast<const uint8_t *>(text);
  size_t lines = 0, undecided = 0;
  for (size_t i = 0; i < pieces; ++i) {
    size_t p = i * (len / pieces);
    const size_t end = p + kPiece + kMtxHalo < len ? p + kPiece : p;
    for (; i > 0 && p < end && t[p] != '\n'; ++p) {
    }
    bool ok = true;
    for (int f = 0; p < end;) {
      if (space(t[p])) {
        if (t[p] == '\n' && f > 0) {
          ++lines;
          undecided += !ok;
          f = 0;
          ok = true;
        }
        ++p;
        continue;
      }
      int32_t index;
      float value;
      if (f < fields) ok &= f < 2 ? parse_index(t + p, &index) : parse_value(t + p, &value);
      ++f;
      while (p < end && !space(t[p])) ++p;
    }
  }
  return undecided * 8 >= lines && undecided * (len / (pieces * kPiece)) > 2 * kMaxLeft;
}

rvsp_status_t status_of(cudaError_t e) {
  return e == cudaErrorMemoryAllocation ? RVSP_ERROR_ALLOCATION_FAILED : RVSP_ERROR_DEVICE;
}

// The entries of text (at least one byte of it, and of limit) into row, col
// and val of limit; *n_out of them.  *parsed stays 0 when the host parser has
// to read it.
rvsp_status_t parse_entries(cudaStream_t s, const char *text, size_t len, int fields,
                            int64_t limit, int32_t *row, int32_t *col, float *val,
                            int64_t *n_out, int *parsed) {
  const int64_t chunks = static_cast<int64_t>((len + kMtxChunk - 1) / kMtxChunk);
  const size_t padded = size_t(chunks) * kMtxChunk + kMtxHalo;
  Scratch sc(s);
  uint8_t *d_text = nullptr;
  int32_t *counts = nullptr;
  int64_t *first = nullptr, *partials = nullptr;
  unsigned long long *meta = nullptr;  // tokens, tokens left
  LeftToken *d_left = nullptr;
  const size_t nc = size_t(chunks);
  int64_t &n = *n_out;
  cudaError_t e = sc.alloc(reinterpret_cast<void **>(&d_text), padded);
  if (e == cudaSuccess) e = sc.alloc(reinterpret_cast<void **>(&counts), nc * sizeof(int32_t));
  if (e == cudaSuccess) e = sc.alloc(reinterpret_cast<void **>(&first), nc * sizeof(int64_t));
  if (e == cudaSuccess)
    e = sc.alloc(reinterpret_cast<void **>(&partials),
                 scan_partials_bytes(static_cast<int32_t>(chunks)));
  if (e == cudaSuccess)
    e = sc.alloc(reinterpret_cast<void **>(&meta), 2 * sizeof(unsigned long long));
  if (e == cudaSuccess)
    e = sc.alloc(reinterpret_cast<void **>(&d_left), kMaxLeft * sizeof(LeftToken));
  if (e != cudaSuccess) return status_of(e);
  cudaMemcpyAsync(d_text, text, len, cudaMemcpyHostToDevice, s);
  cudaMemsetAsync(d_text + len, ' ', padded - len, s);
  cudaMemsetAsync(meta, 0, 2 * sizeof(unsigned long long), s);
  mtx_count_kernel<<<static_cast<unsigned>(chunks), kMtxThreads, 0, s>>>(d_text, counts);
  launch_scan_i64(static_cast<int32_t>(chunks), counts, first, partials,
                  reinterpret_cast<int64_t *>(meta), s);
  if (fields == 2)
    mtx_convert_kernel<2><<<static_cast<unsigned>(chunks), kMtxThreads, 0, s>>>(
        d_text, first, limit, row, col, val, meta + 1, d_left);
  else
    mtx_convert_kernel<3><<<static_cast<unsigned>(chunks), kMtxThreads, 0, s>>>(
        d_text, first, limit, row, col, val, meta + 1, d_left);
  unsigned long long h_meta[2] = {0, 0};
  e = cudaGetLastError();
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(h_meta, meta, sizeof(h_meta), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return status_of(e);
  if (h_meta[1] > kMaxLeft) return RVSP_SUCCESS;
  n = static_cast<int64_t>(h_meta[0]) / fields;
  if (n > limit) n = limit;
  if (h_meta[1] > 0) {
    LeftToken left[kMaxLeft];
    e = cudaMemcpyAsync(left, d_left, size_t(h_meta[1]) * sizeof(LeftToken),
                        cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return status_of(e);
    for (unsigned long long q = 0; q < h_meta[1]; ++q) {
      const int64_t entry = left[q].index / fields;
      const int f = static_cast<int>(left[q].index % fields);
      int32_t iv = 0;
      float fv = 0.0f;
      const int r = convert_left(text, len, left[q].pos, f < 2, &iv, &fv);
      if (r < 0) return RVSP_SUCCESS;
      if (r == 0) {
        if (entry < n) n = entry;
        continue;
      }
      if (f < 2)
        e = cudaMemcpyAsync((f == 0 ? row : col) + entry, &iv, sizeof(iv),
                            cudaMemcpyHostToDevice, s);
      else
        e = cudaMemcpyAsync(val + entry, &fv, sizeof(fv), cudaMemcpyHostToDevice, s);
      if (e != cudaSuccess) return status_of(e);
    }
  }
  *parsed = 1;
  return RVSP_SUCCESS;
}

}  // namespace

}  // namespace rvsp

using namespace rvsp;

extern "C" rvsp_status_t rvsp_cuda_mtx_to_csr(void *stream, const char *text, size_t len,
                                              int fields, int64_t limit, int32_t rows,
                                              int32_t cols, int symmetric,
                                              int32_t *c_row_ptr, int32_t **c_col_out,
                                              float **c_val_out, int32_t *c_nnz_out,
                                              int *parsed) {
  if (!text || !c_row_ptr || !c_col_out || !c_val_out || !c_nnz_out || !parsed)
    return RVSP_ERROR_NULL_POINTER;
  if (rows < 0 || cols < 0 || limit < 0 || limit > int64_t(INT32_MAX) ||
      (fields != 2 && fields != 3))
    return RVSP_ERROR_INVALID_ARGUMENT;
  *parsed = 0;
  *c_col_out = nullptr;
  *c_val_out = nullptr;
  *c_nnz_out = 0;
  const int64_t chunks = static_cast<int64_t>((len + kMtxChunk - 1) / kMtxChunk);
  const char *point = std::localeconv()->decimal_point;
  if (limit == 0 || chunks == 0 || chunks > INT32_MAX / 2 || point[0] != '.' || point[1] ||
      mostly_undecided(text, len, fields))
    return RVSP_SUCCESS;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  rvsp_status_t st = RVSP_SUCCESS;
  {
    Scratch entries(s);
    int32_t *row = nullptr, *col = nullptr;
    float *val = nullptr;
    int64_t n = 0;
    const size_t nl = size_t(limit);
    cudaError_t e = entries.alloc(reinterpret_cast<void **>(&row), nl * sizeof(int32_t));
    if (e == cudaSuccess)
      e = entries.alloc(reinterpret_cast<void **>(&col), nl * sizeof(int32_t));
    if (e == cudaSuccess) e = entries.alloc(reinterpret_cast<void **>(&val), nl * sizeof(float));
    st = e == cudaSuccess ? parse_entries(s, text, len, fields, limit, row, col, val, &n, parsed)
                          : status_of(e);
    if (*parsed)  // (the text's memory is given back by now)
      st = rvsp_cuda_coo_to_csr(stream, rows, cols, n, symmetric, row, col, val, c_row_ptr,
                                c_col_out, c_val_out, c_nnz_out);
  }
  if (st == RVSP_ERROR_ALLOCATION_FAILED) {
    // no room beside the text: the host parser needs less, and gets all of it
    cudaGetLastError();
    *parsed = 0;
    st = RVSP_SUCCESS;
    const cudaMemPool_t pool = scratch_pool();
    if (cudaStreamSynchronize(s) != cudaSuccess) return RVSP_ERROR_DEVICE;
    if (pool) cudaMemPoolTrimTo(pool, 0);
  }
  return st;
}

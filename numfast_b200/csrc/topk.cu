// Top-k of the stable argsort without sorting every row: the first k entries
// of nfc_sort_perm's permutation (the reference's sort -> slice -> gather,
// src/Drivers/CPU/_lib/cpu.py:3170-3200, over the order of _sort_perm,
// cpu.py:1154-1225), by radix selection.
//
//   1. selection   each row's key as an order-preserving unsigned image
//                  (descending = its complement); 11-bit digit histograms
//                  from the top, over the rows whose higher digits match the
//                  prefix chosen so far, find the k-th smallest image: rows
//                  below the prefix are all taken, `need` of the rows on it
//                  (ties) are taken in input order.  A pass stops early once
//                  every row on the prefix is taken, and the passes over the
//                  column stop once the rows on the prefix fit the candidate
//                  buffer (kTkCandCap rows).
//   2. compaction  usual case -- the selection stopped with at most
//                  kTkCandCap rows on the prefix and k <= valid rows: ONE
//                  pass (k_tk_split, 16,384-row tiles, decoupled look-back)
//                  writes the taken rows and every row on the prefix (the
//                  candidates) in input order; the candidates are sorted by
//                  image (stable) and their first `need` join the taken
//                  rows, so the rest of the selection runs on the
//                  candidates, not on the column.  Otherwise (the prefix
//                  group is taken whole, more NULL rows are needed than
//                  exist, or every digit was resolved on the column): per
//                  block of 4,096 rows, counts of taken-below, tie and NULL
//                  rows, one CTA scans them, each block writes its taken
//                  rows' (image, row) pairs in input order and the first
//                  k - valid NULL rows straight into the output tail.
//   3. sort        the k taken pairs by image, stable (radix sort; one CTA
//                  for k <= 2,048), which is the argsort's order of them.
//
// Full passes over the column in the usual case: one histogram (more only
// while the prefix group exceeds the buffer) and the split.
//
// Small k (topk_sampled) needs one pass over the column: the histograms run on
// a sample of the rows, the rows up to a threshold that holds the k-th smallest
// image with near certainty are collected in any order, and every one's place is
// counted against all of them, by (image, row), over the whole chip.  If the
// count shows the threshold too low, or too many rows are on it (ties), the
// passes above run instead; what the sample learned (TkHint) spares them the
// histograms where the k-th image is on its prefix.
//
// Descending float64: every NaN is its own group in the reference's
// _stable_desc_idx, so the NaN block comes first in REVERSE input order: the
// selection takes the last `need` NaN rows and the sorted NaN prefix is
// reversed.  For k above n / 8 the full argsort is cheaper and is used.
#include <algorithm>
#include <cmath>

#include "groupby_core.cuh"
#include "groupby_host.h"

namespace nfc {
namespace {

constexpr int kTkThreads = 256;
constexpr int kTkItems = 16;
constexpr int kTkBlockRows = kTkThreads * kTkItems;  // 4096
constexpr int kTkDigitBits = 11;
constexpr int kTkBins = 1 << kTkDigitBits;
constexpr int64_t kTkCandCap = 1 << 20;  // rows on the prefix that end the full passes

// Order-preserving unsigned image of a key's bits; descending complements it
// (32 bits for int32, 64 for int64 / float64).  float64: -0.0 ties +0.0 and
// every NaN maps past +inf, as in the full argsort.
template <int DT>
NFC_DEV uint64_t tk_image_bits(uint64_t raw, bool desc) {
  uint64_t u;
  if (DT == NFC_I32) {
    u = (uint32_t)raw ^ 0x80000000u;
    return desc ? (~u & 0xFFFFFFFFull) : u;
  }
  if (DT == NFC_I64) {
    u = raw ^ 0x8000000000000000ull;
  } else {
    uint64_t b = raw;
    if (f64_bits_isnan(b)) {
      u = ~0ull;
    } else {
      if (b == 0x8000000000000000ull) b = 0ull;
      u = f64_ord(b);
    }
  }
  return desc ? ~u : u;
}

template <int DT>
NFC_DEV uint64_t tk_image(const void* keys, int64_t i, bool desc) {
  const uint64_t raw = DT == NFC_I32 ? (uint64_t)(uint32_t) static_cast<const int32_t*>(keys)[i]
                                     : static_cast<const uint64_t*>(keys)[i];
  return tk_image_bits<DT>(raw, desc);
}

// Images and validity of rows i0 .. i0+3 (i0 a multiple of 4): one 16-byte
// load of int32 keys or two of 8-byte keys when `vec` (16-byte aligned
// keys), and the rows' four bits of the LSB-first bitmap (one byte).  Rows
// at or past n are invalid.
template <int DT>
NFC_DEV uint32_t tk_load4(const void* __restrict__ keys, const uint8_t* __restrict__ validity, int64_t i0,
                          int64_t n, bool vec, bool desc, uint64_t img[4]) {
  uint32_t ok = i0 + 4 <= n ? 0xFu : (i0 < n ? (1u << (uint32_t)(n - i0)) - 1u : 0u);
  if (validity && ok) ok &= (uint32_t)(__ldg(validity + (i0 >> 3)) >> (i0 & 7)) & 0xFu;
  if (vec && i0 + 4 <= n) {
    if (DT == NFC_I32) {
      const uint4 q = __ldcs(reinterpret_cast<const uint4*>(static_cast<const int32_t*>(keys) + i0));
      img[0] = tk_image_bits<DT>(q.x, desc); img[1] = tk_image_bits<DT>(q.y, desc);
      img[2] = tk_image_bits<DT>(q.z, desc); img[3] = tk_image_bits<DT>(q.w, desc);
    } else {
      const ulonglong2* p = reinterpret_cast<const ulonglong2*>(static_cast<const uint64_t*>(keys) + i0);
      const ulonglong2 a = __ldcs(p), b = __ldcs(p + 1);
      img[0] = tk_image_bits<DT>(a.x, desc); img[1] = tk_image_bits<DT>(a.y, desc);
      img[2] = tk_image_bits<DT>(b.x, desc); img[3] = tk_image_bits<DT>(b.y, desc);
    }
  } else {
#pragma unroll
    for (int r = 0; r < 4; ++r) img[r] = i0 + r < n ? tk_image<DT>(keys, i0 + r, desc) : 0ull;
  }
  return ok;
}

NFC_DEV bool tk_valid(const uint8_t* v, int64_t i) { return !v || ((v[i >> 3] >> (i & 7)) & 1u); }

// Digit histogram of the valid rows on the prefix ((image & mask) == prefix).
// Each thread takes four consecutive rows per step (16-byte loads), two steps
// in flight.  Pairs of warps count into their own copy of the histogram (four
// per CTA), which spreads the atomics of a skewed digit (the sign and
// exponent bits of float64 keys put most rows in a few bins); measured on
// 100M lognormal keys: 255 us, against 315 us merging equal digits of a warp
// with match_any first and 630 us with one shared copy.
template <int DT>
__global__ void __launch_bounds__(kTkThreads) k_tk_hist(const void* __restrict__ keys,
                                                       const uint8_t* __restrict__ validity, int64_t n, bool vec,
                                                       bool desc, uint64_t mask, uint64_t prefix, int shift,
                                                       uint32_t dmask, uint32_t* __restrict__ ghist) {
  constexpr int kCopies = 4;
  __shared__ uint32_t h[kCopies][kTkBins];
  uint32_t* hs = h[(threadIdx.x >> 6) & (kCopies - 1)];
  for (int i = threadIdx.x; i < kCopies * kTkBins; i += blockDim.x) (&h[0][0])[i] = 0u;
  __syncthreads();
  const int64_t ngroups = (n + 3) >> 2;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  constexpr int U = 2;  // groups of four rows in flight per thread
  for (int64_t g0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g0 < ngroups; g0 += U * stride) {
    uint64_t img[U][4];
    uint32_t ok[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t g = g0 + u * stride;
      ok[u] = g < ngroups ? tk_load4<DT>(keys, validity, g * 4, n, vec, desc, img[u]) : 0u;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (((ok[u] >> r) & 1u) && (img[u][r] & mask) == prefix)
          atomicAdd(&hs[(uint32_t)(img[u][r] >> shift) & dmask], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i <= (int)dmask; i += blockDim.x) {
    uint32_t c = 0;
#pragma unroll
    for (int k = 0; k < kCopies; ++k) c += h[k][i];
    if (c) atomicAdd(&ghist[i], c);
  }
}

// Valid rows, rows below the prefix and rows on it -> cnt[0..2].
template <int DT>
__global__ void __launch_bounds__(kTkThreads) k_tk_below(const void* __restrict__ keys,
                                                        const uint8_t* __restrict__ validity, int64_t n, bool vec,
                                                        bool desc, uint64_t mask, uint64_t prefix,
                                                        unsigned long long* __restrict__ cnt) {
  const int64_t ngroups = (n + 3) >> 2;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  constexpr int U = 2;
  uint32_t c[3] = {0u, 0u, 0u};
  for (int64_t g0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g0 < ngroups; g0 += U * stride) {
    uint64_t img[U][4];
    uint32_t ok[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t g = g0 + u * stride;
      ok[u] = g < ngroups ? tk_load4<DT>(keys, validity, g * 4, n, vec, desc, img[u]) : 0u;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if ((ok[u] >> r) & 1u) {
          const uint64_t m = img[u][r] & mask;
          c[0] += 1u;
          c[1] += m < prefix;
          c[2] += m == prefix;
        }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const uint32_t w = warp_sum(c[k]);
    if (lane_id() == 0 && w) atomicAdd(&cnt[k], (unsigned long long)w);
  }
}

// Row class: 0 taken (below the prefix), 1 tie (on the prefix), 2 NULL,
// 3 neither.
template <int DT>
NFC_DEV int tk_class(const void* keys, const uint8_t* validity, int64_t i, bool desc, uint64_t mask,
                     uint64_t prefix) {
  if (!tk_valid(validity, i)) return 2;
  const uint64_t m = tk_image<DT>(keys, i, desc) & mask;
  return m < prefix ? 0 : m == prefix ? 1 : 3;
}

// Per block of kTkBlockRows rows: counts of classes 0, 1, 2 -> cnt[3 b + c].
template <int DT>
__global__ void __launch_bounds__(kTkThreads) k_tk_count(const void* __restrict__ keys,
                                                        const uint8_t* __restrict__ validity, int64_t n, bool desc,
                                                        uint64_t mask, uint64_t prefix, uint32_t* __restrict__ cnt) {
  __shared__ uint32_t s[3][kTkThreads / 32];
  uint32_t c[3] = {0u, 0u, 0u};
  const int64_t base = (int64_t)blockIdx.x * kTkBlockRows;
#pragma unroll 4
  for (int j = 0; j < kTkItems; ++j) {
    const int64_t i = base + j * kTkThreads + threadIdx.x;
    if (i >= n) break;
    const int k = tk_class<DT>(keys, validity, i, desc, mask, prefix);
    if (k < 3) ++c[k];
  }
  const int warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const uint32_t w = warp_sum(c[k]);
    if (lane_id() == 0) s[k][warp] = w;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    uint32_t t = 0;
    for (int w = 0; w < kTkThreads / 32; ++w) t += s[threadIdx.x][w];
    cnt[3 * (int64_t)blockIdx.x + threadIdx.x] = t;
  }
}

// Exclusive scan of the three count columns over nb blocks (one CTA).
__global__ void __launch_bounds__(1024) k_tk_scan(const uint32_t* __restrict__ cnt, int64_t nb,
                                                 uint32_t* __restrict__ pre) {
  __shared__ uint32_t sm[33];
  for (int k = 0; k < 3; ++k) {
    uint32_t carry = 0;
    for (int64_t b0 = 0; b0 < nb; b0 += blockDim.x) {
      const int64_t b = b0 + threadIdx.x;
      const uint32_t v = b < nb ? cnt[3 * b + k] : 0u;
      uint32_t total;
      const uint32_t e = block_excl_scan(v, sm, &total);
      if (b < nb) pre[3 * b + k] = carry + e;
      carry += total;
    }
  }
}

// Each block writes its taken rows, in input order, as (image, row) pairs at
// their place among all taken rows, and its NULL rows of rank < null_take at
// tail[rank].  A tie is taken when its rank among the ties is in
// [tie_lo, tie_lo + need); the number of taken ties before a row follows from
// the tie count before it, so every block knows its base from the scans.
template <int DT, class K>
__global__ void __launch_bounds__(kTkThreads) k_tk_compact(const void* __restrict__ keys,
                                                          const uint8_t* __restrict__ validity, int64_t n, bool desc,
                                                          uint64_t mask, uint64_t prefix,
                                                          const uint32_t* __restrict__ pre, uint32_t tie_lo,
                                                          uint32_t need, uint32_t ksel, uint32_t null_take,
                                                          K* __restrict__ img_out, uint32_t* __restrict__ row_out,
                                                          int32_t* __restrict__ tail, int32_t* err) {
  __shared__ uint32_t sm[33];
  const int64_t b = blockIdx.x;
  uint32_t b_lt = pre[3 * b], b_tie = pre[3 * b + 1], b_null = pre[3 * b + 2];
  const int64_t base = b * kTkBlockRows;
  for (int j = 0; j < kTkItems; ++j) {
    if (base + j * kTkThreads >= n) break;  // uniform across the block
    const int64_t i = base + j * kTkThreads + threadIdx.x;
    const int k = i < n ? tk_class<DT>(keys, validity, i, desc, mask, prefix) : 3;
    const uint32_t v = k == 0 ? 1u : k == 1 ? (1u << 10) : k == 2 ? (1u << 20) : 0u;
    uint32_t tot;
    const uint32_t ex = block_excl_scan(v, sm, &tot);
    const uint32_t lt_before = b_lt + (ex & 1023u);
    const uint32_t tie_before = b_tie + ((ex >> 10) & 1023u);
    const uint32_t taken_ties = min(max(tie_before, tie_lo), tie_lo + need) - tie_lo;
    if (k == 0 || (k == 1 && tie_before >= tie_lo && tie_before < tie_lo + need)) {
      const uint32_t pos = lt_before + (k == 0 ? taken_ties : tie_before - tie_lo);
      if (pos < ksel) {
        img_out[pos] = (K)tk_image<DT>(keys, i, desc);
        row_out[pos] = (uint32_t)i;
      } else {
        atomicExch(err, NFC_ERR_RANGE);
      }
    } else if (k == 2) {
      const uint32_t q = b_null + (ex >> 20);
      if (q < null_take) tail[q] = (int32_t)i;
    }
    b_lt += tot & 1023u;
    b_tie += (tot >> 10) & 1023u;
    b_null += tot >> 20;
  }
}

// One pass, used when the selection stopped with a prefix group of at most
// kTkCandCap rows (and every NULL row is left out: k <= valid rows): taken
// rows (image under the prefix) go to t_img/t_row and every row on the
// prefix to c_img/c_row, both in input order.  Tiles of kTkSplitRows rows
// are claimed in order; warp w of a tile takes its 2,048 contiguous rows in
// 16 steps of four consecutive rows per lane, keeping only two class bits
// per row; the tile's place in both lists comes from one decoupled
// look-back over (taken << 32 | tie) counts, and the few selected rows
// reload their key to write it out.
constexpr int kTkSplitRows = 16384;

template <int DT, class K>
__global__ void __launch_bounds__(kTkThreads) k_tk_split(const void* __restrict__ keys,
                                                        const uint8_t* __restrict__ validity, int64_t n, bool vec,
                                                        bool desc, uint64_t mask, uint64_t prefix, uint32_t n_taken,
                                                        uint32_t n_cand, K* __restrict__ t_img,
                                                        uint32_t* __restrict__ t_row, K* __restrict__ c_img,
                                                        uint32_t* __restrict__ c_row, uint64_t* lb, uint32_t* ticket,
                                                        int32_t* err) {
  constexpr int kWarps = kTkThreads / 32;
  constexpr int kSteps = kTkSplitRows / (kTkThreads * 4);  // 16 steps of 128 rows per warp
  constexpr int U = 4;                                      // steps in flight
  __shared__ int64_t s_tile;
  __shared__ uint32_t s_wt[kWarps][2];
  __shared__ uint64_t s_base;
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
  __syncthreads();
  const int64_t tile = s_tile;
  const int64_t row0 = tile * kTkSplitRows + (int64_t)warp * (kSteps * 128);
  uint64_t tk_bits = 0, tie_bits = 0;  // bit 4 j + r: step j, row r
#pragma unroll
  for (int j0 = 0; j0 < kSteps; j0 += U) {
    uint64_t img[U][4];
    uint32_t ok[U];
#pragma unroll
    for (int u = 0; u < U; ++u) ok[u] = tk_load4<DT>(keys, validity, row0 + (j0 + u) * 128 + lane * 4, n, vec, desc, img[u]);
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (!((ok[u] >> r) & 1u)) continue;
        const uint64_t m = img[u][r] & mask;
        if (m < prefix) tk_bits |= 1ull << (4 * (j0 + u) + r);
        else if (m == prefix) tie_bits |= 1ull << (4 * (j0 + u) + r);
      }
  }
  const uint32_t w_tk = warp_sum((uint32_t)__popcll(tk_bits)), w_tie = warp_sum((uint32_t)__popcll(tie_bits));
  if (lane == 0) { s_wt[warp][0] = w_tk; s_wt[warp][1] = w_tie; }
  __syncthreads();
  if (warp == 0) {
    uint32_t a = 0, b = 0;
    for (int w = 0; w < kWarps; ++w) { a += s_wt[w][0]; b += s_wt[w][1]; }
    const uint64_t base = (uint64_t)lookback_exclusive(lb, tile, ((uint64_t)a << 32) | b, err);  // whole warp
    if (lane == 0) s_base = base;
  }
  __syncthreads();
  if ((w_tk | w_tie) == 0) return;
  uint32_t t_pos = (uint32_t)(s_base >> 32), c_pos = (uint32_t)s_base;
  for (int w = 0; w < warp; ++w) { t_pos += s_wt[w][0]; c_pos += s_wt[w][1]; }
  for (int j = 0; j < kSteps; ++j) {
    const uint32_t tj = (uint32_t)(tk_bits >> (4 * j)) & 0xFu, cj = (uint32_t)(tie_bits >> (4 * j)) & 0xFu;
    if (!__any_sync(0xffffffffu, (tj | cj) != 0u)) continue;
    // Exclusive scan over lanes of both counts at once (<= 128 each per step).
    const uint32_t x = (uint32_t)__popc(tj) | ((uint32_t)__popc(cj) << 16);
    uint32_t incl = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    const uint32_t tot = __shfl_sync(0xffffffffu, incl, 31);
    uint32_t tp = t_pos + ((incl - x) & 0xFFFFu), cp = c_pos + ((incl - x) >> 16);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int64_t i = row0 + j * 128 + lane * 4 + r;
      if ((tj >> r) & 1u) {
        if (tp < n_taken) { t_img[tp] = (K)tk_image<DT>(keys, i, desc); t_row[tp] = (uint32_t)i; }
        else atomicExch(err, NFC_ERR_RANGE);
        ++tp;
      } else if ((cj >> r) & 1u) {
        if (cp < n_cand) { c_img[cp] = (K)tk_image<DT>(keys, i, desc); c_row[cp] = (uint32_t)i; }
        else atomicExch(err, NFC_ERR_RANGE);
        ++cp;
      }
    }
    t_pos += tot & 0xFFFFu;
    c_pos += tot >> 16;
  }
}

// Entries whose image is 0 (descending float64: the NaN rows).
template <class K>
__global__ void __launch_bounds__(kTkThreads) k_tk_zero_count(const K* __restrict__ img, int64_t m,
                                                             unsigned long long* cnt) {
  uint32_t c = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x)
    c += img[i] == (K)0;
  c = warp_sum(c);
  if (lane_id() == 0 && c) atomicAdd(cnt, (unsigned long long)c);
}

__global__ void k_tk_reverse(int32_t* p, int64_t m) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m / 2; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t t = p[i];
    p[i] = p[m - 1 - i];
    p[m - 1 - i] = t;
  }
}

// ---------------------------------------------------------------- sampled threshold
// Bound of the exact form: 557 us of 100M float64 keys go into one histogram
// and one ordered split, both over the whole column, and 50,000 candidates are
// then sorted.  A threshold from a sample costs two small histograms; what is
// left is one pass that reads the column and writes a few thousand rows.
constexpr int kTkCap = 8192;          // rows collected at most (96 KB of shared memory in k_tk_final)
constexpr int64_t kTkExpect = 5000;   // most rows expected under the threshold

constexpr int kTkFinalThreads = 512;
constexpr int kTkLevels = 4;          // digits of the threshold at most

struct TkSampleHead {
  uint64_t prefix, mask;  // threshold: rows with (image & mask) <= prefix
  uint32_t target;        // rank in the sample still to find on the prefix
  uint32_t below;         // sampled rows under the prefix
  uint32_t ready;         // the threshold lets few enough rows through
  uint32_t count;         // rows collected
  uint32_t status;        // 1: the exact passes have to run
  uint32_t failed;        // fewer valid rows in the sample than the target
};
struct TkSample : TkSampleHead {
  uint32_t done[kTkLevels];  // CTAs that have finished each level
  uint32_t hist[kTkLevels][kTkBins];
};

// Histogram of one 11-bit digit of the sampled rows on the prefix; the last
// CTA to finish moves the prefix on to the digit that holds the target rank.
// The sample is one group of four rows out of every `step`, at a hashed place:
// short groups, so that sorted or clustered columns are sampled evenly too.
template <int DT>
__global__ void __launch_bounds__(kTkThreads) k_tk_sample(const void* __restrict__ keys,
                                                         const uint8_t* __restrict__ validity, int64_t n, bool vec,
                                                         bool desc, int level, int shift, uint32_t dmask,
                                                         uint32_t step, uint32_t target, TkSample* st) {
  __shared__ uint32_t h[2][kTkBins];
  __shared__ uint32_t s_scan[33];
  __shared__ int s_last;
  if (level && (st->ready || st->failed)) return;
  const uint64_t prefix = level ? st->prefix : 0ull, mask = level ? st->mask : 0ull;
  uint32_t* hs = h[(threadIdx.x >> 5) & 1];
  for (int i = threadIdx.x; i < 2 * kTkBins; i += kTkThreads) (&h[0][0])[i] = 0u;
  __syncthreads();
  const int64_t ngroups = (n + 3) / 4;
  const int64_t npick = (ngroups + step - 1) / step;
  const int64_t stride = (int64_t)gridDim.x * kTkThreads;
  constexpr int U = 4;
  for (int64_t p0 = blockIdx.x * (int64_t)kTkThreads + threadIdx.x; p0 < npick; p0 += U * stride) {
    uint64_t img[U][4];
    uint32_t ok[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t p = p0 + u * stride;
      const int64_t g = p * step + (step > 1 ? ((uint32_t)p * 0x9E3779B1u >> 8) % step : 0u);
      ok[u] = p < npick && g < ngroups ? tk_load4<DT>(keys, validity, g * 4, n, vec, desc, img[u]) : 0u;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (((ok[u] >> r) & 1u) && (img[u][r] & mask) == prefix)
          atomicAdd(&hs[(uint32_t)(img[u][r] >> shift) & dmask], 1u);
  }
  __syncthreads();
  uint32_t* gh = st->hist[level];
  for (int i = threadIdx.x; i < kTkBins; i += kTkThreads) {
    const uint32_t c = h[0][i] + h[1][i];
    if (c) atomicAdd(&gh[i], c);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&st->done[level], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  constexpr int kPer = kTkBins / kTkThreads;
  uint32_t c[kPer], sum = 0;
  // Read before the scan's barriers: the thread that holds the digit moves the
  // state on after them, while others may still be on their way.
  const uint32_t want = level ? st->target : target, before = level ? st->below : 0u;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    c[j] = __ldcg(&gh[threadIdx.x * kPer + j]);
    sum += c[j];
  }
  uint32_t total;
  uint32_t x = block_excl_scan(sum, s_scan, &total);
  // Fewer sampled valid rows than the target: no digit holds it.
  if (total < want && threadIdx.x == 0) st->failed = 1u;
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    if (x < want && want <= x + c[j]) {
      st->prefix = prefix | ((uint64_t)(threadIdx.x * kPer + j) << shift);
      st->mask = mask | ((uint64_t)dmask << shift);
      st->target = want - x;
      const uint32_t below = before + x;
      st->below = below;
      if ((uint64_t)(below + c[j]) * step <= (uint64_t)(kTkExpect + kTkExpect / 4)) st->ready = 1u;
    }
    x += c[j];
  }
}

// Whether a key's image is at most `top`, on the key itself: one comparison
// with the key at the threshold instead of building every row's image.
template <int DT>
struct TkUnder;
template <>
struct TkUnder<NFC_I32> {
  int32_t t;
  bool desc;
  NFC_DEV TkUnder(uint64_t top, bool d)
      : t((int32_t)((d ? ~(uint32_t)top : (uint32_t)top) ^ 0x80000000u)), desc(d) {}
  NFC_DEV bool operator()(uint32_t raw) const { return desc ? (int32_t)raw >= t : (int32_t)raw <= t; }
};
template <>
struct TkUnder<NFC_I64> {
  int64_t t;
  bool desc;
  NFC_DEV TkUnder(uint64_t top, bool d) : t((int64_t)((d ? ~top : top) ^ 0x8000000000000000ull)), desc(d) {}
  NFC_DEV bool operator()(uint64_t raw) const { return desc ? (int64_t)raw >= t : (int64_t)raw <= t; }
};
// float64: the zeros compare equal, as their images do.  Descending, NaN rows
// come first (image 0) and pass as "not below"; ascending they come last and
// fail "at most" (only a threshold on the NaN image itself lets them in).
// Thresholds outside the images of numbers become the infinity on that side.
template <>
struct TkUnder<NFC_F64> {
  double t;
  bool desc, all;
  NFC_DEV TkUnder(uint64_t top, bool d) : desc(d), all(top == ~0ull) {
    const uint64_t inf = f64_ord(0x7FF0000000000000ull), ninf = f64_ord(0xFFF0000000000000ull);
    const uint64_t u = min(max(d ? ~top : top, ninf), inf);
    t = __longlong_as_double((long long)f64_unord(u));
  }
  NFC_DEV bool operator()(uint64_t raw) const {
    const double v = __longlong_as_double((long long)raw);
    return desc ? !(v < t) : (v <= t || all);
  }
};

// Every valid row up to the threshold, in any order.
template <int DT>
__global__ void __launch_bounds__(kTkThreads, 4) k_tk_collect(const void* __restrict__ keys,
                                                             const uint8_t* __restrict__ validity, int64_t n,
                                                             bool vec, bool desc, TkSample* st,
                                                             uint64_t* __restrict__ c_img,
                                                             uint32_t* __restrict__ c_row) {
  using R = typename std::conditional<DT == NFC_I32, uint32_t, uint64_t>::type;
  if (!st->ready) return;
  const uint64_t image_bits = DT == NFC_I32 ? 0xFFFFFFFFull : ~0ull;
  const TkUnder<DT> under((st->prefix | ~st->mask) & image_bits, desc);
  const R* col = static_cast<const R*>(keys);
  const int lane = lane_id();
  const int64_t ngroups = (n + 3) / 4;
  const int64_t stride = (int64_t)gridDim.x * kTkThreads;
  constexpr int U = 4;
  for (int64_t g0 = blockIdx.x * (int64_t)kTkThreads + (threadIdx.x & ~31u); g0 < ngroups; g0 += U * stride) {
    R raw[U][4];
    uint32_t ok[U], hit = 0;
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i0 = (g0 + u * stride + lane) * 4;
      ok[u] = i0 + 4 <= n ? 0xFu : (i0 < n ? (1u << (uint32_t)(n - i0)) - 1u : 0u);
      if (vec && i0 + 4 <= n) {
        if constexpr (DT == NFC_I32) {
          const uint4 q = __ldcs(reinterpret_cast<const uint4*>(col + i0));
          raw[u][0] = q.x; raw[u][1] = q.y; raw[u][2] = q.z; raw[u][3] = q.w;
        } else {
          const ulonglong2* p = reinterpret_cast<const ulonglong2*>(col + i0);
          const ulonglong2 x = __ldcs(p), y = __ldcs(p + 1);
          raw[u][0] = x.x; raw[u][1] = x.y; raw[u][2] = y.x; raw[u][3] = y.y;
        }
      } else {
#pragma unroll
        for (int r = 0; r < 4; ++r) raw[u][r] = i0 + r < n ? col[i0 + r] : (R)0;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i0 = (g0 + u * stride + lane) * 4;
      if (validity && ok[u]) ok[u] &= (uint32_t)(__ldg(validity + (i0 >> 3)) >> (i0 & 7)) & 0xFu;
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (((ok[u] >> r) & 1u) && under(raw[u][r])) hit |= 1u << (4 * u + r);
    }
    if (!__any_sync(0xffffffffu, hit != 0u)) continue;
    // Rare: one reservation per warp.  Once the buffer is full the exact
    // passes will run, so the rest of the column does not matter.
    const uint32_t mine = (uint32_t)__popc(hit);
    uint32_t incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    uint32_t base = 0;
    if (lane == 31) base = atomicAdd(&st->count, incl);
    base = __shfl_sync(0xffffffffu, base, 31);
    if (base >= (uint32_t)kTkCap) return;
    uint32_t pos = base + incl - mine;
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if ((hit >> (4 * u + r)) & 1u) {
          if (pos < (uint32_t)kTkCap) {
            c_img[pos] = tk_image_bits<DT>(raw[u][r], desc);
            c_row[pos] = (uint32_t)((g0 + u * stride + lane) * 4 + r);
          }
          ++pos;
        }
  }
}

// The collected rows in order of (image, row) -- descending float64 NaN rows
// (image 0) by descending row -- first k rows out.  A row's place is the number
// of rows before it, counted by a warp against all of them: the ~20 M
// comparisons of 5,000 rows are microseconds over the whole chip, where one
// CTA's bitonic sort took 114 us.
__global__ void __launch_bounds__(kTkFinalThreads) k_tk_final(TkSample* st, bool nan_last_first, uint32_t k,
                                                        const uint64_t* __restrict__ c_img,
                                                        const uint32_t* __restrict__ c_row,
                                                        int32_t* __restrict__ perm) {
  extern __shared__ __align__(16) unsigned char tk_smem[];
  const uint32_t cnt = st->count;
  if (!st->ready || cnt < k || cnt > (uint32_t)kTkCap) {
    if (blockIdx.x == 0 && threadIdx.x == 0) st->status = 1u;
    return;
  }
  uint64_t* si = reinterpret_cast<uint64_t*>(tk_smem);
  uint32_t* sr = reinterpret_cast<uint32_t*>(si + kTkCap);
#pragma unroll 4
  for (uint32_t i = threadIdx.x; i < cnt; i += kTkFinalThreads) {
    const uint64_t v = c_img[i];
    const uint32_t r = c_row[i];
    si[i] = v;
    sr[i] = nan_last_first && v == 0ull ? ~r : r;
  }
  __syncthreads();
  const uint32_t lane = lane_id();
  for (uint32_t i = blockIdx.x + gridDim.x * (threadIdx.x >> 5); i < cnt;
       i += gridDim.x * (kTkFinalThreads / 32)) {
    const uint64_t v = si[i];
    const uint32_t r = sr[i];
    uint32_t before = 0;
#pragma unroll 8
    for (uint32_t j = lane; j < cnt; j += 32) {
      const uint64_t w = si[j];
      before += (w < v || (w == v && sr[j] < r)) ? 1u : 0u;
    }
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0 && before < k) perm[before] = (int32_t)(nan_last_first && v == 0ull ? ~r : r);
  }
}

unsigned tk_grid(int64_t n) {
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + kTkThreads - 1) / kTkThreads, (int64_t)num_sms() * 8));
}

}  // namespace
}  // namespace nfc

using namespace nfc;

namespace {

int tk_status(cudaStream_t s, const int32_t* d_err) {
  int32_t h = 0;
  NFC_CUDA(readback(&h, d_err, sizeof(int32_t), s));
  return h;
}

// Sample rank of the threshold when one group in `step` is sampled: it gets six
// standard deviations and 16 rows more than k / step, so that the k-th row is
// missed about once in 1e8 calls on rows that the sample represents (and the
// exact passes then run).
int64_t tk_target(int64_t k, int64_t step) {
  if (step == 1) return k;
  const double q = (double)k / (double)step;
  return (int64_t)(q + 6.0 * std::sqrt(q) + 16.0) + 1;
}

// The sampled form, for k small enough that its rows fit k_tk_final's list.
// *done = 0: not tried, or the threshold did not hold.  Where the sample went
// through all its digits and many rows were still on the prefix (ties),
// hint->mask is set: the k-th image is very likely on hint->prefix.  Where the
// sample was the whole column and had too few valid rows, hint->hist is the
// first digit's histogram.
struct TkHint {
  uint64_t prefix, mask;
  int shift;  // bits below the prefix
  bool whole;
  uint32_t hist[kTkBins];
};

template <int DT>
int topk_sampled(const void* keys, const uint8_t* validity, int64_t n, bool desc, int64_t k, int32_t* perm_out,
                 cudaStream_t s, int* done, TkHint* hint) {
  *done = 0;
  // About a million sampled rows at 64M (their histograms take a tenth of the
  // pass), fewer groups skipped where k needs a sharper threshold.
  int64_t step = std::min<int64_t>(64, std::max<int64_t>(1, n >> 20));
  while (step > 1 && tk_target(k, step) * step > kTkExpect) step = step / 2;
  if (tk_target(k, step) * step > kTkExpect || (step < 8 && n >= (1 << 24))) return NFC_OK;
  Scratch sc(s);
  TkSample* st = nullptr;
  uint64_t* c_img = nullptr;
  uint32_t* c_row = nullptr;
  NFC_CUDA(sc.alloc(&st, 1));
  NFC_CUDA(sc.alloc(&c_img, (size_t)kTkCap));
  NFC_CUDA(sc.alloc(&c_row, (size_t)kTkCap));
  NFC_CUDA(cudaMemsetAsync(st, 0, sizeof(TkSample), s));
  const bool vec = (reinterpret_cast<uintptr_t>(keys) & 15u) == 0;
  const int bits = DT == NFC_I32 ? 32 : 64;
  const unsigned gs = (unsigned)std::max<int64_t>(
      1, std::min<int64_t>((n / 4 / step + 1023) / 1024, (int64_t)num_sms() * 4));
  const uint32_t target = (uint32_t)tk_target(k, step);
  for (int level = 0, shift = bits; level < kTkLevels && shift > 0; ++level) {
    const int dbits = std::min(kTkDigitBits, shift);
    shift -= dbits;
    k_tk_sample<DT><<<gs, kTkThreads, 0, s>>>(keys, validity, n, vec, desc, level, shift, (1u << dbits) - 1u,
                                              (uint32_t)step, target, st);
    NFC_CUDA(cudaGetLastError());
    if (level == 0 && step == 1 && validity) {
      // A whole column of NULL rows need not go through the other kernels (1M
      // rows, 500 valid: 166 us through all of them, 121 this way).
      TkSampleHead h;
      NFC_CUDA(readback(&h, static_cast<TkSampleHead*>(st), sizeof(h), s));
      if (h.failed) {
        hint->whole = true;
        NFC_CUDA(readback(hint->hist, st->hist[0], sizeof(hint->hist), s));
        return NFC_OK;
      }
    }
  }
  const unsigned gc =
      (unsigned)std::max<int64_t>(1, std::min<int64_t>((n / 16 + 255) / 256, (int64_t)num_sms() * 4));
  k_tk_collect<DT><<<gc, kTkThreads, 0, s>>>(keys, validity, n, vec, desc, st, c_img, c_row);
  NFC_CUDA(cudaGetLastError());
  constexpr int smem = kTkCap * 12;
  NFC_CUDA(allow_dynamic_smem<k_tk_final>());
  k_tk_final<<<(unsigned)num_sms(), kTkFinalThreads, smem, s>>>(st, DT == NFC_F64 && desc, (uint32_t)k, c_img, c_row, perm_out);
  NFC_CUDA(cudaGetLastError());
  TkSampleHead h;
  NFC_CUDA(readback(&h, static_cast<TkSampleHead*>(st), sizeof(h), s));
  *done = h.status == 0;
  if (h.status && !h.ready && !h.failed) {
    hint->prefix = h.prefix;
    hint->mask = h.mask;
    hint->shift = std::max(0, bits - kTkLevels * kTkDigitBits);
  }
  return NFC_OK;
}

template <int DT>
int topk_impl(const void* keys, const uint8_t* validity, int64_t n, bool desc, int64_t k, int32_t* perm_out,
              cudaStream_t s) {
  using K = typename std::conditional<DT == NFC_I32, uint32_t, uint64_t>::type;
  TkHint hint;
  hint.mask = 0;
  hint.whole = false;
  {
    int done = 0;
    const int rc = topk_sampled<DT>(keys, validity, n, desc, k, perm_out, s, &done, &hint);
    if (rc || done) return rc;
  }
  Scratch sc(s);
  int32_t* d_err = nullptr;
  uint32_t* hist = nullptr;
  NFC_CUDA(sc.alloc(&d_err, 4));
  NFC_CUDA(sc.alloc(&hist, kTkBins));
  NFC_CUDA(cudaMemsetAsync(d_err, 0, 4 * sizeof(int32_t), s));
  const bool vec = (reinterpret_cast<uintptr_t>(keys) & 15u) == 0;
  // ---- selection: prefix / mask of the k-th smallest image, ties to take.
  const int bits = DT == NFC_I32 ? 32 : 64;
  uint64_t mask = 0, prefix = 0;
  int shift = bits;
  int64_t nv = 0, ksel = 0, need = 0, on_prefix = 0;
  uint32_t hh[kTkBins];
  bool first = true;
  bool use_cand = false, found = false;
  if (hint.mask) {
    // One count over the column in place of its digit histograms, if the k-th
    // image is where the sample says (100M int32 of 1,000 values: three of them).
    unsigned long long* d_cnt = nullptr;
    unsigned long long c[3] = {0, 0, 0};  // valid, below, on the prefix
    NFC_CUDA(sc.alloc(&d_cnt, 3));
    NFC_CUDA(cudaMemsetAsync(d_cnt, 0, sizeof(c), s));
    k_tk_below<DT><<<tk_grid((n + 3) / 4), kTkThreads, 0, s>>>(keys, validity, n, vec, desc, hint.mask, hint.prefix,
                                                               d_cnt);
    NFC_CUDA(cudaGetLastError());
    NFC_CUDA(readback(c, d_cnt, sizeof(c), s));
    if (k < (int64_t)c[0] && (int64_t)c[1] < k && k <= (int64_t)(c[1] + c[2])) {
      first = false;
      nv = (int64_t)c[0];
      ksel = k;
      need = k - (int64_t)c[1];
      on_prefix = (int64_t)c[2];
      prefix = hint.prefix;
      mask = hint.mask;
      shift = hint.shift;
      use_cand = on_prefix != need && on_prefix <= kTkCandCap && shift > 0;
      found = on_prefix == need || use_cand;
    }
  }
  while (shift > 0 && !found) {
    const int dbits = std::min(kTkDigitBits, shift);
    shift -= dbits;
    const uint32_t dmask = (1u << dbits) - 1u;
    if (first && hint.whole) {
      std::copy(hint.hist, hint.hist + kTkBins, hh);
    } else {
      NFC_CUDA(cudaMemsetAsync(hist, 0, sizeof(uint32_t) * (dmask + 1), s));
      k_tk_hist<DT><<<tk_grid((n + 3) / 4), kTkThreads, 0, s>>>(keys, validity, n, vec, desc, mask, prefix, shift,
                                                                dmask, hist);
      NFC_CUDA(cudaGetLastError());
      NFC_CUDA(readback(hh, hist, sizeof(uint32_t) * (dmask + 1), s));
    }
    if (first) {
      first = false;
      for (uint32_t d = 0; d <= dmask; ++d) nv += hh[d];
      ksel = std::min(k, nv);
      need = ksel;
      if (ksel == nv) {  // every valid row is taken: all of them sit on the empty prefix
        on_prefix = nv;
        break;
      }
    }
    int64_t cum = 0;
    uint32_t d = 0;
    while (d < dmask && cum + hh[d] < need) cum += hh[d++];
    need -= cum;
    prefix |= (uint64_t)d << shift;
    mask |= (uint64_t)dmask << shift;
    on_prefix = hh[d];
    if (on_prefix == need) break;  // the whole prefix group is taken
    if (on_prefix <= kTkCandCap && shift > 0) {
      use_cand = true;  // the rest of the selection runs on the prefix group
      break;
    }
  }
  if (on_prefix < need) {
    set_last_error("topk: selection found %lld rows on the prefix for %lld", (long long)on_prefix, (long long)need);
    return NFC_ERR_RANGE;
  }
  // Descending float64 NaNs (image 0) are taken from the end of their block.
  const int64_t tie_lo = (DT == NFC_F64 && desc && prefix == 0) ? on_prefix - need : 0;
  // ---- compaction of the taken rows (and the first k - nv NULL rows).
  const int64_t nb = (n + kTkBlockRows - 1) / kTkBlockRows;
  uint32_t *row = nullptr, *row_alt = nullptr;
  K *img = nullptr, *img_alt = nullptr;
  NFC_CUDA(sc.alloc(&img, (size_t)std::max<int64_t>(1, ksel)));
  NFC_CUDA(sc.alloc(&img_alt, (size_t)std::max<int64_t>(1, ksel)));
  NFC_CUDA(sc.alloc(&row, (size_t)std::max<int64_t>(1, ksel)));
  NFC_CUDA(sc.alloc(&row_alt, (size_t)std::max<int64_t>(1, ksel)));
  if (!use_cand) {
    uint32_t *cnt = nullptr, *pre = nullptr;
    NFC_CUDA(sc.alloc(&cnt, (size_t)(3 * nb)));
    NFC_CUDA(sc.alloc(&pre, (size_t)(3 * nb)));
    k_tk_count<DT><<<(unsigned)nb, kTkThreads, 0, s>>>(keys, validity, n, desc, mask, prefix, cnt);
    NFC_CUDA(cudaGetLastError());
    k_tk_scan<<<1, 1024, 0, s>>>(cnt, nb, pre);
    NFC_CUDA(cudaGetLastError());
    const int64_t null_take = k - ksel;  // NULL rows follow every valid row
    k_tk_compact<DT, K><<<(unsigned)nb, kTkThreads, 0, s>>>(keys, validity, n, desc, mask, prefix, pre,
                                                           (uint32_t)tie_lo, (uint32_t)need, (uint32_t)ksel,
                                                           (uint32_t)null_take, img, row, perm_out + ksel, d_err);
    NFC_CUDA(cudaGetLastError());
  } else {
    // Taken rows (ksel - need of them) straight to img/row; the prefix group
    // to the candidate buffer, sorted by image (stable: input order within
    // equal images); its first `need` entries are the rest of the selection.
    // Descending float64 with the NaN block on the prefix (prefix 0: NaN and
    // +inf rows): when the block is cut, its last `need` rows are taken.
    // ksel < nv here, so no NULL row is part of the output.
    const int64_t cum = ksel - need;
    K *c_img = nullptr, *c_img_alt = nullptr;
    uint32_t *c_row = nullptr, *c_row_alt = nullptr;
    uint64_t* lb = nullptr;
    NFC_CUDA(sc.alloc(&c_img, (size_t)on_prefix));
    NFC_CUDA(sc.alloc(&c_img_alt, (size_t)on_prefix));
    NFC_CUDA(sc.alloc(&c_row, (size_t)on_prefix));
    NFC_CUDA(sc.alloc(&c_row_alt, (size_t)on_prefix));
    const int64_t ns = (n + kTkSplitRows - 1) / kTkSplitRows;
    NFC_CUDA(sc.alloc(&lb, (size_t)ns + 1));
    uint32_t* ticket = reinterpret_cast<uint32_t*>(lb + ns);
    NFC_CUDA(cudaMemsetAsync(lb, 0, sizeof(uint64_t) * (ns + 1), s));
    k_tk_split<DT, K><<<(unsigned)ns, kTkThreads, 0, s>>>(keys, validity, n, vec, desc, mask, prefix, (uint32_t)cum,
                                                         (uint32_t)on_prefix, img, row, c_img, c_row, lb, ticket,
                                                         d_err);
    NFC_CUDA(cudaGetLastError());
    K* ckr = nullptr;
    uint32_t* cvr = nullptr;
    int rc;
    if constexpr (DT == NFC_I32)
      rc = radix_sort_u32(c_img, c_img_alt, c_row, c_row_alt, on_prefix, 32, false, s, sc, &ckr, &cvr);
    else
      rc = radix_sort_u64(c_img, c_img_alt, c_row, c_row_alt, on_prefix, 64, false, s, sc, &ckr, &cvr);
    if (rc) return rc;
    int64_t off = 0;
    if (DT == NFC_F64 && desc && prefix == 0) {
      unsigned long long* d_z = nullptr;
      NFC_CUDA(sc.alloc(&d_z, 1));
      NFC_CUDA(cudaMemsetAsync(d_z, 0, sizeof(unsigned long long), s));
      k_tk_zero_count<K><<<tk_grid(on_prefix), kTkThreads, 0, s>>>(ckr, on_prefix, d_z);
      NFC_CUDA(cudaGetLastError());
      unsigned long long h_z = 0;
      NFC_CUDA(readback(&h_z, d_z, sizeof(h_z), s));
      if ((int64_t)h_z > need) off = (int64_t)h_z - need;
    }
    NFC_CUDA(cudaMemcpyAsync(img + cum, ckr + off, sizeof(K) * need, cudaMemcpyDeviceToDevice, s));
    NFC_CUDA(cudaMemcpyAsync(row + cum, cvr + off, sizeof(uint32_t) * need, cudaMemcpyDeviceToDevice, s));
  }
  // ---- sort of the taken rows by image (stable: they are in input order).
  K* kr = nullptr;
  if (ksel > 0) {
    uint32_t* vr = nullptr;
    int rc;
    if constexpr (DT == NFC_I32)
      rc = radix_sort_u32(img, img_alt, row, row_alt, ksel, 32, false, s, sc, &kr, &vr);
    else
      rc = radix_sort_u64(img, img_alt, row, row_alt, ksel, 64, false, s, sc, &kr, &vr);
    if (rc) return rc;
    NFC_CUDA(cudaMemcpyAsync(perm_out, vr, sizeof(int32_t) * ksel, cudaMemcpyDeviceToDevice, s));
  }
  if (DT == NFC_F64 && desc && ksel > 0) {
    // The taken NaN rows (image 0) lead the sorted selection; reverse them.
    unsigned long long* d_nan = nullptr;
    NFC_CUDA(sc.alloc(&d_nan, 1));
    NFC_CUDA(cudaMemsetAsync(d_nan, 0, sizeof(unsigned long long), s));
    k_tk_zero_count<K><<<tk_grid(ksel), kTkThreads, 0, s>>>(kr, ksel, d_nan);
    NFC_CUDA(cudaGetLastError());
    unsigned long long h_nan = 0;
    NFC_CUDA(readback(&h_nan, d_nan, sizeof(h_nan), s));
    const int64_t m = std::min<int64_t>(ksel, (int64_t)h_nan);
    if (m > 1) {
      k_tk_reverse<<<tk_grid(m / 2 + 1), kTkThreads, 0, s>>>(perm_out, m);
      NFC_CUDA(cudaGetLastError());
    }
  }
  return tk_status(s, d_err);
}

}  // namespace

extern "C" int32_t nfc_sort_topk(int32_t dtype, const void* keys, const uint8_t* validity, int64_t n,
                                 int32_t descending, int64_t k, int32_t* perm_out, void* stream) {
  if (n < 0 || k < 0 || k > n) return NFC_ERR_MALFORMED;
  if (k == 0) return NFC_OK;
  if (!keys || !perm_out) return NFC_ERR_NULL;
  if (dtype != NFC_I32 && dtype != NFC_I64 && dtype != NFC_F64) return NFC_ERR_MALFORMED;
  if (n >= (1ll << 30)) {
    set_last_error("topk: n=%lld >= 2^30", (long long)n);
    return NFC_ERR_UNSUPPORTED;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (k * 8 > n || n < 65536) {
    // Most rows are kept (or few exist): the full argsort, then its first k.
    Scratch sc(s);
    int32_t* full = nullptr;
    NFC_CUDA(sc.alloc(&full, (size_t)n));
    const int32_t rc = nfc_sort_perm(dtype, keys, validity, n, descending, full, stream);
    if (rc) return rc;
    NFC_CUDA(cudaMemcpyAsync(perm_out, full, sizeof(int32_t) * k, cudaMemcpyDeviceToDevice, s));
    return NFC_OK;
  }
  const bool desc = descending != 0;
  if (dtype == NFC_I32) return topk_impl<NFC_I32>(keys, validity, n, desc, k, perm_out, s);
  if (dtype == NFC_I64) return topk_impl<NFC_I64>(keys, validity, n, desc, k, perm_out, s);
  return topk_impl<NFC_F64>(keys, validity, n, desc, k, perm_out, s);
}

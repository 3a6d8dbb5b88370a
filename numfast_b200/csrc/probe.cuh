// Pieces of the probe shared by its kernels: the call's validity bitmaps and
// the in-order reduction of key range, count and sortedness.
#pragma once

#include "groupby_host.h"

namespace nfc {

struct BitmapSet {
  int32_t nbm;
  uint32_t word_aligned;  // bit b: bitmap b is 4-byte aligned
  const uint8_t* bm[NFC_MAX_COLS + 2];  // key, columns, row filter
};

// Validity bits of rows [row0, row0+32) (row0 multiple of 32); only the
// bitmap bytes that cover rows < n are read.
NFC_DEV uint32_t bitmap_word(const uint8_t* bm, bool aligned4, int64_t row0, int64_t rem) {
  const uint8_t* p = bm + (row0 >> 3);
  if (rem >= 32) {
    if (aligned4) return __ldg(reinterpret_cast<const uint32_t*>(p));
    return (uint32_t)p[0] | ((uint32_t)p[1] << 8) | ((uint32_t)p[2] << 16) | ((uint32_t)p[3] << 24);
  }
  uint32_t w = 0;
  for (int i = 0; i < (int)((rem + 7) >> 3); ++i) w |= (uint32_t)p[i] << (8 * i);
  return w;
}

static inline BitmapSet bitmaps_of(const nfc_groupby_args* a) {
  BitmapSet bms{};
  if (a->key_validity) bms.bm[bms.nbm++] = a->key_validity;
  for (int c = 0; c < a->ncols; ++c)
    if (a->cols[c].validity) bms.bm[bms.nbm++] = a->cols[c].validity;
  if (a->row_filter) bms.bm[bms.nbm++] = a->row_filter;
  for (int b = 0; b < bms.nbm; ++b)
    if ((reinterpret_cast<uintptr_t>(bms.bm[b]) & 3u) == 0) bms.word_aligned |= 1u << b;
  return bms;
}

struct ProbeAcc {
  bool has, sorted;
  int32_t first, last, kmin, kmax;
  int64_t n;
};

NFC_DEV ProbeAcc probe_combine(const ProbeAcc& a, const ProbeAcc& b) {
  ProbeAcc r;
  r.has = a.has || b.has;
  r.sorted = a.sorted && b.sorted && !(a.has && b.has && b.first < a.last);
  r.first = a.has ? a.first : b.first;
  r.last = b.has ? b.last : a.last;
  r.kmin = min(a.kmin, b.kmin);
  r.kmax = max(a.kmax, b.kmax);
  r.n = a.n + b.n;
  return r;
}

NFC_DEV ProbeAcc probe_shfl_down(const ProbeAcc& a, int off) {
  ProbeAcc r;
  r.has = __shfl_down_sync(0xffffffffu, (int)a.has, off) != 0;
  r.sorted = __shfl_down_sync(0xffffffffu, (int)a.sorted, off) != 0;
  r.first = __shfl_down_sync(0xffffffffu, a.first, off);
  r.last = __shfl_down_sync(0xffffffffu, a.last, off);
  r.kmin = __shfl_down_sync(0xffffffffu, a.kmin, off);
  r.kmax = __shfl_down_sync(0xffffffffu, a.kmax, off);
  r.n = __shfl_down_sync(0xffffffffu, a.n, off);
  return r;
}

// In-order reduction of a warp's accumulators (lane order = row order).
NFC_DEV ProbeAcc probe_warp_reduce(ProbeAcc acc) {
  const int lane = lane_id();
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const ProbeAcc other = probe_shfl_down(acc, off);
    if ((lane & (2 * off - 1)) == 0) acc = probe_combine(acc, other);
  }
  return acc;
}

}  // namespace nfc

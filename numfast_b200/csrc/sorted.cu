// SORTED strategy: group-by over keys that are nondecreasing in row order.
//
// The reference plans "sorted" whenever the valid keys are nondecreasing
// (src/Runtime/Planner/_lib/planner.py:226) and reduces each run of equal
// keys in one pass (sorted_fused_aggregate, src/Drivers/CPU/_lib/
// groupindex.py:259-304; sorted_runs, numfast-native/src/groupby/sorted.rs:
// 24-56).  The output contract is the one of every strategy: groups
// ascending by key, int64 counts and integer sums, float64 sums, min/max in
// the value dtype, rows with a NULL anywhere dropped.
//
// Here, with no atomics and no aggregation state in global memory:
//   1. k_sorted_prev    one CTA turns the probe records into the last valid
//                       key before every tile (an exclusive "last non-empty"
//                       scan over the 16,384-row blocks the probe summarised);
//   2. k_sorted_agg     one CTA per tile of 2,048 or 4,096 rows, claimed in
//                       order, a thread per 8 or 16 consecutive rows.  A thread finds its
//                       run heads (valid rows whose key differs from the
//                       previous valid row's), sums the rows before its first
//                       head and after its last one into shared memory, and a
//                       decoupled look-back gives the tile its first run
//                       number.  The thread that holds a run's head then adds
//                       what the threads after it have of that run (a whole
//                       warp without heads is one step) and writes the run.
//                       The tile's first run (continued from earlier tiles) and
//                       last run (possibly continued by later ones) leave as
//                       two partial "pieces";
//   3. k_sorted_fix     the pieces are merged in order (segmented scan by run
//                       number): chunks of 1,024 in parallel CTAs, then the
//                       chunks' own edge runs in one CTA.
// Output keys are written by the thread holding each run's head.  float64 sums
// differ from the reference's row loop in the order of their additions (mean
// relative error of a run's sum below 2^-53); everything else is exact.
#include <algorithm>
#include <type_traits>

#include "groupby_host.h"

namespace nfc {
namespace {

constexpr int kSoThreads = 256;                    // threads with rows; one more warp looks back
constexpr int kSoWarps = kSoThreads / 32;
// Consecutive rows per thread and rows per tile: more where a row is little work.
constexpr int so_rows(int nc) { return nc <= 1 ? 16 : 8; }
constexpr int so_tile(int nc) { return kSoThreads * so_rows(nc); }
static_assert(kProbeBlockRows % so_tile(0) == 0 && kProbeBlockRows % so_tile(4) == 0,
              "tiles do not straddle probe records");
constexpr int kFixThreads = 1024;

// ---------------------------------------------------------------- run aggregate
// Integers are kept as int64 bits (sums wrap like the other strategies' int64
// atomics), float64 min/max as the ordered encodings of nfc_common.cuh;
// int32 min/max use int32 identities and 32-bit compares.  A count never
// exceeds the row count (< 2^31).
//
// A float64 sum of rows added one after the other loses with the root of their
// number.  So a thread adds its rows in fours (`rest`, added to the sum by
// seg_add_four), and combining two run aggregates keeps the rounding error of the
// float64 addition in `rest` (seg_close adds it).  Mean relative error of a sum,
// 20M rows in runs of 200: 1.2e-16 with plain chains, 7e-17 as a tree over the
// rows, 4.5e-17 this way; the errors of every single row as well: 4.4e-17, but
// 5-12% of the time.
template <int NC>
struct Seg {
  uint32_t cnt;
  uint64_t sum[NC > 0 ? NC : 1], mn[NC > 0 ? NC : 1], mx[NC > 0 ? NC : 1];
  double rest[NC > 0 ? NC : 1];
};

template <int NC, uint32_t SIG>
NFC_DEV void seg_identity(const ColSet& cs, Seg<NC>& a) {
  a.cnt = 0;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    a.sum[c] = 0;
    a.rest[c] = 0.0;
    if (col_dt<SIG>(cs, c) == NFC_F64) {
      a.mn[c] = ~0ull;
      a.mx[c] = 0ull;
    } else if (col_dt<SIG>(cs, c) == NFC_I32) {
      a.mn[c] = (uint64_t)(int64_t)INT_MAX;
      a.mx[c] = (uint64_t)(int64_t)INT_MIN;
    } else {
      a.mn[c] = (uint64_t)LLONG_MAX;
      a.mx[c] = (uint64_t)LLONG_MIN;
    }
  }
}

NFC_DEV uint64_t i32_min64(uint64_t a, uint64_t b) { return (uint64_t)(int64_t)min((int32_t)a, (int32_t)b); }
NFC_DEV uint64_t i32_max64(uint64_t a, uint64_t b) { return (uint64_t)(int64_t)max((int32_t)a, (int32_t)b); }
NFC_DEV uint64_t f64_add_bits(uint64_t a, uint64_t b) {
  return (uint64_t)__double_as_longlong(__longlong_as_double((long long)a) + __longlong_as_double((long long)b));
}

template <int NC, uint32_t SIG>
NFC_DEV void seg_add_four(const ColSet& cs, Seg<NC>& a) {
#pragma unroll
  for (int c = 0; c < NC; ++c)
    if (col_dt<SIG>(cs, c) == NFC_F64 && (col_ag<SIG>(cs, c) & NFC_AGG_SUM)) {
      a.sum[c] = f64_add_bits(a.sum[c], (uint64_t)__double_as_longlong(a.rest[c]));
      a.rest[c] = 0.0;
    }
}

template <int NC, uint32_t SIG>
NFC_DEV void seg_close(const ColSet& cs, Seg<NC>& a) {
#pragma unroll
  for (int c = 0; c < NC; ++c)
    if (col_dt<SIG>(cs, c) == NFC_F64 && (col_ag<SIG>(cs, c) & NFC_AGG_SUM)) {
      a.sum[c] = (uint64_t)__double_as_longlong(f64_close(__longlong_as_double((long long)a.sum[c]), a.rest[c]));
      a.rest[c] = 0.0;
    }
}

// a = a then b.
template <int NC, uint32_t SIG>
NFC_DEV void seg_combine(const ColSet& cs, Seg<NC>& a, const Seg<NC>& b) {
  a.cnt += b.cnt;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int dt = col_dt<SIG>(cs, c), ag = col_ag<SIG>(cs, c);
    if (dt == NFC_F64) {
      if (ag & NFC_AGG_SUM) {
        double t = __longlong_as_double((long long)a.sum[c]);
        a.rest[c] += b.rest[c] + f64_two_sum(t, __longlong_as_double((long long)b.sum[c]));
        a.sum[c] = (uint64_t)__double_as_longlong(t);
      }
      if (ag & NFC_AGG_MIN) a.mn[c] = min(a.mn[c], b.mn[c]);
      if (ag & NFC_AGG_MAX) a.mx[c] = max(a.mx[c], b.mx[c]);
    } else if (dt == NFC_I32) {
      if (ag & NFC_AGG_SUM) a.sum[c] += b.sum[c];
      if (ag & NFC_AGG_MIN) a.mn[c] = i32_min64(a.mn[c], b.mn[c]);
      if (ag & NFC_AGG_MAX) a.mx[c] = i32_max64(a.mx[c], b.mx[c]);
    } else {
      if (ag & NFC_AGG_SUM) a.sum[c] += b.sum[c];
      if (ag & NFC_AGG_MIN) a.mn[c] = (uint64_t)min((long long)a.mn[c], (long long)b.mn[c]);
      if (ag & NFC_AGG_MAX) a.mx[c] = (uint64_t)max((long long)a.mx[c], (long long)b.mx[c]);
    }
  }
}

// Fold one row: int32 values as their 32-bit word, 8-byte values as bits.
template <int NC, uint32_t SIG>
NFC_DEV void seg_add_row(const ColSet& cs, Seg<NC>& a, const uint64_t* raw) {
  a.cnt += 1;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int dt = col_dt<SIG>(cs, c), ag = col_ag<SIG>(cs, c);
    const uint64_t r = raw[c];
    if (dt == NFC_F64) {
      if (ag & NFC_AGG_SUM) a.rest[c] += __longlong_as_double((long long)r);
      if (ag & (NFC_AGG_MIN | NFC_AGG_MAX)) {
        // One order-preserving word for both lanes (the encodings of
        // nfc_common.cuh); NaN wins both.
        const uint32_t hi = (uint32_t)(r >> 32), lo = (uint32_t)r;
        const uint32_t s = (uint32_t)((int32_t)hi >> 31);
        const uint64_t ord = r ^ (((uint64_t)(s | 0x80000000u) << 32) | s);
        const uint32_t ah = hi & 0x7FFFFFFFu;
        const bool nan = ah > 0x7FF00000u || (ah == 0x7FF00000u && lo != 0u);
        if (ag & NFC_AGG_MIN) a.mn[c] = min(a.mn[c], nan ? (uint64_t)0 : ord);
        if (ag & NFC_AGG_MAX) a.mx[c] = max(a.mx[c], nan ? ~(uint64_t)0 : ord);
      }
    } else if (dt == NFC_I32) {
      if (ag & NFC_AGG_SUM) a.sum[c] += (uint64_t)(int64_t)(int32_t)r;
      if (ag & NFC_AGG_MIN) a.mn[c] = i32_min64(a.mn[c], r);
      if (ag & NFC_AGG_MAX) a.mx[c] = i32_max64(a.mx[c], r);
    } else {
      if (ag & NFC_AGG_SUM) a.sum[c] += r;
      if (ag & NFC_AGG_MIN) a.mn[c] = (uint64_t)min((long long)a.mn[c], (long long)r);
      if (ag & NFC_AGG_MAX) a.mx[c] = (uint64_t)max((long long)a.mx[c], (long long)r);
    }
  }
}

// Shuffles of a run aggregate: only the requested aggregates move, counts
// and int32 min/max as 32-bit words.
template <int NC, uint32_t SIG, bool UP>
NFC_DEV void seg_shfl(const ColSet& cs, const Seg<NC>& a, Seg<NC>& out, int arg) {
  auto sh32 = [&](uint32_t v) { return UP ? __shfl_up_sync(0xffffffffu, v, arg) : __shfl_sync(0xffffffffu, v, arg); };
  auto sh64 = [&](uint64_t v) { return UP ? __shfl_up_sync(0xffffffffu, v, arg) : __shfl_sync(0xffffffffu, v, arg); };
  out.cnt = sh32(a.cnt);
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int ag = col_ag<SIG>(cs, c);
    if (ag & NFC_AGG_SUM) out.sum[c] = sh64(a.sum[c]);
    if (col_dt<SIG>(cs, c) == NFC_F64 && (ag & NFC_AGG_SUM))
      out.rest[c] = __longlong_as_double((long long)sh64((uint64_t)__double_as_longlong(a.rest[c])));
    if (col_dt<SIG>(cs, c) == NFC_I32) {
      if (ag & NFC_AGG_MIN) out.mn[c] = (uint64_t)(int64_t)(int32_t)sh32((uint32_t)a.mn[c]);
      if (ag & NFC_AGG_MAX) out.mx[c] = (uint64_t)(int64_t)(int32_t)sh32((uint32_t)a.mx[c]);
    } else {
      if (ag & NFC_AGG_MIN) out.mn[c] = sh64(a.mn[c]);
      if (ag & NFC_AGG_MAX) out.mx[c] = sh64(a.mx[c]);
    }
  }
}

// All lanes' run aggregates (closed) combined: 32-bit fields by warp reductions, 64-bit
// ones by shuffles.
template <int NC, uint32_t SIG>
NFC_DEV void seg_warp_reduce(const ColSet& cs, const Seg<NC>& a, Seg<NC>& out) {
  out.cnt = __reduce_add_sync(0xffffffffu, a.cnt);
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int dt = col_dt<SIG>(cs, c), ag = col_ag<SIG>(cs, c);
    uint64_t s = a.sum[c], lo = a.mn[c], hi = a.mx[c];
    if (ag & NFC_AGG_SUM) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const uint64_t t = __shfl_xor_sync(0xffffffffu, s, o);
        s = dt == NFC_F64 ? f64_add_bits(s, t) : s + t;
      }
    }
    if (dt == NFC_I32) {
      if (ag & NFC_AGG_MIN) lo = (uint64_t)(int64_t)__reduce_min_sync(0xffffffffu, (int32_t)lo);
      if (ag & NFC_AGG_MAX) hi = (uint64_t)(int64_t)__reduce_max_sync(0xffffffffu, (int32_t)hi);
    } else {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        if (ag & NFC_AGG_MIN) {
          const uint64_t t = __shfl_xor_sync(0xffffffffu, lo, o);
          lo = dt == NFC_F64 ? min(lo, t) : (uint64_t)min((long long)lo, (long long)t);
        }
        if (ag & NFC_AGG_MAX) {
          const uint64_t t = __shfl_xor_sync(0xffffffffu, hi, o);
          hi = dt == NFC_F64 ? max(hi, t) : (uint64_t)max((long long)hi, (long long)t);
        }
      }
    }
    out.sum[c] = s;
    out.rest[c] = 0.0;
    out.mn[c] = lo;
    out.mx[c] = hi;
  }
}

// Output row g of run aggregate a, closed (keys are written at the heads).
template <int NC, uint32_t SIG>
NFC_DEV void seg_emit(const ColSet& cs, const OutSet& o, int64_t g, const Seg<NC>& a) {
  o.counts[g] = (int64_t)a.cnt;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int dt = col_dt<SIG>(cs, c), ag = col_ag<SIG>(cs, c);
    if (ag & NFC_AGG_SUM) static_cast<uint64_t*>(o.sum[c])[g] = a.sum[c];
    if (dt == NFC_I32) {
      if (ag & NFC_AGG_MIN) static_cast<int32_t*>(o.mn[c])[g] = (int32_t)a.mn[c];
      if (ag & NFC_AGG_MAX) static_cast<int32_t*>(o.mx[c])[g] = (int32_t)a.mx[c];
    } else if (dt == NFC_I64) {
      if (ag & NFC_AGG_MIN) static_cast<uint64_t*>(o.mn[c])[g] = a.mn[c];
      if (ag & NFC_AGG_MAX) static_cast<uint64_t*>(o.mx[c])[g] = a.mx[c];
    } else {
      if (ag & NFC_AGG_MIN) static_cast<uint64_t*>(o.mn[c])[g] = f64_min_dec(a.mn[c]);
      if (ag & NFC_AGG_MAX) static_cast<uint64_t*>(o.mx[c])[g] = f64_max_dec(a.mx[c]);
    }
  }
}

// Partial runs at tile (or chunk) edges: slot 2t = the run continued from
// before tile t, slot 2t+1 = the tile's last run; idx -1 = none.
struct Pieces {
  int64_t* idx;
  uint64_t* cnt;
  uint64_t* sum[NFC_MAX_COLS];
  uint64_t* mn[NFC_MAX_COLS];
  uint64_t* mx[NFC_MAX_COLS];
};

template <int NC>
NFC_DEV void piece_store(const Pieces& P, int64_t slot, int64_t idx, const Seg<NC>& a) {
  P.idx[slot] = idx;
  P.cnt[slot] = a.cnt;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    P.sum[c][slot] = a.sum[c];
    P.mn[c][slot] = a.mn[c];
    P.mx[c][slot] = a.mx[c];
  }
}

template <int NC>
NFC_DEV void piece_load(const Pieces& P, int64_t slot, Seg<NC>& a) {
  a.cnt = (uint32_t)P.cnt[slot];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    a.sum[c] = P.sum[c][slot];
    a.rest[c] = 0.0;
    a.mn[c] = P.mn[c][slot];
    a.mx[c] = P.mx[c][slot];
  }
}

// Warp-wide segmented scan.  Lane l holds (f, a): f = a run starts inside
// the lane.  The operator is (f1,a1) then (f2,a2) = (f1|f2, f2 ? a2 : a1+a2).
// (cf, ca) is the warp-uniform open run before lane 0.  Returns in ex the
// exclusive value of every lane (carry included) and advances the carry past
// lane 31.  The scan stops as soon as every lane has met a head.
template <int NC, uint32_t SIG>
NFC_DEV void warp_seg_scan(const ColSet& cs, uint32_t f, const Seg<NC>& a, uint32_t& cf, Seg<NC>& ca, Seg<NC>& ex) {
  const int lane = lane_id();
  uint32_t incf = f;
  Seg<NC> inc = a;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    if (__all_sync(0xffffffffu, incf)) break;
    Seg<NC> y;
    seg_shfl<NC, SIG, true>(cs, inc, y, o);
    const uint32_t yf = __shfl_up_sync(0xffffffffu, incf, o);
    if (lane >= o) {
      if (!incf) {
        seg_combine<NC, SIG>(cs, y, inc);
        inc = y;
      }
      incf |= yf;
    }
  }
  Seg<NC> w;
  seg_shfl<NC, SIG, true>(cs, inc, w, 1);
  const uint32_t wf = __shfl_up_sync(0xffffffffu, incf, 1);
  if (lane == 0 || !wf) {
    ex = ca;
    if (lane != 0) seg_combine<NC, SIG>(cs, ex, w);
  } else {
    ex = w;
  }
  Seg<NC> last;
  seg_shfl<NC, SIG, false>(cs, inc, last, 31);
  const uint32_t lastf = __shfl_sync(0xffffffffu, incf, 31);
  if (lastf) ca = last;
  else seg_combine<NC, SIG>(cs, ca, last);
  cf |= lastf;
}

// Block-wide segmented scan (same operator), blockDim a multiple of 32.
template <int NC, uint32_t SIG>
struct SegScanSmem {
  Seg<NC> tot[32];
  uint32_t totf[32];
  Seg<NC> wcarry[32];
  uint32_t wcarryf[32];
  Seg<NC> carry;
  uint32_t carryf;
};

template <int NC, uint32_t SIG>
NFC_DEV void block_seg_scan(const ColSet& cs, uint32_t f, const Seg<NC>& a, uint32_t& carry_f, Seg<NC>& carry,
                            Seg<NC>& excl, SegScanSmem<NC, SIG>& sm) {
  const int lane = lane_id(), warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  // Within the warp, from an empty carry: wex = the lanes before this one
  // (back to the nearest head), wtot = the whole warp.
  uint32_t wf = 0;
  Seg<NC> wtot, wex;
  seg_identity<NC, SIG>(cs, wtot);
  warp_seg_scan<NC, SIG>(cs, f, a, wf, wtot, wex);
  const bool head_before = (__ballot_sync(0xffffffffu, f) & ((1u << lane) - 1u)) != 0u;
  if (lane == 0) {
    sm.tot[warp] = wtot;
    sm.totf[warp] = wf;
  }
  __syncthreads();
  if (warp == 0) {
    uint32_t tf = 0;
    Seg<NC> t;
    seg_identity<NC, SIG>(cs, t);
    if (lane < nw) {
      t = sm.tot[lane];
      tf = sm.totf[lane];
    }
    uint32_t c2f = carry_f;
    Seg<NC> c2 = carry, ex;
    warp_seg_scan<NC, SIG>(cs, tf, t, c2f, c2, ex);  // ex = carry-in of warp `lane`
    if (lane < nw) sm.wcarry[lane] = ex;
    if (lane == 0) {
      sm.carry = c2;
      sm.carryf = c2f;
    }
  }
  __syncthreads();
  if (head_before) {
    excl = wex;
  } else {
    excl = sm.wcarry[warp];
    seg_combine<NC, SIG>(cs, excl, wex);
  }
  carry = sm.carry;
  carry_f = sm.carryf;
  __syncthreads();
}

// Last valid key before each probe block of kProbeBlockRows rows: prev[i] =
// (1 << 32 | key) or 0 when no valid row precedes it.  One CTA walks the probe
// records in order; it also empties the nq second-level pieces.
__global__ void __launch_bounds__(1024) k_sorted_prev(const ProbeRec* recs, int64_t nrec, uint64_t* prev,
                                                      int64_t* q_idx, int64_t nq) {
  for (int64_t i = threadIdx.x; i < nq; i += blockDim.x) q_idx[i] = -1;
  __shared__ uint64_t s_w[32];
  __shared__ uint64_t s_carry;
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (int64_t base = 0; base < nrec; base += blockDim.x) {
    const int64_t i = base + threadIdx.x;
    uint64_t v = 0;  // inclusive "last valid" of record i
    if (i < nrec) {
      const ProbeRec r = recs[i];
      if (r.flags & 1u) v = (1ull << 32) | (uint32_t)r.last;
    }
    uint64_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t y = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o && !(inc >> 32)) inc = y;
    }
    if (lane == 31) s_w[warp] = inc;
    __syncthreads();
    uint64_t before = s_carry;
    for (int w = 0; w < warp; ++w)
      if (s_w[w] >> 32) before = s_w[w];
    uint64_t ex = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane == 0) ex = 0;
    const uint64_t mine = (ex >> 32) ? ex : before;
    if (i < nrec) prev[i] = mine;
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) s_carry = (inc >> 32) ? inc : mine;
    __syncthreads();
  }
}

// Four rows' values of every column, from row (a multiple of 4) on: 32-bit
// words as they are, 8-byte values as bits; rows at or past n are not read.
template <int NC, uint32_t SIG>
NFC_DEV void load_rows4(const ColSet& cs, int64_t n, bool aligned, int64_t row, uint64_t (&v)[4][NC > 0 ? NC : 1]) {
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    if (aligned && row + 4 <= n) {
      if (col_dt<SIG>(cs, c) == NFC_I32) {
        const int4 x = __ldg(reinterpret_cast<const int4*>(static_cast<const int32_t*>(cs.data[c]) + row));
        v[0][c] = (uint32_t)x.x; v[1][c] = (uint32_t)x.y; v[2][c] = (uint32_t)x.z; v[3][c] = (uint32_t)x.w;
      } else {
        const ulonglong2* q = reinterpret_cast<const ulonglong2*>(static_cast<const uint64_t*>(cs.data[c]) + row);
        const ulonglong2 x = __ldg(q), y = __ldg(q + 1);
        v[0][c] = x.x; v[1][c] = x.y; v[2][c] = y.x; v[3][c] = y.y;
      }
    } else {
#pragma unroll
      for (int r = 0; r < 4; ++r)
        v[r][c] = row + r >= n                       ? 0ull
                  : col_dt<SIG>(cs, c) == NFC_I32 ? (uint64_t)(uint32_t) static_cast<const int32_t*>(cs.data[c])[row + r]
                                                  : static_cast<const uint64_t*>(cs.data[c])[row + r];
    }
  }
}

// A thread's rows of column c (load_rows4's conventions).
template <int kSoRows, uint32_t SIG>
NFC_DEV void load_rows(const ColSet& cs, int c, int64_t n, bool aligned, int64_t row, uint64_t (&v)[kSoRows]) {
  if (aligned && row + kSoRows <= n) {
    if (col_dt<SIG>(cs, c) == NFC_I32) {
      const int4* q = reinterpret_cast<const int4*>(static_cast<const int32_t*>(cs.data[c]) + row);
#pragma unroll
      for (int e = 0; e < kSoRows / 4; ++e) {
        const int4 x = __ldg(q + e);
        v[4 * e] = (uint32_t)x.x; v[4 * e + 1] = (uint32_t)x.y; v[4 * e + 2] = (uint32_t)x.z; v[4 * e + 3] = (uint32_t)x.w;
      }
    } else {
      const ulonglong2* q = reinterpret_cast<const ulonglong2*>(static_cast<const uint64_t*>(cs.data[c]) + row);
#pragma unroll
      for (int e = 0; e < kSoRows / 2; ++e) {
        const ulonglong2 x = __ldg(q + e);
        v[2 * e] = x.x;
        v[2 * e + 1] = x.y;
      }
    }
  } else {
#pragma unroll
    for (int r = 0; r < kSoRows; ++r)
      v[r] = row + r >= n                       ? 0ull
             : col_dt<SIG>(cs, c) == NFC_I32 ? (uint64_t)(uint32_t) static_cast<const int32_t*>(cs.data[c])[row + r]
                                             : static_cast<const uint64_t*>(cs.data[c])[row + r];
  }
}

// Partial runs of the tile's threads, one array per field so that neighbouring
// threads touch neighbouring words.
template <int NC>
struct Partials {
  uint64_t sum[NC > 0 ? NC : 1][kSoThreads];
  uint64_t mn[NC > 0 ? NC : 1][kSoThreads];
  uint64_t mx[NC > 0 ? NC : 1][kSoThreads];
  uint32_t cnt[kSoThreads];
};

template <int NC, uint32_t SIG>
NFC_DEV void part_store(const ColSet& cs, Partials<NC>& p, int t, const Seg<NC>& a) {
  p.cnt[t] = a.cnt;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int ag = col_ag<SIG>(cs, c);
    if (ag & NFC_AGG_SUM) p.sum[c][t] = a.sum[c];
    if (ag & NFC_AGG_MIN) p.mn[c][t] = a.mn[c];
    if (ag & NFC_AGG_MAX) p.mx[c][t] = a.mx[c];
  }
}

template <int NC, uint32_t SIG>
NFC_DEV void part_add(const ColSet& cs, Seg<NC>& a, const Partials<NC>& p, int t) {
  Seg<NC> b;
  b.cnt = p.cnt[t];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int ag = col_ag<SIG>(cs, c);
    b.sum[c] = ag & NFC_AGG_SUM ? p.sum[c][t] : 0ull;
    b.rest[c] = 0.0;
    b.mn[c] = ag & NFC_AGG_MIN ? p.mn[c][t] : 0ull;
    b.mx[c] = ag & NFC_AGG_MAX ? p.mx[c][t] : 0ull;
  }
  seg_combine<NC, SIG>(cs, a, b);
}

// CTAs per SM that the registers of the run aggregates leave room for.
template <int NC, uint32_t SIG>
constexpr int so_ctas() { return NC == 0 ? 4 : NC <= 2 ? 3 : 2; }

template <int NC, uint32_t SIG>
struct SortedSmem {
  union {
    Partials<NC> lead;             // rows before the thread's first head; all its rows when it has none
    uint64_t stage[so_tile(NC)];  // short runs: one output column of the tile's runs
  };
  Seg<NC> wsum[kSoWarps];  // all rows of a warp without heads
  uint64_t wlast[kSoWarps];  // last valid key of the warp (1 << 32 | key), 0 none
  uint32_t wheads[kSoWarps];
  uint32_t wany[kSoWarps];  // bit l: lane l has a head
  uint64_t carry;
  int64_t tile, excl;
};

// What bounds it: 40M rows of one int64 and one float64 sum in runs of 16 are
// 0.88 GB (135 us); the form with a segmented warp scan per 128 rows, four rows
// per lane, was issue bound at 1,145 us (and 16,384-row tiles left most SMs
// without work below 2M rows).
template <int NC, uint32_t SIG>
__global__ void __launch_bounds__(kSoThreads + 32, so_ctas<NC, SIG>())
    k_sorted_agg(const int32_t* __restrict__ keys, const uint32_t* __restrict__ vmask, ColSet cs, int64_t n,
                 bool aligned, const uint64_t* __restrict__ prev, OutSet o, int64_t cap, Pieces P, uint64_t* lb,
                 uint32_t* ticket, int64_t* ng_out, int32_t* err) {
  extern __shared__ __align__(128) unsigned char sm_raw[];
  SortedSmem<NC, SIG>& sm = *reinterpret_cast<SortedSmem<NC, SIG>*>(sm_raw);
  constexpr int kSoRows = so_rows(NC), kSoTile = so_tile(NC);
  const int tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
  if (tid == 0) sm.tile = atomicAdd(ticket, 1u);
  __syncthreads();
  const int64_t tile = sm.tile;
  const int64_t ntiles = (n + kSoTile - 1) / kSoTile;
  if (tile >= ntiles) return;
  const int64_t tbase = tile * kSoTile;
  if (warp == kSoWarps) {
    // The extra warp: last valid key before the tile (usually one of the 32
    // rows before it; else the rows back to the probe block's start, 1,024 at a
    // time, then the probe's own record), then the look-back, while the other
    // warps load and sum.
    const int64_t block = tbase / kProbeBlockRows;
    const int64_t w_lo = block * (kProbeBlockRows / 32);
    uint64_t carry = prev[block];
    int64_t w0 = tbase / 32 - 1;
    if (w0 >= w_lo) {
      const uint32_t bits = vmask ? __ldg(vmask + w0) : 0xFFFFFFFFu;
      const int32_t key = keys[tbase - 32 + lane];
      const int32_t got = __shfl_sync(0xffffffffu, key, bits ? 31 - __clz(bits) : 0);
      if (bits) carry = (1ull << 32) | (uint32_t)got;
      w0 = bits ? w_lo - 1 : w0 - 1;
    }
    for (; w0 >= w_lo; w0 -= 32) {
      const int64_t w = w0 - lane;
      const uint32_t bits = w < w_lo ? 0u : __ldg(vmask + w);  // a bitmap: without one every row is valid
      const unsigned nz = __ballot_sync(0xffffffffu, bits != 0u);
      if (nz) {
        const int l = __ffs(nz) - 1;
        const uint32_t b = __shfl_sync(0xffffffffu, bits, l);
        carry = (1ull << 32) | (uint32_t)keys[(w0 - l) * 32 + (31 - __clz(b))];
        break;
      }
    }
    if (lane == 0) sm.carry = carry;
    __syncthreads();  // carry and the warps' last keys
    __syncthreads();  // head counts
    const uint32_t total = __reduce_add_sync(0xffffffffu, lane < kSoWarps ? sm.wheads[lane] : 0u);
    const int64_t ex = lookback_exclusive(lb, tile, total, err);  // whole warp
    if (lane == 0) {
      sm.excl = ex;
      if (tile == ntiles - 1) *ng_out = ex + total;
    }
    __syncthreads();  // run numbers and partial sums
    return;
  }
  const int64_t row0 = tbase + tid * kSoRows;

  // ---- keys and validity of the thread's rows.
  int32_t k[kSoRows];
  constexpr uint32_t kAll = (1u << kSoRows) - 1u;
  uint32_t vb = row0 + kSoRows <= n ? kAll : row0 < n ? (1u << (uint32_t)(n - row0)) - 1u : 0u;
  if (vmask && vb) vb &= (__ldg(vmask + (row0 >> 5)) >> (row0 & 31)) & kAll;
  if (aligned && row0 + kSoRows <= n) {
#pragma unroll
    for (int e = 0; e < kSoRows / 4; ++e) {
      const int4 x = __ldg(reinterpret_cast<const int4*>(keys + row0) + e);
      k[4 * e] = x.x; k[4 * e + 1] = x.y; k[4 * e + 2] = x.z; k[4 * e + 3] = x.w;
    }
  } else {
#pragma unroll
    for (int r = 0; r < kSoRows; ++r) k[r] = row0 + r < n ? keys[row0 + r] : 0;
  }
  uint64_t last = 0;
#pragma unroll
  for (int r = 0; r < kSoRows; ++r)
    if (vb & (1u << r)) last = (1ull << 32) | (uint32_t)k[r];
  const unsigned has = __ballot_sync(0xffffffffu, vb != 0u);
  const unsigned below = has & lanemask_lt();
  const uint64_t before = __shfl_sync(0xffffffffu, last, below ? 31 - __clz(below) : 0);
  const uint64_t wl = __shfl_sync(0xffffffffu, last, has ? 31 - __clz(has) : 0);
  if (lane == 0) sm.wlast[warp] = has ? wl : 0ull;
  __syncthreads();

  // ---- run heads.
  uint64_t p = before;
  if (!below) {
    p = sm.carry;
    for (int w = 0; w < warp; ++w)
      if (sm.wlast[w]) p = sm.wlast[w];
  }
  uint32_t hb = 0;
#pragma unroll
  for (int r = 0; r < kSoRows; ++r)
    if (vb & (1u << r)) {
      if (p != ((1ull << 32) | (uint32_t)k[r])) hb |= 1u << r;
      p = (1ull << 32) | (uint32_t)k[r];
    }
  const uint32_t hc = (uint32_t)__popc(hb);
  uint32_t hi = hc;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, hi, off);
    if (lane >= off) hi += y;
  }
  const unsigned any = __ballot_sync(0xffffffffu, hb != 0u);
  if (lane == 31) sm.wheads[warp] = hi;
  if (lane == 0) sm.wany[warp] = any;
  __syncthreads();

  // ---- partial sums before the first and from the last head.
  Seg<NC> cur, lead;
  seg_identity<NC, SIG>(cs, cur);
  seg_identity<NC, SIG>(cs, lead);
#pragma unroll
  for (int q = 0; q < kSoRows / 4; ++q) {
    if (((vb >> (4 * q)) & 0xFu) == 0u) continue;
    uint64_t v[4][NC > 0 ? NC : 1];
    load_rows4<NC, SIG>(cs, n, aligned, row0 + 4 * q, v);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const uint32_t bit = 1u << (4 * q + r);
      if (hb & bit) {
        if ((hb & (bit - 1u)) == 0u) {
          seg_add_four<NC, SIG>(cs, cur);
          lead = cur;
        }
        seg_identity<NC, SIG>(cs, cur);
      }
      if (vb & bit) seg_add_row<NC, SIG>(cs, cur, v[r]);
    }
    seg_add_four<NC, SIG>(cs, cur);
  }
  part_store<NC, SIG>(cs, sm.lead, tid, hb ? lead : cur);
  if (any == 0u) {
    Seg<NC> w;
    seg_warp_reduce<NC, SIG>(cs, cur, w);
    if (lane == 0) sm.wsum[warp] = w;
  }
  __syncthreads();
  uint32_t total = 0, mine = 0;
  for (int w = 0; w < kSoWarps; ++w) {
    if (w < warp) mine += sm.wheads[w];
    total += sm.wheads[w];
  }
  const int64_t excl = sm.excl;

  // Adds to `a` what the threads from t on hold of an open run, and closes it;
  // true when the run ends inside the tile.
  auto follow = [&](Seg<NC>& a, int t) {
    bool ends = false;
    while (t < kSoThreads) {
      const uint32_t rest = sm.wany[t >> 5] >> (t & 31);
      if (rest == 0u && (t & 31) == 0) {
        seg_combine<NC, SIG>(cs, a, sm.wsum[t >> 5]);
        t += 32;
        continue;
      }
      part_add<NC, SIG>(cs, a, sm.lead, t);
      if (rest & 1u) {
        ends = true;
        break;
      }
      ++t;
    }
    seg_close<NC, SIG>(cs, a);
    return ends;
  };
  // The run that the tile continues (its rows before the first head).
  if (tid == 0) {
    Seg<NC> run = hb ? lead : any ? cur : sm.wsum[0];
    if (!hb) follow(run, any ? 1 : 32);
    if (run.cnt > 0) piece_store<NC>(P, 2 * tile, excl - 1, run);
    else P.idx[2 * tile] = -1;
    if (total == 0) P.idx[2 * tile + 1] = -1;
  }
  // The run of the thread's last head; the tile's last run stays open.
  const int64_t g = excl + mine + hi - hc;
  Seg<NC> run = cur;
  bool ended = false;
  if (hb) {
    ended = follow(run, tid + 1);
    if (!ended) piece_store<NC>(P, 2 * tile + 1, g + hc - 1, run);
  }
  // Runs never outnumber min(span, valid rows) <= cap for sorted keys; the
  // checks only keep a broken sortedness flag in bounds.
  if (excl + total > cap) {
    if (tid == 0) atomicExch(err, NFC_ERR_RANGE);
    return;
  }
  const uint32_t last_head = hb ? 31u - (uint32_t)__clz(hb) : 0u;
  if (total < kSoTile / 4) {
    // Few runs: every thread writes its own.
    if (hb == 0u) return;
    if (ended) seg_emit<NC, SIG>(cs, o, g + hc - 1, run);
    int64_t gi = g;
#pragma unroll
    for (int r = 0; r < kSoRows; ++r)
      if (hb & (1u << r)) o.ukeys[gi++] = (int64_t)k[r];
    if ((hb & (hb - 1u)) == 0u) return;
    // Runs inside the thread: from each head to the next.
    seg_identity<NC, SIG>(cs, run);
    gi = g - 1;
#pragma unroll
    for (int q = 0; q < kSoRows / 4; ++q) {
      if (4u * q > last_head) continue;
      uint64_t v[4][NC > 0 ? NC : 1];
      load_rows4<NC, SIG>(cs, n, aligned, row0 + 4 * q, v);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const uint32_t bit = 1u << (4 * q + r);
        if (hb & bit) {
          if (gi >= g) {
            seg_add_four<NC, SIG>(cs, run);
            seg_emit<NC, SIG>(cs, o, gi, run);
          }
          ++gi;
          seg_identity<NC, SIG>(cs, run);
        }
        if (vb & bit) seg_add_row<NC, SIG>(cs, run, v[r]);
      }
      seg_add_four<NC, SIG>(cs, run);
    }
    return;
  }
  // Many short runs: threads writing several runs each would scatter 8-byte
  // stores (20M rows in runs of 1.6, six aggregates: 763 us), so the outputs
  // leave column by column through shared memory.
  const uint32_t l0 = mine + hi - hc;
  uint32_t last_key = 0u;  // of the thread's last head
#pragma unroll
  for (int r = 0; r < kSoRows; ++r)
    if (hb & (1u << r)) last_key = (uint32_t)k[r];
  // fill() sets the thread's entries of the stage, store(i, x) writes entry i.
  auto put = [&](auto fill, auto store) {
    __syncthreads();  // the stage is free
    fill();
    __syncthreads();
    for (uint32_t i = tid; i < total; i += kSoThreads) store(i, sm.stage[i]);
  };
  // One aggregate of every run: `first` starts a run's value, `add` folds a
  // row's, `dec` gives what is staged of it, `fin` is that of the thread's last
  // run.  The tile's last run is open; its entry is not written out.
  auto runs_of = [&](uint64_t first, uint64_t fin, auto add, auto dec) {
    uint32_t l = l0;
    uint64_t x = first;
    bool open = false;
#pragma unroll
    for (int r = 0; r < kSoRows; ++r) {
      if (hb & (1u << r)) {
        if (open) sm.stage[l++] = dec(x);
        open = true;
        x = first;
      }
      if (vb & (1u << r)) x = add(x, r);
    }
    if (hb) sm.stage[l] = fin;
  };
  auto same = [](uint64_t x) { return x; };
  // Keys and counts in one go: a run's key is any of its rows' keys.
  put([&] {
        runs_of(0, (uint64_t)run.cnt << 32 | last_key,
                [&](uint64_t x, int r) { return ((x >> 32) + 1) << 32 | (uint32_t)k[r]; }, same);
      },
      [&](uint32_t i, uint64_t x) {
        o.ukeys[excl + i] = (int64_t)(int32_t)(uint32_t)x;
        if (i + 1 < total) o.counts[excl + i] = (int64_t)(x >> 32);
      });
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int dt = col_dt<SIG>(cs, c), ag = col_ag<SIG>(cs, c);
    if (ag == 0) continue;
    uint64_t v[kSoRows];
    load_rows<kSoRows, SIG>(cs, c, n, aligned, row0, v);
    auto to64 = [&](void* dst) {
      uint64_t* d = static_cast<uint64_t*>(dst) + excl;
      return [d, total](uint32_t i, uint64_t x) {
        if (i + 1 < total) d[i] = x;
      };
    };
    if ((ag & NFC_AGG_SUM) && dt == NFC_F64)
      put([&] {
            // In fours, as above.
            double four = 0.0;
            runs_of(0, run.sum[c],
                    [&](uint64_t x, int r) {
                      if ((hb >> r) & 1u) four = 0.0;  // a run starts
                      if ((r & 3) == 0) {
                        x = f64_add_bits(x, (uint64_t)__double_as_longlong(four));
                        four = 0.0;
                      }
                      four += __longlong_as_double((long long)v[r]);
                      return x;
                    },
                    [&](uint64_t x) { return f64_add_bits(x, (uint64_t)__double_as_longlong(four)); });
          },
          to64(o.sum[c]));
    else if (ag & NFC_AGG_SUM)
      put([&] {
            runs_of(0, run.sum[c],
                    [&](uint64_t x, int r) { return x + (dt == NFC_I32 ? (uint64_t)(int64_t)(int32_t)v[r] : v[r]); },
                    same);
          },
          to64(o.sum[c]));
    if (dt == NFC_I32) {
      if (ag & (NFC_AGG_MIN | NFC_AGG_MAX))  // both in one word: maximum above minimum
        put([&] {
              runs_of((uint64_t)0x80000000u << 32 | 0x7FFFFFFFu,
                      (uint64_t)(uint32_t)run.mx[c] << 32 | (uint32_t)run.mn[c],
                      [&](uint64_t x, int r) {
                        const int32_t y = (int32_t)v[r];
                        const int32_t lo = min((int32_t)(uint32_t)x, y), hi = max((int32_t)(x >> 32), y);
                        return (uint64_t)(uint32_t)hi << 32 | (uint32_t)lo;
                      },
                      same);
            },
            [&](uint32_t i, uint64_t x) {
              if (i + 1 >= total) return;
              if (ag & NFC_AGG_MIN) static_cast<int32_t*>(o.mn[c])[excl + i] = (int32_t)(uint32_t)x;
              if (ag & NFC_AGG_MAX) static_cast<int32_t*>(o.mx[c])[excl + i] = (int32_t)(x >> 32);
            });
      continue;
    }
    if (ag & NFC_AGG_MIN)
      put([&] {
            if (dt == NFC_F64)
              runs_of(~0ull, f64_min_dec(run.mn[c]), [&](uint64_t x, int r) { return min(x, f64_min_enc(v[r])); },
                      [](uint64_t x) { return f64_min_dec(x); });
            else
              runs_of((uint64_t)LLONG_MAX, run.mn[c],
                      [&](uint64_t x, int r) { return (uint64_t)min((long long)x, (long long)v[r]); }, same);
          },
          to64(o.mn[c]));
    if (ag & NFC_AGG_MAX)
      put([&] {
            if (dt == NFC_F64)
              runs_of(0ull, f64_max_dec(run.mx[c]), [&](uint64_t x, int r) { return max(x, f64_max_enc(v[r])); },
                      [](uint64_t x) { return f64_max_dec(x); });
            else
              runs_of((uint64_t)LLONG_MIN, run.mx[c],
                      [&](uint64_t x, int r) { return (uint64_t)max((long long)x, (long long)v[r]); }, same);
          },
          to64(o.mx[c]));
  }
}

// Merge pieces (nondecreasing run numbers; -1 = none) by run number.
// With Q.idx null one CTA walks every piece and writes every run.  Otherwise
// CTA b takes chunk b (blockDim pieces): the runs that start and end inside
// it are written, and its first and last runs -- which may continue in the
// neighbouring chunks -- become pieces 2b and 2b+1 of Q for a second pass.
template <int NC, uint32_t SIG>
__global__ void __launch_bounds__(kFixThreads) k_sorted_fix(ColSet cs, Pieces P, int64_t npieces, OutSet o,
                                                            int64_t cap, Pieces Q) {
  __shared__ SegScanSmem<NC, SIG> sm;
  __shared__ int64_t s_wmax[32];
  __shared__ int64_t s_cmax, s_first;
  const int lane = lane_id(), warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const bool level1 = Q.idx != nullptr;
  if (threadIdx.x == 0) {
    s_cmax = -1;
    s_first = -1;
  }
  uint32_t carry_f = 0;
  Seg<NC> carry_a;
  seg_identity<NC, SIG>(cs, carry_a);
  __syncthreads();
  const int64_t begin = level1 ? (int64_t)blockIdx.x * blockDim.x : 0;
  const int64_t end = level1 ? min(npieces, begin + (int64_t)blockDim.x) : npieces;
  for (int64_t base = begin; base < end; base += blockDim.x) {
    const int64_t i = base + threadIdx.x;
    const int64_t idx = i < end ? P.idx[i] : -1;
    Seg<NC> a;
    if (idx >= 0) piece_load<NC>(P, i, a);
    else seg_identity<NC, SIG>(cs, a);
    // Exclusive running max of the run numbers (the run of the previous piece).
    int64_t inc = idx;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, inc, off);
      if (lane >= off) inc = max(inc, y);
    }
    if (lane == 31) s_wmax[warp] = inc;
    __syncthreads();
    int64_t before = s_cmax;
    for (int w = 0; w < warp; ++w) before = max(before, s_wmax[w]);
    int64_t ex = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane == 0) ex = -1;
    const int64_t runmax = max(before, ex);
    const bool head = idx >= 0 && idx > runmax;
    if (level1 && head && runmax < 0) s_first = idx;  // the chunk's first run (one thread)
    int64_t new_cmax = s_cmax;
    for (int w = 0; w < nw; ++w) new_cmax = max(new_cmax, s_wmax[w]);
    Seg<NC> ea;
    block_seg_scan<NC, SIG>(cs, head ? 1u : 0u, a, carry_f, carry_a, ea, sm);  // syncs: s_first visible
    if (head && runmax >= 0) {
      seg_close<NC, SIG>(cs, ea);
      if (level1 && runmax == s_first) piece_store<NC>(Q, 2 * blockIdx.x, runmax, ea);
      else if (runmax < cap) seg_emit<NC, SIG>(cs, o, runmax, ea);
    }
    if (threadIdx.x == 0) s_cmax = new_cmax;
    __syncthreads();
  }
  if (threadIdx.x == 0 && s_cmax >= 0) {
    seg_close<NC, SIG>(cs, carry_a);
    if (level1) piece_store<NC>(Q, s_cmax == s_first ? 2 * blockIdx.x : 2 * blockIdx.x + 1, s_cmax, carry_a);
    else if (s_cmax < cap) seg_emit<NC, SIG>(cs, o, s_cmax, carry_a);
  }
}

template <int NC, uint32_t SIG>
int launch_sorted(const nfc_groupby_args* a, const ColSet& cs, const OutSet& o, const uint32_t* vmask,
                  const uint64_t* prev, const Pieces& P, const Pieces& Q, int64_t ntiles, int64_t nchunks,
                  uint64_t* lb, uint32_t* ticket, int64_t* d_ng, int32_t* d_err, cudaStream_t s, StageTimer* tm) {
  const size_t smem = sizeof(SortedSmem<NC, SIG>);
  NFC_CUDA(allow_dynamic_smem<k_sorted_agg<NC, SIG>>());
  k_sorted_agg<NC, SIG><<<(unsigned)ntiles, kSoThreads + 32, smem, s>>>(a->keys, vmask, cs, a->n, inputs_aligned(a), prev, o,
                                                                   a->out_cap, P, lb, ticket, d_ng, d_err);
  NFC_CUDA(cudaGetLastError());
  tm->launched();
  tm->mark(s);
  Pieces none{};
  if (nchunks > 1) {
    k_sorted_fix<NC, SIG><<<(unsigned)nchunks, kFixThreads, 0, s>>>(cs, P, 2 * ntiles, o, a->out_cap, Q);
    NFC_CUDA(cudaGetLastError());
    k_sorted_fix<NC, SIG><<<1, kFixThreads, 0, s>>>(cs, Q, 2 * nchunks, o, a->out_cap, none);
    tm->launched(2);
  } else {
    k_sorted_fix<NC, SIG><<<1, kFixThreads, 0, s>>>(cs, P, 2 * ntiles, o, a->out_cap, none);
    tm->launched();
  }
  NFC_CUDA(cudaGetLastError());
  tm->mark(s);
  return NFC_OK;
}


Pieces carve_pieces(uint64_t*& q, int64_t np) {
  Pieces P{};
  P.idx = reinterpret_cast<int64_t*>(q); q += np;
  P.cnt = q; q += np;
  for (int c = 0; c < NFC_MAX_COLS; ++c) {
    P.sum[c] = q; q += np;
    P.mn[c] = q; q += np;
    P.mx[c] = q; q += np;
  }
  return P;
}

}  // namespace

int run_sorted(const nfc_groupby_args* a, const ColSet& cs, const OutSet& o, const nfc_probe& p,
               const uint32_t* vmask, const ProbeRec* recs, cudaStream_t s, Scratch& sc, int64_t* d_ng,
               int32_t* d_err, StageTimer* tm) {
  const int64_t n = a->n;
  const int64_t ntiles = (n + so_tile(a->ncols) - 1) / so_tile(a->ncols);
  const int64_t nrec = (n + kProbeBlockRows - 1) / kProbeBlockRows;  // <= ntiles
  const int64_t np = 2 * ntiles;
  const int64_t nchunks = (np + kFixThreads - 1) / kFixThreads;
  const int64_t nq = 2 * nchunks;
  // One allocation: prev[ntiles], lb[ntiles], ticket, tile pieces, chunk pieces.
  const size_t per_piece = 2 + 3 * NFC_MAX_COLS;
  const size_t words = (size_t)ntiles * 2 + 2 + (size_t)(np + nq) * per_piece;
  uint64_t* w = nullptr;
  NFC_CUDA(sc.alloc(&w, words));
  uint64_t* prev = w;
  uint64_t* lb = prev + ntiles;
  uint32_t* ticket = reinterpret_cast<uint32_t*>(lb + ntiles);
  uint64_t* q = lb + ntiles + 2;
  const Pieces P = carve_pieces(q, np);
  const Pieces Q = carve_pieces(q, nq);
  NFC_CUDA(cudaMemsetAsync(lb, 0, sizeof(uint64_t) * ((size_t)ntiles + 2), s));
  k_sorted_prev<<<1, 1024, 0, s>>>(recs, nrec, prev, Q.idx, nq);
  NFC_CUDA(cudaGetLastError());
  tm->launched();
  tm->mark(s);
  const uint32_t sig = sig_of(cs);
  const bool sums = sums_only(cs);
#define NFC_SORTED_LAUNCH(NCV, SIGV) \
  launch_sorted<NCV, SIGV>(a, cs, o, vmask, prev, P, Q, ntiles, nchunks, lb, ticket, d_ng, d_err, s, tm)
  switch (cs.ncols) {
    case 0: return NFC_SORTED_LAUNCH(0, 0);
    case 1:
      if (sig == kSigI32Sum) return NFC_SORTED_LAUNCH(1, kSigI32Sum);
      if (sums) return NFC_SORTED_LAUNCH(1, kSigSums);
      return NFC_SORTED_LAUNCH(1, 0);
    case 2:
      if (sig == kSigI32SumMinMax_F64SumMinMax) return NFC_SORTED_LAUNCH(2, kSigI32SumMinMax_F64SumMinMax);
      if (sums) return NFC_SORTED_LAUNCH(2, kSigSums);
      return NFC_SORTED_LAUNCH(2, 0);
    case 3:
      if (sums) return NFC_SORTED_LAUNCH(3, kSigSums);
      return NFC_SORTED_LAUNCH(3, 0);
    default:
      if (sums) return NFC_SORTED_LAUNCH(4, kSigSums);
      return NFC_SORTED_LAUNCH(4, 0);
  }
#undef NFC_SORTED_LAUNCH
}

}  // namespace nfc

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
//                       order, a thread per 8 or 16 consecutive rows.  A
//                       thread finds its run heads (valid rows whose key
//                       differs from the previous valid row's), sums the rows before its first
//                       head and after its last one and each run in between,
//                       and a decoupled look-back gives the tile its first run
//                       number.  The thread that holds a run's head then adds
//                       what the threads after it have of that run (a whole
//                       warp without heads is one step); the runs are staged
//                       in shared memory and written out column by column.
//                       The tile's first run (continued from earlier tiles) and
//                       last run (possibly continued by later ones) leave as
//                       two partial "pieces";
//   3. k_sorted_fix     the pieces are merged in order (segmented scan by run
//                       number): chunks of a CTA each, then the chunks' own
//                       edge runs in one CTA.
// Every run's output key is staged by the thread holding its head, the last run's
// too, whose values leave as a piece.  float64 sums differ from the reference's
// row loop in the order of their additions (mean relative error of a run's sum
// below 2^-53); everything else is exact.
#include <algorithm>

#include "groupby_host.h"

namespace nfc {
namespace {

constexpr int kSoThreads = 256;                    // threads with rows; one more warp looks back
constexpr int kSoWarps = kSoThreads / 32;
// Consecutive rows per thread and rows per tile: more where a row is little work.
constexpr int so_rows(int nc) { return nc <= 1 ? 16 : 8; }
// float64 rows added in fours (Seg); three and more columns lack the registers.
constexpr bool so_fours(int nc) { return nc <= 2; }
constexpr int so_tile(int nc) { return kSoThreads * so_rows(nc); }
static_assert(kProbeBlockRows % so_tile(0) == 0 && kProbeBlockRows % so_tile(4) == 0,
              "tiles do not straddle probe records");
// Pieces of a chunk in k_sorted_fix; with three and more columns a thread needs more
// than the 64 registers that 1,024 leave it.
constexpr int fix_threads(int nc) { return nc <= 2 ? 1024 : 512; }

// ---------------------------------------------------------------- run aggregate
// Integers are kept as int64 bits (sums wrap like the other strategies' int64
// atomics), float64 min/max as the ordered encodings of nfc_common.cuh;
// int32 min/max use int32 identities and 32-bit compares.  A count never
// exceeds the row count (< 2^31).
//
// A float64 sum of many terms added one after the other loses with the root of
// their number.  So a thread adds its rows in fours (from the second four on in
// `rest`, which seg_add_four adds to the sum), and the aggregates of threads, warps and tiles are
// added up with the rounding errors of the additions (in `rest`; seg_close adds
// them).  Mean relative error of a sum, 20M rows in runs of 200: 1.2e-16 with plain
// chains, 7e-17 as a tree over the rows, 4.5e-17 this way.
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

// Fold one row: int32 values as their 32-bit word, 8-byte values as bits.  first:
// one of the thread's first four rows.
template <int NC, uint32_t SIG>
NFC_DEV void seg_add_row(const ColSet& cs, Seg<NC>& a, const uint64_t* raw, bool first) {
  a.cnt += 1;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int dt = col_dt<SIG>(cs, c), ag = col_ag<SIG>(cs, c);
    const uint64_t r = raw[c];
    if (dt == NFC_F64) {
      if (ag & NFC_AGG_SUM) {
        if (first) a.sum[c] = f64_add_bits(a.sum[c], r);
        else a.rest[c] += __longlong_as_double((long long)r);
      }
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
NFC_DEV void part_load(const ColSet& cs, Seg<NC>& a, const Partials<NC>& p, int t) {
  a.cnt = p.cnt[t];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int ag = col_ag<SIG>(cs, c);
    a.sum[c] = ag & NFC_AGG_SUM ? p.sum[c][t] : 0ull;
    a.rest[c] = 0.0;
    a.mn[c] = ag & NFC_AGG_MIN ? p.mn[c][t] : 0ull;
    a.mx[c] = ag & NFC_AGG_MAX ? p.mx[c][t] : 0ull;
  }
}

template <int NC, uint32_t SIG>
NFC_DEV void part_add(const ColSet& cs, Seg<NC>& a, const Partials<NC>& p, int t) {
  Seg<NC> b;
  part_load<NC, SIG>(cs, b, p, t);
  seg_combine<NC, SIG>(cs, a, b);
}

// The tile's runs on their way out: arrays of `cap` 8-byte entries, key << 32 | count
// first, then every aggregate (with run-time types room for all of a column's;
// with known ones an int32 column's minimum and maximum share an array).  Array f
// starts at f * cap, f known at compile time: a pointer per array would be 26
// registers for four columns, which the rows' loads then lack.
enum { kFSum, kFMin, kFMax };
template <uint32_t SIG>
constexpr bool stage_packs(int c) {
  return SIG != 0 && SIG != kSigSums && ((SIG >> (5 * c)) & 3u) == (uint32_t)NFC_I32 &&
         ((SIG >> (5 * c + 3)) & 3u) == 3u;
}
template <int NC, uint32_t SIG>
constexpr int stage_field(int c, int which) {
  if (SIG == 0) return 1 + 3 * c + which;
  if (SIG == kSigSums) return 1 + c;
  int f = 1;
  for (int i = 0; i < c; ++i) {
    for (int a = 0; a < 3; ++a) f += (SIG >> (5 * i + 2 + a)) & 1u;
    f -= stage_packs<SIG>(i);
  }
  for (int a = 0; a < which; ++a) f += (SIG >> (5 * c + 2 + a)) & 1u;
  return which == kFMax ? f - stage_packs<SIG>(c) : f;
}
static_assert(NFC_AGG_SUM == 1 && NFC_AGG_MIN == 2 && NFC_AGG_MAX == 4, "bit order of the fields");
template <int NC, uint32_t SIG>
constexpr int stage_fields() { return stage_field<NC, SIG>(NC, 0); }

struct Stage {
  uint64_t* base;
  int cap;
  NFC_DEV uint64_t& at(int f, int e) const { return base[f * cap + e]; }
};

template <int NC, uint32_t SIG>
NFC_DEV void stage_put(const ColSet& cs, const Stage& st, int e, const Seg<NC>& a, int32_t key) {
  st.at(0, e) = (uint64_t)(uint32_t)key << 32 | a.cnt;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int ag = col_ag<SIG>(cs, c);
    if (ag & NFC_AGG_SUM) st.at(stage_field<NC, SIG>(c, kFSum), e) = a.sum[c];
    if (stage_packs<SIG>(c)) {
      st.at(stage_field<NC, SIG>(c, kFMin), e) = a.mx[c] << 32 | (uint32_t)a.mn[c];
      continue;
    }
    if (ag & NFC_AGG_MIN) st.at(stage_field<NC, SIG>(c, kFMin), e) = a.mn[c];
    if (ag & NFC_AGG_MAX) st.at(stage_field<NC, SIG>(c, kFMax), e) = a.mx[c];
  }
}

// Entries 0 .. n of the stage to output rows g0 on, the keys of nk.
template <int NC, uint32_t SIG>
NFC_DEV void stage_write(const ColSet& cs, const Stage& st, const OutSet& o, int64_t g0, int nk, int n) {
  const int t = threadIdx.x;
  for (int i = t; i < nk; i += kSoThreads) {
    const uint64_t x = st.at(0, i);
    o.ukeys[g0 + i] = (int64_t)(int32_t)(x >> 32);
    if (i < n) o.counts[g0 + i] = (int64_t)(uint32_t)x;
  }
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int dt = col_dt<SIG>(cs, c), ag = col_ag<SIG>(cs, c);
    if (ag & NFC_AGG_SUM) {
      uint64_t* d = static_cast<uint64_t*>(o.sum[c]) + g0;
      for (int i = t; i < n; i += kSoThreads) d[i] = st.at(stage_field<NC, SIG>(c, kFSum), i);
    }
    if (dt == NFC_I32) {
      if (ag & NFC_AGG_MIN) {
        int32_t* d = static_cast<int32_t*>(o.mn[c]) + g0;
        for (int i = t; i < n; i += kSoThreads) d[i] = (int32_t)st.at(stage_field<NC, SIG>(c, kFMin), i);
      }
      if (ag & NFC_AGG_MAX) {
        int32_t* d = static_cast<int32_t*>(o.mx[c]) + g0;
        for (int i = t; i < n; i += kSoThreads)
          d[i] = (int32_t)(st.at(stage_field<NC, SIG>(c, kFMax), i) >> (stage_packs<SIG>(c) ? 32 : 0));
      }
      continue;
    }
    if (ag & NFC_AGG_MIN) {
      uint64_t* d = static_cast<uint64_t*>(o.mn[c]) + g0;
      for (int i = t; i < n; i += kSoThreads) {
        const uint64_t x = st.at(stage_field<NC, SIG>(c, kFMin), i);
        d[i] = dt == NFC_F64 ? f64_min_dec(x) : x;
      }
    }
    if (ag & NFC_AGG_MAX) {
      uint64_t* d = static_cast<uint64_t*>(o.mx[c]) + g0;
      for (int i = t; i < n; i += kSoThreads) {
        const uint64_t x = st.at(stage_field<NC, SIG>(c, kFMax), i);
        d[i] = dt == NFC_F64 ? f64_max_dec(x) : x;
      }
    }
  }
}

// Shared memory of a CTA.  More stage, fewer turns for short runs, but less L1 for the
// rows' loads: one float64 sum over 20M rows in long runs 254 us at 40 KB, 278 at
// 75; two columns with all aggregates in runs of two 445 us at 40 KB, 392 at 60.
constexpr size_t so_smem(int nc) { return (nc <= 1 ? 44 : nc == 2 ? 60 : 80) * 1024; }

// CTAs per SM that the registers of the run aggregates leave room for.
template <int NC, uint32_t SIG>
constexpr int so_ctas() { return NC == 0 ? 4 : NC <= 2 ? 3 : 2; }

template <int NC, uint32_t SIG>
struct SortedSmem {
  Partials<NC> lead;  // rows before the thread's first head; all its rows when it has none
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
// without work below 2M rows).  Runs leave through a stage in one pass over the
// rows: writing the runs between two heads in a second pass, and output column
// by output column where runs are short, took 60M rows in runs of 2.3 with six
// aggregates 1,160 us, 935 this way; runs of 8 850 and 790.
template <int NC, uint32_t SIG>
__global__ void __launch_bounds__(kSoThreads + 32, so_ctas<NC, SIG>())
    k_sorted_agg(const int32_t* __restrict__ keys, const uint32_t* __restrict__ vmask, ColSet cs, int64_t n,
                 bool aligned, const uint64_t* __restrict__ prev, OutSet o, int64_t out_cap, int cap, Pieces P,
                 uint64_t* lb, uint32_t* ticket, int64_t* ng_out, int32_t* err) {
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

  uint32_t total = 0, mine = 0;
  for (int w = 0; w < kSoWarps; ++w) {
    if (w < warp) mine += sm.wheads[w];
    total += sm.wheads[w];
  }
  const int l0 = (int)(mine + hi - hc);  // the thread's first run, in the tile
  const Stage st{reinterpret_cast<uint64_t*>(sm_raw + ((sizeof(sm) + 15) & ~(size_t)15)), cap};

  // Adds to `a` what the threads from t on hold of an open run, and closes it;
  // true when the run ends inside the tile.
  auto follow = [&](Seg<NC>& a, int t) {
    bool ends = false;
    while (t < kSoThreads && !ends) {
      const uint32_t rest = sm.wany[t >> 5] >> (t & 31);
      if (rest == 0u && (t & 31) == 0) {
        seg_combine<NC, SIG>(cs, a, sm.wsum[t >> 5]);
        t += 32;
      } else {
        part_add<NC, SIG>(cs, a, sm.lead, t);
        ends = rest & 1u;
        ++t;
      }
    }
    seg_close<NC, SIG>(cs, a);
    return ends;
  };

  // The tile's runs leave through the stage.  Where there are more of them than fit
  // (runs of one or two rows), the threads of the later ones take another turn
  // over their rows.
  for (int w0 = 0;; w0 += cap) {
    // The rows before the thread's first head, the runs between two heads, and in
    // `cur` the rows from its last head on (all of them without one).
    Seg<NC> cur;
    seg_identity<NC, SIG>(cs, cur);
    uint32_t e = (uint32_t)(l0 - 1 - w0);  // entry of the open run
    int32_t key = 0;
    const bool turn = w0 == 0 || (hb && l0 + (int)hc > w0 && l0 < w0 + cap);
    if (turn) {
#pragma unroll
      for (int q = 0; q < kSoRows / 4; ++q) {
        if (((vb >> (4 * q)) & 0xFu) == 0u) continue;
        uint64_t v[4][NC > 0 ? NC : 1];
        load_rows4<NC, SIG>(cs, n, aligned, row0 + 4 * q, v);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const uint32_t bit = 1u << (4 * q + r);
          if (hb & bit) {
            if (q > 0 && so_fours(NC)) seg_add_four<NC, SIG>(cs, cur);
            if (hb & (bit - 1u)) {
              if (e < (uint32_t)cap) stage_put<NC, SIG>(cs, st, (int)e, cur, key);
            } else if (w0 == 0) {
              part_store<NC, SIG>(cs, sm.lead, tid, cur);
            }
            seg_identity<NC, SIG>(cs, cur);
            key = k[4 * q + r];
            ++e;
          }
          if (vb & bit) seg_add_row<NC, SIG>(cs, cur, v[r], q == 0 || !so_fours(NC));
        }
        if (q > 0 && so_fours(NC)) seg_add_four<NC, SIG>(cs, cur);
      }
    }
    if (w0 == 0) {
      if (hb == 0u) part_store<NC, SIG>(cs, sm.lead, tid, cur);
      if (any == 0u) {
        Seg<NC> w;
        seg_warp_reduce<NC, SIG>(cs, cur, w);
        if (lane == 0) sm.wsum[warp] = w;
      }
      __syncthreads();
      // The run that the tile continues (its rows before the first head).
      if (tid == 0) {
        Seg<NC> run;
        if (any) part_load<NC, SIG>(cs, run, sm.lead, 0);
        else run = sm.wsum[0];
        if (!hb) follow(run, any ? 1 : 32);
        if (run.cnt > 0) piece_store<NC>(P, 2 * tile, sm.excl - 1, run);
        else P.idx[2 * tile] = -1;
        if (total == 0) P.idx[2 * tile + 1] = -1;
      }
      if (total == 0) return;
    }
    // The run of the thread's last head; the tile's last run stays open.
    if (hb && turn) {
      const bool ended = follow(cur, tid + 1);
      if (e < (uint32_t)cap) stage_put<NC, SIG>(cs, st, (int)e, cur, key);
      if (!ended && w0 == 0) piece_store<NC>(P, 2 * tile + 1, sm.excl + total - 1, cur);
    }
    // Runs never outnumber min(span, valid rows) <= out_cap for sorted keys; the
    // check only keeps a broken sortedness flag in bounds.
    if (sm.excl + total > out_cap) {
      if (tid == 0) atomicExch(err, NFC_ERR_RANGE);
      return;
    }
    __syncthreads();
    const int nk = min((int)total - w0, cap);
    if (warp * 32 < nk) stage_write<NC, SIG>(cs, st, o, sm.excl + w0, nk, min((int)total - 1 - w0, cap));
    if (w0 + cap >= (int)total) return;
    __syncthreads();  // the stage is free
  }
}

// Merge pieces (nondecreasing run numbers; -1 = none) by run number.
// With Q.idx null one CTA walks every piece and writes every run.  Otherwise
// CTA b takes chunk b (blockDim pieces): the runs that start and end inside
// it are written, and its first and last runs -- which may continue in the
// neighbouring chunks -- become pieces 2b and 2b+1 of Q for a second pass.
template <int NC, uint32_t SIG>
__global__ void __launch_bounds__(fix_threads(NC), 1) k_sorted_fix(ColSet cs, Pieces P, int64_t npieces, OutSet o,
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
  // The stage: what leaves the loads some L1 (runs of one row need several turns).
  const size_t base = (sizeof(SortedSmem<NC, SIG>) + 15) & ~(size_t)15, entry = 8 * (size_t)stage_fields<NC, SIG>();
  const size_t room = so_smem(NC) - base;
  const int cap = (int)std::min<size_t>(so_tile(NC), room / entry);
  const size_t smem = base + (size_t)cap * entry;
  NFC_CUDA(allow_dynamic_smem<k_sorted_agg<NC, SIG>>());
  k_sorted_agg<NC, SIG><<<(unsigned)ntiles, kSoThreads + 32, smem, s>>>(a->keys, vmask, cs, a->n, inputs_aligned(a), prev,
                                                                      o, a->out_cap, cap, P, lb, ticket, d_ng, d_err);
  NFC_CUDA(cudaGetLastError());
  tm->launched();
  tm->mark(s);
  Pieces none{};
  if (nchunks > 1) {
    k_sorted_fix<NC, SIG><<<(unsigned)nchunks, fix_threads(NC), 0, s>>>(cs, P, 2 * ntiles, o, a->out_cap, Q);
    NFC_CUDA(cudaGetLastError());
    k_sorted_fix<NC, SIG><<<1, fix_threads(NC), 0, s>>>(cs, Q, 2 * nchunks, o, a->out_cap, none);
    tm->launched(2);
  } else {
    k_sorted_fix<NC, SIG><<<1, fix_threads(NC), 0, s>>>(cs, P, 2 * ntiles, o, a->out_cap, none);
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
  const int64_t nchunks = (np + fix_threads(a->ncols) - 1) / fix_threads(a->ncols);
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

// Shared-memory aggregation state for one CTA's groups, shared by the
// partition aggregate and the shared-hash strategy.
//
// 64-bit shared-memory atomics on integers are emulated, so an int32
// column's sum is kept as two native 32-bit sums of its low and high 16-bit
// halves (exact while a state slot sees at most 65,536 rows) -- or, when
// the caller knows every value of the column lies in [-32767, 32767]
// (bit c of `narrow`), as one signed 32-bit sum in the low array (exact for
// the same 65,536 rows); float64
// min/max use native 64-bit min/max on an order-preserving encoding;
// float64 sums use the 64-bit float add, with ERR also a second array for the
// rounding errors of the additions.  agg_merge folds a slot into the
// global state layout (StateRef) with global atomics.
#pragma once

#include "groupby_core.cuh"

namespace nfc {

template <int NC>
struct AggState {
  uint32_t* cnt;
  uint32_t* slo[NC > 0 ? NC : 1];   // int32 columns: sum of low 16-bit halves
  int32_t* shi[NC > 0 ? NC : 1];    // int32 columns: sum of high 16-bit halves
  uint64_t* s64[NC > 0 ? NC : 1];   // int64 / float64 columns: sum
  double* err[NC > 0 ? NC : 1];     // float64 columns, ERR: rounding errors of the sum
  void* mn[NC > 0 ? NC : 1];
  void* mx[NC > 0 ? NC : 1];
  uint32_t narrow;  // bit c: int32 column c summed with one signed 32-bit atomic
};

template <int NC, uint32_t SIG, bool ERR = false>
NFC_DEV AggState<NC> carve_agg(const ColSet& cs, unsigned char* base, int w, uint32_t narrow = 0u) {
  AggState<NC> st;
  st.narrow = narrow;
  unsigned char* p = base;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    st.slo[c] = nullptr; st.shi[c] = nullptr; st.s64[c] = nullptr; st.mn[c] = nullptr; st.mx[c] = nullptr;
    st.err[c] = nullptr;
    const bool wide = col_dt<SIG>(cs, c) != NFC_I32;
    const int ag = col_ag<SIG>(cs, c);
    if (wide && (ag & NFC_AGG_SUM)) { st.s64[c] = reinterpret_cast<uint64_t*>(p); p += 8 * w; }
    if (ERR && col_dt<SIG>(cs, c) == NFC_F64 && (ag & NFC_AGG_SUM)) { st.err[c] = reinterpret_cast<double*>(p); p += 8 * w; }
    if (wide && (ag & NFC_AGG_MIN)) { st.mn[c] = p; p += 8 * w; }
    if (wide && (ag & NFC_AGG_MAX)) { st.mx[c] = p; p += 8 * w; }
  }
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    if (col_dt<SIG>(cs, c) != NFC_I32) continue;
    const int ag = col_ag<SIG>(cs, c);
    if (ag & NFC_AGG_SUM) {
      st.slo[c] = reinterpret_cast<uint32_t*>(p); p += 4 * w;
      st.shi[c] = reinterpret_cast<int32_t*>(p); p += 4 * w;
    }
    if (ag & NFC_AGG_MIN) { st.mn[c] = p; p += 4 * w; }
    if (ag & NFC_AGG_MAX) { st.mx[c] = p; p += 4 * w; }
  }
  st.cnt = reinterpret_cast<uint32_t*>(p);
  return st;
}

template <int NC, uint32_t SIG, bool ERR = false>
NFC_DEV void agg_init(const ColSet& cs, const AggState<NC>& st, int g) {
  st.cnt[g] = 0u;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int dt = col_dt<SIG>(cs, c), ag = col_ag<SIG>(cs, c);
    if (dt == NFC_I32) {
      if (ag & NFC_AGG_SUM) { st.slo[c][g] = 0u; st.shi[c][g] = 0; }
      if (ag & NFC_AGG_MIN) static_cast<int32_t*>(st.mn[c])[g] = INT_MAX;
      if (ag & NFC_AGG_MAX) static_cast<int32_t*>(st.mx[c])[g] = INT_MIN;
    } else {
      if (ag & NFC_AGG_SUM) st.s64[c][g] = 0ull;
      if (ERR && dt == NFC_F64 && (ag & NFC_AGG_SUM)) st.err[c][g] = 0.0;
      if (dt == NFC_I64) {
        if (ag & NFC_AGG_MIN) static_cast<int64_t*>(st.mn[c])[g] = LLONG_MAX;
        if (ag & NFC_AGG_MAX) static_cast<int64_t*>(st.mx[c])[g] = LLONG_MIN;
      } else {
        if (ag & NFC_AGG_MIN) static_cast<uint64_t*>(st.mn[c])[g] = ~0ull;
        if (ag & NFC_AGG_MAX) static_cast<uint64_t*>(st.mx[c])[g] = 0ull;
      }
    }
  }
}

NFC_DEV void block_fill16(void* p, int vecs, uint64_t v) {
  ulonglong2* q = static_cast<ulonglong2*>(p);
  for (int i = threadIdx.x; i < vecs; i += blockDim.x) q[i] = make_ulonglong2(v, v);
}

// Identities of all w slots with 16-byte stores (whole block; w a multiple of
// 4 and the state 16-byte aligned).  Slot by slot, eight 4- or 8-byte stores
// per slot, the initialisation is a third of a bucket with a few hundred rows.
template <int NC, uint32_t SIG>
NFC_DEV void agg_init_all(const ColSet& cs, const AggState<NC>& st, int w) {
  constexpr uint64_t kMax32 = 0x7FFFFFFF7FFFFFFFull, kMin32 = 0x8000000080000000ull;
  block_fill16(st.cnt, w / 4, 0ull);
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int dt = col_dt<SIG>(cs, c), ag = col_ag<SIG>(cs, c);
    if (dt == NFC_I32) {
      if (ag & NFC_AGG_SUM) {
        block_fill16(st.slo[c], w / 4, 0ull);
        block_fill16(st.shi[c], w / 4, 0ull);
      }
      if (ag & NFC_AGG_MIN) block_fill16(st.mn[c], w / 4, kMax32);
      if (ag & NFC_AGG_MAX) block_fill16(st.mx[c], w / 4, kMin32);
    } else {
      const bool i64 = dt == NFC_I64;
      if (ag & NFC_AGG_SUM) block_fill16(st.s64[c], w / 2, 0ull);
      if (ag & NFC_AGG_MIN) block_fill16(st.mn[c], w / 2, i64 ? (uint64_t)LLONG_MAX : ~0ull);
      if (ag & NFC_AGG_MAX) block_fill16(st.mx[c], w / 2, i64 ? (uint64_t)LLONG_MIN : 0ull);
    }
  }
}

// READ_FIRST: min/max read the slot first and skip the atomic when the value
// cannot win (the stored extreme only moves one way, so a value that does
// not beat it now can never beat the final one).  That pays when slots see
// many rows each; with a few rows per slot (the partition aggregate: ~8 on
// average) the read costs more shared-memory wavefronts than the atomics it
// saves, so that caller issues the atomics directly.
template <int NC, uint32_t SIG, bool READ_FIRST = true>
NFC_DEV void agg_apply(const ColSet& cs, const AggState<NC>& st, uint32_t g, const uint64_t* raw) {
  atomicAdd(&st.cnt[g], 1u);
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int dt = col_dt<SIG>(cs, c), ag = col_ag<SIG>(cs, c);
    const uint64_t r = raw[c];
    if (dt == NFC_I32) {
      const int32_t v = (int32_t)(uint32_t)r;
      if (ag & NFC_AGG_SUM) {
        if ((st.narrow >> c) & 1u) {
          atomicAdd(reinterpret_cast<int*>(st.slo[c]) + g, v);
        } else {
          atomicAdd(&st.slo[c][g], (uint32_t)v & 0xFFFFu);
          atomicAdd(&st.shi[c][g], v >> 16);
        }
      }
      if ((ag & NFC_AGG_MIN) && (!READ_FIRST || v < static_cast<volatile int32_t*>(st.mn[c])[g]))
        atomicMin(static_cast<int*>(st.mn[c]) + g, v);
      if ((ag & NFC_AGG_MAX) && (!READ_FIRST || v > static_cast<volatile int32_t*>(st.mx[c])[g]))
        atomicMax(static_cast<int*>(st.mx[c]) + g, v);
    } else if (dt == NFC_I64) {
      if (ag & NFC_AGG_SUM) atomicAdd(reinterpret_cast<unsigned long long*>(st.s64[c]) + g, (unsigned long long)r);
      if ((ag & NFC_AGG_MIN) && (!READ_FIRST || (long long)r < static_cast<volatile long long*>(st.mn[c])[g]))
        atomicMin(static_cast<long long*>(st.mn[c]) + g, (long long)r);
      if ((ag & NFC_AGG_MAX) && (!READ_FIRST || (long long)r > static_cast<volatile long long*>(st.mx[c])[g]))
        atomicMax(static_cast<long long*>(st.mx[c]) + g, (long long)r);
    } else {
      if (ag & NFC_AGG_SUM) atomicAdd(reinterpret_cast<double*>(st.s64[c]) + g, __longlong_as_double((long long)r));
      if (ag & NFC_AGG_MIN) {
        const unsigned long long e = f64_min_enc(r);
        if (!READ_FIRST || e < static_cast<volatile unsigned long long*>(st.mn[c])[g])
          atomicMin(static_cast<unsigned long long*>(st.mn[c]) + g, e);
      }
      if (ag & NFC_AGG_MAX) {
        const unsigned long long e = f64_max_enc(r);
        if (!READ_FIRST || e > static_cast<volatile unsigned long long*>(st.mx[c])[g])
          atomicMax(static_cast<unsigned long long*>(st.mx[c]) + g, e);
      }
    }
  }
}

// Fold k rows combined by warp_agg_rows (sums as int64 / float64 bits,
// minima / maxima as int64 / ordered float64 lanes) into slot g.  An int32
// sum goes into the split halves as its own low 16 bits and the rest, which
// keeps value = high * 65536 + low and the same bounds as k single rows.
template <int NC, uint32_t SIG, bool ERR = false>
NFC_DEV void agg_apply_group(const ColSet& cs, const AggState<NC>& st, uint32_t g, uint32_t k, const uint64_t* sum,
                             const uint64_t* mn, const uint64_t* mx) {
  atomicAdd(&st.cnt[g], k);
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int dt = col_dt<SIG>(cs, c), ag = col_ag<SIG>(cs, c);
    if (dt == NFC_I32) {
      if (ag & NFC_AGG_SUM) {
        const int64_t s = (int64_t)sum[c];
        if ((st.narrow >> c) & 1u) {
          atomicAdd(reinterpret_cast<int*>(st.slo[c]) + g, (int)s);
        } else {
          atomicAdd(&st.slo[c][g], (uint32_t)(s & 0xFFFF));
          atomicAdd(&st.shi[c][g], (int32_t)(s >> 16));
        }
      }
      if (ag & NFC_AGG_MIN) atomicMin(static_cast<int*>(st.mn[c]) + g, (int)(int64_t)mn[c]);
      if (ag & NFC_AGG_MAX) atomicMax(static_cast<int*>(st.mx[c]) + g, (int)(int64_t)mx[c]);
    } else if (dt == NFC_I64) {
      if (ag & NFC_AGG_SUM) atomicAdd(reinterpret_cast<unsigned long long*>(st.s64[c]) + g, (unsigned long long)sum[c]);
      if (ag & NFC_AGG_MIN) atomicMin(static_cast<long long*>(st.mn[c]) + g, (long long)mn[c]);
      if (ag & NFC_AGG_MAX) atomicMax(static_cast<long long*>(st.mx[c]) + g, (long long)mx[c]);
    } else {
      if (ag & NFC_AGG_SUM) {
        double* dst = reinterpret_cast<double*>(st.s64[c]) + g;
        if (ERR) f64_atomic_add_err(dst, st.err[c] + g, __longlong_as_double((long long)sum[c]));
        else atomicAdd(dst, __longlong_as_double((long long)sum[c]));
      }
      if (ag & NFC_AGG_MIN) atomicMin(static_cast<unsigned long long*>(st.mn[c]) + g, (unsigned long long)mn[c]);
      if (ag & NFC_AGG_MAX) atomicMax(static_cast<unsigned long long*>(st.mx[c]) + g, (unsigned long long)mx[c]);
    }
  }
}

template <int NC, uint32_t SIG>
NFC_DEV int64_t agg_sum_bits(const ColSet& cs, const AggState<NC>& st, int c, int g) {
  if (col_dt<SIG>(cs, c) == NFC_I32) {
    if ((st.narrow >> c) & 1u) return (int64_t)(int32_t)st.slo[c][g];
    return (int64_t)st.shi[c][g] * 65536 + (int64_t)st.slo[c][g];
  }
  return (int64_t)st.s64[c][g];
}

// Merge shared slot g into the global merge state (StateRef layout) slot d.
// LEAVE: without the float64 sums of which that state keeps the errors.
template <int NC, uint32_t SIG, bool LEAVE = false>
NFC_DEV void agg_merge(const ColSet& cs, const StateRef& dst, int64_t d, const AggState<NC>& st, int g) {
  const uint32_t k = st.cnt[g];
  if (k == 0u) return;
  atomicAdd(&dst.cnt[d], k);
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int dt = col_dt<SIG>(cs, c), ag = col_ag<SIG>(cs, c);
    if (ag & NFC_AGG_SUM) {
      if (dt == NFC_F64) {
        if (!(LEAVE && dst.err[c]))
          atomicAdd(static_cast<double*>(dst.sum[c]) + d, __longlong_as_double((long long)st.s64[c][g]));
      } else {
        atomicAdd(static_cast<unsigned long long*>(dst.sum[c]) + d,
                  (unsigned long long)agg_sum_bits<NC, SIG>(cs, st, c, g));
      }
    }
    if (dt == NFC_I32) {
      if (ag & NFC_AGG_MIN) atomicMin(static_cast<int*>(dst.mn[c]) + d, static_cast<const int*>(st.mn[c])[g]);
      if (ag & NFC_AGG_MAX) atomicMax(static_cast<int*>(dst.mx[c]) + d, static_cast<const int*>(st.mx[c])[g]);
    } else if (dt == NFC_I64) {
      if (ag & NFC_AGG_MIN) atomicMin(static_cast<long long*>(dst.mn[c]) + d, static_cast<const long long*>(st.mn[c])[g]);
      if (ag & NFC_AGG_MAX) atomicMax(static_cast<long long*>(dst.mx[c]) + d, static_cast<const long long*>(st.mx[c])[g]);
    } else {
      if (ag & NFC_AGG_MIN)
        atomicMin(static_cast<unsigned long long*>(dst.mn[c]) + d, static_cast<const unsigned long long*>(st.mn[c])[g]);
      if (ag & NFC_AGG_MAX)
        atomicMax(static_cast<unsigned long long*>(dst.mx[c]) + d, static_cast<const unsigned long long*>(st.mx[c])[g]);
    }
  }
}

// Slots 0 .. w of a state into slots d0 on of the global one (whole block, after
// a barrier); slot g is entry g << lg.  The CTAs' float64 partial sums of a slot
// are one chain, and more CTAs make it longer (4M rows over 365 keys, mean relative
// error of a sum: 62 CTAs 1.8e-16, 280 CTAs 3.5e-16), so the global state may keep
// the rounding error of each addition (4.7e-17).  That needs the old value back
// from the atomic; a thread has four of them under way.
template <int NC, uint32_t SIG>
NFC_DEV void agg_merge_all(const ColSet& cs, const StateRef& dst, int64_t d0, const AggState<NC>& st, int w, int lg) {
  for (int g = threadIdx.x; g < w; g += blockDim.x) agg_merge<NC, SIG, true>(cs, dst, d0 + g, st, g << lg);
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    if (col_dt<SIG>(cs, c) != NFC_F64 || !(col_ag<SIG>(cs, c) & NFC_AGG_SUM) || !dst.err[c]) continue;
    double* sum = static_cast<double*>(dst.sum[c]) + d0;
    constexpr int K = 4;
    for (int g0 = threadIdx.x; g0 < w; g0 += K * blockDim.x) {
      double old[K], x[K];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const int g = g0 + k * (int)blockDim.x;
        old[k] = x[k] = 0.0;
        if (g < w && st.cnt[g << lg]) {
          x[k] = __longlong_as_double((long long)st.s64[c][g << lg]);
          old[k] = atomicAdd(sum + g, x[k]);
        }
      }
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const double e = f64_two_sum(old[k], x[k]);
        if (!(e == 0.0)) atomicAdd(dst.err[c] + d0 + g0 + k * (int)blockDim.x, e);
      }
    }
  }
}

// The 2^lg interleaved copies of every slot (slot g of copy r is entry
// (g << lg) + r) combined into the first one (whole block).  As many lanes share
// a slot as the block has to spare, each takes its copies one after the other,
// turned by the slot so that the lanes of a warp meet no bank twice.  (32 lanes to
// a slot and all of it by shuffles: 20 us a CTA for 365 slots of 32 copies.)
// ERR: the state keeps the rounding errors of its float64 sums.
template <int NC, uint32_t SIG, bool ERR = false>
NFC_DEV void fold_copies(const ColSet& cs, const AggState<NC>& st, int slots, int lg) {
  int lanes = 0;
  while (lanes < min(lg, 5) && slots << (lanes + 1) <= (int)blockDim.x) ++lanes;
  const int steps = 1 << (lg - lanes), all = (1 << lg) - 1;
  const int part = lane_id() & ((1 << lanes) - 1);
  for (int e0 = threadIdx.x & ~31; e0 < slots << lanes; e0 += (int)blockDim.x) {
    const int g = (e0 + (int)lane_id()) >> lanes;
    const bool in = g < slots, write = in && part == 0;
    const int first = (in ? g : 0) << lg;
    auto entry = [&](int r) { return first + ((((r + g) << lanes) + part) & all); };
    uint32_t cnt = 0;
    for (int r = 0; r < steps; ++r) cnt += st.cnt[entry(r)];
    for (int o = 1; o < 1 << lanes; o <<= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    __syncwarp();
    if (write) st.cnt[first] = cnt;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int dt = col_dt<SIG>(cs, c), ag = col_ag<SIG>(cs, c);
      if ((ag & NFC_AGG_SUM) && dt == NFC_F64) {
        const double* sum = reinterpret_cast<const double*>(st.s64[c]);
        double s = 0.0, e = 0.0;
        for (int r = 0; r < steps; ++r) {
          if (ERR) e += st.err[c][entry(r)];
          e += f64_two_sum(s, sum[entry(r)]);
        }
        for (int o = 1; o < 1 << lanes; o <<= 1) {
          const double s2 = __shfl_xor_sync(0xffffffffu, s, o), e2 = __shfl_xor_sync(0xffffffffu, e, o);
          e += e2;
          e += f64_two_sum(s, s2);
        }
        if (write) {
          st.s64[c][first] = (uint64_t)__double_as_longlong(ERR ? s : f64_close(s, e));
          if (ERR) st.err[c][first] = e;
        }
      } else if (ag & NFC_AGG_SUM) {
        uint64_t s = 0;
        for (int r = 0; r < steps; ++r) s += (uint64_t)agg_sum_bits<NC, SIG>(cs, st, c, entry(r));
        for (int o = 1; o < 1 << lanes; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (write) {
          if (dt == NFC_I64) {
            st.s64[c][first] = s;
          } else {
            st.slo[c][first] = (uint32_t)s & 0xFFFFu;
            st.shi[c][first] = (int32_t)((int64_t)s >> 16);
          }
        }
      }
      if (!(ag & (NFC_AGG_MIN | NFC_AGG_MAX))) continue;
      if (dt == NFC_I32) {
        int32_t lo = INT_MAX, hi = INT_MIN;
        for (int r = 0; r < steps; ++r) {
          if (ag & NFC_AGG_MIN) lo = min(lo, static_cast<const int32_t*>(st.mn[c])[entry(r)]);
          if (ag & NFC_AGG_MAX) hi = max(hi, static_cast<const int32_t*>(st.mx[c])[entry(r)]);
        }
        for (int o = 1; o < 1 << lanes; o <<= 1) {
          lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
          hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (write && (ag & NFC_AGG_MIN)) static_cast<int32_t*>(st.mn[c])[first] = lo;
        if (write && (ag & NFC_AGG_MAX)) static_cast<int32_t*>(st.mx[c])[first] = hi;
      } else {
        // As signed numbers; the float64 encodings with the top bit turned.
        const uint64_t turn = dt == NFC_F64 ? 1ull << 63 : 0ull;
        int64_t lo = LLONG_MAX, hi = LLONG_MIN;
        for (int r = 0; r < steps; ++r) {
          if (ag & NFC_AGG_MIN) lo = min(lo, (int64_t)(static_cast<const uint64_t*>(st.mn[c])[entry(r)] ^ turn));
          if (ag & NFC_AGG_MAX) hi = max(hi, (int64_t)(static_cast<const uint64_t*>(st.mx[c])[entry(r)] ^ turn));
        }
        for (int o = 1; o < 1 << lanes; o <<= 1) {
          lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
          hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
        if (write && (ag & NFC_AGG_MIN)) static_cast<uint64_t*>(st.mn[c])[first] = (uint64_t)lo ^ turn;
        if (write && (ag & NFC_AGG_MAX)) static_cast<uint64_t*>(st.mx[c])[first] = (uint64_t)hi ^ turn;
      }
    }
    __syncwarp();
  }
}

template <int NC, uint32_t SIG, bool ERR = false>
NFC_DEV void agg_emit(const ColSet& cs, const AggState<NC>& st, int g, const OutSet& o, int64_t pos, int64_t key) {
  o.ukeys[pos] = key;
  o.counts[pos] = (int64_t)st.cnt[g];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int dt = col_dt<SIG>(cs, c), ag = col_ag<SIG>(cs, c);
    if (ERR && dt == NFC_F64 && (ag & NFC_AGG_SUM))
      static_cast<double*>(o.sum[c])[pos] = f64_close(reinterpret_cast<const double*>(st.s64[c])[g], st.err[c][g]);
    else if (ag & NFC_AGG_SUM)
      static_cast<int64_t*>(o.sum[c])[pos] = agg_sum_bits<NC, SIG>(cs, st, c, g);
    if (dt == NFC_I32) {
      if (ag & NFC_AGG_MIN) static_cast<int32_t*>(o.mn[c])[pos] = static_cast<const int32_t*>(st.mn[c])[g];
      if (ag & NFC_AGG_MAX) static_cast<int32_t*>(o.mx[c])[pos] = static_cast<const int32_t*>(st.mx[c])[g];
    } else if (dt == NFC_I64) {
      if (ag & NFC_AGG_MIN) static_cast<int64_t*>(o.mn[c])[pos] = static_cast<const int64_t*>(st.mn[c])[g];
      if (ag & NFC_AGG_MAX) static_cast<int64_t*>(o.mx[c])[pos] = static_cast<const int64_t*>(st.mx[c])[g];
    } else {
      if (ag & NFC_AGG_MIN) static_cast<uint64_t*>(o.mn[c])[pos] = f64_min_dec(static_cast<const uint64_t*>(st.mn[c])[g]);
      if (ag & NFC_AGG_MAX) static_cast<uint64_t*>(o.mx[c])[pos] = f64_max_dec(static_cast<const uint64_t*>(st.mx[c])[g]);
    }
  }
}

// ---------------------------------------------------------------- hot keys
// Rows of a key that takes a large share of a CTA's rows meet on one address:
// every float64 sum and 64-bit min/max is then a serial chain.  Such a key
// gets accumulators in every thread's registers instead (a compare and, on a
// hit, plain arithmetic), reduced per warp and folded into its slot once.
template <int NC>
struct HotAcc {
  uint32_t cnt;
  uint64_t sum[NC > 0 ? NC : 1];
  int32_t mn32[NC > 0 ? NC : 1], mx32[NC > 0 ? NC : 1];
  uint64_t mn64[NC > 0 ? NC : 1], mx64[NC > 0 ? NC : 1];  // int64 as is, float64 as the ordered encodings
};

// Keys held in registers: what two 512-thread CTAs per SM leave room for (the
// slices of 69M Zipf(1.1) rows: four keys at one CTA per SM 1.04 ms, two keys at
// two CTAs 0.76, four keys at two CTAs, spilled, 1.17).  Two and more columns of
// run-time types would need one CTA per SM, and the rows of the other keys then
// lose more than the hot keys gain (40M Zipf(1.1) rows over 30,000 keys, int64 and
// float64 with all aggregates 1.54 ms without, 1.69 with; four columns 2.13 and
// 2.55).
constexpr int kHotKeys = 2;
template <int NC, uint32_t SIG>
constexpr bool hot_columns() { return SIG != 0 || NC == 1; }

template <int NC, uint32_t SIG>
NFC_DEV void hot_init(const ColSet& cs, HotAcc<NC>& a) {
  a.cnt = 0u;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const bool i64 = col_dt<SIG>(cs, c) == NFC_I64;
    a.sum[c] = 0ull;
    a.mn32[c] = INT_MAX;
    a.mx32[c] = INT_MIN;
    a.mn64[c] = i64 ? (uint64_t)LLONG_MAX : ~0ull;
    a.mx64[c] = i64 ? (uint64_t)LLONG_MIN : 0ull;
  }
}

template <int NC, uint32_t SIG>
NFC_DEV void hot_add(const ColSet& cs, HotAcc<NC>& a, const uint64_t* raw) {
  ++a.cnt;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int dt = col_dt<SIG>(cs, c), ag = col_ag<SIG>(cs, c);
    const uint64_t r = raw[c];
    if (dt == NFC_I32) {
      const int32_t v = (int32_t)(uint32_t)r;
      if (ag & NFC_AGG_SUM) a.sum[c] += (uint64_t)(int64_t)v;
      if (ag & NFC_AGG_MIN) a.mn32[c] = min(a.mn32[c], v);
      if (ag & NFC_AGG_MAX) a.mx32[c] = max(a.mx32[c], v);
    } else if (dt == NFC_I64) {
      if (ag & NFC_AGG_SUM) a.sum[c] += r;
      if (ag & NFC_AGG_MIN) a.mn64[c] = (uint64_t)min((long long)a.mn64[c], (long long)r);
      if (ag & NFC_AGG_MAX) a.mx64[c] = (uint64_t)max((long long)a.mx64[c], (long long)r);
    } else {
      if (ag & NFC_AGG_SUM)
        a.sum[c] = (uint64_t)__double_as_longlong(__longlong_as_double((long long)a.sum[c]) +
                                                  __longlong_as_double((long long)r));
      if (ag & NFC_AGG_MIN) a.mn64[c] = min(a.mn64[c], f64_min_enc(r));
      if (ag & NFC_AGG_MAX) a.mx64[c] = max(a.mx64[c], f64_max_enc(r));
    }
  }
}

// One thread's accumulators into slot g.
template <int NC, uint32_t SIG, bool ERR = false>
NFC_DEV void hot_apply(const ColSet& cs, const AggState<NC>& st, uint32_t g, const HotAcc<NC>& a) {
  uint64_t mn[NC > 0 ? NC : 1], mx[NC > 0 ? NC : 1];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const bool narrow = col_dt<SIG>(cs, c) == NFC_I32;
    mn[c] = narrow ? (uint64_t)(int64_t)a.mn32[c] : a.mn64[c];
    mx[c] = narrow ? (uint64_t)(int64_t)a.mx32[c] : a.mx64[c];
  }
  agg_apply_group<NC, SIG, ERR>(cs, st, g, a.cnt, a.sum, mn, mx);
}

// Reduce one hot key over the warp and fold it into slot g (whole warp).
template <int NC, uint32_t SIG, bool ERR = false>
NFC_DEV void hot_flush(const ColSet& cs, const AggState<NC>& st, uint32_t g, const HotAcc<NC>& a) {
  const uint32_t k = __reduce_add_sync(0xffffffffu, a.cnt);
  if (k == 0u) return;
  uint64_t sum[NC > 0 ? NC : 1], mn[NC > 0 ? NC : 1], mx[NC > 0 ? NC : 1];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int dt = col_dt<SIG>(cs, c), ag = col_ag<SIG>(cs, c);
    uint64_t s = a.sum[c];
    if (ag & NFC_AGG_SUM) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const uint64_t t = __shfl_xor_sync(0xffffffffu, s, o);
        s = dt == NFC_F64 ? (uint64_t)__double_as_longlong(__longlong_as_double((long long)s) +
                                                           __longlong_as_double((long long)t))
                          : s + t;
      }
    }
    sum[c] = s;
    if (dt == NFC_I32) {
      mn[c] = (uint64_t)(int64_t)__reduce_min_sync(0xffffffffu, a.mn32[c]);
      mx[c] = (uint64_t)(int64_t)__reduce_max_sync(0xffffffffu, a.mx32[c]);
    } else {
      uint64_t lo = a.mn64[c], hi = a.mx64[c];
      if (ag & (NFC_AGG_MIN | NFC_AGG_MAX)) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const uint64_t l2 = __shfl_xor_sync(0xffffffffu, lo, o), h2 = __shfl_xor_sync(0xffffffffu, hi, o);
          if (dt == NFC_I64) {
            lo = (uint64_t)min((long long)lo, (long long)l2);
            hi = (uint64_t)max((long long)hi, (long long)h2);
          } else {
            lo = min(lo, l2);
            hi = max(hi, h2);
          }
        }
      }
      mn[c] = lo;
      mx[c] = hi;
    }
  }
  if (lane_id() == 0) agg_apply_group<NC, SIG, ERR>(cs, st, g, k, sum, mn, mx);
}

// The up to H slots of [0, w) with the most rows counted so far, at least
// `floor` rows each; 0xFFFFFFFF in the rest.  Whole block; red[33] is shared.
// Slots below 2^16 and counts below 2^16.
template <int H>
NFC_DEV void pick_hot(const uint32_t* cnt, int w, uint32_t floor, uint32_t* red, uint32_t (&hot)[H]) {
  uint32_t last = 0xFFFFFFFFu;
#pragma unroll
  for (int h = 0; h < H; ++h) {
    uint32_t best = 0u;
    for (int g = threadIdx.x; g < w; g += blockDim.x) {
      const uint32_t v = (cnt[g] << 16) | (uint32_t)g;
      if (v < last) best = max(best, v);
    }
    best = __reduce_max_sync(0xffffffffu, best);
    if (lane_id() == 0) red[threadIdx.x >> 5] = best;
    __syncthreads();
    best = red[lane_id() < (blockDim.x >> 5) ? lane_id() : 0];
    best = __reduce_max_sync(0xffffffffu, best);
    __syncthreads();
    hot[h] = (best >> 16) >= floor ? best & 0xFFFFu : 0xFFFFFFFFu;
    last = best;
  }
}

}  // namespace nfc

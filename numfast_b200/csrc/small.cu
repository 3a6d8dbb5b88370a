// Small inputs: the probe and, where the key span fits one CTA's shared
// memory, the whole group-by in one launch.
//
// A group-by of 10,000 rows took 100 us, 27 of them on the device in five
// dependent launches; the rest was launches, allocations, memsets and two
// read-backs.  Up to kSmallRows rows one CTA does everything from registers and
// shared memory and leaves its answer in pinned host memory, so the call is one
// allocation, one launch and one wait.  When the span is too wide the kernel
// has still done the probe's work (range, count, sortedness, combined validity
// bitmap) and the call goes on from there.  10,007 rows over 250 keys: 102 -> 51
// us a call.
//
// Few keys meet on few addresses, and a float64 sum is a compare-and-swap loop
// there (16,384 rows of one key: 615 us with one slot per key, 74 now).  So the
// state has copies where the keys leave room, a warp whose rows all have one key
// adds them as one, and with sorted keys a thread adds its rows run by run.
// Sorted keys also keep the rounding errors of their float64 additions: as one
// chain of atomics per key the sums of 10,000 rows over ten keys were off by
// 6.2e-16 on average, by 8.6e-17 as SORTED's run sums.
#include <algorithm>
#include <cstring>

#include "agg_smem.cuh"
#include "probe.cuh"

namespace nfc {

// Threads (each takes four consecutive rows per step): the shared atomics want all
// the threads a CTA can have, three and four columns need the registers.
template <int NC>
struct SmallShape {
  static constexpr int threads = NC <= 2 ? 1024 : 512;
  static constexpr int warps = threads / 32;
  static constexpr int steps = (int)(kSmallRows / (4 * threads));
  static constexpr int parts = steps * warps / 32;  // partial probe records per lane
  static_assert(parts * 32 == steps * warps && warps <= 32, "one warp reduces the partial records");
};
static_assert(kSmallRows == kProbeBlockRows, "one probe record");
constexpr int kSmCopies = 8;  // log2 of the most copies of the state

template <int NC>
__global__ void __launch_bounds__(SmallShape<NC>::threads, 1)
    k_small(const int32_t* __restrict__ keys, BitmapSet bms, ColSet cs, int n, bool aligned, OutSet o, int64_t out_cap,
            uint32_t state_bytes, uint32_t slot_bytes, uint32_t err_bytes, int max_copies,
            uint32_t* __restrict__ vmask, ProbeRec* __restrict__ rec, SmallResult* __restrict__ res) {
  constexpr int kSmThreads = SmallShape<NC>::threads, kSmWarps = SmallShape<NC>::warps;
  constexpr int kSmSteps = SmallShape<NC>::steps, kSmParts = SmallShape<NC>::parts;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ ProbeAcc s_part[kSmSteps * kSmWarps];
  __shared__ ProbeAcc s_all;
  __shared__ uint32_t s_cnt[kSmWarps];
  const int tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
  const ProbeAcc none{false, true, 0, 0, INT_MAX, INT_MIN, 0};
  // ---- keys and combined validity; one record per warp and step, in row order.
  int32_t key[kSmSteps][4];
  uint32_t valid[kSmSteps];
#pragma unroll
  for (int j = 0; j < kSmSteps; ++j) {
    const int r0 = (j * kSmThreads + tid) * 4;
    const int left = n - r0;
    valid[j] = left >= 4 ? 0xFu : left > 0 ? (1u << left) - 1u : 0u;
    if (left >= 4 && aligned) {
      const int4 k = __ldg(reinterpret_cast<const int4*>(keys + r0));
      key[j][0] = k.x; key[j][1] = k.y; key[j][2] = k.z; key[j][3] = k.w;
    } else {
#pragma unroll
      for (int r = 0; r < 4; ++r) key[j][r] = r < left ? keys[r0 + r] : 0;
    }
#pragma unroll
    for (int b = 0; b < NFC_MAX_COLS + 2; ++b)
      if (b < bms.nbm && valid[j]) valid[j] &= (uint32_t)(__ldg(bms.bm[b] + (r0 >> 3)) >> (r0 & 7));
  }
#pragma unroll
  for (int j = 0; j < kSmSteps; ++j) {
    if (vmask) {
      uint32_t w = valid[j] << (4 * (lane & 7));
#pragma unroll
      for (int off = 1; off < 8; off <<= 1) w |= __shfl_xor_sync(0xffffffffu, w, off);
      const int r0 = (j * kSmThreads + tid) * 4;
      if ((lane & 7) == 0 && r0 < n) vmask[r0 >> 5] = w;
    }
    ProbeAcc acc = none;
#pragma unroll
    for (int r = 0; r < 4; ++r)
      if ((valid[j] >> r) & 1u) acc = probe_combine(acc, ProbeAcc{true, true, key[j][r], key[j][r], key[j][r], key[j][r], 1});
    acc = probe_warp_reduce(acc);
    if (lane == 0) s_part[j * kSmWarps + warp] = acc;
  }
  __syncthreads();
  if (warp == 0) {
    ProbeAcc acc = none;
#pragma unroll
    for (int i = 0; i < kSmParts; ++i) acc = probe_combine(acc, s_part[lane * kSmParts + i]);
    acc = probe_warp_reduce(acc);
    if (lane == 0) s_all = acc;
  }
  __syncthreads();
  const ProbeAcc all = s_all;
  const int64_t m = all.has ? (int64_t)all.kmax - all.kmin + 1 : 0;
  // The state (the rounding errors have their own room), and an output that
  // certainly fits (else the host reports it).
  const bool fits = m > 0 && m * slot_bytes + 16 <= state_bytes && (out_cap >= m || out_cap >= all.n);
  if (tid == 0) {
    *rec = ProbeRec{all.first, all.last, all.kmin, all.kmax, (uint32_t)all.n,
                    (all.has ? 1u : 0u) | (all.sorted ? 2u : 0u)};
    res->probe.n_valid = all.n;
    res->probe.kmin = all.has ? all.kmin : 0;
    res->probe.kmax = all.has ? all.kmax : 0;
    res->probe.sorted = all.sorted ? 1 : 0;
    res->probe.pad = 0;
    res->done = fits ? 1 : 0;
    if (!fits) {
      res->ng = 0;
      __threadfence_system();
    }
  }
  if (!fits) return;
  // ---- aggregate in shared memory (at most 65,536 rows: the split sums hold).
  const int w = (int)m;
  // Copies: as many as fit, as long as a slot of one sees eight rows on average
  // (setting up and folding 4,000 entries takes 4 us).
  int lg = 0;
  while (lg < max_copies && ((size_t)w << (lg + 1)) * (slot_bytes + err_bytes) <= state_bytes && w << (lg + 1) <= n / 8)
    ++lg;
  const AggState<NC> st = carve_agg<NC, 0, true>(cs, smem_raw, w << lg);
  for (int g = tid; g < w << lg; g += kSmThreads) agg_init<NC, 0, true>(cs, st, g);
  __syncthreads();
  const uint32_t copy = (uint32_t)(lane + warp) & ((1u << lg) - 1u);
  auto entry = [&](int32_t k) { return ((uint32_t)(k - all.kmin) << lg) + copy; };
#pragma unroll
  for (int j = 0; j < kSmSteps; ++j) {
    const int r0 = (j * kSmThreads + tid) * 4;
    const unsigned any = __ballot_sync(0xffffffffu, valid[j] != 0u);
    if (any == 0u) continue;
    uint64_t raw[4][NC > 0 ? NC : 1];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const bool narrow = cs.dtype[c] == NFC_I32;
      if (aligned && r0 + 4 <= n) {
        if (narrow) {
          const int4 v = __ldg(reinterpret_cast<const int4*>(static_cast<const int32_t*>(cs.data[c]) + r0));
          raw[0][c] = (uint64_t)(int64_t)v.x; raw[1][c] = (uint64_t)(int64_t)v.y;
          raw[2][c] = (uint64_t)(int64_t)v.z; raw[3][c] = (uint64_t)(int64_t)v.w;
        } else {
          const ulonglong2* p = reinterpret_cast<const ulonglong2*>(static_cast<const uint64_t*>(cs.data[c]) + r0);
          const ulonglong2 x = __ldg(p), y = __ldg(p + 1);
          raw[0][c] = x.x; raw[1][c] = x.y; raw[2][c] = y.x; raw[3][c] = y.y;
        }
      } else {
#pragma unroll
        for (int r = 0; r < 4; ++r)
          raw[r][c] = r0 + r >= n ? 0ull
                      : narrow    ? (uint64_t)(int64_t) static_cast<const int32_t*>(cs.data[c])[r0 + r]
                                  : static_cast<const uint64_t*>(cs.data[c])[r0 + r];
      }
    }
    // One key in the whole warp: added as one.
    int32_t k0 = key[j][0];
    bool same = true;
#pragma unroll
    for (int r = 1; r < 4; ++r) {
      if ((valid[j] & ((1u << r) - 1u)) == 0u) k0 = key[j][r];
      else if ((valid[j] >> r) & 1u) same &= key[j][r] == k0;
    }
    const int32_t wk = __shfl_sync(0xffffffffu, k0, __ffs(any) - 1);
    if (__all_sync(0xffffffffu, valid[j] == 0u || (same && k0 == wk))) {
      HotAcc<NC> acc;
      hot_init<NC, 0>(cs, acc);
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if ((valid[j] >> r) & 1u) hot_add<NC, 0>(cs, acc, raw[r]);
      hot_flush<NC, 0, true>(cs, st, entry(wk), acc);
    } else if (all.sorted) {
      HotAcc<NC> acc;
      hot_init<NC, 0>(cs, acc);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (!((valid[j] >> r) & 1u)) continue;
        hot_add<NC, 0>(cs, acc, raw[r]);
        // The run ends with the thread's last row or before another key.
        const uint32_t later = valid[j] >> (r + 1);
        int32_t next = key[j][r];
#pragma unroll
        for (int q = 3; q > r; --q)
          if ((valid[j] >> q) & 1u) next = key[j][q];
        if (later == 0u || next != key[j][r]) {
          hot_apply<NC, 0, true>(cs, st, entry(key[j][r]), acc);
          hot_init<NC, 0>(cs, acc);
        }
      }
    } else {
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if ((valid[j] >> r) & 1u) agg_apply<NC, 0>(cs, st, entry(key[j][r]), raw[r]);
    }
  }
  __syncthreads();
  if (lg > 0) {
    fold_copies<NC, 0, true>(cs, st, w, lg);
    __syncthreads();
  }
  // ---- present groups in key order: warp w owns consecutive slots.
  const int per = ((w + kSmWarps - 1) / kSmWarps + 31) & ~31;
  const int g0 = min(w, warp * per), g1 = min(w, g0 + per);
  uint32_t c = 0;
  for (int g = g0; g < g1; g += 32) c += __popc(__ballot_sync(0xffffffffu, g + lane < g1 && st.cnt[(g + lane) << lg] != 0u));
  if (lane == 0) s_cnt[warp] = c;
  __syncthreads();
  const uint32_t mine = lane < kSmWarps ? s_cnt[lane] : 0u;
  int64_t pos = __reduce_add_sync(0xffffffffu, lane < warp ? mine : 0u);
  const uint32_t total = __reduce_add_sync(0xffffffffu, mine);
  const unsigned lt = lanemask_lt();
  for (int g = g0; g < g1; g += 32) {
    const bool pres = g + lane < g1 && st.cnt[(g + lane) << lg] != 0u;
    const unsigned bal = __ballot_sync(0xffffffffu, pres);
    if (pres) agg_emit<NC, 0, true>(cs, st, (g + lane) << lg, o, pos + __popc(bal & lt), (int64_t)all.kmin + g + lane);
    pos += __popc(bal);
  }
  if (tid == 0) {
    res->ng = total;
    __threadfence_system();
  }
}

template <int NC>
static int launch_small(const nfc_groupby_args* a, const ColSet& cs, const OutSet& o, uint32_t* vmask, ProbeRec* rec,
                        SmallResult* res, cudaStream_t s) {
  constexpr int kState = 96 * 1024;
  const size_t slot = state_bytes_per_slot(cs);
  const size_t errs = state_err_bytes_per_slot(cs);
  bool wide = false;  // 32-bit atomics alone keep up on few keys
  for (int c = 0; c < cs.ncols; ++c) wide |= cs.dtype[c] != NFC_I32 && cs.aggs[c] != 0;
  const int smem = kState + (int)(errs * (kState / slot));  // 8,191 slots of one float64 sum: 160 KB
  NFC_CUDA(allow_dynamic_smem<k_small<NC>>());
  k_small<NC><<<1, SmallShape<NC>::threads, smem, s>>>(a->keys, bitmaps_of(a), cs, (int)a->n, inputs_aligned(a), o,
                                                       a->out_cap, kState, (uint32_t)slot, (uint32_t)errs,
                                                       wide ? kSmCopies : 0, vmask, rec, res);
  NFC_CUDA(cudaGetLastError());
  return NFC_OK;
}

int run_small(const nfc_groupby_args* a, const ColSet& cs, const OutSet& o, cudaStream_t s, Scratch& sc,
              uint32_t** vmask_out, const ProbeRec** recs_out, SmallResult* out, StageTimer* tm) {
  SmallResult* res = reinterpret_cast<SmallResult*>(pinned_readback());
  if (!res) return NFC_ERR_UNSUPPORTED;  // the caller probes as usual
  const size_t words = (size_t)((a->n + 31) / 32 + 1);
  // One allocation: the probe record, then the bitmap at a 256-byte boundary.
  unsigned char* buf = nullptr;
  NFC_CUDA(sc.alloc(&buf, 256 + words * 4));
  ProbeRec* rec = reinterpret_cast<ProbeRec*>(buf);
  uint32_t* vmask = bitmaps_of(a).nbm > 0 ? reinterpret_cast<uint32_t*>(buf + 256) : nullptr;
  tm->mark(s);
  int rc;
  switch (cs.ncols) {
    case 0: rc = launch_small<0>(a, cs, o, vmask, rec, res, s); break;
    case 1: rc = launch_small<1>(a, cs, o, vmask, rec, res, s); break;
    case 2: rc = launch_small<2>(a, cs, o, vmask, rec, res, s); break;
    case 3: rc = launch_small<3>(a, cs, o, vmask, rec, res, s); break;
    default: rc = launch_small<4>(a, cs, o, vmask, rec, res, s); break;
  }
  if (rc) return rc;
  tm->launched();
  tm->mark(s);
  NFC_CUDA(cudaStreamSynchronize(s));
  std::memcpy(out, res, sizeof(*out));
  *vmask_out = vmask;
  *recs_out = rec;
  return NFC_OK;
}

}  // namespace nfc

// Distinct values by partition: unique keys and grouped COUNT DISTINCT without
// a sort of the rows.
//
// The partition passes (partition.cu) bring the rows into buckets of
// consecutive keys, a few thousand rows each; one CTA per bucket then finds
// what is distinct in shared memory and writes it at the bucket's place
// (decoupled look-back over the buckets), in ascending key order.
//   unique          a bit per key of the bucket; a key's rank is the number of
//                   bits below it, which addresses its first row and count
//   count distinct  a hash set of the bucket's (key, value) records, a counter
//                   per key
// Against the sorted forms (radix_sort.cu) that is two passes of 8-byte records
// instead of four of pairs (or of one per eight bits of the pair), and no run
// pass: 200M keys over the full int32 range 5.85 -> 3.89 ms, COUNT DISTINCT of
// 50M rows over 1M keys 2.10 -> 1.28 ms.  Rows that do not spread over the
// buckets (few keys, skew), small inputs and unaligned columns stay with the sort:
// a bucket has to fit one CTA, the scatter passes copy 16-byte vectors.
#include <algorithm>

#include "groupby_host.h"

namespace nfc {
namespace {

constexpr int kDpThreads = 512;
constexpr int kDpWarps = kDpThreads / 32;
// Where the sort takes over, us partitioned / sorted: unique of 1.1M rows over 1M
// keys 264 / 239, 2.1M 284 / 295, 3M 304 / 338, 20M 597 / 830.
constexpr int64_t kDpMinRows = 1 << 21;

struct DpArgs {
  const uint64_t* rec;  // key low part | payload << 32
  const int64_t* offs;
  int32_t nb, wb;
  int64_t kmin, m;  // span
  uint64_t* lb;
  uint32_t* ticket;
  int64_t* ng_out;
  int32_t* err;
};

// The bucket's place among the outputs.  The whole CTA looks back, 512 buckets
// at a time: the CTAs of a wave reach this point together, and a warp's walk
// over the 444 of them, 32 at a time, is 14 loads one after the other (unique of
// 200M rows 1,470 -> 1,425 us, with the totals published before the counts).
// dp_publish makes the bucket's total known; dp_base returns the place to every
// thread.
NFC_DEV void dp_publish(const DpArgs& a, int32_t b, uint32_t total) {
  if (threadIdx.x == 0) lb_store(a.lb + b, (b == 0 ? kLbInc : kLbAgg) | (uint64_t)total);
}

struct DpWalk {
  uint64_t sum[kDpWarps];
  int32_t state[kDpWarps];  // 0 totals only, 1 ends at an inclusive one, 2 one is not published yet
};

NFC_DEV int64_t dp_base(const DpArgs& a, int32_t b, uint32_t total, DpWalk* sw) {
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  uint64_t excl = 0;
  if (b > 0) {  // the same for every thread, as is every branch below
    int32_t j = b - 1;
    uint32_t spins = 0;
    while (true) {
      const int32_t t = j - (int32_t)threadIdx.x;
      const uint64_t w = t >= 0 ? ld_volatile_u64(a.lb + t) : kLbInc;
      const uint64_t flag = w & ~kLbVal;
      const unsigned inc = __ballot_sync(0xffffffffu, flag == kLbInc);
      const unsigned pending = __ballot_sync(0xffffffffu, flag == 0);
      const unsigned upto = inc ? (((inc & (0u - inc)) << 1) - 1u) : 0xffffffffu;  // lanes 0 .. first inclusive
      const uint64_t v = warp_sum((upto >> lane) & 1u ? (w & kLbVal) : 0ull);
      if (lane == 0) {
        sw->sum[warp] = v;
        sw->state[warp] = (pending & upto) ? 2 : inc ? 1 : 0;
      }
      __syncthreads();
      const int32_t st = lane < kDpWarps ? sw->state[lane] : 0;
      const unsigned done = __ballot_sync(0xffffffffu, st == 1), wait = __ballot_sync(0xffffffffu, st == 2);
      const unsigned stop = done | wait;
      const unsigned use = stop ? (((stop & (0u - stop)) << 1) - 1u) : 0xffffffffu;  // warps 0 .. first that stops
      const uint64_t part = warp_sum(lane < kDpWarps && ((use >> lane) & 1u) ? sw->sum[lane] : 0ull);
      __syncthreads();
      if (wait & use) {  // read these again
        if (++spins > kSpinLimit) {
          if (threadIdx.x == 0) atomicExch(a.err, NFC_ERR_TIMEOUT);
          break;
        }
        continue;
      }
      excl += part;
      if (done & use) break;
      j -= kDpThreads;
    }
  }
  if (threadIdx.x == 0) {
    if (b > 0) {
      __threadfence();
      lb_store(a.lb + b, kLbInc | (excl + total));
    }
    if (b == a.nb - 1) *a.ng_out = (int64_t)(excl + total);
  }
  return (int64_t)excl;
}

// The CTA's bucket; -1 when an earlier kernel gave up on a wait.
NFC_DEV int32_t dp_claim(const DpArgs& a, int32_t* s_bucket) {
  if (threadIdx.x == 0) *s_bucket = (int32_t)atomicAdd(a.ticket, 1u);
  return sync_failed(a.err) ? -1 : *s_bucket;
}

// How the rows are cut up.  wb: the widest bucket (2^wb keys, lo <= wb <= hi) of
// no more than `rows` rows on average, or wider where that makes more than
// kDpMaxBuckets; none if a bucket then has less than min_rows rows on average.
constexpr int kDpMaxBuckets = 32768;

struct DpRule {
  int64_t rows, min_rows, max_rows;
  int lo, hi;
  __host__ __device__ int width(int64_t m, int64_t nv) const {
    auto buckets = [m](int w) { return (m + (1ll << w) - 1) >> w; };
    int wb = lo;
    while (wb < hi && buckets(wb + 1) * rows >= nv) ++wb;
    while (wb < hi && buckets(wb) > kDpMaxBuckets) ++wb;
    const int64_t nb = buckets(wb);
    return nb > kDpMaxBuckets || nb * min_rows > nv || nb * max_rows < nv ? -1 : wb;
  }
};

// Looks at up to 8,192 rows before anything reads them all: are there few rows
// per bucket, or does one bucket hold far more than max_rows of them?  Then the
// caller sorts, some 25 us later instead of a probe and a histogram later (200M
// zipf keys: 0.37 of 6 ms).  What it lets through by chance the histogram finds.
constexpr int kDpSampleThreads = 1024, kDpSamplesPerThread = 8;

__global__ void __launch_bounds__(kDpSampleThreads) k_dp_sample(const int32_t* __restrict__ keys,
                                                               const uint8_t* __restrict__ validity, int64_t n,
                                                               int samples, DpRule rule, int32_t* __restrict__ ok) {
  extern __shared__ __align__(16) uint32_t dp_cnt[];  // kDpMaxBuckets u16
  __shared__ int32_t s_lo, s_hi, s_wb;
  __shared__ uint32_t s_n, s_max;
  const int tid = threadIdx.x;
  if (tid == 0) {
    s_lo = 0x7FFFFFFF;
    s_hi = -0x7FFFFFFF - 1;
    s_n = s_max = 0u;
  }
  for (int i = tid; i < kDpMaxBuckets / 2; i += kDpSampleThreads) dp_cnt[i] = 0u;
  __syncthreads();
  int32_t key[kDpSamplesPerThread];
  uint32_t have = 0;
  int32_t lo = 0x7FFFFFFF, hi = -0x7FFFFFFF - 1;
#pragma unroll
  for (int j = 0; j < kDpSamplesPerThread; ++j) {
    const int i = j * kDpSampleThreads + tid;
    key[j] = 0;
    if (i < samples) {
      const int64_t r = (int64_t)i * n / samples;
      if (!validity || bit_at(validity, r)) {
        key[j] = __ldg(keys + r);
        have |= 1u << j;
        lo = min(lo, key[j]);
        hi = max(hi, key[j]);
      }
    }
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  const uint32_t c = __reduce_add_sync(0xffffffffu, (uint32_t)__popc(have));
  if (lane_id() == 0) {
    atomicMin(&s_lo, lo);
    atomicMax(&s_hi, hi);
    atomicAdd(&s_n, c);
  }
  __syncthreads();
  const int64_t nv = n * s_n / samples;
  if (tid == 0) s_wb = s_n ? rule.width((int64_t)s_hi - s_lo + 1, nv) : -1;
  __syncthreads();
  if (s_wb < 0) {  // the same for every thread
    if (tid == 0) *ok = 0;
    return;
  }
  uint32_t most = 0;
#pragma unroll
  for (int j = 0; j < kDpSamplesPerThread; ++j)
    if (have >> j & 1u) {
      const uint32_t b = ((uint32_t)key[j] - (uint32_t)s_lo) >> s_wb;
      const uint32_t old = atomicAdd(&dp_cnt[b >> 1], 1u << (16 * (b & 1)));
      most = max(most, (old >> (16 * (b & 1)) & 0xFFFFu) + 1u);
    }
  most = __reduce_max_sync(0xffffffffu, most);
  if (lane_id() == 0) atomicMax(&s_max, most);
  __syncthreads();
  // A bucket of max_rows rows has `share` sampled ones on average.
  const int64_t share = rule.max_rows * samples / n;
  if (tid == 0) *ok = s_max <= 12 + share + share / 2 ? 1 : 0;
}

// ---------------------------------------------------------------- unique
// 200M rows in 32,768 buckets of 2^17 keys: 1,425 us, 3.4 TB/s; issue (62%) and the latency of the
// record loads and shared atomics, with three CTAs per SM (two, with 32-bit
// counts and ranks: 2,017 us).
// Shared memory: bits[words] | first[most] | count[most] u16 | prefix[words]
// u16; words = keys of a bucket / 32 (a multiple of 4), most = an upper bound of
// the distinct keys of one (even, below 2^16 as its rows are).
__global__ void __launch_bounds__(kDpThreads, 3) k_dp_unique(DpArgs a, int32_t most, int32_t* __restrict__ uniq,
                                                            int32_t* __restrict__ first_out,
                                                            int64_t* __restrict__ counts, int32_t* __restrict__ inv) {
  extern __shared__ __align__(16) uint32_t dp_smem[];
  __shared__ uint32_t s_scan[33];
  __shared__ DpWalk s_walk;
  __shared__ int32_t s_bucket;
  const int32_t b = dp_claim(a, &s_bucket);
  if (b < 0) return;
  const int32_t words = (1 << a.wb) >> 5;
  uint32_t* bits = dp_smem;
  uint32_t* first = bits + words;
  uint32_t* cnt = first + most;
  uint16_t* prefix = reinterpret_cast<uint16_t*>(cnt + most / 2);
  const int64_t r0 = a.offs[b];
  const int n = (int)(a.offs[b + 1] - r0);
  const uint64_t* __restrict__ rec = a.rec + r0;
  for (int i = threadIdx.x; i < words; i += kDpThreads) bits[i] = 0u;
  for (int i = threadIdx.x; i < min(n, most); i += kDpThreads) first[i] = 0xFFFFFFFFu;
  for (int i = threadIdx.x; i < min((n + 1) / 2, most / 2); i += kDpThreads) cnt[i] = 0u;
  __syncthreads();
#pragma unroll 4
  for (int i = threadIdx.x; i < n; i += kDpThreads) {
    const uint32_t k = (uint32_t)__ldg(rec + i);
    atomicOr(&bits[k >> 5], 1u << (k & 31));
  }
  __syncthreads();
  // Ranks: 4 words a thread and step (one 16-byte read, one 8-byte write; a
  // thread's words one after the other would be an 8-way bank conflict).
  uint32_t total = 0;
  for (int w0 = 0; w0 < words; w0 += 4 * kDpThreads) {
    const int w = w0 + 4 * threadIdx.x;
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (w < words) v = *reinterpret_cast<const uint4*>(bits + w);
    const uint32_t c0 = __popc(v.x), c1 = c0 + __popc(v.y), c2 = c1 + __popc(v.z), c3 = c2 + __popc(v.w);
    uint32_t t;
    const uint32_t x = total + block_excl_scan(c3, s_scan, &t);
    if (w < words)
      *reinterpret_cast<uint2*>(prefix + w) = make_uint2(x | ((x + c0) << 16), (x + c1) | ((x + c2) << 16));
    total += t;
    __syncthreads();
  }
  dp_publish(a, b, total);
  auto rank_of = [&](uint32_t k) {
    return (uint32_t)prefix[k >> 5] + (uint32_t)__popc(bits[k >> 5] & ((1u << (k & 31)) - 1u));
  };
#pragma unroll 4
  for (int i = threadIdx.x; i < n; i += kDpThreads) {
    const uint64_t r = __ldg(rec + i);
    const uint32_t q = rank_of((uint32_t)r);
    atomicMin(&first[q], (uint32_t)(r >> 32));
    atomicAdd(&cnt[q >> 1], 1u << (16 * (q & 1)));
  }
  __syncthreads();
  const int64_t base = dp_base(a, b, total, &s_walk);
  for (uint32_t i = threadIdx.x; i < total; i += kDpThreads) {
    first_out[base + i] = (int32_t)first[i];
    counts[base + i] = (int64_t)reinterpret_cast<const uint16_t*>(cnt)[i];
  }
  const int64_t key0 = a.kmin + ((int64_t)b << a.wb);
  for (int w = threadIdx.x; w < words; w += kDpThreads) {
    int64_t o = base + prefix[w];
    for (uint32_t v = bits[w]; v; v &= v - 1u) uniq[o++] = (int32_t)(key0 + 32 * w + __ffs(v) - 1);
  }
  if (inv)
    for (int i = threadIdx.x; i < n; i += kDpThreads) {
      const uint64_t r = __ldg(rec + i);
      inv[(uint32_t)(r >> 32)] = (int32_t)(base + rank_of((uint32_t)r));
    }
}

// ---------------------------------------------------------------- count distinct
// 47.5M records in 7,813 buckets: 551 us, bound by the walks' shared-memory
// round trips and the 64-bit compare-and-swap of each new pair (with linear
// probing and a loop per record 1,538; at half that load 710).
// Shared memory: set[slots] u64 | distinct[keys of a bucket] u32.  A record is
// its own hash key (the key part is below 2^wb, so all ones is free).
constexpr uint64_t kDpEmpty = ~0ull;

__global__ void __launch_bounds__(kDpThreads, 3) k_dp_count(DpArgs a, int lg_slots, int64_t* __restrict__ ukeys,
                                                           int64_t* __restrict__ nunique) {
  extern __shared__ __align__(16) uint64_t dp_set[];
  __shared__ uint32_t s_warp[kDpWarps];
  __shared__ DpWalk s_walk;
  __shared__ int32_t s_bucket;
  const int32_t b = dp_claim(a, &s_bucket);
  if (b < 0) return;
  const int32_t slots = 1 << lg_slots, W = 1 << a.wb;
  uint32_t* distinct = reinterpret_cast<uint32_t*>(dp_set + slots);
  const int64_t r0 = a.offs[b];
  const int n = (int)(a.offs[b + 1] - r0);
  const uint64_t* __restrict__ rec = a.rec + r0;
  for (int i = threadIdx.x; i < slots / 2; i += kDpThreads)
    reinterpret_cast<ulonglong2*>(dp_set)[i] = make_ulonglong2(kDpEmpty, kDpEmpty);
  for (int i = threadIdx.x; i < W; i += kDpThreads) distinct[i] = 0u;
  __syncthreads();
  // Each lane walks through its own records, one slot an iteration, the next
  // record loaded ahead: lanes with short walks go on while others still probe
  // (a loop per record lasts as long as the longest of 32 walks).
  const uint32_t mask = (uint32_t)slots - 1u;
  auto hash = [](uint64_t r) {
    return (((uint32_t)(r >> 32) * 0x9E3779B1u) ^ ((uint32_t)r * 0x85EBCA77u)) * 0xC2B2AE3Du;
  };
  int i = threadIdx.x;
  uint64_t r = i < n ? __ldg(rec + i) : 0ull, next = i + kDpThreads < n ? __ldg(rec + i + kDpThreads) : 0ull;
  uint32_t f = hash(r), h = f >> (32 - lg_slots);
  while (i < n) {
    uint64_t cur = *reinterpret_cast<volatile uint64_t*>(&dp_set[h]);
    if (cur == kDpEmpty) {
      cur = atomicCAS(reinterpret_cast<unsigned long long*>(&dp_set[h]), (unsigned long long)kDpEmpty,
                      (unsigned long long)r);
      if (cur == kDpEmpty) {
        atomicAdd(&distinct[(uint32_t)r], 1u);
        cur = r;
      }
    }
    // An odd step reaches every slot, and more slots than records stay free.
    h = (h + (f << 1 | 1u)) & mask;
    if (cur == r) {
      i += kDpThreads;
      r = next;
      next = i + kDpThreads < n ? __ldg(rec + i + kDpThreads) : 0ull;
      f = hash(r);
      h = f >> (32 - lg_slots);
    }
  }
  __syncthreads();
  // Present keys in order: warp w owns a run of consecutive ones.
  const int wbk = (int)min((int64_t)W, a.m - ((int64_t)b << a.wb));
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  const int per = ((wbk + kDpWarps - 1) / kDpWarps + 31) & ~31;
  const int g0 = min(wbk, warp * per), g1 = min(wbk, g0 + per);
  uint32_t c = 0;
  for (int g = g0; g < g1; g += 32) c += __popc(__ballot_sync(0xffffffffu, g + lane < g1 && distinct[g + lane] != 0u));
  if (lane == 0) s_warp[warp] = c;
  __syncthreads();
  uint32_t total = 0, mine = 0;
  for (int w = 0; w < kDpWarps; ++w) {
    if (w < warp) mine += s_warp[w];
    total += s_warp[w];
  }
  dp_publish(a, b, total);
  int64_t pos = dp_base(a, b, total, &s_walk) + mine;
  const int64_t key0 = a.kmin + ((int64_t)b << a.wb);
  const unsigned lt = lanemask_lt();
  for (int g = g0; g < g1; g += 32) {
    const uint32_t d = g + lane < g1 ? distinct[g + lane] : 0u;
    const unsigned bal = __ballot_sync(0xffffffffu, d != 0u);
    if (d) {
      ukeys[pos + __popc(bal & lt)] = key0 + g + lane;
      nunique[pos + __popc(bal & lt)] = (int64_t)d;
    }
    pos += __popc(bal);
  }
}

int dp_spread(const nfc_groupby_args* g, const DpRule& rule, cudaStream_t s, Scratch& sc, int32_t* ok) {
  int32_t* d_ok = nullptr;
  NFC_CUDA(sc.alloc(&d_ok, 4));
  const int samples = (int)std::min<int64_t>(kDpSampleThreads * kDpSamplesPerThread, g->n / 256);
  const size_t smem = kDpMaxBuckets * sizeof(uint16_t);
  NFC_CUDA(allow_dynamic_smem<k_dp_sample>());
  k_dp_sample<<<1, kDpSampleThreads, smem, s>>>(g->keys, g->key_validity, g->n, samples, rule, d_ok);
  NFC_CUDA(cudaGetLastError());
  NFC_CUDA(readback(ok, d_ok, sizeof(*ok), s));
  return NFC_OK;
}

// Sample, probe, partition and bucket descriptors, shared by both calls.
int dp_prepare(const nfc_groupby_args* g, int32_t dtype, const void* values, const DpRule& rule, cudaStream_t s,
               Scratch& sc, DpArgs* a, int64_t* most, int64_t* nv) {
  int32_t ok = 0;
  {
    Scratch tmp(s);
    const int rc = dp_spread(g, rule, s, tmp, &ok);
    if (rc) return rc;
  }
  if (!ok) return NFC_ERR_UNSUPPORTED;
  StageTimer tm;
  uint32_t* vmask = nullptr;
  nfc_probe p{};
  int rc = run_probe(g, s, sc, &vmask, &p, &tm);
  if (rc) return rc;
  *nv = p.n_valid;
  if (p.n_valid < kDpMinRows) return NFC_ERR_UNSUPPORTED;
  const int64_t m = p.kmax - p.kmin + 1;
  const int wb = rule.width(m, p.n_valid);
  if (wb < 0) return NFC_ERR_UNSUPPORTED;
  int64_t* words = nullptr;  // ng | err | ticket
  NFC_CUDA(sc.alloc(&words, 4));
  NFC_CUDA(cudaMemsetAsync(words, 0, 4 * sizeof(int64_t), s));
  a->ng_out = words;
  a->err = reinterpret_cast<int32_t*>(words + 1);
  a->ticket = reinterpret_cast<uint32_t*>(words + 2);
  PartRecords pr{};
  rc = partition_records(g, dtype, values, p, vmask, wb, rule.max_rows, s, sc, a->err, &pr);
  if (rc) return rc;
  NFC_CUDA(sc.alloc(&a->lb, (size_t)pr.nb));
  NFC_CUDA(cudaMemsetAsync(a->lb, 0, sizeof(uint64_t) * (size_t)pr.nb, s));
  a->rec = pr.rec;
  a->offs = pr.offs;
  a->nb = pr.nb;
  a->wb = wb;
  a->kmin = p.kmin;
  a->m = m;
  *most = pr.most;
  return NFC_OK;
}

int64_t dp_finish(const DpArgs& a, cudaStream_t s) {
  int64_t h[2] = {0, 0};
  NFC_CUDA(readback(h, a.ng_out, sizeof(h), s));
  const int32_t status = (int32_t)h[1];
  if (status) {
    set_last_error("device status %d", status);
    return status;
  }
  return h[0];
}

}  // namespace

// Rows per bucket: up to 6,400, which three CTAs per SM hold at 2^17 keys (200M
// keys of the full range).  Below 1,024 the fixed cost of a bucket (some 8 us of
// a CTA) takes the gain; above 28,672 the first rows and counts of 2^17 keys
// no longer fit one CTA, and a CTA's time would show as a tail.
int64_t unique_by_partition(const int32_t* keys, int64_t n, int32_t* uniq_out, int32_t* first_out,
                            int64_t* counts_out, int32_t* inv_out, cudaStream_t s) {
  if (n < kDpMinRows || !aligned16(keys)) return NFC_ERR_UNSUPPORTED;
  Scratch sc(s);
  nfc_groupby_args g{};
  g.n = n;
  g.keys = keys;
  DpArgs a{};
  int64_t most = 0, nv = 0;
  const int rc = dp_prepare(&g, kRowId, nullptr, DpRule{6400, 1024, 28672, 7, 17}, s, sc, &a, &most, &nv);
  if (rc) return rc;
  most = (std::min<int64_t>(most, 1ll << a.wb) + 3) & ~3ll;
  const size_t smem = ((size_t)1 << a.wb) / 32 * 6 + (size_t)most * 6;
  NFC_CUDA(allow_dynamic_smem<k_dp_unique>());
  k_dp_unique<<<(unsigned)a.nb, kDpThreads, smem, s>>>(a, (int32_t)most, uniq_out, first_out, counts_out, inv_out);
  NFC_CUDA(cudaGetLastError());
  return dp_finish(a, s);
}

// Rows per bucket: up to 6,200, so that the set of the largest bucket has 8,192
// slots (64 KB, three CTAs per SM) and is at most 4/5 full.  16,384 slots leave
// one CTA per SM; that is for inputs of more than 32,768 such buckets.
int64_t count_distinct_by_partition(const int32_t* keys, const uint8_t* key_validity, const int32_t* values,
                                    const uint8_t* value_validity, int64_t n, int64_t out_cap, int64_t* ukeys_out,
                                    int64_t* nunique_out, cudaStream_t s) {
  if (n < kDpMinRows || !aligned16(keys) || !aligned16(values)) return NFC_ERR_UNSUPPORTED;
  Scratch sc(s);
  nfc_value_col col{};
  col.dtype = NFC_I32;
  col.data = values;
  col.validity = value_validity;
  nfc_groupby_args g{};
  g.n = n;
  g.keys = keys;
  g.key_validity = key_validity;
  g.ncols = 1;
  g.cols = &col;
  DpArgs a{};
  int64_t most = 0, nv = 0;
  const int rc = dp_prepare(&g, NFC_I32, values, DpRule{6200, 512, 13000, 0, 13}, s, sc, &a, &most, &nv);
  if (rc) return rc;
  // Outputs that may not hold every key are written once they are known to.
  const int64_t bound = std::min<int64_t>(a.m, nv);
  int64_t *uk = ukeys_out, *nu = nunique_out;
  if (out_cap < bound) {
    NFC_CUDA(sc.alloc(&uk, (size_t)(2 * bound)));
    nu = uk + bound;
  }
  int lg = 10;
  while ((4ll << lg) / 5 < most) ++lg;
  const size_t smem = ((size_t)8 << lg) + ((size_t)4 << a.wb);
  NFC_CUDA(allow_dynamic_smem<k_dp_count>());
  k_dp_count<<<(unsigned)a.nb, kDpThreads, smem, s>>>(a, lg, uk, nu);
  NFC_CUDA(cudaGetLastError());
  const int64_t ng = dp_finish(a, s);
  if (ng <= 0 || out_cap >= bound) return ng;
  if (ng > out_cap) {
    set_last_error("group_count_distinct: %lld groups > out_cap %lld", (long long)ng, (long long)out_cap);
    return NFC_ERR_RANGE;
  }
  NFC_CUDA(cudaMemcpyAsync(ukeys_out, uk, sizeof(int64_t) * ng, cudaMemcpyDeviceToDevice, s));
  NFC_CUDA(cudaMemcpyAsync(nunique_out, nu, sizeof(int64_t) * ng, cudaMemcpyDeviceToDevice, s));
  NFC_CUDA(cudaStreamSynchronize(s));
  return ng;
}

}  // namespace nfc

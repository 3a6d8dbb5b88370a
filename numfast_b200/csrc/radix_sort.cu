// Stable LSD radix sort of u32 / u64 keys with an optional u32 payload.
//
// One reduction over the keys finds the bits in which they differ; passes of
// up to 8 bits cover just those.  A pass is three kernels:
//   k_rs_count    digit counts of every tile and of every group of 16 tiles
//   k_rs_scan     exclusive prefix of each digit's counts over the groups
//   k_rs_scatter  one CTA per tile: rank, stage in digit order, write out
// so no CTA waits for another one, and tiles that run at the same time write
// next to each other: the 2 x 256 places where the output grows are shared by
// all of them and their lines fill up in L2.  (With chunks of consecutive
// tiles per CTA every CTA grows its own 512 places; half-written lines then
// leave L2 and come back: 200M u32 pairs in chunks of four tiles, 2.9 GB read
// instead of 1.6 and 1.60 ms a scatter instead of 1.10 at the same tile.)
#include <algorithm>

#include "groupby_host.h"

namespace nfc {

constexpr int kRsDigits = 256;
constexpr int kRsCountThreads = 512;
constexpr int kRsCopies = 8;  // digit counters per bin in k_rs_count

// ---------------------------------------------------------------- differing bits
// OR over all keys of (key ^ keys[0]).
template <class K>
__global__ void __launch_bounds__(256) k_rs_vary(const K* __restrict__ keys, int64_t n, unsigned long long* out) {
  constexpr int VEC = 16 / sizeof(K);
  constexpr int U = 4;
  const K k0 = keys[0];
  K acc = 0;
  int64_t done = 0;
  const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  if ((reinterpret_cast<uintptr_t>(keys) & 15u) == 0) {
    const int64_t nvec = n / VEC;
    for (int64_t v0 = t0; v0 < nvec; v0 += stride * U) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t v = v0 + u * stride;
        if (v < nvec) {
          if constexpr (sizeof(K) == 4) {
            const uint4 q = __ldcs(reinterpret_cast<const uint4*>(keys) + v);
            acc |= (q.x ^ k0) | (q.y ^ k0) | (q.z ^ k0) | (q.w ^ k0);
          } else {
            const ulonglong2 q = __ldcs(reinterpret_cast<const ulonglong2*>(keys) + v);
            acc |= (q.x ^ k0) | (q.y ^ k0);
          }
        }
      }
    }
    done = nvec * VEC;
  }
  for (int64_t i = done + t0; i < n; i += stride) acc |= keys[i] ^ k0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc |= __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane_id() == 0 && acc) atomicOr(out, (unsigned long long)acc);
}

// ---------------------------------------------------------------- geometry
constexpr int kRsThreads = 256;
constexpr int kRsWarps = kRsThreads / 32;
template <class K>
struct RsTile {
  static constexpr int items = 16;  // keys per thread
  static constexpr int rows = kRsThreads * items;
  static constexpr int ctas = sizeof(K) == 4 ? 4 : 3;  // per SM: the most that run without spills
};
constexpr uint32_t kRsGroup = 16;        // tiles per group, where there are enough tiles for every SM
constexpr uint32_t kRsDirectTiles = 32;  // up to here the scatter adds up the tile counts itself

// ---------------------------------------------------------------- counts
// tcount[t * 256 + d] = keys of tile t with digit d; gcount[d * ngroups + g] =
// the same per group.  Each bin has eight counters picked by lane, so equal
// digits in a warp meet at most four at a time.
template <class K>
__global__ void __launch_bounds__(kRsCountThreads) k_rs_count(const K* __restrict__ keys, int64_t n, int shift,
                                                              uint32_t dmask, K xr, bool aligned,
                                                              uint32_t gtiles, uint16_t* __restrict__ tcount,
                                                              uint32_t* __restrict__ gcount, uint32_t ngroups) {
  constexpr int kTile = RsTile<K>::rows;
  constexpr int VEC = 16 / sizeof(K);
  constexpr int U = kTile / (VEC * kRsCountThreads);
  static_assert(U * VEC * kRsCountThreads == kTile, "whole vectors per thread");
  __shared__ __align__(16) uint32_t h[kRsDigits * kRsCopies];
  for (int i = threadIdx.x; i < kRsDigits * kRsCopies; i += kRsCountThreads) h[i] = 0u;
  const uint32_t copy = threadIdx.x & (kRsCopies - 1);
  auto add = [&](K k) { atomicAdd(&h[(((uint32_t)((k ^ xr) >> shift) & dmask) * kRsCopies) + copy], 1u); };
  const int64_t t0 = (int64_t)blockIdx.x * gtiles;
  const int64_t t1 = min((n + kTile - 1) / kTile, t0 + gtiles);
  uint32_t sum = 0;
  uint4 q[U];
  auto full = [&](int64_t t) { return aligned && (t + 1) * kTile <= n; };
  auto load = [&](int64_t t) {
#pragma unroll
    for (int u = 0; u < U; ++u)
      q[u] = __ldg(reinterpret_cast<const uint4*>(keys + t * kTile) + u * kRsCountThreads + threadIdx.x);
  };
  if (full(t0)) load(t0);
  __syncthreads();
  for (int64_t t = t0; t < t1; ++t) {
    if (full(t)) {
      uint4 c[U];
#pragma unroll
      for (int u = 0; u < U; ++u) c[u] = q[u];
      if (t + 1 < t1 && full(t + 1)) load(t + 1);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if constexpr (sizeof(K) == 4) {
          add(c[u].x); add(c[u].y); add(c[u].z); add(c[u].w);
        } else {
          add((uint64_t)c[u].x | ((uint64_t)c[u].y << 32));
          add((uint64_t)c[u].z | ((uint64_t)c[u].w << 32));
        }
      }
    } else {
      const int64_t b = min(n, (t + 1) * kTile);
      for (int64_t i = t * kTile + threadIdx.x; i < b; i += kRsCountThreads) add(keys[i]);
    }
    __syncthreads();
    if (threadIdx.x < kRsDigits) {
      uint32_t s = 0;
#pragma unroll
      for (int c = 0; c < kRsCopies; c += 4) {
        uint4* p = reinterpret_cast<uint4*>(&h[threadIdx.x * kRsCopies + c]);
        const uint4 v = *p;
        s += v.x + v.y + v.z + v.w;
        *p = make_uint4(0, 0, 0, 0);
      }
      tcount[t * kRsDigits + threadIdx.x] = (uint16_t)s;
      sum += s;
    }
    __syncthreads();
  }
  if (ngroups && threadIdx.x < kRsDigits) gcount[(size_t)threadIdx.x * ngroups + blockIdx.x] = sum;
}

// Block d: counts of digit d over the groups -> exclusive prefix; totals[d].
__global__ void __launch_bounds__(256) k_rs_scan(uint32_t* __restrict__ gcount, uint32_t ngroups,
                                                 uint32_t* __restrict__ totals) {
  __shared__ uint32_t s_scan[33];
  uint32_t* row = gcount + (size_t)blockIdx.x * ngroups;
  uint32_t carry = 0;
  for (uint32_t c0 = 0; c0 < ngroups; c0 += 1024) {
    uint32_t v[4], t = 0;
    const uint32_t i0 = c0 + threadIdx.x * 4;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      v[e] = i0 + e < ngroups ? row[i0 + e] : 0u;
      t += v[e];
    }
    uint32_t total;
    uint32_t x = carry + block_excl_scan(t, s_scan, &total);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (i0 + e < ngroups) row[i0 + e] = x;
      x += v[e];
    }
    carry += total;
  }
  if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// ---------------------------------------------------------------- scatter
// CTAs of 256 threads, one thread per digit.  The work is spread over the ALU
// (votes and masks of the ranking), shared memory (staging) and DRAM, none of
// them full; several small CTAs per SM let one rank while others load, stage
// or write.  A scatter of 200M u32 pairs takes 0.97 ms (3.2 GB, 3.3 TB/s), of
// 28.5M u64 pairs 0.182 ms, of 50M u64 keys 0.216 ms; with the counts a pass is
// 1.15, 0.235 and 0.29 ms, against 1.60, 0.29 and 0.42 ms for one look-back
// kernel with two 512-thread CTAs per SM.  24 keys per thread: 2-10% slower.
template <class K, bool HAS_VALS>
struct RsSmem {
  K keys[RsTile<K>::rows];
  uint32_t vals[HAS_VALS ? RsTile<K>::rows : 4];
  uint16_t wh[kRsWarps][kRsDigits];  // per warp: digit counts, then first places in the tile
  uint32_t gofs[kRsDigits];          // output place of a staged element minus its place in the tile
  uint32_t wt[2][kRsWarps];
};

// Lanes whose digit equals this lane's: a vote per digit bit, as GPU radix sorts
// commonly rank (CUB's among them), and the lanes whose bit is not this lane's
// collected with one three-input operation on the vote and this lane's bit as a
// mask.  A fixed cost for any digits, where __match_any_sync goes through the
// distinct values (200M u32 pairs sorted in 6.9 against 5.6 ms).  In PTX because
// the compiler's own choice for the same steps takes 2-4% longer sorts.
NFC_DEV unsigned match_digit8(uint32_t d) {
  uint32_t differ = 0u;
#pragma unroll
  for (int b = 0; b < 8; ++b)
    asm volatile(
        "{\n"
        " .reg .pred set;\n"
        " .reg .b32 mine, all;\n"
        " and.b32 mine, %1, %2;\n"
        " setp.ne.u32 set, mine, 0;\n"
        " selp.b32 mine, 0xffffffff, 0, set;\n"
        " vote.sync.ballot.b32 all, set, 0xffffffff;\n"
        " lop3.b32 %0, %0, all, mine, 0xF6;\n"
        "}"
        : "+r"(differ)
        : "r"(d), "r"(1u << b));
  return ~differ;
}

// 4 bytes from global straight to shared memory, no register held meanwhile.
NFC_DEV void cp_async4(uint32_t* dst, const uint32_t* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}

// Keys are read as kin[i] ^ xr and written flipped; IOTA: the payload is the
// input index.  Elements past n carry the largest digit and, being last in
// order, the last places of the tile, which are not written out.
template <class K, bool HAS_VALS, bool IOTA>
__global__ void __launch_bounds__(kRsThreads, RsTile<K>::ctas)
    k_rs_scatter(const K* __restrict__ kin, K* __restrict__ kout, const uint32_t* __restrict__ vin,
                 uint32_t* __restrict__ vout, int64_t n, int shift, uint32_t dmask, K xr,
                 const uint16_t* __restrict__ tcount, const uint32_t* __restrict__ prefix,
                 const uint32_t* __restrict__ totals, uint32_t gtiles, uint32_t ngroups) {
  constexpr int kItems = RsTile<K>::items;
  constexpr int kTile = RsTile<K>::rows;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RsSmem<K, HAS_VALS>& S = *reinterpret_cast<RsSmem<K, HAS_VALS>*>(smem_raw);
  const int tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
  const uint32_t tile = blockIdx.x;
  const int64_t t0 = (int64_t)tile * kTile;
  const int tile_n = n - t0 < kTile ? (int)(n - t0) : kTile;
  const int wofs = warp * (32 * kItems) + lane;
  constexpr K kPad = ~(K)0;

  K key[kItems];
  {
    const K* p = kin + t0 + wofs;
    if (tile_n == kTile) {
#pragma unroll
      for (int j = 0; j < kItems; ++j) key[j] = __ldcs(p + j * 32) ^ xr;
    } else {
#pragma unroll
      for (int j = 0; j < kItems; ++j) key[j] = wofs + j * 32 < tile_n ? (K)(__ldcs(p + j * 32) ^ xr) : kPad;
    }
  }
  // First output place of this thread's digit: the digits before it, the
  // groups before this one, the tiles of the group before this one.
  uint32_t first = 0, dtotal = 0;
  uint32_t tg = 0;
  if (ngroups) {
    const uint32_t group = tile / gtiles;
    tg = group * gtiles;
    first = __ldg(prefix + (size_t)tid * ngroups + group);
    dtotal = __ldg(totals + tid);
  }
#pragma unroll 4
  for (uint32_t t = tg; t < tile; ++t) first += __ldg(tcount + (size_t)t * kRsDigits + tid);
  if (!ngroups) {
    dtotal = first;
#pragma unroll 4
    for (uint32_t t = tile; t < gridDim.x; ++t) dtotal += __ldg(tcount + (size_t)t * kRsDigits + tid);
  }
  // Inclusive warp scan of `t`; the warps' totals go to S.wt[slot].
  auto warp_scan = [&](uint32_t t, int slot) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    if (lane == 31) S.wt[slot][warp] = t;
    return t;
  };
  auto warps_before = [&](int slot) {
    uint32_t x = 0;
    for (int w = 0; w < warp; ++w) x += S.wt[slot][w];
    return x;
  };
  first += warp_scan(dtotal, 0) - dtotal;
  // Each warp clears and counts in its own row; nobody else reads it before
  // the first barrier.
  reinterpret_cast<uint4*>(&S.wh[warp][0])[lane] = make_uint4(0, 0, 0, 0);
  __syncwarp();
  // Rank of each key among its warp's earlier keys of the same digit.
  uint32_t rank[kItems / 2];
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    const uint32_t dg = (uint32_t)(key[j] >> shift) & dmask;
    const unsigned peers = match_digit8(dg);
    const unsigned before = peers & lanemask_lt();
    uint32_t c = S.wh[warp][dg];
    __syncwarp();
    if (before == 0u) S.wh[warp][dg] = (uint16_t)(c + __popc(peers));
    __syncwarp();
    c += __popc(before);
    if (j & 1) rank[j / 2] |= c << 16;
    else rank[j / 2] = c;
  }
  __syncthreads();
  // Digit counts of the warps -> first place of each (warp, digit) in the tile.
  {
    uint32_t c[kRsWarps], sum = 0;
#pragma unroll
    for (int w = 0; w < kRsWarps; ++w) {
      c[w] = S.wh[w][tid];
      sum += c[w];
    }
    uint32_t p = warp_scan(sum, 1) - sum;
    __syncthreads();
    p += warps_before(1);
    S.gofs[tid] = first + warps_before(0) - p;
#pragma unroll
    for (int w = 0; w < kRsWarps; ++w) {
      S.wh[w][tid] = (uint16_t)p;
      p += c[w];
    }
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    const uint32_t dg = (uint32_t)(key[j] >> shift) & dmask;
    const uint32_t p = S.wh[warp][dg] + ((rank[j / 2] >> (16 * (j & 1))) & 0xFFFFu);
    S.keys[p] = key[j];
    if (HAS_VALS) {
      if (IOTA) S.vals[p] = (uint32_t)(t0 + wofs + j * 32);
      else if (wofs + j * 32 < tile_n) cp_async4(&S.vals[p], vin + t0 + wofs + j * 32);
    }
  }
  if (HAS_VALS && !IOTA) asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  auto put = [&](int i) {
    const K k = S.keys[i];
    const uint32_t dst = S.gofs[(uint32_t)(k >> shift) & dmask] + (uint32_t)i;
    kout[dst] = k;
    if (HAS_VALS) vout[dst] = S.vals[i];
  };
  if (tile_n == kTile) {
#pragma unroll 4
    for (int j = 0; j < kItems; ++j) put(j * kRsThreads + tid);
  } else {
    for (int i = tid; i < tile_n; i += kRsThreads) put(i);
  }
}

// Inputs of at most kSmallSort keys (the distinct keys of a low-cardinality
// hash group-by, small argsorts) are sorted by one CTA: a bitonic network in
// shared memory over (masked key, input index) pairs, which makes it stable,
// then a gather of the full keys and values.  One launch and no host round
// trip, where the multi-pass sort costs a histogram read-back and up to
// eight more launches.
constexpr int kSmallSort = 2048;

template <class K>
__global__ void __launch_bounds__(1024) k_sort_small(const K* __restrict__ kin, const uint32_t* __restrict__ vin,
                                                     bool iota, int n, K mask, K xr, K* __restrict__ kout,
                                                     uint32_t* __restrict__ vout) {
  __shared__ K sk[kSmallSort];
  __shared__ uint32_t si[kSmallSort];
  int m = 1;
  while (m < n) m <<= 1;
  // Padding (index >= n) holds the largest key and sorts after every real key.
  for (int i = threadIdx.x; i < m; i += blockDim.x) {
    sk[i] = i < n ? ((kin[i] ^ xr) & mask) : ~(K)0;
    si[i] = (uint32_t)i;
  }
  __syncthreads();
  for (int size = 2; size <= m; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int t = threadIdx.x; t < (m >> 1); t += blockDim.x) {
        const int lo = 2 * t - (t & (stride - 1));  // pair (lo, lo + stride), bit 'stride' of lo clear
        const int hi = lo + stride;
        const K a = sk[lo], b = sk[hi];
        const uint32_t ia = si[lo], ib = si[hi];
        const bool gt = a > b || (a == b && ia > ib);
        if (gt == ((lo & size) == 0)) {  // ascending where bit 'size' of lo is clear
          sk[lo] = b;
          sk[hi] = a;
          si[lo] = ib;
          si[hi] = ia;
        }
      }
      __syncthreads();
    }
  }
  for (int r = threadIdx.x; r < n; r += blockDim.x) {
    const uint32_t i = si[r];
    kout[r] = kin[i] ^ xr;
    if (vout) vout[r] = iota ? i : vin[i];
  }
}

template <class K>
__global__ void k_xor_copy(const K* __restrict__ in, K xr, int64_t n, K* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = in[i] ^ xr;
}

__global__ void k_iota(uint32_t* v, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    v[i] = (uint32_t)i;
}

// Scratch of one sort: counts per tile and group, digit totals.
struct RsCounts {
  uint16_t* tcount;
  uint32_t* gcount;
  uint32_t* totals;
  uint32_t ntiles, gtiles, ngroups;  // ngroups 0: tile counts only
};

template <class K, bool HAS_VALS, bool IOTA>
static int launch_scatter(const K* kin, K* kout, const uint32_t* vin, uint32_t* vout, int64_t n, int shift,
                          uint32_t dmask, K xr, const RsCounts& rc, cudaStream_t s) {
  constexpr size_t smem = sizeof(RsSmem<K, HAS_VALS>);
  NFC_CUDA(allow_dynamic_smem<k_rs_scatter<K, HAS_VALS, IOTA>>());
  k_rs_scatter<K, HAS_VALS, IOTA><<<rc.ntiles, kRsThreads, smem, s>>>(kin, kout, vin, vout, n, shift, dmask, xr,
                                                                     rc.tcount, rc.gcount, rc.totals, rc.gtiles,
                                                                     rc.ngroups);
  NFC_CUDA(cudaGetLastError());
  return NFC_OK;
}

// src (when not null) is a read-only key column that the first pass reads as
// src[i] ^ in_xor; keys / keys_alt are then only the ping-pong buffers, and
// the result never aliases src.
template <class K>
static int radix_sort_impl(K* keys, K* keys_alt, uint32_t* vals, uint32_t* vals_alt, int64_t n, int key_bits,
                           bool iota_vals, cudaStream_t s, Scratch& sc, K** keys_result, uint32_t** vals_result,
                           const K* src = nullptr, K in_xor = 0) {
  if (!src) {
    src = keys;
    in_xor = 0;
  }
  *keys_result = keys;
  *vals_result = vals;
  if (n <= 0) return NFC_OK;
  const bool has_vals = vals != nullptr;
  const K mask = key_bits >= (int)(8 * sizeof(K)) ? ~(K)0 : (K)(((K)1 << key_bits) - 1);
  if (n <= kSmallSort) {
    k_sort_small<K><<<1, 1024, 0, s>>>(src, vals, iota_vals, (int)n, mask, in_xor, keys_alt,
                                       has_vals ? vals_alt : nullptr);
    NFC_CUDA(cudaGetLastError());
    *keys_result = keys_alt;
    if (has_vals) *vals_result = vals_alt;
    return NFC_OK;
  }
  if (n >= (1ll << 30)) {
    set_last_error("radix sort: n=%lld >= 2^30", (long long)n);
    return NFC_ERR_UNSUPPORTED;
  }
  constexpr int64_t kTile = RsTile<K>::rows;
  RsCounts rc;
  rc.ntiles = (uint32_t)((n + kTile - 1) / kTile);
  // Few tiles: one per count CTA, and no scan at all where a scatter thread
  // can add up its digit over the tiles (50,000 u64 pairs: 20 -> 14 us a pass).
  rc.gtiles = rc.ntiles >= kRsGroup * (uint32_t)num_sms() ? kRsGroup : 1u;
  rc.ngroups = rc.ntiles <= kRsDirectTiles ? 0u : (rc.ntiles + rc.gtiles - 1) / rc.gtiles;
  unsigned long long* d_vary = nullptr;
  NFC_CUDA(sc.alloc(&d_vary, 1 + kRsDigits / 2 + (size_t)rc.ngroups * (kRsDigits / 2) +
                                 (size_t)rc.ntiles * (kRsDigits / 4)));
  rc.totals = reinterpret_cast<uint32_t*>(d_vary + 1);
  rc.gcount = rc.totals + kRsDigits;
  rc.tcount = reinterpret_cast<uint16_t*>(rc.gcount + (size_t)rc.ngroups * kRsDigits);
  NFC_CUDA(cudaMemsetAsync(d_vary, 0, sizeof(unsigned long long), s));
  k_rs_vary<K><<<(unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 8191) / 8192, (int64_t)num_sms() * 8)), 256, 0,
                 s>>>(src, n, d_vary);
  NFC_CUDA(cudaGetLastError());
  unsigned long long vary = 0;
  NFC_CUDA(readback(&vary, d_vary, sizeof(vary), s));
  vary &= (unsigned long long)mask;
  const K* kin = src;
  K* kout = src == keys ? keys_alt : keys;
  K xr = in_xor;
  uint32_t* vin = vals;
  uint32_t* vout = vals_alt;
  bool need_iota = has_vals && iota_vals;
  while (vary) {
    // The next pass covers eight bits from the lowest differing bit left.
    const int shift = __builtin_ctzll(vary);
    const uint32_t dmask = (uint32_t)(mask >> shift) & (kRsDigits - 1);
    vary &= shift + 8 >= 64 ? 0ull : ~0ull << (shift + 8);
    k_rs_count<K><<<(rc.ntiles + rc.gtiles - 1) / rc.gtiles, kRsCountThreads, 0, s>>>(
        kin, n, shift, dmask, xr, (reinterpret_cast<uintptr_t>(kin) & 15u) == 0, rc.gtiles, rc.tcount, rc.gcount,
        rc.ngroups);
    NFC_CUDA(cudaGetLastError());
    if (rc.ngroups) {
      k_rs_scan<<<kRsDigits, 256, 0, s>>>(rc.gcount, rc.ngroups, rc.totals);
      NFC_CUDA(cudaGetLastError());
    }
    int st;
    if (!has_vals)
      st = launch_scatter<K, false, false>(kin, kout, nullptr, nullptr, n, shift, dmask, xr, rc, s);
    else if (need_iota)
      st = launch_scatter<K, true, true>(kin, kout, nullptr, vout, n, shift, dmask, xr, rc, s);
    else
      st = launch_scatter<K, true, false>(kin, kout, vin, vout, n, shift, dmask, xr, rc, s);
    if (st) return st;
    need_iota = false;
    xr = 0;
    K* written = kout;
    kout = written == keys ? keys_alt : keys;
    kin = written;
    std::swap(vin, vout);
  }
  const unsigned g1 = (unsigned)std::min<int64_t>((n + 255) / 256, (int64_t)num_sms() * 8);
  if (kin == src && src != keys) {
    // No differing bits: the result is the source itself, flipped into the first buffer.
    k_xor_copy<K><<<g1, 256, 0, s>>>(src, in_xor, n, keys);
    NFC_CUDA(cudaGetLastError());
    kin = keys;
  }
  if (need_iota) {
    // No differing bits: the input order is already sorted.
    k_iota<<<g1, 256, 0, s>>>(vin, n);
    NFC_CUDA(cudaGetLastError());
  }
  *keys_result = const_cast<K*>(kin);
  *vals_result = vin;
  return NFC_OK;
}

int radix_sort_u32(uint32_t* keys, uint32_t* keys_alt, uint32_t* vals, uint32_t* vals_alt, int64_t n, int key_bits,
                   bool iota_vals, cudaStream_t s, Scratch& sc, uint32_t** kr, uint32_t** vr) {
  return radix_sort_impl<uint32_t>(keys, keys_alt, vals, vals_alt, n, key_bits, iota_vals, s, sc, kr, vr);
}
int radix_sort_u32_from(const uint32_t* src, uint32_t in_xor, uint32_t* keys, uint32_t* keys_alt, uint32_t* vals,
                        uint32_t* vals_alt, int64_t n, int key_bits, bool iota_vals, cudaStream_t s, Scratch& sc,
                        uint32_t** kr, uint32_t** vr) {
  return radix_sort_impl<uint32_t>(keys, keys_alt, vals, vals_alt, n, key_bits, iota_vals, s, sc, kr, vr, src, in_xor);
}
int radix_sort_u64(uint64_t* keys, uint64_t* keys_alt, uint32_t* vals, uint32_t* vals_alt, int64_t n, int key_bits,
                   bool iota_vals, cudaStream_t s, Scratch& sc, uint64_t** kr, uint32_t** vr) {
  return radix_sort_impl<uint64_t>(keys, keys_alt, vals, vals_alt, n, key_bits, iota_vals, s, sc, kr, vr);
}

}  // namespace nfc

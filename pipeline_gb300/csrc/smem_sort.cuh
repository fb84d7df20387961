// Shared-memory sorting of one CTA's keys: the one-launch build and sort, the
// bucket sort of batched builds (bins), the bucket kernels of the learned sort and
// the digit passes of the one-launch sort (radix).
#pragma once

#include "common.cuh"

namespace octgb {

constexpr int kRsBits = 8;  // radix-sort digit width
constexpr int kRsBins = 1 << kRsBits;

template <int WARPS>
struct RadixSmem {
  uint16_t whist[WARPS][kRsBins];  // per-warp digit counts, then offsets
  uint32_t dstart[kRsBins];        // first position of each digit
  uint32_t warp_tot[32];
  uint32_t total;
};

// One digit pass of a[0, cnt) to b (cnt <= WARPS * 32 * ITEMS, WARPS * 32
// threads): digit (key - kmin) >> shift & mask, mask <= 255. Warp w ranks its
// contiguous ITEMS * 32 keys at most. STABLE: by ballot multi-split (peers =
// lanes with the same digit), so ties keep input order. S.dstart is left at
// the digits' first positions. Ends with a barrier.
template <int WARPS, int ITEMS, bool STABLE>
__device__ __forceinline__ void smem_radix_pass(const uint32_t* a, uint32_t* b, int cnt,
                                                uint32_t kmin, int shift, uint32_t mask,
                                                RadixSmem<WARPS>& S) {
  constexpr int kThreads = WARPS * 32;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const uint32_t lt = lanemask_lt();
  // every warp takes `items` rows of 32 keys (the last warps may be partial)
  const int items = (cnt + WARPS * 32 - 1) / (WARPS * 32);
  const int seg = items * 32;
  for (int k = tid; k < WARPS * kRsBins / 2; k += kThreads)
    reinterpret_cast<uint32_t*>(S.whist)[k] = 0;
  __syncthreads();
  uint32_t rk[ITEMS / 2];  // two 16-bit ranks per register; keys are re-read
  uint16_t* wh = S.whist[wid];
  if (!STABLE) {
    // A shared-memory atomic on the warp's 16-bit digit counter (the upper or
    // lower half of its 32-bit word; a warp counts at most ITEMS * 32 keys, so
    // no carry reaches the other half) ranks a key.
    uint32_t* wh32 = reinterpret_cast<uint32_t*>(wh);
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
      if (it >= items) break;
      const int idx = wid * seg + it * 32 + lane;
      uint32_t r = 0;
      if (idx < cnt) {
        const uint32_t dg = ((a[idx] - kmin) >> shift) & mask;
        const uint32_t sh = 16u * (dg & 1u);
        r = (atomicAdd(&wh32[dg >> 1], 1u << sh) >> sh) & 0xffffu;
      }
      if (it & 1) rk[it >> 1] |= r << 16;
      else rk[it >> 1] = r;
    }
  } else {
    // peers from two 4-bit half-digit equality tables (lane v: lanes whose half
    // equals v), fetched by shuffle
    constexpr int kHalf = kRsBits / 2;
    uint32_t lane_bits[kHalf];
#pragma unroll
    for (int b = 0; b < kHalf; ++b) lane_bits[b] = 0u - ((uint32_t)(lane >> b) & 1u);
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
      if (it >= items) break;
      const int idx = wid * seg + it * 32 + lane;
      const bool valid = idx < cnt;
      const uint32_t key = valid ? a[idx] : 0u;
      const uint32_t dg = ((key - kmin) >> shift) & mask;
      uint32_t eq_lo = 0xffffffffu, eq_hi = 0xffffffffu;
#pragma unroll
      for (int bit = 0; bit < kHalf; ++bit) {
        eq_lo &= ~(__ballot_sync(0xffffffffu, (dg >> bit) & 1u) ^ lane_bits[bit]);
        eq_hi &= ~(__ballot_sync(0xffffffffu, (dg >> (kHalf + bit)) & 1u) ^ lane_bits[bit]);
      }
      const uint32_t peers = __ballot_sync(0xffffffffu, valid) &
                             __shfl_sync(0xffffffffu, eq_lo, (int)(dg & ((1u << kHalf) - 1u))) &
                             __shfl_sync(0xffffffffu, eq_hi, (int)(dg >> kHalf));
      const uint32_t before = valid ? wh[dg] : 0u;
      const uint32_t r = before + __popc(peers & lt);
      if (it & 1) rk[it >> 1] |= r << 16;
      else rk[it >> 1] = r;
      __syncwarp();
      if (valid && (peers & lt) == 0) wh[dg] = (uint16_t)(before + __popc(peers));
      __syncwarp();
    }
  }
  __syncthreads();
  // per digit: exclusive offsets over warps, then digit starts over digits
  uint32_t tot = 0;
  if (tid < kRsBins) {
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const uint32_t c = S.whist[w][tid];
      S.whist[w][tid] = (uint16_t)tot;
      tot += c;
    }
  }
  const uint32_t start = block_exclusive_sum<kThreads>(tid < kRsBins ? tot : 0u, S.warp_tot,
                                                       &S.total);
  if (tid < kRsBins) S.dstart[tid] = start;
  __syncthreads();
#pragma unroll
  for (int it = 0; it < ITEMS; ++it) {
    if (it >= items) break;
    const int idx = wid * seg + it * 32 + lane;
    if (idx < cnt) {
      const uint32_t key = a[idx];
      const uint32_t dg = ((key - kmin) >> shift) & mask;
      const uint32_t r = (rk[it >> 1] >> ((it & 1) * 16)) & 0xffffu;
      b[S.dstart[dg] + S.whist[wid][dg] + r] = key;
    }
  }
  __syncthreads();
}

// LSD radix sort of a[0, cnt) on the low `bits` bits of key - kmin, ping-pong
// between a and b. Returns the sorted array.
template <int WARPS, int ITEMS>
__device__ uint32_t* smem_radix_sort(uint32_t* a, uint32_t* b, int cnt, uint32_t kmin, int bits,
                                     RadixSmem<WARPS>& S) {
  for (int shift = 0; shift < bits; shift += kRsBits) {
    // the first pass needs no stability (the keys arrive in any order)
    if (shift == 0)
      smem_radix_pass<WARPS, ITEMS, false>(a, b, cnt, kmin, shift, kRsBins - 1, S);
    else
      smem_radix_pass<WARPS, ITEMS, true>(a, b, cnt, kmin, shift, kRsBins - 1, S);
    uint32_t* t = a;
    a = b;
    b = t;
  }
  return a;
}

// First i in [lo, hi) with start[i] >= x, or hi.
__device__ __forceinline__ int first_at_least(const uint32_t* start, int lo, int hi, uint32_t x) {
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (start[mid] < x) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

constexpr uint32_t kBinNet = 8;     // keys in a bin up to which the networks of 16 place them
constexpr uint32_t kBinCut = 32;    // keys in a bin up to which the bins stay as they are
constexpr int kBinFewItems = 2;        // keys per thread that compare within their bins
constexpr uint32_t kBinCompare = 128;  // of at most as many keys
constexpr uint32_t kBinWarp = 512;  // keys in a bin that a warp sorts
constexpr uint32_t kBinList = 2048;    // larger bins' list, words
constexpr uint32_t kBinValues = 2048;  // values counted
constexpr uint32_t kBinAux = kBinList + kBinValues + 1;  // words of smem_bin_sort's scratch
constexpr int kBinPad = 16;         // words behind smem_bin_sort's b

// Word j of the binned keys lives at bin_swz(j): threads that read 16
// consecutive words each as four 16-byte loads then meet all banks.
__device__ __forceinline__ uint32_t bin_swz(uint32_t j) { return j ^ (((j >> 5) & 3u) << 2); }

// Sixteen keys in registers sorted by Batcher's odd-even merge exchange
// (Knuth, The Art of Computer Programming 3, 5.2.2, algorithm M): 63 exchanges.
__device__ __forceinline__ void sort16(uint32_t (&v)[16]) {
#pragma unroll
  for (int p = 8; p > 0; p >>= 1) {
    int q = 8, r = 0, d = p;
#pragma unroll
    for (int round = 0; round < 4; ++round) {
#pragma unroll
      for (int i = 0; i < 16 - d; ++i)
        if ((i & p) == r) {
          const uint32_t lo = min(v[i], v[i + d]);
          v[i + d] = max(v[i], v[i + d]);
          v[i] = lo;
        }
      if (q == p) break;
      d = q - p;
      q >>= 1;
      r = p;
    }
  }
}

// Words [s, s + m) of the binned keys (m <= 32 * K) sorted by the calling warp:
// bitonic, word k * 32 + lane in register k.
template <int K>
__device__ __forceinline__ void warp_sort_bin(uint32_t* b, uint32_t s, uint32_t m) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t v[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const uint32_t j = (uint32_t)k * 32u + lane;
    v[k] = j < m ? b[bin_swz(s + j)] : 0xffffffffu;
  }
  bool same = true;  // one value: nothing to do
  const uint32_t first = __shfl_sync(0xffffffffu, v[0], 0);
#pragma unroll
  for (int k = 0; k < K; ++k) same &= (uint32_t)k * 32u + lane >= m || v[k] == first;
  if (__all_sync(0xffffffffu, same)) return;
#pragma unroll
  for (int size = 2; size <= 32 * K; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (stride >= 32) {
          const int o = k | (stride >> 5);
          if (o != k) {
            const bool up = ((k << 5) & size) == 0;
            const uint32_t lo = min(v[k], v[o]), hi = max(v[k], v[o]);
            v[k] = up ? lo : hi;
            v[o] = up ? hi : lo;
          }
        } else {
          const uint32_t y = __shfl_xor_sync(0xffffffffu, v[k], stride);
          const bool up = ((((uint32_t)k << 5) | lane) & (uint32_t)size) == 0u;
          const bool lower = (lane & (uint32_t)stride) == 0u;
          v[k] = up == lower ? min(v[k], y) : max(v[k], y);
        }
      }
    }
  }
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const uint32_t j = (uint32_t)k * 32u + lane;
    if (j < m) b[bin_swz(s + j)] = v[k];
  }
}

// a[0, rows * WARPS * 32) to its exclusive prefix sums (WARPS * 32 threads): a
// warp takes `rows` rows of 32 words, so no two lanes meet a bank. Ends with a
// barrier.
template <int WARPS>
__device__ __forceinline__ void smem_exclusive_rows(uint32_t* a, int rows, uint32_t* warp_tot,
                                                    uint32_t* total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t* row = a + wid * rows * 32 + lane;
  uint32_t sum = 0;
  for (int k = 0; k < rows; ++k) sum += row[k * 32];
  sum = __reduce_add_sync(0xffffffffu, sum);
  uint32_t run = block_exclusive_sum<WARPS * 32>(lane == 0 ? sum : 0u, warp_tot, total);
  run = __shfl_sync(0xffffffffu, run, 0);
#pragma unroll 4
  for (int k = 0; k < rows; ++k) {
    const uint32_t c = row[k * 32];
    uint32_t inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    row[k * 32] = run + inc - c;
    run += __shfl_sync(0xffffffffu, inc, 31);
  }
  __syncthreads();
}

// bins[v] counted by the calling (whole) warp; v 0xffffffff: none. The lanes that
// agree with the first count together, so one frequent value costs a warp one
// atomic.
__device__ __forceinline__ void warp_count(uint32_t* bins, uint32_t v) {
  const uint32_t lane = threadIdx.x & 31u, v0 = __shfl_sync(0xffffffffu, v, 0);
  const uint32_t same = __ballot_sync(0xffffffffu, v == v0);
  if (v != 0xffffffffu && (lane == 0u || v != v0)) atomicAdd(&bins[v], lane ? 1u : __popc(same));
}

// The bin [from, from + m) of b with at most kBinValues values, in order, by
// counting them (cnt: kBinValues words).
template <int WARPS>
__device__ __forceinline__ void smem_count_bin(uint32_t* b, uint32_t from, uint32_t m,
                                               uint32_t* cnt, uint32_t* low, uint32_t* warp_tot,
                                               uint32_t* total) {
  constexpr uint32_t kThreads = WARPS * 32;
  static_assert(kBinValues % kThreads == 0, "whole rows");
  const uint32_t tid = threadIdx.x, lane = tid & 31u;
  for (uint32_t v = tid; v < kBinValues; v += kThreads) cnt[v] = 0u;
  if (tid == 0) *low = 0xffffffffu;
  __syncthreads();
  uint32_t lo = 0xffffffffu;
  for (uint32_t j = tid; j < m; j += kThreads) lo = min(lo, b[bin_swz(from + j)]);
  lo = __reduce_min_sync(0xffffffffu, lo);
  if (lane == 0) atomicMin(low, lo);
  __syncthreads();
  lo = *low;
  for (uint32_t j = tid; j < ((m + 31u) & ~31u); j += kThreads) {
    const uint32_t v = j < m ? b[bin_swz(from + j)] - lo : 0xffffffffu;
    warp_count(cnt, v < kBinValues ? v : 0xffffffffu);
  }
  __syncthreads();
  smem_exclusive_rows<WARPS>(cnt, kBinValues / kThreads, warp_tot, total);
  for (uint32_t j = tid; j < m; j += kThreads) {
    uint32_t v = 0, top = kBinValues - 1u;  // the last value that starts at or before j
    while (v < top) {
      const uint32_t mid = (v + top + 1u) >> 1;
      if (cnt[mid] <= j) v = mid;
      else top = mid - 1u;
    }
    b[bin_swz(from + j)] = lo + v;
  }
  __syncthreads();
}

// The keys k[0, cnt), word bin_swz(j) each, nearly in order, put in order: each
// lies in its bin, start[j] to start[j + 1] (cnt after the last), and no other
// bin's key does. Sixteens are sorted in registers, then the sixteens that
// start in their middles: that places the keys of bins of at most eight (one
// that belongs across a border lies within eight words of it), and no key
// leaves its bin. more: larger bins are sorted too, by a warp each, beyond
// kBinWarp keys by the CTA (then the bin has at most kBinValues values).
template <int WARPS, int ITEMS>
__device__ __forceinline__ void smem_sort_bins(uint32_t* k, const uint32_t* start, int cnt,
                                               bool more, uint32_t* aux, uint32_t* warp_tot,
                                               uint32_t* total, uint32_t* s_span) {
  constexpr int kThreads = WARPS * 32;
  const int tid = threadIdx.x, wid = tid >> 5;
  // the last sixteen and the one after it: keys that stay behind all others
  const int end = ((cnt + 15) & ~15) + 8;
  if (cnt + tid < end) k[bin_swz((uint32_t)(cnt + tid))] = 0xffffffffu;
  if (tid < 2) s_span[tid] = 0u;
  uint4* k4 = reinterpret_cast<uint4*>(k);
  static_assert(ITEMS <= 16, "one sixteen per thread");
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    __syncthreads();
    const int at = tid * 16 + half * 8;
    if (at < cnt) {
      uint32_t v[16];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint4 q = k4[bin_swz((uint32_t)(at + 4 * c)) >> 2];
        v[4 * c] = q.x;
        v[4 * c + 1] = q.y;
        v[4 * c + 2] = q.z;
        v[4 * c + 3] = q.w;
      }
      sort16(v);
#pragma unroll
      for (int c = 0; c < 4; ++c)
        k4[bin_swz((uint32_t)(at + 4 * c)) >> 2] =
            make_uint4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
    }
  }
  __syncthreads();
  if (!more) return;
  // the larger bins, listed first: they lie side by side, in few warps' rows
  uint32_t* list = aux;  // start | keys << 16
  uint32_t* values = list + kBinList;
  static_assert(kThreads * ITEMS / kBinNet <= kBinList, "every larger bin fits");
  for (int j = tid; j < cnt; j += kThreads) {
    const uint32_t s = start[j], e = j + 1 < cnt ? start[j + 1] : (uint32_t)cnt, m = e - s;
    if (m > kBinWarp) list[kBinList - 1u - atomicAdd(&s_span[1], 1u)] = s | m << 16;
    else if (m > kBinNet) list[atomicAdd(&s_span[0], 1u)] = s | m << 16;
  }
  __syncthreads();
  const uint32_t bins = s_span[0], giants = s_span[1];
  for (uint32_t i = wid; i < bins; i += WARPS) {
    const uint32_t from = list[i] & 0xffffu, m = list[i] >> 16;
    if (m <= 32u) warp_sort_bin<1>(k, from, m);
    else if (m <= 64u) warp_sort_bin<2>(k, from, m);
    else if (m <= 128u) warp_sort_bin<4>(k, from, m);
    else if (m <= 256u) warp_sort_bin<8>(k, from, m);
    else warp_sort_bin<16>(k, from, m);
  }
  for (uint32_t i = 0; i < giants; ++i) {
    const uint32_t from = list[kBinList - 1u - i] & 0xffffu, m = list[kBinList - 1u - i] >> 16;
    bool same = true;
    for (uint32_t j = tid; j < m; j += kThreads) same &= k[bin_swz(from + j)] == k[bin_swz(from)];
    if (!__syncthreads_and(same))
      smem_count_bin<WARPS>(k, from, m, values, values + kBinValues, warp_tot, total);
  }
  __syncthreads();
}

// keys[0, cnt) (cnt <= WARPS * 32 * ITEMS, WARPS * 32 threads) sorted in a or b:
// returns which (both 16-byte aligned, with kBinPad words behind each). place_of:
// a key's bin, 0 to cnt - 1 and rising with the key, and how far into the bin
// its value lies, in units of 2^-32. As many bins as keys that follow the keys'
// density hold about one each: one count, one scan and one scatter then bring a
// key to within its bin's size of its place. Where a bin has more than kBinCut
// keys, every bin is cut into as many as it has keys, and the keys are counted
// once more: what is large after that is mostly one value. aux: kBinAux words,
// s_span: two.
// (By 1,024 threads 16,384 even keys take 13 us; 22 us with comparisons within
// the bins and a scan of 16 bins per thread.)
template <int WARPS, int ITEMS, class PlaceOf>
__device__ __forceinline__ uint32_t* smem_bin_sort(const uint32_t* keys, int cnt, uint32_t* a,
                                                   uint32_t* b, uint32_t* aux,
                                                   uint32_t* warp_tot, uint32_t* total,
                                                   uint32_t* s_span, PlaceOf place_of) {
  constexpr int kThreads = WARPS * 32;
  const int tid = threadIdx.x, lane = tid & 31;
  const int items = (cnt + kThreads - 1) / kThreads;
  // a key's rank in its bin; after a cut its bin below that
  uint32_t key[ITEMS], rank[ITEMS];
  for (int j = tid; j < items * kThreads; j += kThreads) a[j] = 0u;
#pragma unroll
  for (int it = 0; it < ITEMS; ++it) {
    if (it >= items) break;
    const int j = it * kThreads + tid;
    key[it] = j < cnt ? keys[j] : 0u;
  }
  if (tid == 0) s_span[0] = 0u;
  __syncthreads();
  uint32_t most = 0;
#pragma unroll
  for (int it = 0; it < ITEMS; ++it) {
    if (it >= items) break;
    uint32_t r = 0, into;
    if (it * kThreads + tid < cnt) r = atomicAdd(&a[place_of(key[it], into)], 1u);
    most = max(most, r);
    rank[it] = r;
  }
  most = __reduce_max_sync(0xffffffffu, most);
  if (lane == 0 && most >= kBinNet) atomicMax(&s_span[0], most);
  __syncthreads();
  const bool more = s_span[0] != 0u, cut = s_span[0] >= kBinCut;
  smem_exclusive_rows<WARPS>(a, items, warp_tot, total);  // bin counts to bin starts
  if (items <= kBinFewItems && s_span[0] < kBinCompare) {
    // few keys: each finds its place by comparing with its bin's others, in
    // fewer steps than the forms below need whatever the keys
#pragma unroll
    for (int it = 0; it < kBinFewItems; ++it)
      if (it * kThreads + tid < cnt) {
        uint32_t into;
        b[a[place_of(key[it], into)] + rank[it]] = key[it];
      }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < kBinFewItems; ++it) {
      const int j = it * kThreads + tid;
      if (j >= cnt) break;
      uint32_t into;
      const uint32_t x = b[j], bin = place_of(x, into);
      const int s = (int)a[bin], e = (int)bin + 1 < cnt ? (int)a[bin + 1] : cnt;
      uint32_t place = (uint32_t)s;
#pragma unroll 4
      for (int q = s; q < e; ++q) {
        const uint32_t y = b[q];
        place += y < x || (y == x && q < j) ? 1u : 0u;
      }
      key[it] = x;
      rank[it] = place;
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < kBinFewItems; ++it)
      if (it * kThreads + tid < cnt) a[rank[it]] = key[it];
    __syncthreads();
    return a;
  }
  if (cut) {
    for (int j = tid; j < items * kThreads; j += kThreads) b[j] = 0u;
    __syncthreads();
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
      if (it >= items) break;
      if (it * kThreads + tid < cnt) {
        uint32_t into;
        const uint32_t bin = place_of(key[it], into), s = a[bin];
        const uint32_t m = ((int)bin + 1 < cnt ? a[bin + 1] : (uint32_t)cnt) - s;
        const uint32_t sub = s + __umulhi(into, m);
        rank[it] = sub | atomicAdd(&b[sub], 1u) << 16;
      }
    }
    __syncthreads();
    smem_exclusive_rows<WARPS>(b, items, warp_tot, total);
  }
  uint32_t* start = cut ? b : a;
  uint32_t* dst = cut ? a : b;
#pragma unroll
  for (int it = 0; it < ITEMS; ++it) {
    if (it >= items) break;
    if (it * kThreads + tid < cnt) {
      uint32_t into;
      const uint32_t at = cut ? b[rank[it] & 0xffffu] + (rank[it] >> 16)
                              : a[place_of(key[it], into)] + rank[it];
      dst[bin_swz(at)] = key[it];
    }
  }
  smem_sort_bins<WARPS, ITEMS>(dst, start, cnt, more, aux, warp_tot, total, s_span);
  for (int j = tid; j < cnt; j += kThreads) start[j] = dst[bin_swz((uint32_t)j)];
  __syncthreads();
  return start;
}

// cnt keys written in order from how often each of their values occurs:
// bins[v], v < values (room a multiple of WARPS * 32, values or more; zero from
// values on), counts top | v. A warp writes consecutive positions; a position's
// value is the last that starts at or before it, searched by doubled steps from
// the lane's last one. All threads call it, behind a barrier.
template <int WARPS>
__device__ __forceinline__ void smem_emit_counts(uint32_t* bins, uint32_t values, uint32_t room,
                                                 uint32_t cnt, uint32_t top, uint32_t* dst,
                                                 uint32_t* warp_tot, uint32_t* total) {
  constexpr uint32_t kThreads = WARPS * 32;
  const uint32_t tid = threadIdx.x, lane = tid & 31u;
  smem_exclusive_rows<WARPS>(bins, (int)(room / kThreads), warp_tot, total);
  const uint32_t span = ((cnt + kThreads - 1u) / kThreads) * 32u;
  const uint32_t p0 = (tid >> 5) * span, p1 = min(p0 + span, cnt);
  uint32_t v = 0;
  for (uint32_t p = p0 + lane; p < p1; p += 32u) {
    uint32_t step = 1;
    while (v + step < values && bins[v + step] <= p) {
      v += step;
      step <<= 1;
    }
    while (step >>= 1)
      if (v + step < values && bins[v + step] <= p) v += step;
    dst[p] = top | v;
  }
  __syncthreads();
}

// Bitmap words [seg0, seg1) of this warp: lanes take consecutive words.
// Pass 0 returns the warp's popcount; pass 1 emits keys at base + rank, into
// shared memory (stage) or global memory.
__device__ __forceinline__ uint32_t bitmap_emit(const uint32_t* bm, int seg0, int seg1,
                                                uint32_t kmin, bool emit, uint32_t base,
                                                uint32_t* dst) {
  const int lane = threadIdx.x & 31;
  uint32_t run = 0;
  for (int w0 = seg0; w0 < seg1; w0 += 32) {
    const int w = w0 + lane;
    uint32_t bits = w < seg1 ? bm[w] : 0u;
    const uint32_t c = __popc(bits);
    uint32_t inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (emit) {
      uint32_t pos = base + run + inc - c;
      const uint32_t kw = kmin + ((uint32_t)w << 5);
      while (bits) {
        const int bit = __ffs(bits) - 1;
        bits &= bits - 1;
        dst[pos++] = kw + (uint32_t)bit;
      }
    }
    run += __shfl_sync(0xffffffffu, inc, 31);
  }
  return run;
}

// Sorted keys a[seg0, seg1) of this warp (a[-1] read for run heads).
__device__ __forceinline__ uint32_t heads_emit(const uint32_t* a, int seg0, int seg1, bool emit,
                                               uint32_t base, uint32_t* dst) {
  const int lane = threadIdx.x & 31;
  uint32_t run = 0;
  for (int i0 = seg0; i0 < seg1; i0 += 32) {
    const int i = i0 + lane;
    const bool head = i < seg1 && (i == 0 || a[i] != a[i - 1]);
    const uint32_t m = __ballot_sync(0xffffffffu, head);
    if (emit && head) dst[base + run + __popc(m & lanemask_lt())] = a[i];
    run += __popc(m);
  }
  return run;
}

}  // namespace octgb

// Sorting keys alone (stage 2: k_SimpleRadixSort, reference
// kernels/02_sort.cpp:13-58 and kernels/cuda/02_sort.cu:208-338) as one
// cooperative launch of at most one CTA per SM.
//
// Digit passes move every key three or four times, each pass behind a
// histogram, a scan and their launches. Here a key moves twice: to its bucket,
// then, sorted with its neighbours in shared memory, to its place. Phases, with
// a grid barrier between them (up to eight CTAs are one cluster):
//
//   count    keys per bucket (their top 12 bits); the CTA's place in each
//            bucket from the global count's atomic add
//   split    only when a bucket holds more than a CTA sorts: such buckets are
//            cut by further bits, and the keys counted again
//   scatter  bucket bases (every CTA scans the counts), the keys to their
//            buckets in the other buffer
//   sort     a CTA takes the buckets that start in its share of the positions,
//            as many at a time as fit shared memory, through smem_bin_sort;
//            a cut bucket that still does not fit by counting its values
//            (2^15 at most)
//
// Equal keys are alike, so their order is free: unless a key has bits above
// key_bits, which the sort passes over. Such keys, and buckets beyond the
// limits above (a few values that hold much of a large array), take stable 8-bit
// digit passes inside the same launch, or are left to passes behind it.
//
// Measured against the launched digit passes, us: 20,000 even 32-bit keys 99 ->
// 20, 130,000 99 -> 22, 1,048,576 102 -> 33, 4M 157 -> 75; Morton codes of points
// around 64 centres 99 -> 48 at 1M; one value 92 -> 68 at 130,000, 157 -> 48 at 4M.
// Up to some 100,000 keys the phases' latencies are what is left, later the
// scatter's 4-byte stores (a third at 8.4M: an SM stores about one sector a
// cycle) and the shared-memory work of the sort phase.
#include <algorithm>

#include "kernels.cuh"
#include "smem_sort.cuh"

namespace octgb {

constexpr int kSoThreads = 1024;
constexpr int kSoWarps = kSoThreads / 32;
constexpr int kSoItems = 16;
constexpr int kSoCap = kSoThreads * kSoItems;  // keys a CTA sorts in shared memory
constexpr int kSoTopBits = 12;
constexpr int kSoTop = 1 << kSoTopBits;
constexpr int kSoIds = 8192;      // buckets after the split, at most
constexpr int kSoCountBits = 15;  // values counted: the two key arrays as one table
constexpr int kSoMaxGrid = 256;
constexpr int kSoMaxCluster = 8;
constexpr int kSoStretch = 14336; // positions whose buckets are sorted together (mostly at once)
constexpr int kSoMinPer = 1024;   // keys per CTA at least
// Up to kSoAny keys the launch sorts whatever it is given: none of 20 distributions
// is slower than by launched passes by more than 3% (4M keys: even 157 us by passes
// and 75 here, codes around 64 centres 155 and 132, a cloud a sixteenth of its box
// thick 155 and 116, a few values 146 to 164 and 141 to 144). Beyond, passes are
// faster for uneven keys (8.4M: codes around 64 centres 235 and 242, ten values
// that hold nine tenths 223 and 292), but not for even ones (232 and 160): up to
// kSoEven the launch leaves keys that a look finds uneven to passes behind it, which
// otherwise are four launches that return at once (even 232 and 190; uneven within
// 1% of the passes alone). Larger arrays take passes alone (16.7M: even keys would
// gain an eighth, uneven ones lose 4%).
constexpr int kSoAny = 4000000;
// Whole builds take it to where the MSD form begins (4,190,000 points, build: even 373
// us by passes and 299, codes around 64 centres 357 and 333, a few values 240 and 234;
// at that end alone a cloud in one sixteenth of one axis has its 256 buckets just above
// what a CTA sorts: 313 and 336, at 4.1M 307 and 274).
constexpr int kSoBuild = (1 << 22) - 1;
// Keys of one digit (10 bits) take a single launched pass, as fast for any of them
// (45 us up to 250,000, 54 at 1M): the launch is faster for even ones (26 to 50) but
// not where a value holds half of them or more (35 to 66), so it takes arrays up to
// kSoOneDigit, those of one cluster. Two digits are worth it throughout: 70 us up to
// 250,000 by passes and 24 to 72 here, 81 at 1.5M and 38 to 72.
constexpr int kSoOneDigit = kSoMaxCluster * kSoMinPer;
constexpr int kSoEven = 1 << 23;
// The look: 1,024 keys of the array. Few values hold much of it if more than kSoFew
// are alike in all but 12 bits; such keys take the digit passes in here at once, not
// after two counts (20 us of 155 at 4M and of 106 at 1.5M; even keys lose 1 us, and
// smaller arrays little by the counts). It is uneven, for kSoEven, if more than
// kSoTopMost are alike in the top 10 bits or kSoPairs meet another in a cell of 2^12
// values (even keys: 32 by the table's size).
constexpr int kSoLook = 1 << 20;
constexpr uint32_t kSoFew = 16;
constexpr uint32_t kSoTopMost = 14;
constexpr int kSoPairs = 80;
constexpr int kSoCellBits = 14;

struct SoLayout {
  size_t hist_off, zero_bytes, ids_off, mat_off, total;
  int grid;
};

static SoLayout so_layout(int n) {
  SoLayout L{};
  L.grid = std::max(1, std::min((n + kSoMinPer - 1) / kSoMinPer,
                                std::min(device_sm_count(), kSoMaxGrid)));
  L.hist_off = 256;
  L.zero_bytes = L.hist_off + 4 * (size_t)kSoTop;
  L.ids_off = L.zero_bytes;
  L.mat_off = L.ids_off + 4 * (size_t)kSoIds;
  L.total = L.mat_off + 8 * (size_t)kRsBins * L.grid;
  return L;
}

struct SoArgs {
  uint32_t* keys;
  uint32_t* alt;
  int n;
  int key_bits;  // the keys' significant bits
  int low_bits;  // bits that order the keys, should some have more
  GridBarrier bar;
  uint32_t* high;  // keys have bits above key_bits
  uint32_t* next;  // stretches taken, beyond one per CTA
  uint32_t* hist;  // [kSoTop] zeroed
  uint32_t* ids;   // [kSoIds]
  uint32_t* mat;   // [2][grid][kRsBins]
  uint32_t* status;
  const uint32_t* gate;  // device flag: 0 returns at once
  uint32_t* defer;  // nullptr, or a zeroed flag: keys left to passes set it
};

struct SoSmem {
  // two key arrays; before that the buckets' places
  __align__(16) uint32_t ab[2 * (kSoCap + kBinPad)];
  uint32_t start[kSoIds + 1];   // first position of each bucket
  uint32_t tab[kSoTop];         // a top bucket's first bucket | log2(buckets) << 16
  RadixSmem<kSoWarps> radix;
};
static_assert(sizeof(RadixSmem<kSoWarps>) >= 4 * kBinAux, "the bin sort's scratch");
static_assert(kSoIds <= 2 * kSoCap && (1 << kSoCountBits) <= 2 * kSoCap, "aliases of ab");

// src[0, cnt), keys of one bucket whose values differ in their low `bits` bits
// only (bits <= kSoCountBits), sorted to dst by counting the values in bins.
__device__ __forceinline__ void so_count_sort(const uint32_t* src, uint32_t cnt, uint32_t* dst,
                                              int bits, uint32_t* bins, uint32_t* warp_tot,
                                              uint32_t* total) {
  const int tid = threadIdx.x, lane = tid & 31;
  const uint32_t values = 1u << bits, mask = values - 1u;
  const uint32_t room = max(values, (uint32_t)kSoThreads);
  for (uint32_t v = tid; v < room; v += kSoThreads) bins[v] = 0u;
  const uint32_t top = src[0] & ~mask;
  __syncthreads();
  for (uint32_t i0 = tid & ~31u; i0 < cnt; i0 += 4 * kSoThreads) {
    uint32_t k[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t i = i0 + (uint32_t)q * kSoThreads + lane;
      k[q] = i < cnt ? src[i] & mask : 0xffffffffu;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) warp_count(bins, k[q]);
  }
  __syncthreads();
  smem_emit_counts<kSoWarps>(bins, values, room, cnt, top, dst, warp_tot, total);
}

template <bool CLUSTER>
__global__ void __launch_bounds__(kSoThreads, 1) sort_once_kernel(SoArgs A) {
  if (A.gate && *A.gate == 0u) return;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  SoSmem& M = *reinterpret_cast<SoSmem*>(sm_raw);
  __shared__ uint32_t s_warp[32], s_total, s_span[2], s_next[2];
  __shared__ int s_ok;
  const int tid = threadIdx.x;
  const uint32_t G = gridDim.x, cta = blockIdx.x;
  uint32_t phase = 0;
  auto barrier = [&]() {
    const bool ok = grid_barrier<CLUSTER>(A.bar, ++phase, &s_ok);
    if (!ok && tid == 0) raise_status(A.status, kStatusSpinTimeout);
    return ok;
  };
  const uint32_t n = (uint32_t)A.n;
  const uint32_t per = (n + G - 1u) / G;
  const uint32_t t0 = min(cta * per, n), t1 = min(t0 + per, n);
  const bool one = per <= (uint32_t)kSoCap;  // the CTA's keys stay in registers
  const int shift = max(A.key_bits - kSoTopBits, 0);
  uint32_t* base = M.ab;
  uint32_t key[kSoItems], rank2[kSoItems / 2];
  // The keys from t on (at most kSoCap of the CTA's) to `key`; f(item, key) for
  // the valid ones.
  auto load = [&](uint32_t t) {
#pragma unroll
    for (int it = 0; it < kSoItems; ++it) {
      const uint32_t i = t + (uint32_t)it * kSoThreads + tid;
      if (t + (uint32_t)it * kSoThreads >= t1) break;
      key[it] = i < t1 ? A.keys[i] : 0u;
    }
  };
  auto each = [&](uint32_t t, auto f) {
#pragma unroll
    for (int it = 0; it < kSoItems; ++it) {
      if (t + (uint32_t)it * kSoThreads >= t1) break;
      if (t + (uint32_t)it * kSoThreads + tid < t1) f(it, key[it]);
    }
  };
  auto keep_rank = [&](int it, uint32_t r) {
    if (it & 1) rank2[it / 2] |= r << 16;
    else rank2[it / 2] = r;
  };
  // Counts of every bucket of the CTA's keys in base (with the ranks of keys
  // that stay), then the CTA's place in each bucket from the global counts.
  auto count = [&](int buckets, uint32_t* global, auto id_of) {
    for (uint32_t t = t0; t < t1; t += kSoCap) {
      if (!one || t != t0 || phase == 0) load(t);
      if (one) {
        each(t, [&](int it, uint32_t k) { keep_rank(it, atomicAdd(&base[id_of(k)], 1u)); });
      } else {
        each(t, [&](int, uint32_t k) { atomicAdd(&base[id_of(k)], 1u); });
      }
    }
    __syncthreads();
    for (int b = tid; b < buckets; b += kSoThreads) {
      const uint32_t c = base[b];
      if (c) base[b] = atomicAdd(global + b, c);
    }
  };
  auto top_of = [&](uint32_t k) { return (k >> shift) & (uint32_t)(kSoTop - 1); };

  // ---- look
  bool lsd = false;
  if (A.n > kSoLook) {  // (every CTA looks at the same keys)
    const uint32_t k = A.keys[(unsigned long long)tid * n / kSoThreads];
    const uint32_t hash = (k >> 12) * 0x9e3779b1u;
    for (int b = tid; b < kSoTop; b += kSoThreads) M.tab[b] = 0u;
    for (int b = tid; A.defer && b < 1 << kSoCellBits; b += kSoThreads) M.ab[b] = 0u;
    __syncthreads();
    if (A.defer) {
      const uint32_t top = (k >> max(A.key_bits - 10, 0)) & 1023u;
      const bool met = atomicAdd(&M.ab[hash >> (32 - kSoCellBits)], 1u) > 0u;
      lsd = __syncthreads_or(atomicAdd(&M.tab[top], 1u) >= kSoTopMost) != 0;
      lsd |= __syncthreads_count(met) >= kSoPairs;
    } else {
      lsd = __syncthreads_or(atomicAdd(&M.tab[hash >> (32 - kSoTopBits)], 1u) >= kSoFew) != 0;
    }
  }
  auto deferred = [&]() {
    if (lsd && A.defer && cta == 0 && tid == 0) *A.defer = 1u;
    return lsd && A.defer;
  };
  if (deferred()) return;

  // ---- count
  for (int b = tid; b < kSoTop; b += kSoThreads) base[b] = 0u;
  for (int b = (int)cta * kSoThreads + tid; b < kSoIds; b += (int)G * kSoThreads) A.ids[b] = 0u;
  if (CLUSTER) {  // no memset was launched
    for (int b = (int)cta * kSoThreads + tid; b < kSoTop; b += (int)G * kSoThreads) A.hist[b] = 0u;
    if (cta == 0 && tid == 0) *A.high = 0u;
    grid_barrier<CLUSTER>(A.bar, 0, &s_ok);
  }
  __syncthreads();
  if (!lsd) {
    bool high = false;
    count(kSoTop, A.hist, [&](uint32_t k) {
      high |= A.key_bits < 32 && (k >> A.key_bits) != 0u;
      return top_of(k);
    });
    if (__syncthreads_or(high) && tid == 0) *A.high = 1u;
    if (!barrier()) return;
    lsd = *reinterpret_cast<volatile uint32_t*>(A.high) != 0u;
  }

  // ---- bucket bases; buckets that don't fit are split
  constexpr int kPer = kSoTop / kSoThreads;
  static_assert(kPer == 4, "one 16-byte load of counts per thread");
  const uint4 q4 = reinterpret_cast<const uint4*>(A.hist)[tid];
  const uint32_t c4[kPer] = {q4.x, q4.y, q4.z, q4.w};
  const uint32_t c_most = max(max(c4[0], c4[1]), max(c4[2], c4[3]));
  const bool split = __syncthreads_or(c_most > (uint32_t)kSoCap) != 0 && !lsd;
  int ids = kSoTop;
  // (uniform branches: every thread of every CTA sees the same counts)
  auto id_of = [&](uint32_t k) {
    if (!split) return top_of(k);
    const uint32_t t = M.tab[top_of(k)], sub = t >> 16;
    return (t & 0xffffu) + ((k >> (shift - (int)sub)) & ((1u << sub) - 1u));
  };
  if (!lsd && !split) {
    uint32_t ex = block_exclusive_sum<kSoThreads>(c4[0] + c4[1] + c4[2] + c4[3], s_warp, &s_total);
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      M.start[kPer * tid + k] = ex;
      base[kPer * tid + k] += ex;
      ex += c4[k];
    }
    if (tid == 0) M.start[kSoTop] = n;
  }
  if (split) {
    // buckets of about `unit` keys, and of few enough values to be counted
    const uint32_t unit = max((uint32_t)kSoCap / 4, n >> 11);
    uint32_t sub[kPer], mine = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      uint32_t l = 0;
      if (c4[k] > (uint32_t)kSoCap) {
        l = (uint32_t)max(shift - kSoCountBits, 0);
        while ((unit << l) < c4[k]) ++l;
        l = min(l, (uint32_t)shift);
      }
      sub[k] = l;
      mine += 1u << l;
    }
    uint32_t ex = block_exclusive_sum<kSoThreads>(mine, s_warp, &s_total);
    ids = (int)min(s_total, (uint32_t)kSoIds + 1u);
    lsd = ids > kSoIds;
    if (!lsd) {
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        M.tab[kPer * tid + k] = ex | sub[k] << 16;
        ex += 1u << sub[k];
      }
      for (int b = tid; b < ids; b += kSoThreads) base[b] = 0u;
      __syncthreads();
      count(ids, A.ids, id_of);
      if (!barrier()) return;
      constexpr int kEach = kSoIds / kSoThreads;
      uint32_t c[kEach], sum = 0, most = 0;
#pragma unroll
      for (int k = 0; k < kEach; ++k) {
        const int b = tid * kEach + k;
        c[k] = b < ids ? A.ids[b] : 0u;
        sum += c[k];
        most = max(most, c[k]);
      }
      // one CTA counts a bucket: one with far more keys than the CTA's share
      // would be waited for
      const uint32_t limit = max(8u * (uint32_t)kSoCap, 4u * per);
      lsd = __syncthreads_or(most > limit) != 0;
      uint32_t at = block_exclusive_sum<kSoThreads>(sum, s_warp, &s_total);
#pragma unroll
      for (int k = 0; k < kEach; ++k) {
        const int b = tid * kEach + k;
        if (b < ids) {
          M.start[b] = at;
          base[b] += at;
        }
        at += c[k];
      }
      if (tid == 0) M.start[ids] = n;
    }
  }
  __syncthreads();
  if (deferred()) return;

  if (!lsd) {
    // ---- scatter
    for (uint32_t t = t0; t < t1; t += kSoCap) {
      if (one) {
        each(t, [&](int it, uint32_t k) {
          A.alt[base[id_of(k)] + ((rank2[it / 2] >> (16 * (it & 1))) & 0xffffu)] = k;
        });
      } else {
        load(t);
        each(t, [&](int, uint32_t k) { A.alt[atomicAdd(&base[id_of(k)], 1u)] = k; });
      }
    }
    if (!barrier()) return;

    // ---- sort the buckets that start in a stretch of the positions: the CTA's
    // share, or stretches from a counter (the next one's number is fetched while
    // one is worked on)
    const uint32_t most = split ? (uint32_t)kSoStretch / 2u : (uint32_t)kSoStretch;
    const uint32_t rounds = (per + most - 1u) / most;
    const uint32_t stretch = one ? per : (per + rounds - 1u) / rounds;
    uint32_t k = cta;
    for (int turn = 0; (unsigned long long)k * stretch < n; turn ^= 1) {
      if (!one && tid == 0) s_next[turn] = G + atomicAdd(A.next, 1u);
      const uint32_t w0 = k * stretch, w1 = min(w0 + stretch, n);
      int i = first_at_least(M.start, 0, ids, w0);
      const int end = first_at_least(M.start, i, ids, w1);
      while (i < end) {
        const uint32_t lo = M.start[i];
        // as many buckets as fit: all up to the first that starts past the end
        int e = first_at_least(M.start, i + 1, end + 1, lo + (uint32_t)kSoCap + 1u) - 1;
        e = min(max(e, i + 1), end);
        const uint32_t cnt = M.start[e] - lo;
        if (cnt > (uint32_t)kSoCap) {
          // one bucket, cut as far as it takes: its values fit the table
          const uint32_t t = M.tab[top_of(A.alt[lo])];
          so_count_sort(A.alt + lo, cnt, A.keys + lo, shift - (int)(t >> 16), M.ab, s_warp,
                        &s_total);
        } else if (cnt > 0) {
          auto place_of = [&](uint32_t k, uint32_t& into) {
            const uint32_t b = id_of(k), s = M.start[b], c = M.start[b + 1] - s;
            const int rem = split ? shift - (int)(M.tab[top_of(k)] >> 16) : shift;
            const uint32_t part = rem ? k << (32 - rem) : 0u;
            into = part * c;
            return s - lo + __umulhi(part, c);
          };
          const uint32_t* sorted =
              smem_bin_sort<kSoWarps, kSoItems>(A.alt + lo, (int)cnt, M.ab, M.ab + kSoCap + kBinPad,
                                                reinterpret_cast<uint32_t*>(&M.radix), s_warp,
                                                &s_total, s_span, place_of);
          for (uint32_t j = tid; j < cnt; j += kSoThreads) A.keys[lo + j] = sorted[j];
          __syncthreads();
        }
        i = e;
      }
      if (one) break;
      __syncthreads();
      k = s_next[turn];
    }
    return;
  }

  // ---- stable digit passes: a CTA's tiles in order, one digit's keys of
  // earlier CTAs before its own
  uint32_t* src = A.keys;
  uint32_t* dst = A.alt;
  uint32_t* dbase = M.start;  // [kRsBins] next position of each digit
  const int passes = (A.low_bits + kRsBits - 1) / kRsBits;
  for (int p = 0; p < passes; ++p) {
    const int sh = p * kRsBits;
    const int width = min(max(A.low_bits - sh, 0), kRsBits);
    const uint32_t mask = (1u << width) - 1u;
    if (tid < kRsBins) dbase[tid] = 0u;
    __syncthreads();
    for (uint32_t i0 = t0 + (uint32_t)(tid & ~31); i0 < t1; i0 += 4 * kSoThreads) {
      uint32_t d[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t i = i0 + (uint32_t)(q * kSoThreads + (tid & 31));
        d[q] = i < t1 ? (src[i] >> sh) & mask : 0xffffffffu;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) warp_count(dbase, d[q]);
    }
    __syncthreads();
    uint32_t* mat = A.mat + (size_t)(p & 1) * G * kRsBins;  // (a skipped pass has no second barrier)
    if (tid < kRsBins) mat[cta * kRsBins + tid] = dbase[tid];
    if (!barrier()) return;
    bool same = false;  // all keys have one digit: nothing moves
    {
      // four threads per digit: keys of it in all CTAs, and in earlier ones
      const uint32_t d = tid & (kRsBins - 1), part = tid / kRsBins;
      uint32_t all = 0, before = 0;
      for (uint32_t g = part; g < G; g += kSoThreads / kRsBins) {
        const uint32_t c = mat[g * kRsBins + d];
        all += c;
        before += g < cta ? c : 0u;
      }
      uint32_t* sums = M.tab;  // [2][kSoThreads]
      sums[tid] = all;
      sums[kSoThreads + tid] = before;
      __syncthreads();
      all = before = 0;
      if (tid < kRsBins)
        for (int q = 0; q < kSoThreads; q += kRsBins) {
          all += sums[q + tid];
          before += sums[kSoThreads + q + tid];
        }
      same = tid < kRsBins && all == n;
      const uint32_t ex = block_exclusive_sum<kSoThreads>(all, s_warp, &s_total);
      if (tid < kRsBins) dbase[tid] = ex + before;
    }
    if (__syncthreads_or(same)) continue;
    for (uint32_t t = t0; t < t1; t += kSoCap) {
      const int cnt = (int)min(t1 - t, (uint32_t)kSoCap);
      uint32_t* a = M.ab;
      uint32_t* b = M.ab + kSoCap;
      for (int j = tid; j < cnt; j += kSoThreads) a[j] = src[t + j];
      __syncthreads();
      smem_radix_pass<kSoWarps, kSoItems, true>(a, b, cnt, 0u, sh, mask, M.radix);
      for (int j = tid; j < cnt; j += kSoThreads) {
        const uint32_t d = (b[j] >> sh) & mask;
        dst[dbase[d] + (uint32_t)j - M.radix.dstart[d]] = b[j];
      }
      __syncthreads();
      if (tid < kRsBins) {
        const uint32_t next = tid + 1 < kRsBins ? M.radix.dstart[tid + 1] : (uint32_t)cnt;
        dbase[tid] += next - M.radix.dstart[tid];
      }
      __syncthreads();
    }
    if (!barrier()) return;
    uint32_t* other = src;
    src = dst;
    dst = other;
  }
  if (src != A.keys)
    for (uint32_t i = t0 + tid; i < t1; i += kSoThreads) A.keys[i] = src[i];
}

// zeroed: the first zero_bytes of the layout (cleared here unless `cleared`),
// rest: what follows them.
static cudaError_t launch_sort_once(uint32_t* keys, uint32_t* alt, int n, int key_bits,
                                    int low_bits, void* zeroed, void* rest, uint32_t* status,
                                    cudaStream_t s, const uint32_t* gate = nullptr,
                                    bool cleared = false, uint32_t* defer = nullptr,
                                    uint32_t absent = 0,
                                    unsigned long long limit_ns = kWaitLimitNs) {
  const SoLayout L = so_layout(n);
  char* w = static_cast<char*>(zeroed);
  char* r = static_cast<char*>(rest) - L.zero_bytes;
  SoArgs A{};
  A.keys = keys;
  A.alt = alt;
  A.n = n;
  A.key_bits = key_bits;
  A.low_bits = low_bits;
  A.bar = GridBarrier{reinterpret_cast<uint32_t*>(w), absent, limit_ns};
  A.high = A.bar.arrivals + 1;
  A.next = A.bar.arrivals + 2;
  A.hist = reinterpret_cast<uint32_t*>(w + L.hist_off);
  A.ids = reinterpret_cast<uint32_t*>(r + L.ids_off);
  A.mat = reinterpret_cast<uint32_t*>(r + L.mat_off);
  A.status = status;
  A.gate = gate;
  A.defer = defer;
  const int smem = (int)sizeof(SoSmem);
  const bool cluster = L.grid <= kSoMaxCluster;
  auto kernel = cluster ? sort_once_kernel<true> : sort_once_kernel<false>;
  cudaError_t e = set_smem_limit(kernel, smem);
  if (e == cudaSuccess && !cluster && !cleared) e = cudaMemsetAsync(w, 0, L.zero_bytes, s);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(L.grid);
  c.blockDim = dim3(kSoThreads);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at[1];
  if (cluster) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {(unsigned)L.grid, 1u, 1u};
  } else {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  }
  c.attrs = at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, A);
}

static bool sort_once_takes(int n, int most) {
  const SortConfig c = get_sort_config(), d = kSortConfigDefault;
  return n > 1 && n <= most && c.radix_bits == d.radix_bits && c.warps == d.warps &&
         c.items == d.items && c.scan == d.scan;
}

// Past kSoAny: the launch's zeroed scratch and the plan's control block, cleared
// together, then the rest of the launch's scratch and the look-back words (past
// kSoEven as much beside the plan as there, so that more keys never need less).
size_t sort_keys_bytes(int n, int key_bits) {
  const size_t plan = sort_plan(n, key_bits).bytes;
  if (n <= 1) return plan;
  const int m = std::min(n, kSoEven);
  const size_t once = so_layout(m).total;
  return n <= kSoAny ? std::max(plan, once)
                     : once + align_up(plan, 256) + sort_few_lookback_bytes(sort_plan(m, key_bits));
}

__global__ void __launch_bounds__(1024)
    copy_gated_kernel(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst, int n,
                      const uint32_t* __restrict__ gate) {
  chain_enter();
  if (*gate == 0u) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    dst[i] = src[i];
}

cudaError_t launch_copy_gated(const uint32_t* src, uint32_t* dst, int n, const uint32_t* gate,
                              cudaStream_t s) {
  return launch_chained(copy_gated_kernel, dim3(device_sm_count() * 2), dim3(1024), 0, s, src, dst,
                        n, gate);
}

cudaError_t launch_sort_keys(uint32_t* keys, uint32_t* alt, int n, int key_bits, void* workspace,
                             uint32_t* status, cudaStream_t s) {
  const SortPlan p = sort_plan(n, key_bits);
  const SoLayout L = so_layout(n);
  const int low_bits = std::min(32, p.passes * p.radix_bits);
  char* w = static_cast<char*>(workspace);
  uint32_t* result = keys;
  if (sort_once_takes(n, p.passes > 1 ? kSoAny : kSoOneDigit)) {
    const cudaError_t e =
        launch_sort_once(keys, alt, n, key_bits, low_bits, w, w + L.zero_bytes, status, s);
    if (e != cudaErrorCooperativeLaunchTooLarge) return e;
    (void)cudaGetLastError();  // a context with fewer SMs: the passes
  } else if (n > kSoAny && sort_once_takes(n, kSoEven) && sort_few_ok(p)) {
    char* plan = w + align_up(L.zero_bytes, 256);
    char* rest = plan + align_up(p.bytes, 256);
    uint32_t* defer = reinterpret_cast<uint32_t*>(w) + 3;
    cudaError_t e = cudaMemsetAsync(w, 0, (size_t)(plan - w) + p.zero_bytes, s);
    if (e == cudaSuccess)
      e = launch_sort_once(keys, alt, n, key_bits, low_bits, w, rest, status, s, nullptr, true,
                           defer);
    if (e == cudaSuccess)
      e = launch_sort_passes_few(keys, alt, &p, plan, rest + (L.total - L.zero_bytes), status,
                                 defer, nullptr, s, &result);
    if (e == cudaSuccess && result != keys) e = launch_copy_gated(result, keys, n, defer, s);
    if (e != cudaErrorCooperativeLaunchTooLarge) return e;
    (void)cudaGetLastError();
  }
  cudaError_t e = cudaMemsetAsync(w, 0, p.zero_bytes, s);
  if (e == cudaSuccess) e = launch_histogram(keys, &p, w, s);
  if (e == cudaSuccess) e = launch_sort_passes(keys, alt, &p, w, status, s, &result);
  if (e == cudaSuccess && result != keys)
    e = cudaMemcpyAsync(keys, result, sizeof(uint32_t) * (size_t)n, cudaMemcpyDeviceToDevice, s);
  return e;
}

constexpr int kSoDiagKeys = (kSoMaxCluster + 1) * kSoMinPer;  // the fewest of a cooperative grid
size_t diag_grid_wait_bytes() {
  return 2 * sizeof(uint32_t) * (size_t)kSoDiagKeys + so_layout(kSoDiagKeys).total;
}
cudaError_t launch_diag_grid_wait(void* workspace, uint32_t* status, unsigned long long limit_ns,
                                  cudaStream_t s) {
  uint32_t* keys = static_cast<uint32_t*>(workspace);
  uint32_t* alt = keys + kSoDiagKeys;
  char* w = reinterpret_cast<char*>(alt + kSoDiagKeys);
  const cudaError_t e = cudaMemsetAsync(keys, 0, sizeof(uint32_t) * (size_t)kSoDiagKeys, s);
  return e == cudaSuccess
             ? launch_sort_once(keys, alt, kSoDiagKeys, 30, 30, w,
                                w + so_layout(kSoDiagKeys).zero_bytes, status, s, nullptr, false,
                                nullptr, 1u, limit_ns)
             : e;
}

bool sort_once_in_plan(const SortPlan& p) {
  const SoLayout L = so_layout(p.n);
  return sort_once_takes(p.n, kSoBuild) && msd_plan_ok(p) &&
         p.zero_bytes - p.tile_part_off >= 2 * align_up(L.zero_bytes, 256) &&
         p.bytes - p.tile_hist_off >= L.total - L.zero_bytes;
}

cudaError_t launch_sort_once_in_plan(uint32_t* keys, uint32_t* alt, const SortPlan& p, void* ctrl,
                                     uint32_t* status, cudaStream_t s) {
  char* c = static_cast<char*>(ctrl);  // the split sums and the tile histograms
  return launch_sort_once(keys, alt, p.n, 30, 30, c + p.tile_part_off, c + p.tile_hist_off, status,
                          s, nullptr, true);
}

size_t sort_keys_gated_zero_bytes(int n) {
  return std::max(sort_plan(n, 30).zero_bytes, (size_t)256 + 4 * kSoTop);
}

size_t sort_keys_gated_bytes(int n) {
  const size_t least = std::max(sort_plan(n, 30).bytes, sort_keys_gated_zero_bytes(n));
  return n > 1 && n <= kSoAny ? std::max(least, so_layout(n).total) : least;
}

// A sort that mostly does not run (gate 0) should cost little then: one launch,
// or four where that is the slower sort, instead of eleven (5, 14 and 32 us
// behind a learned sort that fits; whole build of 239,010 points 196 -> 157, of
// 16.7M 867 -> 829).
cudaError_t launch_sort_keys_gated(uint32_t* keys, uint32_t* alt, int n, void* workspace,
                                   void* lookback, uint32_t* status, const uint32_t* gate,
                                   cudaStream_t s, uint32_t** result) {
  *result = keys;
  if (sort_once_takes(n, kSoAny)) {
    const cudaError_t e = launch_sort_once(
        keys, alt, n, 30, 30, workspace, static_cast<char*>(workspace) + so_layout(n).zero_bytes,
        status, s, gate, true);
    if (e != cudaErrorCooperativeLaunchTooLarge) return e;
    (void)cudaGetLastError();
  }
  const SortPlan p = sort_plan(n, 30);
  if (sort_few_ok(p))
    return launch_sort_passes_few(keys, alt, &p, workspace, lookback, status, gate, nullptr, s,
                                  result);
  const cudaError_t e = launch_histogram_gated(keys, &p, workspace, gate, s);
  return e == cudaSuccess
             ? launch_sort_passes_gated(keys, alt, &p, workspace, status, gate, s, result)
             : e;
}

}  // namespace octgb

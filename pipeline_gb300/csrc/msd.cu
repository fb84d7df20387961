// Stages 2-3 of the whole build in MSD form, for large clouds whose keys
// spread evenly over the top digit (k_SimpleRadixSort + k_CountUnique,
// reference kernels/02_sort.cpp:13-58 and kernels/03_unique.cpp:2-16: the
// sorted unique codes are the same whichever way they are found).
//
//   gate     from the Morton kernel's top-digit histogram (bits 20..29): the
//            MSD form runs when n >= 2^22, no top-digit bucket holds more than
//            32x the mean and the work below stays within 8 reads a key;
//            otherwise the LSD passes and the run-head unique run. Both forms
//            are launched; the unused one's kernels return at once (a device
//            flag each). The gate also cuts the buckets into items: a bucket
//            well above the mean is 2 to 16 items, each the keys of an equal
//            part of its values
//   scatter  one unstable radix pass on the top digit: the LSD form's pass-0
//            launches, which take the top digit's shift, bases and split sums
//            when the MSD flag is set, so bucket b holds the keys
//            [b << 20, (b + 1) << 20) in any order;
//   buckets  one CTA per SM takes items from a counter, the long ones
//            first: a bitmap of the item's values (2^20 bits, 128 KiB of
//            shared memory, for a whole bucket) marks its keys; the set bits,
//            read in order, are the item's sorted unique keys (duplicates mark
//            the same bit), staged behind the bitmap and copied to the next
//            free place of the other key buffer;
//   pack     a scan of the unique counts, then one CTA per item copies its
//            run to its output offset with the delta of each code to the
//            next (the radix tree's input) and lowers the minima of the tree
//            tiles it touches: the same outputs as the LSD form's unique
//            stage.
//
// An item of a cut bucket reads the whole bucket and keeps its part: two to
// three reads a key on mixtures of 64 Gaussians, far less than a stable pass
// costs. Such a cloud took the LSD form before (nine launches, ranking-bound
// stable passes): whole build of 10,000,003 points around 64
// centres 656 -> 608 us, of which the bucket kernel is 126 (a lane that walks
// alone sets its warp's pace, so dense stretches are shared out by rank); 16.7M
// uniform points 803.5 -> 802.9 us. Where the lines lie (whole builds, mixtures
// of 8 to 64 Gaussians, LSD -> MSD form, us): largest bucket of 13 means 395 ->
// 373 at 4.2M points, 715 -> 639 at 10M, 1,055 -> 951 at 16.8M; 30 means 380 ->
// 369, 661 -> 630, 952 -> 904; 53 means (6 to 7 reads a key) 361 -> 369, 618 ->
// 620, 907 -> 899. Cuts of 16,384 to 49,152 keys measure alike from 8M points
// on; 24,576 is the best at 4.2M (380 against 392 with 49,152: an item is long
// against 1/152 of such a cloud).
#include <algorithm>

#include "kernels.cuh"
#include "tree.cuh"

namespace octgb {

constexpr int kMsdSpanBits = 20;                       // key bits below the top digit
constexpr int kMsdBuckets = 1 << (30 - kMsdSpanBits);  // 1,024
constexpr int kMsdWords = 1 << (kMsdSpanBits - 5);     // bitmap words per bucket
constexpr int kMsdThreads = 1024;
constexpr int kMsdStage = 22528;  // run keys staged in shared memory behind the bitmap
constexpr int kMsdWarpWords = kMsdWords / (kMsdThreads / 32);
constexpr int kMsdMinN = 1 << 22;
constexpr uint32_t kMsdSkew = 32;      // largest bucket, in means
constexpr uint32_t kMsdReads = 8;      // bucket keys read per key, at most
constexpr uint32_t kMsdCut = 24576;    // keys from which a bucket is cut (or 4x the mean)
constexpr int kMsdMaxCutLog = 4;  // 32 means, cut at 4
constexpr int kMsdLaneWalk = 64;       // keys in a thread's words that it walks alone
// Items: a cut bucket of c keys has at most 3 c / (4 means) (c > 4 means), so
// all of them at most 768, plus one for every other bucket.
constexpr int kMsdMaxItems = 2048;
constexpr int kPackThreads = 512;

static_assert(kMsdBuckets == kMsdThreads, "one gate thread per bucket");
static_assert(kMsdWarpWords == 32 * 32, "a warp's words are 32 rows of 32");

int msd_min_n() { return kMsdMinN; }
// Runs start at multiples of four words: at most three words lost an item.
size_t msd_run_slack() { return 4 * (size_t)kMsdMaxItems; }

// Items in key order: bucket | part << 10 | log2(parts) << 16.
struct MsdScratch {
  uint32_t* item;   // [kMsdMaxItems]
  uint32_t* order;  // [kMsdMaxItems] items of buckets above twice the mean, then the others
  uint32_t* run;    // [kMsdMaxItems] start of the item's run
  uint32_t* count;  // [kMsdMaxItems] its unique keys
  uint32_t* off;    // [kMsdMaxItems + 1] its output offset
  int* next;        // [kMsdMaxItems] start of the next run with keys, or -1
  uint32_t* items;  // how many
};
size_t msd_scratch_bytes() { return sizeof(uint32_t) * (6 * (size_t)kMsdMaxItems + 8); }
static MsdScratch msd_scratch(void* base) {
  uint32_t* p = static_cast<uint32_t*>(base);
  MsdScratch M;
  M.item = p;
  M.order = p + kMsdMaxItems;
  M.run = p + 2 * kMsdMaxItems;
  M.count = p + 3 * kMsdMaxItems;
  M.next = reinterpret_cast<int*>(p + 4 * kMsdMaxItems);
  M.off = p + 5 * kMsdMaxItems;
  M.items = p + 6 * kMsdMaxItems + 4;
  return M;
}

__global__ void __launch_bounds__(kMsdBuckets)
    msd_gate_kernel(const uint32_t* __restrict__ top_hist, int n, uint32_t* __restrict__ flags,
                    MsdScratch M, uint32_t* __restrict__ top_base) {
  chain_enter();
  __shared__ uint32_t s_max[32], warp_tot[32], total;
  __shared__ unsigned long long s_reads[32];
  const int b = threadIdx.x;
  const uint32_t cnt = top_hist[b];
  const uint32_t mean = ((uint32_t)n + kMsdBuckets - 1) / kMsdBuckets;
  const uint32_t cut = max(kMsdCut, 4 * mean);
  int ls = 0;  // parts of about two thirds of the cut
  if (cnt > cut)
    while (ls < kMsdMaxCutLog && ((unsigned long long)cnt * 3 / 2) > ((unsigned long long)cut << ls))
      ++ls;
  const uint32_t parts = cnt ? 1u << ls : 0u;
  const uint32_t most = __reduce_max_sync(0xffffffffu, cnt);
  unsigned long long reads = (unsigned long long)cnt * parts;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) reads += __shfl_xor_sync(0xffffffffu, reads, o);
  if ((b & 31) == 0) {
    s_max[b >> 5] = most;
    s_reads[b >> 5] = reads;
  }
  const uint32_t id = block_exclusive_sum<kMsdBuckets>(parts, warp_tot, &total);
  const uint32_t items = total;
  // the long items first, so that none starts when the others are done
  const bool is_long = cnt > 2 * mean;
  const uint32_t of_long = block_exclusive_sum<kMsdBuckets>(is_long ? parts : 0u, warp_tot, &total);
  const uint32_t place = is_long ? of_long : total + (id - of_long);
  if (top_base) top_base[b] = block_exclusive_sum<kMsdBuckets>(cnt, warp_tot, &total);
  if (items <= (uint32_t)kMsdMaxItems)
    for (uint32_t k = 0; k < parts; ++k) {
      M.item[id + k] = (uint32_t)b | k << 10 | (uint32_t)ls << 16;
      M.order[place + k] = id + k;
    }
  if (b == 0) {
    unsigned long long mx = 0, rd = 0;
    for (int w = 0; w < 32; ++w) {
      mx = max(mx, (unsigned long long)s_max[w]);
      rd += s_reads[w];
    }
    const bool msd = n >= kMsdMinN && mx <= (unsigned long long)kMsdSkew * mean &&
                     rd <= (unsigned long long)kMsdReads * (uint32_t)n &&
                     items <= (uint32_t)kMsdMaxItems;
    flags[0] = msd ? 1u : 0u;  // MSD form
    flags[1] = msd ? 0u : 1u;  // LSD form
    *M.items = items;
  }
}

// Bitmap word x lives at x ^ (((x >> 5) & 7) << 2): the 32 words of a lane's
// 1,024-value chunk stay together, and the eight lanes of a 16-byte shared
// load phase read eight different bank groups.
__device__ __forceinline__ uint32_t msd_swz(uint32_t x) { return x ^ (((x >> 5) & 7u) << 2); }

// The keys of bucket b (WHOLE), or those of them in part `part` of 2^ls (its
// values' top bits), marked in the bitmap. Returns false in a thread that saw a
// key of another bucket (never past the bitmap).
template <bool WHOLE>
__device__ __forceinline__ bool msd_mark(const uint32_t* __restrict__ keys, uint32_t cnt, int b,
                                         uint32_t part, int ls, uint32_t* bm, int tid) {
  bool good = true;
  constexpr int kBatch = WHOLE ? 8 : 16;  // keys in flight per thread
  const int bits = kMsdSpanBits - ls;
  for (uint32_t i0 = 0; i0 < cnt; i0 += kBatch * kMsdThreads) {
    uint32_t k[kBatch];
#pragma unroll
    for (int q = 0; q < kBatch; ++q) {
      const uint32_t i = i0 + (uint32_t)(q * kMsdThreads + tid);
      k[q] = i < cnt ? keys[i] : 0xffffffffu;  // no code reaches it
    }
#pragma unroll
    for (int q = 0; q < kBatch; ++q) {
      if (k[q] == 0xffffffffu) continue;
      if ((k[q] >> kMsdSpanBits) != (uint32_t)b) {
        good = false;
        continue;
      }
      const uint32_t v = k[q] & ((1u << kMsdSpanBits) - 1u);
      if (WHOLE) {
        atomicOr(&bm[msd_swz(v >> 5)], 1u << (v & 31u));
      } else if ((v >> bits) == part) {
        atomicOr(&bm[(v & ((1u << bits) - 1u)) >> 5], 1u << (v & 31u));
      }
    }
  }
  return good;
}

// One item: its sorted unique keys to the next free place of `out` (cursor),
// the place and count to run and count.
__device__ __forceinline__ void msd_item(const uint32_t* __restrict__ keys, uint32_t cnt,
                                         uint32_t item, uint32_t* bm, uint32_t* s_wsum,
                                         uint32_t* s_wmax, uint32_t* s_pre, uint32_t* s_nz,
                                         uint32_t* s_pos, uint32_t* __restrict__ out,
                                         uint32_t* cursor, uint32_t* run, uint32_t* count,
                                         uint32_t* __restrict__ status, int tid, int lane, int w) {
  const int b = (int)(item & 1023u), ls = (int)(item >> 16);
  const uint32_t part = (item >> 10) & 63u;
  const bool whole = ls == 0;
  const int words = kMsdWords >> ls;
  uint4* s_bm4 = reinterpret_cast<uint4*>(bm);
  for (int i = tid; i < words / 4; i += kMsdThreads) s_bm4[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  const bool good = whole ? msd_mark<true>(keys, cnt, b, part, ls, bm, tid)
                          : msd_mark<false>(keys, cnt, b, part, ls, bm, tid);
  if (__syncthreads_or(!good) && tid == 0) raise_status(status, kStatusRange);
  // Thread tid owns values [tid * 1024, tid * 1024 + 1024) of a whole bucket,
  // its 32 words read into registers in value order; of a part the words
  // [tid * per, tid * per + per).
  const int c = tid;
  const int per = max(words / kMsdThreads, 1);
  uint32_t own = 0, nz = 0;  // set bits, and the words that have any
  if (whole) {
    uint32_t wd[32];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint4 v = s_bm4[c * 8 + (j ^ (c & 7))];
      wd[4 * j] = v.x;
      wd[4 * j + 1] = v.y;
      wd[4 * j + 2] = v.z;
      wd[4 * j + 3] = v.w;
    }
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      own += __popc(wd[k]);
      nz |= (wd[k] != 0u ? 1u : 0u) << k;
    }
  } else if (c * per < words) {
    for (int k = 0; k < per; ++k) {
      const uint32_t v = bm[c * per + k];
      own += __popc(v);
      nz |= (v != 0u ? 1u : 0u) << k;
    }
  }
  uint32_t inc = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  const uint32_t most_w = __reduce_max_sync(0xffffffffu, own);
  if (lane == 31) {
    s_wsum[w] = inc;
    s_wmax[w] = most_w;
  }
  if (tid == 0) bulk_wait_read();  // the previous item's copy has read the stage
  __syncthreads();
  uint32_t pos = inc - own, total = 0;
#pragma unroll 8
  for (int k = 0; k < kMsdThreads / 32; ++k) {
    const uint32_t v = s_wsum[k];
    if (k < w) pos += v;
    total += v;
  }
  const uint32_t most = __reduce_max_sync(0xffffffffu, s_wmax[lane]);
  const bool even = most <= (uint32_t)kMsdLaneWalk;
  if (!even) {
    s_pre[tid] = pos;
    s_nz[tid] = nz;
  }
  // `total` and `most` are the same in every thread, so the branches on them
  // are uniform. A run that fits is staged behind the bitmap, its place fetched
  // meanwhile; a longer one goes straight out.
  const bool staged = total <= (uint32_t)kMsdStage;
  if (tid == 0) {
    const uint32_t at = atomicAdd(cursor, (total + 3u) & ~3u);
    *s_pos = at;
    *run = at;
    *count = total;
  }
  if (!staged || !even) __syncthreads();
  uint32_t* stage = bm + kMsdWords;
  uint32_t* dst = staged ? stage : out + *s_pos;
  const uint32_t kc = ((uint32_t)b << kMsdSpanBits) | (part << (kMsdSpanBits - ls));
  const uint32_t step = (uint32_t)(whole ? 32 : per);  // words per thread
  if (even) {
    // A lane walks its own set bits in one loop (words re-read from the
    // bitmap), so a warp runs as many rounds as its fullest lane has keys.
    uint32_t bits = 0, kw = 0;
    for (uint32_t e = 0; e < own; ++e) {
      if (bits == 0u) {
        const int k = __ffs(nz) - 1;
        nz &= nz - 1u;
        const uint32_t x = (uint32_t)c * step + (uint32_t)k;
        kw = kc | (x << 5);
        bits = bm[whole ? msd_swz(x) : x];
      }
      const int bit = __ffs(bits) - 1;
      bits &= bits - 1u;
      dst[pos + e] = kw | (uint32_t)bit;
    }
  } else {
    // Dense stretches: the set bits are shared out evenly instead. Thread t
    // takes ranks [t q, t q + q), q odd (so that the stores of a warp meet
    // different banks); a rank's thread's words by search in the prefixes, the
    // word among them by counting.
    const uint32_t q = ((total + kMsdThreads - 1u) / kMsdThreads) | 1u;
    uint32_t e = (uint32_t)tid * q;
    const uint32_t end = min(e + q, total);
    uint32_t bits = 0, left = 0, x = 0, x0 = 0;
    for (; e < end; ++e) {
      if (bits == 0u) {
        uint32_t skip = 0;
        if (left == 0u) {  // another thread's words
          int lo = 0, hi = kMsdThreads - 1;
          while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (s_pre[mid] <= e) lo = mid;
            else hi = mid - 1;
          }
          skip = e - s_pre[lo];
          left = s_nz[lo];
          x0 = (uint32_t)lo * step;
        }
        while (true) {
          x = x0 + (uint32_t)(__ffs(left) - 1);
          left &= left - 1u;
          bits = bm[whole ? msd_swz(x) : x];
          const uint32_t n = __popc(bits);
          if (skip < n) break;
          skip -= n;
        }
        for (; skip; --skip) bits &= bits - 1u;
      }
      const int bit = __ffs(bits) - 1;
      bits &= bits - 1u;
      dst[e] = kc | (x << 5) | (uint32_t)bit;
    }
  }
  if (staged) {
    bulk_fence_writes();
    __syncthreads();
    // one bulk copy of whole 16-byte words (the TMA engine writes it while the
    // CTA goes on to the next item's bitmap)
    if (tid == 0 && total) bulk_store_s2g(out + *s_pos, stage, ((total + 3u) & ~3u) * 4u);
  }
}

__global__ void __launch_bounds__(kMsdThreads, 1)
    msd_bucket_kernel(const uint32_t* __restrict__ keys, uint32_t* __restrict__ out,
                      const uint32_t* __restrict__ top_base, const uint32_t* __restrict__ top_hist,
                      MsdScratch M, uint32_t* counters, const uint32_t* __restrict__ gate,
                      uint32_t* __restrict__ status) {
  chain_enter();
  if (*gate == 0) return;
  extern __shared__ uint4 s_bm4[];
  uint32_t* bm = reinterpret_cast<uint32_t*>(s_bm4);
  __shared__ uint32_t s_wsum[kMsdThreads / 32], s_wmax[kMsdThreads / 32], s_pre[kMsdThreads];
  __shared__ uint32_t s_nz[kMsdThreads];
  __shared__ uint32_t s_pos, s_next[2];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const uint32_t items = *M.items;
  // one CTA per SM (its shared memory); the next item's number is fetched
  // while the current one is worked on
  uint32_t k = blockIdx.x;
  for (int turn = 0; k < items; turn ^= 1) {
    if (tid == 0) s_next[turn] = gridDim.x + atomicAdd(counters, 1u);
    const uint32_t id = M.order[k], item = M.item[id], b = item & 1023u;
    msd_item(keys + top_base[b], top_hist[b], item, bm, s_wsum, s_wmax, s_pre, s_nz, &s_pos, out, counters + 1,
             M.run + id, M.count + id, status, tid, lane, w);
    __syncthreads();  // the next item clears the bitmap
    k = s_next[turn];
  }
  if (tid == 0) bulk_wait_all();  // the runs are written before the kernel ends
}

__global__ void __launch_bounds__(1024)
    msd_pack_scan_kernel(MsdScratch M, int* __restrict__ d_unique, TreeScratch S,
                         const uint32_t* __restrict__ gate) {
  chain_enter();
  if (*gate == 0) return;
  __shared__ uint32_t warp_tot[32];
  __shared__ uint32_t total;
  __shared__ int s_ne[kMsdMaxItems + 1];
  const int items = (int)*M.items;
  const int t = threadIdx.x, i0 = 2 * t, i1 = 2 * t + 1;
  static_assert(kMsdMaxItems == 2 * 1024, "two items per thread");
  const uint32_t c0 = i0 < items ? M.count[i0] : 0u, c1 = i1 < items ? M.count[i1] : 0u;
  const uint32_t ex = block_exclusive_sum<1024>(c0 + c1, warp_tot, &total);
  if (i0 < items) M.off[i0] = ex;
  if (i1 < items) M.off[i1] = ex + c0;
  // the next item with keys (suffix minimum of the non-empty ids)
  s_ne[i0] = c0 > 0 ? i0 : kMsdMaxItems;
  s_ne[i1] = c1 > 0 ? i1 : kMsdMaxItems;
  if (t == 0) s_ne[kMsdMaxItems] = kMsdMaxItems;
  __syncthreads();
  for (int d = 1; d < items; d <<= 1) {
    const int v0 = min(s_ne[i0], s_ne[min(i0 + d, kMsdMaxItems)]);
    const int v1 = min(s_ne[i1], s_ne[min(i1 + d, kMsdMaxItems)]);
    __syncthreads();
    s_ne[i0] = v0;
    s_ne[i1] = v1;
    __syncthreads();
  }
  if (i0 < items) M.next[i0] = s_ne[i0 + 1] < items ? (int)M.run[s_ne[i0 + 1]] : -1;
  if (i1 < items) M.next[i1] = s_ne[i1 + 1] < items ? (int)M.run[s_ne[i1 + 1]] : -1;
  if (t == 0) *d_unique = (int)total;
  // the tree scratch of the LSD form's unique stage: no tile sums yet, every
  // tile minimum absent until the pack lowers it
  const int pad = (int)align_up((size_t)S.tiles, kTtMinBlock);
  for (int k = t; k < pad; k += 1024) S.tile_min[k] = (uint8_t)kTtAbsent;
  for (int k = t; k < S.tiles; k += 1024) S.tile_sum[k] = 0;
}

constexpr int kPackTiles = 1028;  // tree tiles one run can touch (2^20 codes: 257)

__device__ __forceinline__ void msd_pack_run(const uint32_t* __restrict__ keys, uint32_t start,
                                             uint32_t u, uint32_t o0, uint32_t U, int ns,
                                             uint32_t* __restrict__ codes, const TreeScratch& S,
                                             uint32_t* s_tmin, int tid) {
  const uint32_t* src = keys + start;
  const uint32_t after = ns >= 0 ? keys[ns] : 0u;  // read only when a code follows the run
  const uint32_t t0 = o0 / kTtTile;
  const uint32_t nt = min((o0 + u - 1) / kTtTile - t0 + 1, (uint32_t)kPackTiles);
  for (uint32_t k = tid; k < nt; k += kPackThreads) s_tmin[k] = kTtAbsent;
  __syncthreads();
  const uint32_t lane = tid & 31, warp = tid >> 5;
  constexpr uint32_t kRows = 8;  // a warp takes 8 x 32 consecutive codes per round
  constexpr uint32_t kSpan = kRows * 32;
  // whole warps iterate together (the shuffles and warp minima need every lane)
  for (uint32_t j0 = warp * kSpan; j0 < u; j0 += (kPackThreads / 32) * kSpan) {
    uint32_t k[kRows];
#pragma unroll
    for (uint32_t q = 0; q < kRows; ++q) {
      const uint32_t j = j0 + q * 32 + lane;
      k[q] = j < u ? src[j] : 0u;
    }
    // the code after this round's last: the next round's first, or the next run's
    const uint32_t jn = j0 + kSpan;
    const uint32_t tail = jn < u ? src[jn] : after;
    uint32_t ma = kTtAbsent, mb = kTtAbsent;
    const uint32_t ta = (o0 + j0) / kTtTile;  // the round's 256 positions: one tile or two
#pragma unroll
    for (uint32_t q = 0; q < kRows; ++q) {
      const uint32_t j = j0 + q * 32 + lane;
      const uint32_t o = o0 + j;
      const uint32_t down = __shfl_down_sync(0xffffffffu, k[q], 1);
      const uint32_t next_row = q + 1 < kRows ? __shfl_sync(0xffffffffu, k[q + 1 < kRows ? q + 1 : q], 0)
                                              : tail;
      const uint32_t nxt = j + 1u < u ? (lane < 31 ? down : next_row) : after;
      if (j < u) {
        codes[o] = k[q];
        if (o + 1u < U) {
          const uint32_t d = tt_delta(k[q], nxt);
          S.D[o] = (uint8_t)d;
          if (o / kTtTile == ta) ma = min(ma, d);
          else mb = min(mb, d);
        }
      }
    }
    ma = __reduce_min_sync(0xffffffffu, ma);
    mb = __reduce_min_sync(0xffffffffu, mb);
    if (lane == 0) {
      if (ma < kTtAbsent) {
        if (ta - t0 < nt) atomicMin(&s_tmin[ta - t0], ma);
        else atomic_min_u8(S.tile_min + ta, ma);  // beyond the shared table
      }
      if (mb < kTtAbsent) {
        if (ta + 1 - t0 < nt) atomicMin(&s_tmin[ta + 1 - t0], mb);
        else atomic_min_u8(S.tile_min + ta + 1, mb);
      }
    }
  }
  __syncthreads();
  for (uint32_t k = tid; k < nt; k += kPackThreads)
    if (s_tmin[k] < kTtAbsent) atomic_min_u8(S.tile_min + t0 + k, s_tmin[k]);
}

// A CTA per item: its run goes to the codes from its output offset, with each
// code's delta to the next one (the next run's first code after the run's
// last) and the touched tree tiles' minima.
__global__ void __launch_bounds__(kPackThreads)
    msd_pack_kernel(const uint32_t* __restrict__ keys, MsdScratch M,
                    const int* __restrict__ d_unique, uint32_t* __restrict__ codes, TreeScratch S,
                    const uint32_t* __restrict__ gate) {
  chain_enter();
  if (*gate == 0) return;
  __shared__ uint32_t s_tmin[kPackTiles];
  const uint32_t i = blockIdx.x;
  if (i >= *M.items) return;
  const uint32_t u = M.count[i];
  if (u != 0)
    msd_pack_run(keys, M.run[i], u, M.off[i], (uint32_t)*d_unique, M.next[i], codes, S, s_tmin,
                 threadIdx.x);
}

cudaError_t launch_msd_gate(const uint32_t* top_hist, int n, uint32_t* flags, void* scratch,
                            uint32_t* top_base, cudaStream_t s) {
  return launch_chained(msd_gate_kernel, dim3(1), dim3(kMsdBuckets), 0, s, top_hist, n, flags,
                        msd_scratch(scratch), top_base);
}

cudaError_t launch_msd_buckets(const uint32_t* keys, uint32_t* runs, const uint32_t* top_base,
                               const uint32_t* top_hist, void* scratch, uint32_t* counters,
                               const uint32_t* gate, uint32_t* status, cudaStream_t s) {
  constexpr int smem = sizeof(uint32_t) * (kMsdWords + kMsdStage);
  const cudaError_t e = set_smem_limit(msd_bucket_kernel, smem);
  if (e != cudaSuccess) return e;
  // one CTA fits an SM
  return launch_chained(msd_bucket_kernel, dim3(device_sm_count()), dim3(kMsdThreads), smem, s,
                        keys, runs, top_base, top_hist, msd_scratch(scratch), counters, gate,
                        status);
}

cudaError_t launch_msd_pack(const uint32_t* runs, int n, uint32_t* codes_out, int* d_unique,
                            void* scratch, void* tree_scratch, const uint32_t* gate,
                            cudaStream_t s) {
  const MsdScratch M = msd_scratch(scratch);
  const TreeScratch S = tree_scratch_carve(tree_scratch, n);
  cudaError_t e =
      launch_chained(msd_pack_scan_kernel, dim3(1), dim3(1024), 0, s, M, d_unique, S, gate);
  if (e != cudaSuccess) return e;
  return launch_chained(msd_pack_kernel, dim3(kMsdMaxItems), dim3(kPackThreads), 0, s, runs, M,
                        d_unique, codes_out, S, gate);
}

}  // namespace octgb

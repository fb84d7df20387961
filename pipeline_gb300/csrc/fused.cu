// The whole build of a small or medium cloud as one cooperative launch.
//
// Launched stage by stage, such a build is a chain of some twenty kernels of
// 2 to 17 us that each leave most of the chip idle: launches, tail waits and
// latencies, not work. Here one grid of at most one CTA per SM runs the stages
// as phases with a grid barrier between them (1 to 2 us; up to eight CTAs are
// one cluster with its hardware barrier, about half that). Launched on a
// stream, before and after: 130 -> 33 us at 4,096 uniform points, 147 -> 47 at
// a lidar frame of 122,880, 188 -> 103 at 1,048,576, 228 -> 162 at 1.8M. What
// is left is the phases' latencies (2 to 4 us each) up to some 100,000 points
// and the half-full SMs after that. The limit of 12,288 points per SM leaves
// a quarter of the sort's 16,384 codes for the bucket that straddles the end
// of a CTA's share; the build is still the faster one there.
//
//   codes    each CTA's points to Morton codes, kept in registers; a code
//            equal to the one before it in its warp is dropped (only unique
//            codes are needed, and scan-ordered clouds repeat them in runs);
//            counts per top-12-bit bucket, the CTA's place in each bucket
//            taken from the global count's atomic add
//   scatter  bucket bases (every CTA scans the 4,096 counts), the codes to
//            their buckets
//   cut      only when a bucket holds far more codes than a CTA's share (a cloud
//            in a small part of its box): such buckets are cut by further bits,
//            and the codes counted again before they are scattered
//   sort     a CTA takes the buckets that start in its share of the codes:
//            sorted in shared memory and made unique; a bucket too large for
//            that (few values then) by a bitmap, which takes any number of codes
//   codes    every run to its place (a scan of the CTAs' counts), the deltas
//            of adjacent codes and the tiles' smallest
//   tree     tree_nodes_tile, one tile per CTA (1,024 positions at least)
//   prefix   prefix_slots_tile over the same tiles, each CTA summing the tile
//            sums before its own
//   emit, finalize  emit_slots per radix node, finalize_slots per slot
//
// The outputs are those of the tiled kernels, byte for byte.
//
// Grid barriers are bounded like every other wait: a CTA that gives up raises
// OCT_STATUS_SPIN_TIMEOUT and returns, and so do the others in turn. Memory
// that the kernel itself wrote is read through plain loads only (no
// read-only-cache loads): the barrier's acquire makes it visible.
#include <algorithm>

#include "octree.cuh"
#include "smem_sort.cuh"
#include "tree_tile.cuh"

namespace octgb {

constexpr int kFuThreads = 1024;
constexpr int kFuWarps = kFuThreads / 32;
constexpr int kFuItems = 16;                       // codes per thread at most
constexpr int kFuCap = kFuThreads * kFuItems;      // codes a CTA sorts in shared memory
constexpr int kFuShare = 12288;                    // codes per CTA at most (the rest is slack)
constexpr int kFuBucketBits = 12;
constexpr int kFuBuckets = 1 << kFuBucketBits;
constexpr int kFuSpanBits = 30 - kFuBucketBits;    // values of a bucket: a 32 KiB bitmap
// Codes from which a bucket is cut. A bucket that is not costs its CTA 1.5 ns for
// each of its unique codes (their stores, and later their places) and up to 47 us
// here; the cut costs a build that takes it 6 (a frame's size) to 12 us (1.9M). With
// it clouds in one such bucket take 49 us (122,880 points), 59 (400,000), 72 (1M) and
// 90 (1.86M) where one CTA took 162, 310, 413 and 537, and the stage-by-stage build
// 150, 154, 164 and 188.
constexpr uint32_t kFuCut = 32768;
constexpr uint32_t kFuUnit = 2048;                 // codes of the parts that even ones give
constexpr int kFuIds = 7168;                       // buckets after the cut, at most
constexpr int kFuTile = 1024;                      // tree and prefix tiles: multiples of this
constexpr int kFuMaxGrid = 256;
constexpr int kFuMaxCluster = 8;                   // the portable cluster size
constexpr int kFuMinPer = 1024;                    // points per CTA at least
static_assert(kFuBuckets + 2 * (kFuMaxGrid * kFuShare / (int)kFuUnit) <= kFuIds,
              "a bucket of c codes has fewer than 2 c / kFuUnit parts");
static_assert(kFuMaxCluster * kFuMinPer <= (int)kFuCut, "a cluster's codes need no cut");

struct FusedLayout {
  size_t misc_off, hist_off, zero_bytes, ids_off, cta_off, keys_off, min_off, sum_off, d_off, tags_off,
      total;
};

static FusedLayout fused_layout(int n, int cap) {
  FusedLayout L{};
  const size_t tiles = ((size_t)n + kFuTile - 1) / kFuTile + 1;
  size_t o = 0;
  auto take = [&](size_t bytes) {
    const size_t at = o;
    o = align_up(o + bytes, 256);
    return at;
  };
  L.misc_off = take(256);
  L.hist_off = take(4 * (size_t)kFuBuckets);
  L.zero_bytes = o;
  L.ids_off = take(4 * (size_t)kFuIds);
  L.cta_off = take(8 * (size_t)kFuMaxGrid);
  L.keys_off = take(4 * (size_t)n);
  L.min_off = take(align_up(tiles, kTtMinBlock));
  L.sum_off = take(4 * tiles);
  L.d_off = take((size_t)n + kFuShare + 512);  // the last tile is read whole
  L.tags_off = take(oct_tags_bytes(cap));
  L.total = o;
  return L;
}

struct FusedArgs {
  const float4* pts;
  int n;
  float min_coord, range;
  GridBarrier bar;
  uint32_t* hist;    // [kFuBuckets] zeroed
  uint32_t* ids;     // [kFuIds] counts after the cut
  uint32_t* status;
  int* max_slot;
  uint32_t* cta_count;  // [grid] unique codes of a CTA's run
  uint32_t* cta_first;  // [grid] its first code
  uint32_t* keys;       // [n] bucketed codes
  TreeScratch S;        // at most one tile per CTA
  TreeOut tree;
  uint32_t* codes;
  int* ps;
  OctArgs oct;
  SlotTags tags;
  int* d_counts;
};

struct FusedSort {
  __align__(16) uint32_t a[kFuCap + kBinPad];
  __align__(16) uint32_t b[kFuCap + kBinPad];
  uint32_t start[kFuIds + 1];  // first position of each bucket
  uint16_t tab[kFuBuckets + 2];  // after a cut: a bucket's first part
  union {
    uint32_t base[kFuIds];  // counts, then the CTA's place in each bucket
    uint32_t aux[kBinAux];
  };
};
// 196 KiB of an SM's 256: the rest is the L1 cache of the tree and octree phases
// (with 228 KiB taken a build of 1M points took 4 us more).
static_assert(sizeof(FusedSort) <= 196 * 1024 - 3072, "leaves the next L1 size");
union FusedSmem {
  FusedSort s;
  TreeSmem<kFuShare, kFuThreads> tree;
  PrefixSmem<kFuThreads, kFuShare / kFuThreads> prefix;
  int nodes[kFuThreads * kNodeWords];
  uint32_t spread[1024];
};

// grid_barrier whose CTAs report a wait that ran out, in counts that CTA 0
// cleared when it started. (Should it get there only after others gave up at the
// first barrier, it waits for them in vain at the second and reports it itself.)
template <bool CLUSTER>
__device__ __forceinline__ bool fused_barrier(const FusedArgs& A, uint32_t phase, int* s_ok) {
  const bool ok = grid_barrier<CLUSTER>(A.bar, phase, s_ok);
  if (!ok && threadIdx.x == 0) {
    raise_status(A.status, kStatusSpinTimeout);
    atomicOr(reinterpret_cast<uint32_t*>(A.d_counts) + 3, kStatusSpinTimeout);
  }
  return ok;
}

// Heads of the sorted keys a[0, cnt) (first of each run of equal keys) to
// dst, in order; returns their number. All threads call it.
__device__ __forceinline__ uint32_t fused_unique(const uint32_t* a, int cnt, uint32_t* dst,
                                                 uint32_t* warp_tot, uint32_t* total) {
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per = ((cnt + kFuWarps - 1) / kFuWarps + 31) & ~31;
  const int seg0 = min(wid * per, cnt), seg1 = min(seg0 + per, cnt);
  const uint32_t mine = heads_emit(a, seg0, seg1, false, 0, nullptr);
  const uint32_t ex = block_exclusive_sum<kFuThreads>(lane == 0 ? mine : 0u, warp_tot, total);
  const uint32_t base = __shfl_sync(kFull, ex, 0);
  heads_emit(a, seg0, seg1, true, base, dst);
  __syncthreads();
  return *total;
}

// First positions of the buckets of counts c (EACH per thread, in order; ex: codes
// before the thread's), added to the CTA's places; in s_cut the CTA's share
// [w0, w1) of the `kept` codes as whole buckets: lo, hi, start of the last.
template <int EACH>
__device__ __forceinline__ void fused_starts(FusedSort& M, const uint32_t (&c)[EACH], uint32_t ex,
                                             uint32_t w0, uint32_t w1, uint32_t kept,
                                             uint32_t* s_cut) {
  const int tid = threadIdx.x;
  if (tid == 0) {
    s_cut[0] = w0 == 0 ? 0u : kept;
    s_cut[1] = kept;
    s_cut[2] = kept;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < EACH; ++k) {
    // a boundary inside or at the end of this bucket moves to its end
    if (ex < w0 && w0 <= ex + c[k]) s_cut[0] = ex + c[k];
    if (ex < w1 && w1 <= ex + c[k]) {
      s_cut[1] = ex + c[k];
      s_cut[2] = ex;
    }
    M.start[EACH * tid + k] = ex;
    M.base[EACH * tid + k] += ex;
    ex += c[k];
  }
  if (tid == kFuThreads - 1) M.start[EACH * kFuThreads] = ex;
  __syncthreads();
}

// Bucket of code k after a cut, and the bits of its values.
__device__ __forceinline__ uint32_t fused_part(const FusedSort& M, uint32_t k, int& bits) {
  const uint32_t b = k >> kFuSpanBits, t = M.tab[b], n = M.tab[b + 1u] - t;  // a power of two
  bits = kFuSpanBits - (31 - __clz(n));
  return t + ((k >> bits) & (n - 1u));
}

// Sorted unique codes of a bucket of any size by bitmap (bm: 2^bits bits of
// shared memory, bits >= 5), over the front of its own range keys[0, cnt).
__device__ uint32_t fused_bitmap_bucket(uint32_t* keys, uint32_t cnt, int bits, uint32_t* bm,
                                        uint32_t* warp_tot, uint32_t* total) {
  const int words = 1 << (bits - 5);
  const int per = (words + kFuThreads - 1) / kFuThreads;
  const uint32_t mask = (1u << bits) - 1u;
  const int tid = threadIdx.x;
  for (int w = tid; w < words; w += kFuThreads) bm[w] = 0u;
  const uint32_t top = keys[0] & ~mask;
  __syncthreads();
  for (uint32_t i0 = tid; i0 < cnt; i0 += 4 * kFuThreads) {
    uint32_t k[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t i = i0 + (uint32_t)q * kFuThreads;
      k[q] = i < cnt ? keys[i] & mask : 0xffffffffu;
    }
    uint32_t seen[4];  // (a value that comes often would be a chain of atomics)
#pragma unroll
    for (int q = 0; q < 4; ++q)
      seen[q] = k[q] != 0xffffffffu ? *(volatile uint32_t*)&bm[k[q] >> 5] : 0xffffffffu;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (!(seen[q] >> (k[q] & 31u) & 1u)) atomicOr(&bm[k[q] >> 5], 1u << (k[q] & 31u));
  }
  __syncthreads();
  const int w0 = min(tid * per, words), w1 = min(w0 + per, words);
  uint32_t own = 0;
#pragma unroll 8
  for (int w = w0; w < w1; ++w) own += __popc(bm[w]);
  uint32_t pos = block_exclusive_sum<kFuThreads>(own, warp_tot, total);
#pragma unroll 1
  for (int w = w0; w < w1; ++w) {
    uint32_t set = bm[w];
    while (set) {
      const int bit = __ffs(set) - 1;
      set &= set - 1u;
      keys[pos++] = top | ((uint32_t)w << 5) | (uint32_t)bit;
    }
  }
  __syncthreads();
  return *total;
}

// CLUSTER: the grid is one cluster, and no bucket is cut.
template <bool CLUSTER>
__global__ void __launch_bounds__(kFuThreads, 1) fused_build_kernel(FusedArgs A) {
  extern __shared__ __align__(16) unsigned char sm_raw[];
  FusedSmem& M = *reinterpret_cast<FusedSmem*>(sm_raw);
  __shared__ uint32_t s_warp[32], s_total;
  __shared__ uint32_t s_cut[4];  // lo, hi, start of the straddling bucket
  __shared__ uint32_t s_off[kFuMaxGrid];
  __shared__ int s_next, s_ok;
  __shared__ bool s_parts;
  const int tid = threadIdx.x, lane = tid & 31;
  const uint32_t G = gridDim.x, cta = blockIdx.x;
  uint32_t phase = 0;

  // ---- codes and bucket counts
  if (cta == 0 && tid < 4) A.d_counts[tid] = 0;
  if (tid == 0) s_parts = false;  // (barriers follow)
  const int per = (int)(((uint32_t)A.n + G - 1u) / G);
  const int t0 = (int)min((long long)cta * per, (long long)A.n), t1 = min(t0 + per, A.n);
  uint32_t code[kFuItems];
  uint32_t rank2[kFuItems / 2];  // 16-bit ranks in the bucket, 0xffff: dropped
  {
    uint32_t* cnt = M.s.base;
    uint32_t* lut = M.spread;
    for (int b = tid; b < kFuBuckets; b += kFuThreads) cnt[b] = 0u;
    if (CLUSTER) {  // no memset was launched
      for (int b = (int)cta * kFuThreads + tid; b < kFuBuckets; b += (int)G * kFuThreads)
        A.hist[b] = 0u;
      if (cta == 0 && tid == 0) {
        *A.status = 0u;
        *A.max_slot = 0;
      }
    }
    for (int b = (int)cta * kFuThreads + tid; !CLUSTER && b < kFuIds; b += (int)G * kFuThreads)
      A.ids[b] = 0u;
    fill_spread_lut(lut);
    // tile sums and minima start empty (used three barriers later)
    const int pad = (int)align_up((size_t)A.S.tiles, kTtMinBlock);
    for (int k = (int)cta * kFuThreads + tid; k < pad; k += (int)G * kFuThreads) {
      A.S.tile_min[k] = (uint8_t)kTtAbsent;
      if (k < A.S.tiles) A.S.tile_sum[k] = 0;
    }
    __syncthreads();
    const float scale = __fdiv_rn(1024.0f, A.range);
    bool bad = false;
#pragma unroll
    for (int h = 0; h < kFuItems; h += 4) {
      if (h * kFuThreads < per) {
        float4 p[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = t0 + (h + u) * kFuThreads + tid;
          if (i < t1) p[u] = ld_stream_f4(A.pts + i);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = t0 + (h + u) * kFuThreads + tid;
          uint32_t c = 0, r = 0xffffu;
          if (i < t1) {
            bool ok;
            c = morton_code_lut(p[u].x, p[u].y, p[u].z, A.min_coord, A.range, scale, lut, ok);
            bad |= !ok;
          }
          // the valid lanes are a prefix of the warp
          const uint32_t prev = __shfl_up_sync(kFull, c, 1);
          if (i < t1 && (lane == 0 || prev != c)) r = atomicAdd(&cnt[c >> kFuSpanBits], 1u);
          code[h + u] = c;
          if (u & 1) rank2[(h + u) / 2] |= r << 16;
          else rank2[(h + u) / 2] = r;
        }
      }
    }
    const bool any_bad = __syncthreads_or(bad);
    if (CLUSTER) fused_barrier<CLUSTER>(A, 0, &s_ok);  // the counts are cleared
    if (any_bad && tid == 0) raise_status(A.status, kStatusRange);
    // the CTA's place in each bucket
#pragma unroll
    for (int k = 0; k < kFuBuckets / kFuThreads; ++k) {
      const int b = k * kFuThreads + tid;
      const uint32_t c = cnt[b];
      if (c) cnt[b] = atomicAdd(A.hist + b, c);
    }
  }
  if (!fused_barrier<CLUSTER>(A, ++phase, &s_ok)) return;

  // ---- scatter into buckets; this CTA's share of them
  uint32_t lo, hi, cut, share;
  bool parts;  // (the same in every CTA: all read the same counts)
  {
    constexpr int kPer = kFuBuckets / kFuThreads;
    static_assert(kPer == 4, "one 16-byte load of counts per thread");
    const uint4 q = reinterpret_cast<const uint4*>(A.hist)[tid];
    const uint32_t c[kPer] = {q.x, q.y, q.z, q.w};
    if (max(max(c[0], c[1]), max(c[2], c[3])) > kFuCut) s_parts = true;
    const uint32_t ex =
        block_exclusive_sum<kFuThreads>(c[0] + c[1] + c[2] + c[3], s_warp, &s_total);
    const uint32_t kept = s_total;
    share = (kept + G - 1u) / G;
    const uint32_t w0 = min(cta * share, kept), w1 = min(w0 + share, kept);
    parts = !CLUSTER && s_parts;  // (the sum's barriers)
    if (!parts) {
      fused_starts(M.s, c, ex, w0, w1, kept, s_cut);
    } else {
      uint32_t sub[kPer], mine = 0;
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        sub[k] = 0;
        if (c[k] > kFuCut)
          while ((kFuUnit << sub[k]) < c[k]) ++sub[k];
        mine += 1u << sub[k];
      }
      uint32_t id = block_exclusive_sum<kFuThreads>(mine, s_warp, &s_total);
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        M.s.tab[kPer * tid + k] = (uint16_t)id;
        id += 1u << sub[k];
      }
      if (tid == kFuThreads - 1) M.s.tab[kFuBuckets] = (uint16_t)id;
      for (int b = tid; b < kFuIds; b += kFuThreads) M.s.base[b] = 0u;
      __syncthreads();
#pragma unroll
      for (int it = 0; it < kFuItems; ++it) {
        if (it * kFuThreads >= per) break;
        const int sh = 16 * (it & 1);
        if (((rank2[it / 2] >> sh) & 0xffffu) != 0xffffu) {
          int bits;
          const uint32_t r = atomicAdd(&M.s.base[fused_part(M.s, code[it], bits)], 1u);
          rank2[it / 2] = (rank2[it / 2] & ~(0xffffu << sh)) | r << sh;
        }
      }
      __syncthreads();
      for (int b = tid; b < kFuIds; b += kFuThreads) {
        const uint32_t n = M.s.base[b];
        if (n) M.s.base[b] = atomicAdd(A.ids + b, n);
      }
      if (!fused_barrier<CLUSTER>(A, ++phase, &s_ok)) return;
      constexpr int kEach = kFuIds / kFuThreads;
      uint32_t p[kEach], sum = 0;
#pragma unroll
      for (int k = 0; k < kEach; ++k) {
        p[k] = A.ids[kEach * tid + k];
        sum += p[k];
      }
      fused_starts(M.s, p, block_exclusive_sum<kFuThreads>(sum, s_warp, &s_total), w0, w1, kept,
                   s_cut);
    }
    lo = s_cut[0];
    hi = max(s_cut[1], lo);
    cut = max(s_cut[2], lo);
    auto scatter = [&](auto bucket_of) {
#pragma unroll
      for (int it = 0; it < kFuItems; ++it) {
        if (it * kFuThreads >= per) break;
        const uint32_t r = (rank2[it / 2] >> (16 * (it & 1))) & 0xffffu;
        if (r != 0xffffu) A.keys[M.s.base[bucket_of(code[it])] + r] = code[it];
      }
    };
    if (parts)
      scatter([&](uint32_t k) {
        int bits;
        return fused_part(M.s, k, bits);
      });
    else
      scatter([](uint32_t k) { return k >> kFuSpanBits; });
  }
  if (!fused_barrier<CLUSTER>(A, ++phase, &s_ok)) return;

  // ---- sort and unique: [lo, cut) with the straddling bucket [cut, hi), which
  // goes alone by bitmap (a few us whatever it holds) when it is large beside
  // the CTA's share or both do not fit
  const uint32_t* run;
  uint32_t u_small, u_big = 0;
  {
    const bool big = hi - lo > (uint32_t)kFuCap ||
                     (hi - cut > 2u * (uint32_t)kFuThreads && hi - cut > 2u * share);
    const int cnt = (int)min((big ? cut : hi) - lo, (uint32_t)kFuCap);
    // every bucket has as many bins as codes, spread evenly over its values
    auto place_in = [&](uint32_t b, uint32_t part, uint32_t& into) {
      const uint32_t s = M.s.start[b], c = M.s.start[b + 1] - s;
      into = part * c;
      return s - lo + __umulhi(part, c);
    };
    auto sort = [&](auto place_of) {
      return smem_bin_sort<kFuWarps, kFuItems>(A.keys + lo, cnt, M.s.a, M.s.b, M.s.aux, s_warp,
                                               &s_total, s_cut, place_of);
    };
    // (two sorts: one that asks for every code costs 5 us of 104 at 1M points)
    uint32_t* sorted =
        parts ? sort([&](uint32_t k, uint32_t& into) {
          int bits;
          const uint32_t b = fused_part(M.s, k, bits);
          return place_in(b, k << (32 - bits), into);
        })
              : sort([&](uint32_t k, uint32_t& into) {
                  return place_in(k >> kFuSpanBits, k << (32 - kFuSpanBits), into);
                });
    uint32_t* other = sorted == M.s.a ? M.s.b : M.s.a;
    u_small = fused_unique(sorted, cnt, other, s_warp, &s_total);
    run = other;
    __syncthreads();
    if (big) {
      int bits = kFuSpanBits;
      if (parts) fused_part(M.s, A.keys[cut], bits);
      u_big = fused_bitmap_bucket(A.keys + cut, hi - cut, bits, sorted, s_warp, &s_total);
    }
    if (tid == 0) {
      A.cta_count[cta] = u_small + u_big;
      A.cta_first[cta] = u_small ? run[0] : u_big ? A.keys[cut] : 0u;
    }
  }
  if (!fused_barrier<CLUSTER>(A, ++phase, &s_ok)) return;

  // ---- unique codes and deltas to their places
  int n_unique, tile;
  {
    const uint32_t mine = tid < (int)G ? A.cta_count[tid] : 0u;
    uint32_t* tmin = M.s.base;  // smallest deltas of the tiles this run touches
    for (int k = tid; k < kFuBuckets; k += kFuThreads) tmin[k] = kTtAbsent;
    if (tid == 0) s_next = 0x7fffffff;
    const uint32_t ex = block_exclusive_sum<kFuThreads>(mine, s_warp, &s_total);
    if (tid < (int)G) s_off[tid] = ex;
    if (tid < (int)G && tid > (int)cta && mine > 0) atomicMin(&s_next, tid);
    __syncthreads();
    n_unique = (int)s_total;
    // one tile per CTA where that fills the chip
    tile = (int)((s_total + G * kFuTile - 1u) / (G * kFuTile)) * kFuTile;
    const uint32_t off = s_off[cta], u = u_small + u_big;
    const uint32_t after = s_next < (int)G ? A.cta_first[s_next] : 0u;
    const uint32_t* far = A.keys + cut;
    auto at = [&](uint32_t j) { return j < u_small ? run[j] : far[j - u_small]; };
    const uint32_t t_first = off / (uint32_t)tile;
    uint32_t ta = t_first, ta_end = (t_first + 1u) * (uint32_t)tile;
    for (uint32_t j0 = tid & ~31u; j0 < u; j0 += kFuThreads) {
      const uint32_t j = j0 + lane;
      uint32_t d = kTtAbsent;
      const uint32_t pos = off + j;
      if (j < u) {
        const uint32_t c = at(j);
        A.codes[pos] = c;
        if (pos + 1u < (uint32_t)n_unique) {
          d = tt_delta(c, j + 1u < u ? at(j + 1u) : after);
          A.S.D[pos] = (uint8_t)d;
        }
      }
      // the warp's 32 positions lie in one tile or two
      while (off + j0 >= ta_end) {
        ++ta;
        ta_end += (uint32_t)tile;
      }
      const uint32_t ma = __reduce_min_sync(kFull, pos < ta_end ? d : kTtAbsent);
      const uint32_t mb = __reduce_min_sync(kFull, pos < ta_end ? kTtAbsent : d);
      if (lane == 0 && ma < kTtAbsent) atomicMin(&tmin[ta - t_first], ma);
      if (lane == 0 && mb < kTtAbsent) atomicMin(&tmin[ta + 1u - t_first], mb);
    }
    __syncthreads();
    const uint32_t touched = u ? (off + u - 1u) / (uint32_t)tile - t_first + 1u : 0u;
    for (uint32_t k = tid; k < touched; k += kFuThreads)
      if (tmin[k] < kTtAbsent) atomic_min_u8(A.S.tile_min + t_first + k, tmin[k]);
  }
  if (!fused_barrier<CLUSTER>(A, ++phase, &s_ok)) return;

  // ---- radix tree and edge counts
  const int n_brt = max(n_unique - 1, 0);
  const int tiles = (n_brt + tile - 1) / tile;  // at most one per CTA
  if ((int)cta < tiles) {
    const TileInfo I{(int)cta, 0, tiles - 1, n_brt, (int)cta * tile, 0};
    tree_nodes_tile(M.tree, SizedTile{tile}, I, A.codes, A.S, A.tree);
  }
  if (!fused_barrier<CLUSTER>(A, ++phase, &s_ok)) return;

  // ---- prefix sums, octree tags
  if ((int)cta < tiles) {
    const uint32_t sum = tid < (int)cta ? (uint32_t)A.S.tile_sum[tid] : 0u;
    block_exclusive_sum<kFuThreads>(sum, s_warp, &s_total);
    const uint32_t before = s_total;
    __syncthreads();
    prefix_slots_tile(M.prefix, A.tree.ec, A.ps, n_brt, (int)cta * tile, before, A.tags,
                      A.max_slot, tile / kFuThreads);
    if (tid == 0) bulk_wait_all();
  }
  if (!fused_barrier<CLUSTER>(A, ++phase, &s_ok)) return;

  // ---- octree
  const int n_oct = n_brt >= 1 ? *A.max_slot + 1 : 0;
  const bool octree = A.oct.cap > 0;
  const bool fits = n_oct <= A.oct.cap;
  if (octree) {
    if (!fits) {
      if (cta == 0 && tid == 0) raise_status(A.status, kStatusCapacity);
    } else {
      for (int i = (int)cta * kFuThreads + tid; i < n_brt; i += (int)G * kFuThreads)
        emit_slots(i, A.oct, A.tags, n_brt, n_oct);
    }
    if (!fused_barrier<CLUSTER>(A, ++phase, &s_ok)) return;
  }
  if (cta == 0 && tid == kFuThreads - 1) {  // every status bit is up
    A.d_counts[0] = n_unique;
    A.d_counts[1] = n_brt;
    A.d_counts[2] = n_oct;
    atomicOr(A.d_counts + 3, (int)*reinterpret_cast<volatile uint32_t*>(A.status));
  }
  if (octree) {
    if (fits && n_brt >= 1) {
      const int root_level = A.tree.prefix_n[0] / 3;
      for (int blk = (int)cta * kFuThreads; blk < n_oct; blk += (int)G * kFuThreads) {
        const int p = blk + tid;
        if (p < n_oct)
          finalize_slots(p, A.oct, A.tags, n_brt, root_level, M.nodes + tid * kNodeWords);
        store_node_block(M.nodes, A.oct.nodes + blk, min(kFuThreads, n_oct - blk));
      }
      if (tid == 0) bulk_wait_all();
    }
  }
}

size_t fused_workspace_bytes(int n, int cap) { return fused_layout(n, cap).total; }

static int fused_grid(int n) {
  return std::max(1, std::min((n + kFuMinPer - 1) / kFuMinPer,
                              std::min(device_sm_count(), kFuMaxGrid)));
}
bool fused_is_cluster(int n) { return fused_grid(n) <= kFuMaxCluster; }

int fused_max_points() { return device_sm_count() * kFuShare; }

cudaError_t launch_fused_build(const float4* pts, int n, float min_coord, float range,
                               uint32_t* codes, const OctArgs& oct, int* ec, int* ps,
                               int* d_counts, void* workspace, cudaStream_t s,
                               const GridBarrier* bar) {
  const FusedLayout L = fused_layout(n, oct.cap);
  char* w = static_cast<char*>(workspace);
  const int grid = fused_grid(n);
  FusedArgs A{};
  A.pts = pts;
  A.n = n;
  A.min_coord = min_coord;
  A.range = range;
  A.status = reinterpret_cast<uint32_t*>(w + L.misc_off);
  A.bar = bar ? *bar : GridBarrier{nullptr, 0u, kWaitLimitNs};
  A.bar.arrivals = A.status + 1;
  A.max_slot = reinterpret_cast<int*>(A.status + 2);
  A.hist = reinterpret_cast<uint32_t*>(w + L.hist_off);
  A.ids = reinterpret_cast<uint32_t*>(w + L.ids_off);
  A.cta_count = reinterpret_cast<uint32_t*>(w + L.cta_off);
  A.cta_first = A.cta_count + kFuMaxGrid;
  A.keys = reinterpret_cast<uint32_t*>(w + L.keys_off);
  A.S.D = reinterpret_cast<uint8_t*>(w + L.d_off);
  A.S.tile_min = reinterpret_cast<uint8_t*>(w + L.min_off);
  A.S.tile_sum = reinterpret_cast<int*>(w + L.sum_off);
  A.S.tiles = (n + kFuTile - 1) / kFuTile;
  A.tree = TreeOut{const_cast<uint8_t*>(oct.prefix_n), const_cast<uint8_t*>(oct.hll),
                   const_cast<uint8_t*>(oct.hlr), const_cast<int*>(oct.left_child),
                   const_cast<int*>(oct.parent), ec};
  A.codes = codes;
  A.ps = ps;
  A.oct = oct;
  A.tags = slot_tags(oct_tags_carve(w + L.tags_off, oct.cap), 0, oct.cap);
  A.d_counts = d_counts;
  const int smem = (int)sizeof(FusedSmem);
  const bool cluster = fused_is_cluster(n);
  auto kernel = cluster ? fused_build_kernel<true> : fused_build_kernel<false>;
  cudaError_t e = set_smem_limit(kernel, smem);
  if (e != cudaSuccess) return e;
  if (!cluster) e = cudaMemsetAsync(w + L.misc_off, 0, L.zero_bytes, s);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(kFuThreads);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at[1];
  if (cluster) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {(unsigned)grid, 1u, 1u};
  } else {
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
  }
  c.attrs = at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, A);
}

}  // namespace octgb

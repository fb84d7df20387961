// Second half of a batched build's sort (stage 2: k_SimpleRadixSort per cloud,
// reference kernels/02_sort.cpp:13-58): the keys of every cloud lie in its
// top-digit buckets (2^20 values each, in any order) and are brought in order.
//
// One launch in place of two stable digit passes (tile histogram, scan, ranked
// scatter each): a key moves once more instead of twice, and its place comes
// from smem_bin_sort instead of ballots. Two CTAs of 512 threads per SM take
// units, even stretches of at most kBatchUnit positions of a cloud, from a
// counter: the buckets that start in a unit, as many at a time as fit shared
// memory. A bucket that does not fit (bs_large) is the CTA's in whose unit it
// starts: its keys are counted and scattered by eight further bits, and the parts
// sorted where they then lie; a part that still does not fit has its 2^12 values
// counted. That takes some 90 us for 49,152 keys, which is why batch_build keeps
// larger clouds, whose buckets may be as large, to digit passes.
#include "kernels.cuh"
#include "smem_sort.cuh"

namespace octgb {

constexpr int kBsThreads = 512;
constexpr int kBsWarps = kBsThreads / 32;
constexpr int kBsItems = 16;
constexpr uint32_t kBsCap = kBsThreads * kBsItems;  // keys a CTA sorts in shared memory
constexpr int kBsBuckets = 1024;
constexpr int kBsSpan = 20;  // key bits below the top digit
constexpr int kBsPartBits = 8;
constexpr int kBsParts = 1 << kBsPartBits;
constexpr int kBsPartSpan = kBsSpan - kBsPartBits;

struct BsSmem {
  __align__(16) uint32_t a[kBsCap + kBinPad];
  __align__(16) uint32_t b[kBsCap + kBinPad];
  uint32_t aux[kBinAux];
  uint32_t start[kBsBuckets + 1];  // the cloud's buckets
  uint32_t part[kBsParts + 1];     // the parts of a large bucket
  uint32_t warp[32];
  uint32_t total, span[2], next[2];
};
static_assert((1 << kBsPartSpan) <= kBsCap, "a part's values fit a key array");

// f(key) for the keys of src[0, cnt), whole warps (0xffffffff past the end).
template <class F>
__device__ __forceinline__ void bs_each(const uint32_t* src, uint32_t cnt, F f) {
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t i0 = threadIdx.x & ~31u; i0 < cnt; i0 += 4 * kBsThreads) {
    uint32_t k[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t i = i0 + (uint32_t)q * kBsThreads + lane;
      k[q] = i < cnt ? src[i] : 0xffffffffu;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) f(k[q]);
  }
}

// keys[0, cnt) in global memory, whose bins follow `start` over values of `span`
// bits below bucket id_of(key), in order to dst (keys or elsewhere). lo: start's
// value at the first key.
template <class IdOf>
__device__ __forceinline__ void bs_sort(BsSmem& M, const uint32_t* keys, uint32_t cnt,
                                        const uint32_t* start, uint32_t lo, int span, IdOf id_of,
                                        uint32_t* dst) {
  auto place_of = [&](uint32_t k, uint32_t& into) {
    const uint32_t i = id_of(k), s = start[i], c = start[i + 1] - s, part = k << (32 - span);
    into = part * c;
    return s - lo + __umulhi(part, c);
  };
  const uint32_t* sorted = smem_bin_sort<kBsWarps, kBsItems>(
      keys, (int)cnt, M.a, M.b, M.aux, M.warp, &M.total, M.span, place_of);
  for (uint32_t j = threadIdx.x; j < cnt; j += kBsThreads) dst[j] = sorted[j];
  __syncthreads();
}

// A bucket that does not fit: src[0, cnt) scattered to dst by eight further
// bits, the parts sorted in place.
__device__ __noinline__ void bs_large(BsSmem& M, const uint32_t* src, uint32_t* dst,
                                      uint32_t cnt) {
  const uint32_t tid = threadIdx.x;
  auto part_of = [](uint32_t k) { return (k >> kBsPartSpan) & (uint32_t)(kBsParts - 1); };
  uint32_t* cursor = M.a;
  cursor[tid] = 0u;
  __syncthreads();
  bs_each(src, cnt, [&](uint32_t k) { warp_count(cursor, k == 0xffffffffu ? k : part_of(k)); });
  __syncthreads();
  smem_exclusive_rows<kBsWarps>(cursor, 1, M.warp, &M.total);
  if (tid <= (uint32_t)kBsParts) M.part[tid] = tid < (uint32_t)kBsParts ? cursor[tid] : cnt;
  __syncthreads();
  bs_each(src, cnt, [&](uint32_t k) {
    if (k != 0xffffffffu) dst[atomicAdd(&cursor[part_of(k)], 1u)] = k;
  });
  __syncthreads();
  for (int i = 0; i < kBsParts;) {
    const uint32_t at = M.part[i];
    int e = first_at_least(M.part, i + 1, kBsParts + 1, at + kBsCap + 1u) - 1;
    e = max(e, i + 1);
    const uint32_t n = M.part[e] - at;
    if (n > kBsCap) {
      constexpr uint32_t kValues = 1u << kBsPartSpan;
      for (uint32_t v = tid; v < kValues; v += kBsThreads) M.a[v] = 0u;
      const uint32_t top = dst[at] & ~(kValues - 1u);
      __syncthreads();
      bs_each(dst + at, n, [&](uint32_t k) {
        warp_count(M.a, k == 0xffffffffu ? k : k & (kValues - 1u));
      });
      __syncthreads();
      smem_emit_counts<kBsWarps>(M.a, kValues, kValues, n, top, dst + at, M.warp, &M.total);
    } else if (n > 0) {
      bs_sort(M, dst + at, n, M.part, at, kBsPartSpan, part_of, dst + at);
    }
    i = e;
  }
}

// units: {lo, hi, cloud, 0}; base: [clouds][1024] bucket starts; start: the
// clouds' ([clouds + 1]); next: a zeroed word.
__global__ void __launch_bounds__(kBsThreads, 2)
    batch_bucket_sort_kernel(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst,
                             const int4* __restrict__ units, int n_units,
                             const uint32_t* __restrict__ base, const int* __restrict__ start,
                             uint32_t* next, const uint32_t* __restrict__ gate) {
  if (gate && *gate == 0u) return;
  extern __shared__ __align__(16) unsigned char sm_raw[];
  BsSmem& M = *reinterpret_cast<BsSmem*>(sm_raw);
  const int tid = threadIdx.x;
  int cloud = -1;
  uint32_t u = blockIdx.x;
  // (the next unit's number is fetched while one is worked on)
  for (int turn = 0; u < (uint32_t)n_units; turn ^= 1) {
    if (tid == 0) M.next[turn] = gridDim.x + atomicAdd(next, 1u);
    const int4 t = units[u];
    if (t.z != cloud) {
      cloud = t.z;
      for (int k = tid; k < kBsBuckets; k += kBsThreads)
        M.start[k] = base[(size_t)cloud * kBsBuckets + k];
      if (tid == 0) M.start[kBsBuckets] = (uint32_t)start[cloud + 1];
      __syncthreads();
    }
    const uint32_t lo = (uint32_t)t.x, hi = (uint32_t)t.y;
    int i = first_at_least(M.start, 0, kBsBuckets, lo);
    const int end = first_at_least(M.start, i, kBsBuckets, hi);
    while (i < end) {
      const uint32_t at = M.start[i];
      int e = first_at_least(M.start, i + 1, end + 1, at + kBsCap + 1u) - 1;
      e = min(max(e, i + 1), end);
      const uint32_t n = M.start[e] - at;
      if (n > kBsCap)
        bs_large(M, src + at, dst + at, n);
      else if (n > 0)
        bs_sort(M, src + at, n, M.start, at, kBsSpan,
                [](uint32_t k) { return k >> kBsSpan; }, dst + at);
      i = e;
    }
    __syncthreads();
    u = M.next[turn];
  }
}

cudaError_t launch_batch_bucket_sort(const uint32_t* src, uint32_t* dst, const int4* units,
                                     int n_units, const uint32_t* base, const int* start,
                                     uint32_t* next, const uint32_t* gate, cudaStream_t s) {
  if (n_units <= 0) return cudaSuccess;
  const int smem = (int)sizeof(BsSmem);
  const cudaError_t e = set_smem_limit(batch_bucket_sort_kernel, smem);
  if (e != cudaSuccess) return e;
  const int grid = n_units < 2 * device_sm_count() ? n_units : 2 * device_sm_count();
  batch_bucket_sort_kernel<<<grid, kBsThreads, smem, s>>>(src, dst, units, n_units, base, start,
                                                          next, gate);
  return cudaGetLastError();
}

}  // namespace octgb

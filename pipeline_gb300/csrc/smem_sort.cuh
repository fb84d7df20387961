// Shared-memory sorting of one CTA's keys: the bucket kernels of the learned
// sort and the fused build.
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

// Stable LSD radix sort of a[0, cnt) (cnt <= WARPS * 32 * ITEMS, WARPS * 32
// threads) on the low `bits` bits of key - kmin, 8-bit digits, ping-pong
// between a and b. Warp w ranks its contiguous ITEMS * 32 keys at most with ballot multi-split (peers = lanes
// with the same digit), so ties keep input order. Returns the sorted array.
template <int WARPS, int ITEMS>
__device__ uint32_t* smem_radix_sort(uint32_t* a, uint32_t* b, int cnt, uint32_t kmin, int bits,
                                     RadixSmem<WARPS>& S) {
  constexpr int kThreads = WARPS * 32;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const uint32_t lt = lanemask_lt();
  // every warp takes `items` rows of 32 keys (the last warps may be partial)
  const int items = (cnt + WARPS * 32 - 1) / (WARPS * 32);
  const int seg = items * 32;
  // peers from two 4-bit half-digit equality tables (lane v: lanes whose half
  // equals v), fetched by shuffle
  constexpr int kHalf = kRsBits / 2;
  uint32_t lane_bits[kHalf];
#pragma unroll
  for (int b = 0; b < kHalf; ++b) lane_bits[b] = 0u - ((uint32_t)(lane >> b) & 1u);
  for (int shift = 0; shift < bits; shift += kRsBits) {
    for (int k = tid; k < WARPS * kRsBins / 2; k += kThreads)
      reinterpret_cast<uint32_t*>(S.whist)[k] = 0;
    __syncthreads();
    uint32_t rk[ITEMS / 2];  // two 16-bit ranks per register; keys are re-read
    uint16_t* wh = S.whist[wid];
    if (shift == 0) {
      // The first pass needs no stability (the bucket's keys arrive in any
      // order): a shared-memory atomic on the warp's 16-bit digit counter
      // (the upper or lower half of its 32-bit word; a warp counts at most
      // ITEMS * 32 keys, so no carry reaches the other half) ranks a key.
      uint32_t* wh32 = reinterpret_cast<uint32_t*>(wh);
#pragma unroll
      for (int it = 0; it < ITEMS; ++it) {
        if (it >= items) break;
        const int idx = wid * seg + it * 32 + lane;
        uint32_t r = 0;
        if (idx < cnt) {
          const uint32_t dg = (a[idx] - kmin) & (kRsBins - 1);
          const uint32_t sh = 16u * (dg & 1u);
          r = (atomicAdd(&wh32[dg >> 1], 1u << sh) >> sh) & 0xffffu;
        }
        if (it & 1) rk[it >> 1] |= r << 16;
        else rk[it >> 1] = r;
      }
    } else {
#pragma unroll
      for (int it = 0; it < ITEMS; ++it) {
        if (it >= items) break;
        const int idx = wid * seg + it * 32 + lane;
        const bool valid = idx < cnt;
        const uint32_t key = valid ? a[idx] : 0u;
        const uint32_t dg = ((key - kmin) >> shift) & (kRsBins - 1);
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
        const uint32_t dg = ((key - kmin) >> shift) & (kRsBins - 1);
        const uint32_t r = (rk[it >> 1] >> ((it & 1) * 16)) & 0xffffu;
        b[S.dstart[dg] + S.whist[wid][dg] + r] = key;
      }
    }
    __syncthreads();
    uint32_t* t = a;
    a = b;
    b = t;
  }
  return a;
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

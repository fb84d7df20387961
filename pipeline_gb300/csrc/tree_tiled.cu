// Stage 4 (and stage 5's edge counts) for strictly increasing codes below
// 2^31, from the deltas of adjacent codes.
//
// For such codes the radix tree of k_BuildRadixTree
// (kernels/04_radix_tree.cpp:39-121) is the Cartesian tree of the adjacent
// deltas D[q] = delta(codes[q], codes[q + 1]), q in [0, n): the node whose
// split (gamma) is q covers the codes that share their first D[q] + 1 bits
// with codes[q], i.e. [a + 1, b], where a is the nearest position left of q
// with a smaller delta and b the nearest one right of q (-1 / n when there is
// none). Its index is a + 1 when D[a] > D[b] (it is its parent's right child)
// and b otherwise (the left child). Inside any node's range the smallest delta
// occurs exactly once, so these are the ranges and splits the reference's
// exact searches find. Only radix node 0 differs: the reference starts it at
// d = 1, l = n - 1 (range [0, n - 1]), so its split is the smallest delta of
// [0, n - 2] and its right end is n - 1. When that is not the overall
// smallest delta (the delta at n - 1 is), the root is "short": node n - 1
// covers the same range and the reference's node 0 writes no children's
// parents.
//
// The parent of node i is the node split at a or b, whichever has the larger
// delta, so the edge count prefix_n[i]/3 - prefix_n[parent[i]]/3
// (kernels/05_edge_count.cpp:3-16) is computed here as well.
//
// Kernels over tiles of 4,096 positions:
//   tree_tiles_kernel     D as bytes and each tile's smallest D, from the
//                         codes (learned build, the C entry);
//   unique_count_kernel,  stage 3 of the whole and batched builds: run heads
//   unique_deltas_kernel  of the sorted keys counted per tile and scanned,
//                         then compacted, each unique code also writing D for
//                         the code before it and the tiles' smallest D (per
//                         cloud in the batched build: tile maps OneKeys /
//                         CloudKeys);
//   tree_nodes_kernel     nearest smaller deltas inside each 32-position
//                         chunk from five ballots over the bits of D (one
//                         lane-parallel table of masks per chunk), across the
//                         tile's chunks from prefix / suffix tables in shared
//                         memory, across tiles (rare: only the tile's running
//                         minima) by a peek at the adjacent tile's edge, then
//                         warp-wide scans of the tile minima and of the found
//                         tile's deltas; then every output of the node split
//                         at each position.
#include <climits>

#include "tree_tile.cuh"

namespace octgb {

constexpr int kTtAThreads = 256;
constexpr int kTtBThreads = 512;

static int tt_tiles(int n) { return ((n > 1 ? n : 1) + kTtTile - 1) / kTtTile; }

size_t tree_scratch_bytes_tiles(int tiles) {
  const size_t t = (size_t)(tiles > 1 ? tiles : 1);
  return align_up(t * kTtTile, 256) + align_up(align_up(t, kTtMinBlock), 256) +
         4 * align_up(t * sizeof(int), 256);
}

TreeScratch tree_scratch_carve_tiles(void* base, int tiles) {
  const size_t t = (size_t)(tiles > 1 ? tiles : 1);
  char* p = static_cast<char*>(base);
  TreeScratch S;
  S.tiles = (int)t;
  S.D = reinterpret_cast<uint8_t*>(p);
  p += align_up(t * kTtTile, 256);
  S.tile_min = reinterpret_cast<uint8_t*>(p);
  p += align_up(align_up(t, kTtMinBlock), 256);
  S.tile_sum = reinterpret_cast<int*>(p);
  p += align_up(t * sizeof(int), 256);
  S.tile_prefix = reinterpret_cast<uint32_t*>(p);
  p += align_up(t * sizeof(int), 256);
  S.tile_heads = reinterpret_cast<int*>(p);
  p += align_up(t * sizeof(int), 256);
  S.tile_upos = reinterpret_cast<uint32_t*>(p);
  return S;
}

size_t tree_scratch_bytes(int n) { return tree_scratch_bytes_tiles(tt_tiles(n)); }
TreeScratch tree_scratch_carve(void* base, int n) { return tree_scratch_carve_tiles(base, tt_tiles(n)); }

// One cloud: tile t covers positions [4096 t, 4096 t + 4096).
struct OneCloud {
  int n_host;
  const int* d_unique;
  int tiles;
  __device__ __forceinline__ TileInfo operator()(int t) const {
    TileInfo I;
    I.t = t;
    I.t_first = 0;
    I.t_last = tiles - 1;
    I.n = d_unique ? max(*d_unique - 1, 0) : n_host;
    I.lo = t * kTtTile;
    I.cs = 0;
    return I;
  }
};

// Batched clouds: tile descriptors {first, end, cloud, first tile of cloud}.
struct CloudTiles {
  const int4* tiles;
  const int* start;
  const int* unique_c;
  __device__ __forceinline__ TileInfo operator()(int t) const {
    const int4 d = tiles[t];
    TileInfo I;
    I.t = t;
    I.cs = start[d.z];
    I.t_first = d.w;
    I.t_last = d.w + (start[d.z + 1] - I.cs + kTtTile - 1) / kTtTile - 1;
    I.n = max(unique_c[d.z] - 1, 0);
    I.lo = d.x - I.cs;
    return I;
  }
};

template <class Map>
__global__ void __launch_bounds__(kTtAThreads)
    tree_tiles_kernel(Map map, const uint32_t* __restrict__ codes_all, TreeScratch S) {
  chain_enter();
  constexpr int kWarps = kTtAThreads / 32;
  __shared__ uint32_t s_min[kWarps];
  const TileInfo I = map(blockIdx.x);
  const int n = I.n, t = I.t, t0 = I.lo;
  const uint32_t* codes = codes_all + I.cs;
  uint8_t* Dt = S.D + (size_t)t * kTtTile;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (t == 0) {  // whole blocks of the tile-minimum array; the padding never matches
    const int pad = (int)align_up((size_t)S.tiles, kTtMinBlock);
    for (int k = S.tiles + (int)threadIdx.x; k < pad; k += kTtAThreads)
      S.tile_min[k] = (uint8_t)kTtAbsent;
  }
  uint32_t dmin = kTtAbsent;
  if (t0 < n) {
    // a thread takes 4 consecutive positions per step: 16-byte code loads,
    // 4-byte delta stores; the code after the fourth comes from the next lane
    const uint4* c4 = reinterpret_cast<const uint4*>(codes);
    const bool vec = (reinterpret_cast<uintptr_t>(codes) & 15) == 0;
    for (int base = t0 + 4 * (int)threadIdx.x; base < t0 + kTtTile; base += 4 * kTtAThreads) {
      uint32_t c[5];
      if (vec && base + 4 <= n + 1) {
        const uint4 v = c4[base >> 2];
        c[0] = v.x;
        c[1] = v.y;
        c[2] = v.z;
        c[3] = v.w;
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) c[k] = base + k <= n ? codes[base + k] : 0u;
      }
      c[4] = __shfl_down_sync(kFull, c[0], 1);
      if (lane == 31) c[4] = base + 4 <= n ? codes[base + 4] : 0u;
      uint32_t packed = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t d = base + k < n ? tt_delta(c[k], c[k + 1]) : kTtAbsent;
        dmin = min(dmin, d);
        packed |= d << (8 * k);
      }
      *reinterpret_cast<uint32_t*>(Dt + (base - t0)) = packed;
    }
  } else {
    for (int k = threadIdx.x; k < kTtTile / 4; k += kTtAThreads)
      reinterpret_cast<uint32_t*>(Dt)[k] = kTtAbsent * 0x01010101u;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dmin = min(dmin, __shfl_xor_sync(kFull, dmin, o));
  if (lane == 0) s_min[warp] = dmin;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t m = kTtAbsent;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) m = min(m, s_min[w]);
    S.tile_min[t] = (uint8_t)m;
    S.tile_sum[t] = 0;
  }
}

template <class Map>
__global__ void __launch_bounds__(kTtBThreads)
    tree_nodes_kernel(Map map, const uint32_t* __restrict__ codes, TreeScratch S, TreeOut o) {
  chain_enter();
  __shared__ TreeSmem<kTtTile, kTtBThreads> M;
  tree_nodes_tile(M, FixedTile<kTtTile>{}, map(blockIdx.x), codes, S, o);
}

// ------------------------------------------------------ unique + deltas --
// A tile's keys stay in registers, a warp taking 16 rows of 32 consecutive
// ones: loads are coalesced at any alignment (a batch's clouds start anywhere),
// a key's predecessor comes by shuffle, run heads are ballots and their places
// population counts, so a row's heads leave as consecutive words with no stage.
// Bound by load latency and the stores. 512-cloud batch (74M keys): count
// 119 -> 66 us, compaction 295 -> 217 us against 16
// consecutive keys per thread staged through shared memory.
constexpr int kUdThreads = 256;
constexpr int kUdWarps = kUdThreads / 32;
constexpr int kUdRows = kTtTile / kUdThreads;  // 16 rows per warp

// A 4,096-key tile of sorted keys: keys [lo, hi) of the cloud starting at cs,
// whose unique codes go to the tree tiles from t_first on.
struct KeyTile {
  int lo, hi, cs, t_first, cloud;
  bool last;  // the cloud's last tile
};

// One cloud of n keys.
struct OneKeys {
  int n;
  __device__ __forceinline__ KeyTile operator()(int t) const {
    KeyTile K;
    K.lo = t * kTtTile;
    K.hi = min(K.lo + kTtTile, n);
    K.cs = 0;
    K.t_first = 0;
    K.cloud = 0;
    K.last = K.hi >= n;
    return K;
  }
};

// Batched clouds: tile descriptors {first, end, cloud, first tile of cloud}.
struct CloudKeys {
  const int4* tiles;
  int n_tiles;
  const int* start;
  __device__ __forceinline__ KeyTile operator()(int t) const {
    const int4 d = tiles[t];
    KeyTile K;
    K.lo = d.x;
    K.hi = d.y;
    K.cs = start[d.z];
    K.t_first = d.w;
    K.cloud = d.z;
    K.last = t == n_tiles - 1 || tiles[t + 1].z != d.z;
    return K;
  }
};

// A warp's rows of a tile: its keys, and the heads of its runs as ballots.
struct WarpRows {
  uint32_t key[kUdRows];
  uint32_t first_prev;  // the key before the warp's first (any value for the cloud's first)
  int j0;               // index of the lane's first key
};
__device__ __forceinline__ void load_rows(WarpRows& R, const uint32_t* __restrict__ keys,
                                          const KeyTile& K) {
  const int lane = threadIdx.x & 31, w0 = K.lo + (int)(threadIdx.x >> 5) * 32 * kUdRows;
  R.j0 = w0 + lane;
  R.first_prev = w0 > K.cs && w0 < K.hi ? ld_now_u32(keys + w0 - 1) : 0u;  // one address per warp
  if (w0 + 32 * kUdRows <= K.hi) {
#pragma unroll
    for (int r = 0; r < kUdRows; ++r) R.key[r] = ld_now_u32(keys + R.j0 + 32 * r);
  } else {
#pragma unroll
    for (int r = 0; r < kUdRows; ++r) {
      const int j = R.j0 + 32 * r;
      R.key[r] = j < K.hi ? keys[j] : 0u;
    }
  }
}
// The lane's predecessor in row r, and the row's heads.
__device__ __forceinline__ uint32_t row_prev(const WarpRows& R, int r) {
  const uint32_t up = __shfl_up_sync(kFull, R.key[r], 1);
  const uint32_t before = r > 0 ? __shfl_sync(kFull, R.key[r > 0 ? r - 1 : 0], 31) : R.first_prev;
  return (threadIdx.x & 31) ? up : before;
}
__device__ __forceinline__ uint32_t row_heads(const WarpRows& R, int r, uint32_t prev,
                                              const KeyTile& K) {
  const int j = R.j0 + 32 * r;
  return __ballot_sync(kFull, j < K.hi && (j == K.cs || R.key[r] != prev));
}

// Run heads of sorted keys per tile; also resets the tree tiles' edge-count
// sums and smallest deltas.
template <class Map>
__global__ void __launch_bounds__(kUdThreads)
    unique_count_kernel(const uint32_t* __restrict__ keys, Map map, int n_tiles, TreeScratch S,
                        const uint32_t* __restrict__ gate) {
  chain_enter();
  if (gate && *gate == 0) return;
  __shared__ int s_cnt[kUdWarps];
  const int tid = threadIdx.x;
  // CTAs walk the tiles (a capped grid: a gated-off launch schedules few CTAs)
  for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
    const KeyTile K = map(t);
    if (t == 0) {
      const int pad = (int)align_up((size_t)S.tiles, kTtMinBlock);
      for (int k = S.tiles + tid; k < pad; k += kUdThreads) S.tile_min[k] = (uint8_t)kTtAbsent;
    }
    if (tid == 0) {
      S.tile_min[t] = (uint8_t)kTtAbsent;
      S.tile_sum[t] = 0;
    }
    WarpRows R;
    load_rows(R, keys, K);
    int cnt = 0;
#pragma unroll
    for (int r = 0; r < kUdRows; ++r) cnt += __popc(row_heads(R, r, row_prev(R, r), K));
    if ((tid & 31) == 0) s_cnt[tid >> 5] = cnt;
    __syncthreads();
    if (tid == 0) {
      int total = 0;
      for (int w = 0; w < kUdWarps; ++w) total += s_cnt[w];
      S.tile_heads[t] = total;
    }
    __syncthreads();  // s_cnt is the next tile's
  }
}

// Compaction from the tile prefixes; each unique code at (cloud) position
// o >= 1 also writes D[o - 1], the delta to the code before it (the last key
// of the previous run), and the tiles' smallest deltas. With unique_c, each
// cloud's last tile writes the cloud's U.
template <class Map>
__global__ void __launch_bounds__(kUdThreads, 4)
    unique_deltas_kernel(const uint32_t* __restrict__ keys, Map map, uint32_t* __restrict__ out,
                         int n_tiles, TreeScratch S, int* __restrict__ unique_c,
                         const uint32_t* __restrict__ gate) {
  chain_enter();
  if (gate && *gate == 0) return;
  __shared__ int s_cnt[2][kUdWarps];
  __shared__ uint32_t s_min[2][2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int turn = 0;
  for (int t = blockIdx.x; t < n_tiles; t += gridDim.x, turn ^= 1) {
    const KeyTile K = map(t);
    if (K.hi <= K.lo) continue;  // uniform in the CTA
    WarpRows R;
    load_rows(R, keys, K);
    const int base = (int)(S.tile_upos[t] - S.tile_upos[K.t_first]);
    int cnt = 0;
#pragma unroll
    for (int r = 0; r < kUdRows; ++r) cnt += __popc(row_heads(R, r, row_prev(R, r), K));
    if (lane == 0) s_cnt[turn][warp] = cnt;
    if (tid < 2) s_min[turn][tid] = kTtAbsent;
    __syncthreads();  // (the other turn's arrays are read before the barrier after next)
    int pos = base, total = base;
#pragma unroll
    for (int w = 0; w < kUdWarps; ++w) {
      const int c = s_cnt[turn][w];
      pos += w < warp ? c : 0;
      total += c;
    }
    // Deltas go to positions base - 1 .. total - 2 (the cloud's first code
    // has none), i.e. the cloud's tree tiles ta and at most ta + 1.
    const int ta = max(base - 1, 0) / kTtTile, tb = (ta + 1) * kTtTile;
    uint8_t* D = S.D + (size_t)K.t_first * kTtTile;
    uint32_t ma = kTtAbsent, mb = kTtAbsent;
#pragma unroll
    for (int r = 0; r < kUdRows; ++r) {
      const uint32_t prev = row_prev(R, r);
      const uint32_t heads = row_heads(R, r, prev, K);
      if (heads >> lane & 1u) {
        const int o = pos + __popc(heads & lanemask_lt());
        out[K.cs + o] = R.key[r];
        if (o > 0) {
          const uint32_t d = tt_delta(prev, R.key[r]);
          D[o - 1] = (uint8_t)d;
          if (o - 1 < tb) ma = min(ma, d);
          else mb = min(mb, d);
        }
      }
      pos += __popc(heads);
    }
    ma = __reduce_min_sync(kFull, ma);
    mb = __reduce_min_sync(kFull, mb);
    if (lane == 0) {
      if (ma < kTtAbsent) atomicMin(&s_min[turn][0], ma);
      if (mb < kTtAbsent) atomicMin(&s_min[turn][1], mb);
    }
    __syncthreads();
    if (tid < 2 && s_min[turn][tid] < kTtAbsent)
      atomic_min_u8(S.tile_min + K.t_first + ta + tid, s_min[turn][tid]);
    if (tid == 0 && unique_c && K.last) unique_c[K.cloud] = total;
  }
}

// Grid of the whole build's (gated) unique kernels: the tiles, capped at 8
// CTAs per SM.
static int unique_grid(int tiles) {
  const int cap = device_sm_count() * 8;
  return tiles < cap ? tiles : cap;
}

cudaError_t launch_unique_deltas(const uint32_t* sorted, int n, uint32_t* codes_out, int* d_unique,
                                 void* tree_scratch, cudaStream_t s, const uint32_t* gate) {
  if (n <= 0) return cudaMemsetAsync(d_unique, 0, sizeof(int), s);
  const TreeScratch S = tree_scratch_carve(tree_scratch, n);
  const OneKeys map{n};
  cudaError_t e = launch_chained(unique_count_kernel<OneKeys>, dim3(unique_grid(S.tiles)),
                                 dim3(kUdThreads), 0, s, sorted, map, S.tiles, S, gate);
  if (e == cudaSuccess)
    e = launch_tile_counts_scan(S.tiles, S.tile_heads, S.tile_upos, d_unique, s, gate);
  if (e != cudaSuccess) return e;
  return launch_chained(unique_deltas_kernel<OneKeys>, dim3(unique_grid(S.tiles)), dim3(kUdThreads),
                        0, s, sorted, map, codes_out, S.tiles, S, nullptr, gate);
}

cudaError_t launch_batch_unique_deltas(const uint32_t* sorted, const int4* tiles, int n_tiles,
                                       const int* start, uint32_t* codes_out, int* unique_c,
                                       void* scratch, cudaStream_t s) {
  if (n_tiles <= 0) return cudaSuccess;
  const TreeScratch S = tree_scratch_carve_tiles(scratch, n_tiles);
  const CloudKeys map{tiles, n_tiles, start};
  cudaError_t e = launch_chained(unique_count_kernel<CloudKeys>, dim3(n_tiles), dim3(kUdThreads), 0,
                                 s, sorted, map, n_tiles, S, nullptr);
  if (e == cudaSuccess) e = launch_tile_counts_scan(n_tiles, S.tile_heads, S.tile_upos, nullptr, s);
  if (e != cudaSuccess) return e;
  return launch_chained(unique_deltas_kernel<CloudKeys>, dim3(n_tiles), dim3(kUdThreads), 0, s,
                        sorted, map, codes_out, n_tiles, S, unique_c, nullptr);
}

cudaError_t launch_batch_radix_tree_from_deltas(const int4* tiles, int n_tiles, const int* start,
                                                const int* unique_c, const uint32_t* codes,
                                                uint8_t* prefix_n, uint8_t* hll, uint8_t* hlr,
                                                int* left_child, int* parent, int* ec,
                                                void* scratch, cudaStream_t s) {
  if (n_tiles <= 0) return cudaSuccess;
  const TreeScratch S = tree_scratch_carve_tiles(scratch, n_tiles);
  const CloudTiles map{tiles, start, unique_c};
  const TreeOut o{prefix_n, hll, hlr, left_child, parent, ec};
  return launch_chained(tree_nodes_kernel<CloudTiles>, dim3(n_tiles), dim3(kTtBThreads), 0, s, map,
                        codes, S, o);
}

cudaError_t launch_radix_tree_from_deltas(int n_host, const int* d_unique, const uint32_t* codes,
                                          uint8_t* prefix_n, uint8_t* hll, uint8_t* hlr,
                                          int* left_child, int* parent, int* ec, void* scratch,
                                          cudaStream_t s) {
  if (n_host <= 0) return cudaSuccess;
  const TreeScratch S = tree_scratch_carve(scratch, n_host);
  const OneCloud map{n_host, d_unique, S.tiles};
  const TreeOut o{prefix_n, hll, hlr, left_child, parent, ec};
  return launch_chained(tree_nodes_kernel<OneCloud>, dim3(S.tiles), dim3(kTtBThreads), 0, s, map,
                        codes, S, o);
}

cudaError_t launch_radix_tree_sorted(int n_host, const int* d_unique, const uint32_t* codes,
                                     uint8_t* prefix_n, uint8_t* hll, uint8_t* hlr,
                                     int* left_child, int* parent, int* ec, void* scratch,
                                     cudaStream_t s) {
  if (n_host <= 0) return cudaSuccess;
  const TreeScratch S = tree_scratch_carve(scratch, n_host);
  const OneCloud map{n_host, d_unique, S.tiles};
  cudaError_t e = launch_chained(tree_tiles_kernel<OneCloud>, dim3(S.tiles), dim3(kTtAThreads), 0,
                                 s, map, codes, S);
  if (e != cudaSuccess) return e;
  const TreeOut o{prefix_n, hll, hlr, left_child, parent, ec};
  return launch_chained(tree_nodes_kernel<OneCloud>, dim3(S.tiles), dim3(kTtBThreads), 0, s, map,
                        codes, S, o);
}

}  // namespace octgb

// One tile of the delta-based radix tree (csrc/tree_tiled.cu has the method):
// the device code shared by the tiled kernels and the fused build.
#pragma once

#include "tree.cuh"

namespace octgb {

constexpr uint32_t kFull = 0xffffffffu;

// Where a tile sits: tiles never cross clouds, and a cloud's tiles start at
// its first position and cover 4,096 positions each; positions are
// cloud-local, arrays are indexed from the cloud's start cs.
struct TileInfo {
  int t;        // tile
  int t_first;  // first and last tile of its cloud
  int t_last;
  int n;        // radix nodes of the cloud
  int lo;       // first position of the tile
  int cs;       // cloud start in the concatenated arrays
};

// Delta of cloud position p in the tile-major delta array.
__device__ __forceinline__ size_t d_index(const TileInfo& I, int p, int tile) {
  return (size_t)I.t_first * tile + (size_t)p;
}

// Positions of a tile: a constant, or chosen per build (a multiple of 512).
template <int N>
struct FixedTile {
  static constexpr bool kFixed = true;
  __device__ __forceinline__ constexpr operator int() const { return N; }
};
struct SizedTile {
  static constexpr bool kFixed = false;
  int n;
  __device__ __forceinline__ operator int() const { return n; }
};

// Lanes whose 5-bit value is below v, from the ballots b[k] of the values'
// bits and v's bits as masks (m[k] all ones where v has bit k).
__device__ __forceinline__ uint32_t lanes_below(const uint32_t (&b)[5], const uint32_t (&m)[5]) {
  uint32_t eq = kFull, lt = 0;
#pragma unroll
  for (int k = 4; k >= 0; --k) {
    lt |= eq & ~b[k] & m[k];
    eq &= ~(b[k] ^ m[k]);
  }
  return lt;
}

__device__ __forceinline__ void bit_masks(uint32_t v, uint32_t (&m)[5]) {
#pragma unroll
  for (int k = 0; k < 5; ++k) m[k] = 0u - ((v >> k) & 1u);
}

__device__ __forceinline__ void value_ballots(uint32_t d, uint32_t (&b)[5]) {
#pragma unroll
  for (int k = 0; k < 5; ++k) b[k] = __ballot_sync(kFull, (d >> k) & 1u);
}

// Bytes here are at most 31 and so is x: (byte | 0x80) - x keeps the high
// bit exactly when byte >= x, with no borrow between bytes.
__device__ __forceinline__ uint32_t high_bits_below(uint32_t w, uint32_t x4) {
  return ~((w | 0x80808080u) - x4) & 0x80808080u;
}

// Bit j set when byte j of w (16 bytes) is below x.
__device__ __forceinline__ uint32_t bytes_below(const uint4& w, uint32_t x) {
  const uint32_t x4 = x * 0x01010101u;
  const uint32_t v[4] = {w.x, w.y, w.z, w.w};
  uint32_t m = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    // gather the four high bits (7, 15, 23, 31) into bits 21..24
    const uint32_t h = ((high_bits_below(v[k], x4) >> 7) * 0x00204081u) >> 21;
    m |= (h & 0xFu) << (4 * k);
  }
  return m;
}

// Largest tile in [lo, hi] whose smallest delta is below x, or -1 (whole warp).
__device__ __forceinline__ int tiles_scan_left(const uint8_t* tmin, int lo, int hi, uint32_t x,
                               int lane) {
  if (hi < lo) return -1;
  for (int blk = hi / kTtMinBlock; blk >= lo / kTtMinBlock; --blk) {
    const uint4 w = reinterpret_cast<const uint4*>(tmin + (size_t)blk * kTtMinBlock)[lane];
    uint32_t m = bytes_below(w, x);
    const int base = blk * kTtMinBlock + lane * 16;
    if (base > hi || base + 15 < lo) m = 0;
    if (base + 15 > hi && base <= hi) m &= (2u << (hi - base)) - 1u;
    if (base < lo && base + 15 >= lo) m &= ~((1u << (lo - base)) - 1u);
    const uint32_t any = __ballot_sync(kFull, m != 0);
    if (any) {
      const int L = 31 - __clz(any);
      const uint32_t mL = __shfl_sync(kFull, m, L);
      return blk * kTtMinBlock + L * 16 + 31 - __clz(mL);
    }
  }
  return -1;
}

// Smallest tile in [lo, hi] whose smallest delta is below x, or -1 (whole warp).
__device__ __forceinline__ int tiles_scan_right(const uint8_t* tmin, int lo, int hi, uint32_t x,
                                int lane) {
  if (hi < lo) return -1;
  for (int blk = lo / kTtMinBlock; blk <= hi / kTtMinBlock; ++blk) {
    const uint4 w = reinterpret_cast<const uint4*>(tmin + (size_t)blk * kTtMinBlock)[lane];
    uint32_t m = bytes_below(w, x);
    const int base = blk * kTtMinBlock + lane * 16;
    if (base > hi || base + 15 < lo) m = 0;
    if (base + 15 > hi && base <= hi) m &= (2u << (hi - base)) - 1u;
    if (base < lo && base + 15 >= lo) m &= ~((1u << (lo - base)) - 1u);
    const uint32_t any = __ballot_sync(kFull, m != 0);
    if (any) {
      const int L = __ffs(any) - 1;
      const uint32_t mL = __shfl_sync(kFull, m, L);
      return blk * kTtMinBlock + L * 16 + __ffs(mL) - 1;
    }
  }
  return -1;
}

// Last (first) position of tile tt's deltas below x; the tile holds one. Four
// 512-byte blocks are read at a time, so a search is one or two round trips.
template <class Tile>
__device__ int tile_last_below(const TreeScratch& S, const TileInfo& I, int tt, uint32_t x,
                               int lane, Tile TILE) {
  const uint8_t* Dt = S.D + (size_t)tt * TILE;
  for (int blk = TILE / 512 - 1; blk >= 0; blk -= 4) {
    uint4 w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      w[q] = reinterpret_cast<const uint4*>(Dt + max(blk - q, 0) * 512)[lane];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t m = bytes_below(w[q], x);
      const uint32_t any = __ballot_sync(kFull, m != 0);
      if (any && blk - q >= 0) {
        const int L = 31 - __clz(any);
        const uint32_t mL = __shfl_sync(kFull, m, L);
        return (tt - I.t_first) * TILE + (blk - q) * 512 + L * 16 + 31 - __clz(mL);
      }
    }
  }
  return -1;
}

template <class Tile>
__device__ int tile_first_below(const TreeScratch& S, const TileInfo& I, int tt, uint32_t x,
                                int lane, Tile TILE) {
  const uint8_t* Dt = S.D + (size_t)tt * TILE;
  const int last = TILE / 512 - 1;
  for (int blk = 0; blk <= last; blk += 4) {
    uint4 w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      w[q] = reinterpret_cast<const uint4*>(Dt + min(blk + q, last) * 512)[lane];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t m = bytes_below(w[q], x);
      const uint32_t any = __ballot_sync(kFull, m != 0);
      if (any) {
        const int L = __ffs(any) - 1;
        const uint32_t mL = __shfl_sync(kFull, m, L);
        // from n on: the last tile's unused tail, so the tile holds no match
        return min((tt - I.t_first) * TILE + min(blk + q, last) * 512 + L * 16 + __ffs(mL) - 1,
                   I.n);
      }
    }
  }
  return I.n;
}

struct TreeOut {
  uint8_t* prefix_n;
  uint8_t* hll;
  uint8_t* hlr;
  int* left_child;
  int* parent;
  int* ec;  // optional
};

// Radix node 0 as the reference builds it (range [0, n - 1]) with split q.
__device__ __forceinline__ void emit_root(const TreeOut& o, int n, int q, uint32_t x,
                                          bool short_root) {
  const bool ll = q == 0, lr = q + 1 == n - 1;
  o.prefix_n[0] = (uint8_t)x;
  o.left_child[0] = q;
  o.hll[0] = ll;
  o.hlr[0] = lr;
  o.parent[0] = 0;
  if (short_root || lr) o.parent[n - 1] = 0;
  if (!short_root) {
    if (!ll) o.parent[q] = 0;
    if (!lr && q + 1 < n) o.parent[q + 1] = 0;
  }
  if (o.ec) o.ec[0] = 0;
}

template <int MAX, int THREADS>
struct TreeSmem {  // tiles of at most MAX positions
  static constexpr int kChunks = MAX / 32, kWarps = THREADS / 32;
  __align__(16) uint8_t D[MAX];
  int16_t pl[kChunks][32];  // last tile position before the chunk with D < v
  int16_t sf[kChunks][32];  // first tile position after the chunk with D < v
  int16_t wl[kWarps][32], wf[kWarps][32];
  uint8_t pv[MAX], nv[MAX];  // nearest smaller lane in the chunk, or 0xFF
  // Sized tiles: per value v the nearest position before (after) the tile
  // with D < v (-1 / n when there is none) and its delta.
  int ext_l[32], ext_r[32];
  int8_t ext_ld[32], ext_rd[32];
};

// The nodes split at the tile's positions (THREADS threads; the caller puts a
// barrier before M is used again). No pointer here is __restrict__: in the
// fused build the same kernel wrote what they point to.
template <class Tile, int MAX, int THREADS>
__device__ __forceinline__ void tree_nodes_tile(TreeSmem<MAX, THREADS>& M, Tile TILE,
                                                const TileInfo& I, const uint32_t* codes,
                                                const TreeScratch& S, TreeOut o) {
  constexpr int kWarps = TreeSmem<MAX, THREADS>::kWarps;
  constexpr int kMost = TreeSmem<MAX, THREADS>::kChunks / kWarps;
  const int kPer = Tile::kFixed ? kMost : (TILE / 32 + kWarps - 1) / kWarps;  // chunks per warp
  const int n = I.n, t = I.t, t0 = I.lo;
  if (t0 >= n) return;
  // the cloud's arrays
  codes += I.cs;
  o.prefix_n += I.cs;
  o.hll += I.cs;
  o.hlr += I.cs;
  o.left_child += I.cs;
  o.parent += I.cs;
  if (o.ec) o.ec += I.cs;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (n < 2) {  // a single node: the reference's search steps
    if (tid == 0) {
      radix_node(0, n, GlobalCodes{codes}, o.prefix_n, o.hll, o.hlr, o.left_child, o.parent);
      if (o.ec) o.ec[0] = 0;
    }
    return;
  }
  for (int j = tid; j < TILE / 16; j += THREADS)
    reinterpret_cast<uint4*>(M.D)[j] = reinterpret_cast<const uint4*>(S.D + (size_t)t * TILE)[j];
  if constexpr (!Tile::kFixed) {
    // One warp per value answers every query that leaves the tile at once. (A
    // tiled build's many tiles answer those few on demand below; here each
    // tile is a CTA's whole work and the searches, one after another in the
    // first and last warps, took 5 to 10 us of a 12 to 17 us phase.)
    static_assert(Tile::kFixed || kWarps == 32, "one warp per value");
    const uint32_t v = (uint32_t)warp;
    const int tl = tiles_scan_left(S.tile_min, I.t_first, t - 1, v, lane);
    const int tr = tiles_scan_right(S.tile_min, t + 1, I.t_last, v, lane);
    const int pl = tl >= 0 ? tile_last_below(S, I, tl, v, lane, TILE) : -1;
    const int pr = tr >= 0 ? tile_first_below(S, I, tr, v, lane, TILE) : n;
    if (lane == 0) {
      M.ext_l[v] = pl;
      M.ext_ld[v] = pl >= 0 ? (int8_t)S.D[d_index(I, pl, TILE)] : (int8_t)-1;
      M.ext_r[v] = pr;
      M.ext_rd[v] = pr < n ? (int8_t)S.D[d_index(I, pr, TILE)] : (int8_t)-1;
    }
  }
  __syncthreads();
  if (t0 + TILE > n) {  // the cloud's last tile: positions from n on are absent
    for (int j = n - t0 + tid; j < TILE; j += THREADS) M.D[j] = (uint8_t)kTtAbsent;
    __syncthreads();
  }

  const uint32_t below_me = (1u << lane) - 1u;
  const uint32_t above_me = ~below_me << 1;  // lanes > lane (lane 31: none)
  uint32_t lm[5];
  bit_masks((uint32_t)lane, lm);
  // this warp's chunks (of a sized tile: those inside it)
  const int mine = Tile::kFixed ? kMost : min(kPer, TILE / 32 - warp * kPer);
  int cf[kMost];
  int run = -1;
#pragma unroll
  for (int k = 0; k < kMost; ++k) {
    if (!Tile::kFixed && k >= mine) break;
    const int c = warp * kPer + k;
    const uint32_t d = M.D[32 * c + lane];
    uint32_t b[5];
    value_ballots(d, b);
    // lane v: the lanes whose delta is below v; a lane's own query is lane d's
    const uint32_t lt_lane = lanes_below(b, lm);
    const uint32_t lt_own = __shfl_sync(kFull, lt_lane, (int)d);
    const uint32_t l = lt_own & below_me, r = lt_own & above_me;
    M.pv[32 * c + lane] = l ? (uint8_t)(31 - __clz(l)) : (uint8_t)0xFF;
    M.nv[32 * c + lane] = r ? (uint8_t)(__ffs(r) - 1) : (uint8_t)0xFF;
    M.pl[c][lane] = (int16_t)run;
    if (lt_lane) run = 32 * c + 31 - __clz(lt_lane);
    cf[k] = lt_lane ? 32 * c + __ffs(lt_lane) - 1 : TILE;
  }
  int runf = TILE;
#pragma unroll
  for (int k = kMost - 1; k >= 0; --k) {
    if (!Tile::kFixed && k >= mine) continue;
    const int c = warp * kPer + k;
    M.sf[c][lane] = (int16_t)runf;
    runf = min(runf, cf[k]);
  }
  M.wl[warp][lane] = (int16_t)run;
  M.wf[warp][lane] = (int16_t)runf;
  __syncthreads();
  {
    int cl = -1, cr = TILE;
    for (int w = 0; w < warp; ++w) cl = max(cl, (int)M.wl[w][lane]);
    for (int w = warp + 1; w < kWarps; ++w) cr = min(cr, (int)M.wf[w][lane]);
#pragma unroll
    for (int k = 0; k < kMost; ++k) {
      if (!Tile::kFixed && k >= mine) break;
      const int c = warp * kPer + k;
      M.pl[c][lane] = (int16_t)max((int)M.pl[c][lane], cl);
      M.sf[c][lane] = (int16_t)min((int)M.sf[c][lane], cr);
    }
  }
  __syncwarp();

  int own_sum = 0;  // edge counts of this tile's nodes emitted here
  // Per chunk, the common case without branches: both neighbours inside the
  // tile (shared-memory tables); lanes needing another tile, the root or an
  // edge count of another tile take warp-uniform guarded blocks.
#pragma unroll 1
  for (int k = 0; k < mine; ++k) {
    const int c = warp * kPer + k;
    const int j = 32 * c + lane;
    const int q = t0 + j;
    const bool live = q < n;
    const uint32_t xv = M.D[j];
    const uint32_t pv = M.pv[j], nv = M.nv[j];
    const int pl = M.pl[c][xv], sf = M.sf[c][xv];
    // -2: not in this tile
    int a = pv != 0xFF ? t0 + 32 * c + (int)pv : (pl >= 0 ? t0 + pl : -2);
    int b = nv != 0xFF ? t0 + 32 * c + (int)nv : (sf < TILE ? t0 + sf : -2);
    int da = M.D[max(a - t0, 0)], db = M.D[min(max(b - t0, 0), TILE - 1)];
    // Neighbours outside the tile (the tile's running minima only): the edge
    // of the adjacent tile first, then one warp-wide scan of the tile minima
    // per query and of the found tile's deltas.
    if constexpr (!Tile::kFixed) {
      if (a == -2) {
        a = M.ext_l[xv];
        da = M.ext_ld[xv];
      }
      if (b == -2) {
        b = M.ext_r[xv];
        db = M.ext_rd[xv];
      }
    } else if (__any_sync(kFull, live && (a == -2 || b == -2))) {
      const bool fa = live && a == -2, fb = live && b == -2;
      if (fa) {
        if (t == I.t_first) {
          a = -1;
        } else {
          const uint4 w = *reinterpret_cast<const uint4*>(S.D + (size_t)t * TILE - 16);
          const uint32_t m = bytes_below(w, xv);
          if (m) a = t0 - 16 + 31 - __clz(m);
        }
      }
      if (fb) {
        if (t == I.t_last) {
          b = n;
        } else {
          const uint4 w = *reinterpret_cast<const uint4*>(S.D + (size_t)(t + 1) * TILE);
          const uint32_t m = bytes_below(w, xv);
          // a match from n on lies in the last tile's unused tail: none there
          if (m) b = min(t0 + TILE + __ffs(m) - 1, n);
        }
      }
      uint32_t need = __ballot_sync(kFull, live && a == -2);
      while (need) {
        const int src = __ffs(need) - 1;
        need &= need - 1;
        const uint32_t qx = __shfl_sync(kFull, xv, src);
        const int tt = tiles_scan_left(S.tile_min, I.t_first, t - 1, qx, lane);
        const int ans = tt >= 0 ? tile_last_below(S, I, tt, qx, lane, TILE) : -1;
        if (lane == src) a = ans;
      }
      need = __ballot_sync(kFull, live && b == -2);
      while (need) {
        const int src = __ffs(need) - 1;
        need &= need - 1;
        const uint32_t qx = __shfl_sync(kFull, xv, src);
        const int tt = tiles_scan_right(S.tile_min, t + 1, I.t_last, qx, lane);
        const int ans = tt >= 0 ? tile_first_below(S, I, tt, qx, lane, TILE) : n;
        if (lane == src) b = ans;
      }
      if (fa && a >= 0) da = S.D[d_index(I, a, TILE)];
      if (fb && b < n) db = S.D[d_index(I, b, TILE)];
    }
    if (a < 0) da = -1;
    if (b >= n) db = -1;
    // a < 0 and b >= n: the smallest delta overall (the proper root), which
    // gives radix node 0 unless it sits at n - 1 (a short root: node 0 then
    // comes from the split of [0, n - 2], with a < 0 and b == n - 1).
    const bool top = a < 0 && b >= n;
    const bool short_root = a < 0 && b == n - 1;
    if (live && !top) {
      const int i = a < 0 ? b : (b >= n ? a + 1 : (da > db ? a + 1 : b));
      const bool ll = a + 1 == q, lr = b == q + 1;
      o.prefix_n[i] = (uint8_t)xv;
      o.left_child[i] = q;
      o.hll[i] = ll;
      o.hlr[i] = lr;
      if (!ll) o.parent[q] = i;
      if (!lr) o.parent[q + 1] = i;
      if (o.ec) {
        // the larger neighbour delta is the parent's (>= 0 whenever read)
        const int e = short_root ? 0 : (int)(xv / 3u) - (int)((uint32_t)max(da, db) / 3u);
        o.ec[i] = e;
        const bool own = (uint32_t)(i - t0) < (uint32_t)TILE;
        own_sum += own ? e : 0;
        if (!own) atomicAdd(S.tile_sum + I.t_first + i / TILE, e);
      }
    }
    if (__any_sync(kFull, live && (top || short_root))) {
      if (live && top && q <= n - 2) emit_root(o, n, q, xv, false);
      if (live && short_root) emit_root(o, n, q, xv, true);
    }
  }
  if (o.ec) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) own_sum += __shfl_xor_sync(kFull, own_sum, off);
    if (lane == 0 && own_sum != 0) atomicAdd(S.tile_sum + t, own_sum);
  }
}

}  // namespace octgb

// Octree stage (7-8) device functions shared by the single-cloud and the
// batched builds: sequence tags, per-node write emission, per-slot finalize.
#pragma once

#include "kernels.cuh"

namespace octgb {

constexpr uint32_t kLinkTag = 0x80000000u;

struct Sizes {
  int n_brt, n_oct;
  bool fits;
};

__device__ __forceinline__ Sizes read_sizes(const OctArgs& a) {
  Sizes z;
  z.n_brt = a.d_unique ? max(*a.d_unique - 1, 0) : a.n_brt_host;
  if (a.d_max_slot)
    z.n_oct = z.n_brt >= 1 ? *a.d_max_slot + 1 : 0;
  else
    z.n_oct = a.n_oct_host;
  z.fits = z.n_oct <= a.cap;
  return z;
}

__device__ __forceinline__ void put_child(const OctTags& t, int slot, int which, uint32_t tag,
                                          int n_oct, uint32_t* status) {
  if ((unsigned)slot >= (unsigned)n_oct) {
    raise_status(status, kStatusCapacity);
    return;
  }
  atomicMax(&t.child[(size_t)slot * 8 + which], tag);
}

// Every write radix node i makes (MakeOctNodes for i >= 1 when mode has
// kOctMake, LinkLeafNodes when it has kOctLink), as tags.
//
// Loads are grouped by dependency so each round is issued at once: the node's
// own entries; then its parent's count and parent link and the codes of its
// leaf children; then the rest of the walk up to the first radix node with
// octree nodes (usually none); then that node's octree offset. At most one
// walk applies: MakeOctNodes walks from parent[i] when i has octree nodes,
// LinkLeafNodes walks from i, i.e. from parent[i] when i has none.
__device__ __forceinline__ void emit_node(int mode, int i, const OctArgs& a, const OctTags& t,
                                          const Sizes& z, uint32_t* status) {
  const int pn = a.prefix_n[i];
  const int k = a.counts[i];
  const int par = a.parent[i];
  const bool make = (mode & kOctMake) && i >= 1 && k > 0;
  const bool ll = (mode & kOctLink) && a.hll[i];
  const bool lr = (mode & kOctLink) && a.hlr[i];
  const bool link = ll || lr;
  int base = 0, lc = 0;
  uint32_t code = 0;
  if (make) {
    base = a.offsets[i];
    code = a.codes[i];
  }
  if (link) lc = a.left_child[i];
  const int L = pn / 3;
  // walk start: the parent (MakeOctNodes; LinkLeafNodes of a node without
  // octree nodes other than 0) or i itself (LinkLeafNodes otherwise)
  const bool walk_link = link && k == 0 && i != 0;
  const bool walk = make || walk_link;
  int wc = 0, wp = 0;
  uint32_t cl = 0, cr = 0;
  const bool lc_ok = (unsigned)lc < (unsigned)z.n_brt;  // leaf index lc + 1 <= n_brt
  const bool par_ok = (unsigned)par < (unsigned)z.n_brt;
  if (walk && par_ok) {
    wc = a.counts[par];
    wp = a.parent[par];
  }
  if (link && lc_ok) {
    if (ll) cl = a.codes[lc];
    if (lr) cr = a.codes[lc + 1];
  }

  if (make) {
    // include/shared/oct.h:24-90
    for (int j = 0; j < k - 1; ++j) {
      const int level = L - j;
      const uint32_t pre = code >> (30 - 3 * level);
      const int which = (int)(pre & 7u);
      const int up = base + j + 1;
      put_child(t, up, which, (((uint32_t)i << 4) | (uint32_t)j) + 1u, z.n_oct, status);
      if ((unsigned)up < (unsigned)z.n_oct) atomicOr(&t.mask[up], 1u << which);
      if ((unsigned)(base + j) < (unsigned)z.n_oct) atomicMax(&t.owner[base + j], (uint32_t)i);
    }
    int rp = par;
    bool bad = !par_ok;
    if (!bad && wc == 0) {
      int counter = 0;
      rp = wp;
      bad = (unsigned)rp >= (unsigned)z.n_brt;
      if (!(++counter > 30))
        while (!bad && a.counts[rp] == 0) {
          rp = a.parent[rp];
          bad = (unsigned)rp >= (unsigned)z.n_brt;
          if (++counter > 30) break;
        }
    }
    if (bad) {  // malformed parent[]: never read out of bounds
      raise_status(status, kStatusWalkLimit);
      rp = 0;
    }
    const int top = L - k + 1;
    const int which = (int)((code >> (30 - 3 * top)) & 7u);
    const int oct_parent = a.offsets[rp];
    put_child(t, oct_parent, which, (((uint32_t)i << 4) | (uint32_t)(k - 1)) + 1u, z.n_oct,
              status);
    if ((unsigned)oct_parent < (unsigned)z.n_oct) atomicOr(&t.mask[oct_parent], 1u << which);
    const int slot = base + k - 1;
    if ((unsigned)slot < (unsigned)z.n_oct) atomicMax(&t.owner[slot], (uint32_t)i);
    else raise_status(status, kStatusCapacity);
  }
  if (link) {
    // include/shared/oct.h:92-134, walk bounded at radix node 0.
    int rn = i;
    if (walk_link) {
      int steps = 0;
      if (!par_ok) {
        raise_status(status, kStatusWalkLimit);
      } else {
        rn = par;
        ++steps;
        int cnt = wc, up = wp;
        while (cnt == 0 && rn != 0) {
          if ((unsigned)up >= (unsigned)z.n_brt || ++steps > 64) {
            raise_status(status, kStatusWalkLimit);
            break;
          }
          rn = up;
          cnt = a.counts[rn];
          up = a.parent[rn];
        }
      }
    }
    // rn == i with octree nodes: its offset is already in base (a load here
    // would wait behind the MakeOctNodes atomics, which the compiler may not
    // move it above).
    const int dst = (make && rn == i) ? base : a.offsets[rn];
    const uint32_t sh = (uint32_t)(30 - 3 * (L + 1)) & 31u;
    if (!lc_ok) {
      raise_status(status, kStatusWalkLimit);
      return;
    }
    if (ll) put_child(t, dst, (int)((cl >> sh) & 7u), kLinkTag | ((uint32_t)i << 1), z.n_oct, status);
    if (lr)
      put_child(t, dst, (int)((cr >> sh) & 7u), kLinkTag | ((uint32_t)i << 1) | 1u, z.n_oct,
                status);
  }
}

// range / 2^k as the reference computes it (float division by (float)(1 << k)).
// For k in [0, 30] the divisor is the exact power of two, and the correctly
// rounded quotient equals the correctly rounded product range * 2^-k.
__device__ __forceinline__ float cell_size(float range, int k) {
  if (k >= 0 && k <= 30) return __fmul_rn(range, __int_as_float((127 - k) << 23));
  return __fdiv_rn(range, (float)(1 << k));
}

// ------------------------------------------------------------- slot tags --
// The whole and batched builds' form of the same tags (trees built by this
// library, stages 7 and 8 together, up to kSlotTagMaxPoints points). Two facts
// let finalize turn a tag into its value without looking anything up:
//   - among radix nodes with octree nodes (k >= 1) the inclusive prefix grows
//     by at least one from each to the next, so (prefix, step) orders their
//     writes as (node, step) does, and names the value: prefix + step;
//   - a leaf lies at its parent's own index or at the far end of the parent's
//     range, usually a few codes away, so a link tag carries that distance
//     behind its order key.
//   MakeOctNodes  step j of the node with prefix s : (s << 4) | j     (s < 2^27, s >= 1)
//   LinkLeafNodes of node i : 0x80000000 | (i << (b + 1)) | (2^b + off), the
//     leaf being i + off, off <= 0 for the left leaf and >= 0 for the right
//     one (never 0 for both: i is one end of the node's range). The field's
//     ends, 0 and all ones, stand for a leaf too far off: read left_child[i].
//     b is what the cloud's node numbers leave (6 bits at 16.7M points, where
//     about one slot in a hundred looks up)
// The corner's writer needs no tag either: slots [s, s + k) belong to the node
// with prefix s, later nodes overwrite, and the prefix sum's tiles note each
// slot's node and step (SlotTags::node). The masks take one byte per slot.
// Against node tags (owner tag, 4-byte mask, two table reads per child):
// emit 0.202 -> 0.186 ms (285 -> 236 warp instructions per 32 nodes; bound by its L2
// dependent loads), finalize 0.152 -> 0.132 ms (416 -> 288 per 32 slots; bound by
// DRAM, 5.8 TB/s) at 16.7M uniform points.
constexpr uint32_t kNoNode = 15u;  // SlotTags::node: no node's slots reach this one (0: open)

__device__ __forceinline__ int link_off_bits(int n_brt) {
  return min(__clz(n_brt) - 2, 16);  // 31 tag bits, one of them the side
}

__device__ __forceinline__ void slot_put(const SlotTags& t, int slot, uint32_t which,
                                         uint32_t tag) {
  atomicMax(t.child + ((uint32_t)slot * 8u + which), tag);
}
__device__ __forceinline__ void slot_mark(const SlotTags& t, int slot, uint32_t which) {
  int sh;
  uint32_t* w = t.mask_word(slot, sh);
  atomicOr(w, 1u << (sh + (int)which));
}

// Inclusive prefix sum of one tile of edge counts of a cloud, with the
// slot tags' preparation of the slots it covers: child tags and masks zeroed,
// each slot's radix node written. The tile's own slots are (ex, ex + total];
// the next nine may hold the last node's further steps and are cleared as
// well (the next tile clears them again: zeros either way, and nothing else
// writes tags in this kernel).
//
// Bound: DRAM writes (the tags take 33 B per slot beside 8 B per node). The
// child tags are zeroed by bulk copies of a zeroed 4 KB block (the TMA engine
// writes them), which leaves the load/store units to the counts: 0.084 -> 0.067 ms
// at 16.7M uniform points against the node tags and 16-byte stores.
constexpr int kPfThreads = 256;
constexpr int kPfItems = 16;
constexpr int kPfTile = kPfThreads * kPfItems;  // the radix-tree tiles
constexpr int kPfZero = 4096;                   // bytes of the zero block
constexpr int kMaxSteps = 10;                   // octree levels one radix node can span

template <int THREADS, int ITEMS>
struct PrefixSmem {
  static constexpr int kTile = THREADS * ITEMS;
  __align__(16) uint4 zero[kPfZero / 16];
  __align__(16) uint32_t node[kTile];  // by slot after the tile's prefix: (tile's node + 1) << 4 | step
  int v[kTile + kTile / 32];  // padded: entry j at j + j / 32
  uint32_t warp[32];
  uint32_t total;
  int max_slot;
};

__device__ __forceinline__ int pf_pad(int j) { return j + (j >> 5); }

// ec, ps: the cloud's arrays; the tile's nodes are [lo, min(lo + kTile, n)), its
// exclusive prefix ex. max_slot: raised to the largest slot stages 7-8 write.
// All threads call it; ends with a barrier. The zeroing copies may still be on
// their way then: thread 0 waits for them (bulk_wait_all) before its kernel
// ends, or before a barrier after which the tags are written.
template <int THREADS, int ITEMS>
__device__ __forceinline__ void prefix_slots_tile(PrefixSmem<THREADS, ITEMS>& S, const int* ec,
                                                  int* ps, int n, int lo, uint32_t ex,
                                                  const SlotTags& t, int* max_slot,
                                                int items = ITEMS) {
  constexpr int kTile = THREADS * ITEMS;  // at most; the tile has THREADS * items
  const int tid = threadIdx.x;
  const int valid = min(THREADS * items, n - lo);
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    if (k >= items) break;
    const int j = k * THREADS + tid;
    S.v[pf_pad(j)] = j < valid ? ec[lo + j] : 0;
  }
  if (tid < kPfZero / 16) S.zero[tid] = make_uint4(0u, 0u, 0u, 0u);
  for (int q = tid; q < kTile / 4; q += THREADS)
    reinterpret_cast<uint4*>(S.node)[q] = make_uint4(0u, 0u, 0u, 0u);
  if (tid == 0) S.max_slot = 0;
  bulk_fence_writes();
  __syncthreads();
  int v[ITEMS];
  uint32_t sum = 0;
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    v[k] = k < items ? S.v[pf_pad(tid * items + k)] : 0;
    sum += (uint32_t)v[k];
  }
  const uint32_t off = block_exclusive_sum<THREADS>(sum, S.warp, &S.total);
  const uint32_t total = S.total;
  const uint32_t cap = (uint32_t)t.cap;
  if (ex < cap) {
    const uint32_t hi = min(ex + min(total, cap) + (uint32_t)(kMaxSteps - 1), cap - 1u);
    if (tid == 0) {
      char* dst = reinterpret_cast<char*>(t.child + (size_t)ex * 8);
      const size_t bytes = ((size_t)hi - ex + 1) * 32;
      for (size_t b = 0; b < bytes; b += kPfZero)
        bulk_store_s2g(dst + b, S.zero, (uint32_t)min((size_t)kPfZero, bytes - b));
    }
    clear_mask_range(t, (int)ex, (int)hi, tid, THREADS);
  }
  // (Bounds on run, v and total: counts of a malformed tree, see emit_slots.)
  // The stage takes the tile's slots; there are more than it holds only when many
  // nodes span several levels, and it then takes them kTile at a time.
  uint32_t run = ex + off;
  int mx = 0;
  uint32_t multi = 0;  // items that span several levels
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    if (k >= items) break;
    const int j = tid * items + k;
    run += (uint32_t)v[k];
    S.v[pf_pad(j)] = (int)run;  // each thread rewrites only its own entries
    const int i = lo + j;
    const uint32_t q = run - ex - 1u;
    const bool makes = i > 0 && v[k] > 0;  // entries past the last node are 0
    if (makes) mx = max(mx, (int)run + v[k] - 1);
    if (makes && v[k] > 1) multi |= 1u << k;
    // the node's own slot: later nodes win over earlier nodes' further steps
    if (makes && q < (uint32_t)kTile) atomicMax(&S.node[q], (uint32_t)(j + 1) << 4);
    if (i == n - 1) mx = max(mx, (int)run);
  }
  // further steps, one such node of each lane at a time
  while (multi) {
    const int j = tid * items + __ffs(multi) - 1;
    multi &= multi - 1u;
    const uint32_t q = (uint32_t)S.v[pf_pad(j)] - ex - 1u;
    const uint32_t k = (uint32_t)min(ec[lo + j], kMaxSteps);
    for (uint32_t h = 1; h < k && q + h < min(total, (uint32_t)kTile); ++h)
      atomicMax(&S.node[q + h], ((uint32_t)(j + 1) << 4) | h);
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((tid & 31) == 0 && mx > 0) atomicMax(&S.max_slot, mx);
  __syncthreads();
  if (tid == 0) atomicMax(max_slot, S.max_slot);
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    if (k >= items) break;
    const int j = k * THREADS + tid;
    if (j < valid) ps[lo + j] = S.v[pf_pad(j)];
  }
  for (uint32_t q = tid; q < min(total, (uint32_t)kTile); q += THREADS) {
    const uint32_t slot = ex + 1u + q;
    const uint32_t e = S.node[q];
    // the tile before may reach its first few slots: left open
    const uint32_t none = q < (uint32_t)kMaxSteps && lo > 0 ? 0u : kNoNode;
    if (slot < cap) t.node[slot] = e ? e + ((uint32_t)(lo - 1) << 4) : none;
  }
  // (6M points in pairs of neighbours: 127 us and 215 in finalize when such a tile
  // left its slots to finalize's search, 88 and 153 this way)
#pragma unroll 1
  for (uint32_t w = kTile; w < min(total, (uint32_t)(kTile * kMaxSteps)); w += kTile) {
    __syncthreads();
    for (int q = tid; q < kTile / 4; q += THREADS)
      reinterpret_cast<uint4*>(S.node)[q] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
#pragma unroll 1
    for (int k = 0; k < items; ++k) {
      const int j = tid * items + k;
      if (j >= valid || lo + j == 0) continue;
      const uint32_t q = (uint32_t)S.v[pf_pad(j)] - ex - 1u;
      if (q >= w + (uint32_t)kTile || q + (uint32_t)kMaxSteps <= w) continue;
      const int steps = min(ec[lo + j], kMaxSteps);
      for (int h = 0; h < steps; ++h) {
        const uint32_t s = q + (uint32_t)h;
        if (s - w < (uint32_t)kTile && s < total)
          atomicMax(&S.node[s - w], ((uint32_t)(j + 1) << 4) | (uint32_t)h);
      }
    }
    __syncthreads();
    for (uint32_t q = tid; q < min(total - w, (uint32_t)kTile); q += THREADS) {
      const uint32_t slot = ex + 1u + w + q, e = S.node[q];
      if (slot < cap) t.node[slot] = e ? e + ((uint32_t)(lo - 1) << 4) : kNoNode;
    }
  }
  // slot 0 (the root's) and the slots after the last node's prefix have none
  if (lo == 0 && tid == 0 && cap > 0) t.node[0] = 0u;
  if (lo + THREADS * items >= n && tid < kMaxSteps) {
    const uint32_t slot = ex + total + 1u + (uint32_t)tid;
    if (slot < cap) t.node[slot] = 0u;
  }
  if (tid == 0) bulk_wait_read();  // the zero block may go
  __syncthreads();
}

// The octree writes of one radix node. The tree is this library's own, so a
// walk to the first node with octree nodes ends there or at node 0 after at
// most 30 steps, every index is below n_brt and every slot below n_oct
// (n_oct - 1 is the largest slot written). The clamps on indexes and slots only
// matter after a status bit was raised (a sort whose look-back timed out leaves
// no tree): nothing goes out of bounds.
struct EmitNode {
  int i, k, base;        // node, octree nodes, prefix
  uint32_t code, level;  // the node's own code; prefix length / 3
};

// MakeOctNodes (include/shared/oct.h:24-90) of a node with octree nodes; up:
// the slot of the first node above it that has some.
__device__ __forceinline__ void emit_make(const EmitNode& e, uint32_t up, const SlotTags& t,
                                          uint32_t top_slot) {
  const uint32_t s16 = (uint32_t)e.base << 4;
  for (int j = 0; j < e.k - 1; ++j) {
    const uint32_t which = (e.code >> (30 - 3 * ((int)e.level - j))) & 7u;
    const int slot = (int)min((uint32_t)(e.base + j + 1), top_slot);
    slot_put(t, slot, which, s16 | (uint32_t)j);
    slot_mark(t, slot, which);
  }
  const uint32_t which = (e.code >> (30 - 3 * ((int)e.level - e.k + 1))) & 7u;
  const int slot = (int)min(up, top_slot);
  slot_put(t, slot, which, s16 | (uint32_t)(e.k - 1));
  slot_mark(t, slot, which);
}

// LinkLeafNodes (include/shared/oct.h:92-134, the walk ended at radix node 0)
// of one leaf, code c: node i's left leaf is leaf i - back, its right one
// i + ahead.
__device__ __forceinline__ void emit_leaf(int i, uint32_t level, uint32_t dst, uint32_t c,
                                          uint32_t field, int bits, const SlotTags& t,
                                          uint32_t top_slot) {
  const uint32_t sh = (uint32_t)(27 - 3 * (int)level) & 31u;
  slot_put(t, (int)min(dst, top_slot), (c >> sh) & 7u,
           kLinkTag | ((uint32_t)i << (bits + 1)) | field);
}
__device__ __forceinline__ uint32_t left_field(uint32_t back, int bits) {
  return (1u << bits) - min(back, 1u << bits);
}
__device__ __forceinline__ uint32_t right_field(uint32_t ahead, int bits) {
  return (1u << bits) + min(ahead, (1u << bits) - 1u);
}

// The slot of the first node with octree nodes from rn up, in global memory.
__device__ __forceinline__ uint32_t root_slot(uint32_t rn, const OctArgs& a, uint32_t last) {
  rn = min(rn, last);
  int c = a.counts[rn];
  uint32_t next = (uint32_t)a.parent[rn];
  for (int step = 0; c == 0 && rn != 0u && step < 32; ++step) {
    rn = min(next, last);
    c = a.counts[rn];
    next = (uint32_t)a.parent[rn];
  }
  return (uint32_t)a.offsets[rn];
}

// Node i straight from global memory (the fused build).
__device__ __forceinline__ void emit_slots(int i, const OctArgs& a, const SlotTags& t, int n_brt,
                                           int n_oct) {
  const uint32_t last = (uint32_t)n_brt - 1u, top_slot = (uint32_t)n_oct - 1u;
  EmitNode e;
  e.i = i;
  e.level = a.prefix_n[i] / 3u;
  e.k = min(a.counts[i], kMaxSteps);
  const uint32_t par = (uint32_t)a.parent[i];
  const bool ll = a.hll[i] != 0, lr = a.hlr[i] != 0;
  const bool make = e.k > 0 && i >= 1;
  e.base = 0;
  uint32_t lc = 0;
  if (make) {
    e.base = a.offsets[i];
    e.code = a.codes[i];
  }
  if (ll || lr) lc = min((uint32_t)a.left_child[i], last);
  uint32_t up = 0;
  if (make || ((ll || lr) && e.k == 0 && i != 0)) up = root_slot(par, a, last);
  uint32_t cl = 0, cr = 0;
  if (ll) cl = a.codes[lc];
  if (lr) cr = a.codes[lc + 1u];
  if (make) emit_make(e, up, t, top_slot);
  const uint32_t dst = make ? (uint32_t)e.base : up;
  const int bits = link_off_bits(n_brt);
  if (ll) emit_leaf(i, e.level, dst, cl, left_field((uint32_t)i - lc, bits), bits, t, top_slot);
  if (lr)
    emit_leaf(i, e.level, dst, cr, right_field(lc + 1u - (uint32_t)i, bits), bits, t, top_slot);
}

// A tile of radix nodes in shared memory: a node's parents and leaves lie close
// to it (98% in its tile), so one round of bulk copies takes the place of four
// to seven dependent rounds of loads, and what several nodes need is found once.
constexpr int kEmitThreads = 256;
constexpr int kEmitTile = 1024;  // nodes: four per thread
constexpr int kEmitRoom = kEmitTile + 32;

struct EmitSmem {
  __align__(16) int counts[kEmitRoom];
  __align__(16) int parent[kEmitRoom];
  __align__(16) int offsets[kEmitRoom];
  __align__(16) uint32_t codes[kEmitRoom];
  __align__(16) int left[kEmitRoom];
  __align__(16) uint8_t pn[kEmitRoom];
  __align__(16) uint8_t hll[kEmitRoom];
  __align__(16) uint8_t hlr[kEmitRoom];
  unsigned long long bar;
};

// Brings nodes [lo, lo + n) (n <= kEmitTile, and the code after the last) of a
// cloud into M. first: the cloud's place in the batch's arrays (`a` is the
// cloud's view of them), total: entries of those arrays. Copies start at the
// sixteenth entry at or before the tile, so every array's start is 16-byte
// aligned when the arrays are; what the arrays' end leaves of the last sixteen,
// or everything when they are not aligned, comes by plain loads. Returns the
// tile's place in M; the block has passed a barrier. Thread 0 set M.bar up;
// phase is the parity of earlier calls. False in ok when the wait ran out (the
// caller returns).
__device__ __forceinline__ uint32_t load_emit_tile(EmitSmem& M, const OctArgs& a, uint32_t first,
                                                   uint32_t lo, uint32_t n, uint32_t total,
                                                   uint32_t phase, uint32_t* status, bool& ok) {
  const uint32_t start = first + lo;
  const uint32_t shift = start & 15u;
  const uint32_t need = shift + n + 1u;  // entries from start - shift on
  const uintptr_t any = reinterpret_cast<uintptr_t>(a.counts - first) |
                        reinterpret_cast<uintptr_t>(a.parent - first) |
                        reinterpret_cast<uintptr_t>(a.offsets - first) |
                        reinterpret_cast<uintptr_t>(a.codes - first) |
                        reinterpret_cast<uintptr_t>(a.left_child - first) |
                        reinterpret_cast<uintptr_t>(a.prefix_n - first) |
                        reinterpret_cast<uintptr_t>(a.hll - first) |
                        reinterpret_cast<uintptr_t>(a.hlr - first);
  const uint32_t room = total - (start - shift);  // entries to the arrays' end
  const uint32_t bulk = (any & 15u) ? 0u : min((need + 15u) & ~15u, room & ~15u);
  const int o = (int)lo - (int)shift;  // the first copied entry, from the cloud's start
  if (threadIdx.x == 0) {
    mbar_expect(&M.bar, bulk * 23u);
    if (bulk) {
      bulk_load_g2s(M.counts, a.counts + o, bulk * 4u, &M.bar);
      bulk_load_g2s(M.parent, a.parent + o, bulk * 4u, &M.bar);
      bulk_load_g2s(M.offsets, a.offsets + o, bulk * 4u, &M.bar);
      bulk_load_g2s(M.codes, a.codes + o, bulk * 4u, &M.bar);
      bulk_load_g2s(M.left, a.left_child + o, bulk * 4u, &M.bar);
      bulk_load_g2s(M.pn, a.prefix_n + o, bulk, &M.bar);
      bulk_load_g2s(M.hll, a.hll + o, bulk, &M.bar);
      bulk_load_g2s(M.hlr, a.hlr + o, bulk, &M.bar);
    }
  }
  for (uint32_t j = bulk + threadIdx.x; j < min(need, room); j += kEmitThreads) {
    const int q = o + (int)j;
    M.counts[j] = a.counts[q];
    M.parent[j] = a.parent[q];
    M.offsets[j] = a.offsets[q];
    M.codes[j] = a.codes[q];
    M.left[j] = a.left_child[q];
    M.pn[j] = a.prefix_n[q];
    M.hll[j] = a.hll[q];
    M.hlr[j] = a.hlr[q];
  }
  __syncthreads();
  ok = true;
  for (int tries = 0; tries < 2 && !mbar_try_wait(&M.bar, phase); ++tries) {
    WaitBound wait(kWaitLimitNs);
    bool done = false;
    while (!done && !wait.expired()) done = mbar_try_wait(&M.bar, phase);
    if (done) break;
    // give up, but first wait once more for the copies to leave this memory
    raise_status(status, kStatusSpinTimeout);
    ok = false;
  }
  return shift;
}

// Every write of the tile's nodes [lo, lo + n), in M from place `shift` on
// (load_emit_tile). Two rounds: first each node without octree nodes finds the
// slot of the node above it that has some and keeps it in place of its own
// prefix, which nobody needs; then every node's links go to its own entry and
// its MakeOctNodes write to its parent's. At 16.7M uniform points 0.186 ->
// 0.177 ms against one thread per node on global memory; bound by its L2
// reductions (0.105 ms without them).
__device__ __forceinline__ void emit_tile(EmitSmem& M, const OctArgs& a, const SlotTags& t,
                                          uint32_t lo, uint32_t n, uint32_t shift, int n_brt,
                                          int n_oct) {
  const uint32_t last = (uint32_t)n_brt - 1u, top_slot = (uint32_t)n_oct - 1u;
  const int bits = link_off_bits(n_brt);
  for (uint32_t j = threadIdx.x; j < n; j += kEmitThreads) {
    if (M.counts[shift + j] != 0 || lo + j == 0u) continue;
    uint32_t rn = (uint32_t)M.parent[shift + j], slot = 0;
    for (int step = 0;; ++step) {
      const uint32_t u = rn - lo;
      if (u >= n || step == 32) {
        slot = root_slot(rn, a, last);
        break;
      }
      if (M.counts[shift + u] != 0 || rn == 0u) {
        slot = (uint32_t)M.offsets[shift + u];
        break;
      }
      rn = (uint32_t)M.parent[shift + u];
    }
    M.offsets[shift + j] = (int)slot;
  }
  __syncthreads();
  for (uint32_t j = threadIdx.x; j < n; j += kEmitThreads) {
    const uint32_t at = shift + j;
    EmitNode e;
    e.i = (int)(lo + j);
    e.k = min(M.counts[at], kMaxSteps);
    e.base = M.offsets[at];  // or the slot its links go to
    e.code = M.codes[at];
    e.level = M.pn[at] / 3u;
    if (e.k > 0 && e.i >= 1) {
      const uint32_t par = (uint32_t)M.parent[at], u = par - lo;
      emit_make(e, u < n ? (uint32_t)M.offsets[shift + u] : root_slot(par, a, last), t, top_slot);
    }
    const uint32_t lc = min((uint32_t)M.left[at], last), v = lc - lo;
    if (M.hll[at])
      emit_leaf(e.i, e.level, (uint32_t)e.base, v <= n ? M.codes[shift + v] : a.codes[lc],
                left_field((uint32_t)e.i - lc, bits), bits, t, top_slot);
    if (M.hlr[at])
      emit_leaf(e.i, e.level, (uint32_t)e.base, v < n ? M.codes[shift + v + 1u] : a.codes[lc + 1u],
                right_field(lc + 1u - (uint32_t)e.i, bits), bits, t, top_slot);
  }
}

// The 15 words of slot p, from the slot tags.
__device__ __forceinline__ void finalize_slots(int p, const OctArgs& a, const SlotTags& t,
                                               int n_brt, int root_level, int* w) {
  const uint32_t last = (uint32_t)n_brt - 1u;
  const uint4* c4 = reinterpret_cast<const uint4*>(t.child);
  const uint4 ta = c4[2 * (uint32_t)p], tb = c4[2 * (uint32_t)p + 1u];
  const uint32_t m = t.mask[(uint32_t)t.at + (uint32_t)p];
  uint32_t own = p > 0 ? t.node[p] : 0u;
  if (own == 0u && p > 0) {
    // not in a tile's own slots (a tile's first few): the nearest node before it
    // whose slots reach p
    for (int d = 1; d < kMaxSteps && d < p; ++d) {
      const uint32_t e = t.node[p - d];
      if ((e & 15u) == 0u && e != 0u && a.counts[min(e >> 4, last)] > d) {
        own = e + (uint32_t)d;
        break;
      }
    }
  }
  const int j = (int)(own & 15u);
  own = min(own >> 4, last);  // 0: none
  // slot 0 is the root's: the corner of node 0's cell, the whole range
  const bool owned = own != 0u || p == 0;
  int pn = 0;
  uint32_t code = 0;
  if (owned) {
    pn = a.prefix_n[own];
    code = a.codes[own];
  }
  const uint32_t tags[8] = {ta.x, ta.y, ta.z, ta.w, tb.x, tb.y, tb.z, tb.w};
  const int b = link_off_bits(n_brt);
  const uint32_t field = (2u << b) - 1u;
  uint32_t far = 0;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    // both kinds by selects (a warp holds both): 0 for no tag
    const uint32_t g = tags[c];
    const bool link = (int)g < 0;
    const uint32_t x = g & ~kLinkTag;
    const uint32_t m = link ? field : 15u;
    const uint32_t low = x & m;
    const uint32_t high = x >> (link ? b + 1 : 4);
    w[c] = (int)(high + low - (link ? 1u << b : 0u));
    far |= link && ((low + 1u) & m) < 2u ? 1u << c : 0u;
  }
  while (far) {
    const int c = __ffs(far) - 1;
    far &= far - 1u;
    const uint32_t g = t.child[(uint32_t)p * 8u + (uint32_t)c];
    w[c] = a.left_child[min((g & ~kLinkTag) >> (b + 1), last)] + (int)(g & 1u);
  }
  float4 corner = make_float4(0.f, 0.f, 0.f, 0.f);
  float cell = 0.f;
  if (owned) {
    const int level = p == 0 ? root_level : pn / 3 - j;
    const int sh = 30 - 3 * level;
    corner = decode_corner((code >> sh) << sh, a.min_coord, a.range);
    cell = p == 0 ? a.range : cell_size(a.range, level - root_level);
  }
  w[8] = __float_as_int(corner.x);
  w[9] = __float_as_int(corner.y);
  w[10] = __float_as_int(corner.z);
  w[11] = __float_as_int(corner.w);
  w[12] = __float_as_int(cell);
  w[13] = (int)m;
  w[14] = 0;
}

// One thread per slot computes the node; the block stages its 256 nodes
// (15 KB) in shared memory and writes them as consecutive 32-bit words, so
// every warp store is one contiguous 128-byte line.
constexpr int kFinThreads = 256;
constexpr int kNodeWords = 15;

// The 15 words of slot p (children, corner, cell_size, masks) into w.
__device__ __forceinline__ void finalize_slot(bool fresh, int p, const OctArgs& a,
                                              const OctTags& t, int root_level, int* w) {
  const uint4* c4 = reinterpret_cast<const uint4*>(t.child);
  const uint4 ta = c4[2 * p], tb = c4[2 * p + 1];
  const uint32_t tags[8] = {ta.x, ta.y, ta.z, ta.w, tb.x, tb.y, tb.z, tb.w};
  const oct_node* nd = a.nodes + p;
  const uint32_t m = t.mask[p];
  const uint32_t own = t.owner[p];
  // Every table read below depends only on the tags: issue them all at once.
  int base[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const uint32_t g = tags[c];
    const int* src = (g & kLinkTag) ? a.left_child + ((g & ~kLinkTag) >> 1)
                                    : a.offsets + ((g - 1u) >> 4);
    base[c] = 0;
    if (g != 0) base[c] = __ldg(src);
  }
  int own_off = 0, own_pn = 0;
  uint32_t own_code = 0;
  if (own != 0) {
    own_off = __ldg(a.offsets + own);
    own_pn = __ldg(a.prefix_n + own);
    own_code = __ldg(a.codes + own);
  }
  uint32_t link_bits = 0;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const uint32_t g = tags[c];
    int v;
    if (g == 0) {
      v = fresh ? 0 : nd->children[c];
    } else if (g & kLinkTag) {
      v = base[c] + (int)(g & 1u);
      link_bits |= 1u << c;
    } else {
      v = base[c] + (int)((g - 1u) & 15u);
    }
    w[c] = v;
  }
  float4 corner;
  float cell;
  if (own != 0) {
    const int j = p - own_off;
    const int level = own_pn / 3 - j;
    const int sh = 30 - 3 * level;
    corner = decode_corner((own_code >> sh) << sh, a.min_coord, a.range);
    cell = cell_size(a.range, level - root_level);
  } else if (fresh && p == 0) {
    const int sh = 30 - 3 * root_level;
    corner = decode_corner((a.codes[0] >> sh) << sh, a.min_coord, a.range);
    cell = a.range;
  } else if (fresh) {
    corner = make_float4(0.f, 0.f, 0.f, 0.f);
    cell = 0.f;
  } else {
    corner = make_float4(nd->corner.x, nd->corner.y, nd->corner.z, nd->corner.w);
    cell = nd->cell_size;
  }
  w[8] = __float_as_int(corner.x);
  w[9] = __float_as_int(corner.y);
  w[10] = __float_as_int(corner.z);
  w[11] = __float_as_int(corner.w);
  w[12] = __float_as_int(cell);
  if (fresh) {
    w[13] = (int)m;
    w[14] = 0;
  } else {
    w[13] = nd->child_node_mask | (int)m;
    w[14] = nd->child_leaf_mask & ~(int)link_bits;
  }
}

// The block's staged nodes to dst[0, count): one bulk copy (the TMA engine
// writes it) when dst is 16-byte aligned and the block a whole number of
// 16-byte words, else vector and word stores. The block's threads call it
// after staging; the stage is free again when it returns, the copy done when
// thread 0 has waited for it (bulk_wait_all), as it does before its kernel ends.
__device__ __forceinline__ void store_node_block(const int* s_nodes, oct_node* nodes, int count) {
  bulk_fence_writes();
  __syncthreads();
  int* dst = reinterpret_cast<int*>(nodes);
  const int words = count * kNodeWords;
  const bool aligned = (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
  if (aligned && (words & 3) == 0) {
    if (threadIdx.x == 0) {
      bulk_store_s2g(dst, s_nodes, (uint32_t)words * 4u);
      bulk_wait_read();
    }
  } else {
    const int quads = aligned ? words >> 2 : 0;
    const uint4* src4 = reinterpret_cast<const uint4*>(s_nodes);
    uint4* dst4 = reinterpret_cast<uint4*>(dst);
    for (int k = threadIdx.x; k < quads; k += blockDim.x) dst4[k] = src4[k];
    for (int k = 4 * quads + threadIdx.x; k < words; k += blockDim.x) dst[k] = s_nodes[k];
  }
  __syncthreads();
}

}  // namespace octgb

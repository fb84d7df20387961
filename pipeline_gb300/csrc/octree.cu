// Stages 7-8: octree nodes and leaf links.
//
// Replaces k_MakeOctNodes / k_LinkLeafNodes (reference
// include/kernels/07_octree.hpp:5-25, include/shared/oct.h:9-134; GPU form
// kernels/cuda/07_octree.cu:8-67) and the caller's root set-up
// (apps/cpu_demo/main.cpp:125-132).
//
// The reference's node slots come from an inclusive prefix sum, so the slot
// ranges of consecutive radix nodes overlap and several radix nodes write the
// same OctNode fields; its parallel loops then race. The contract is the
// result of a sequential run in ascending radix-node order (LinkLeaf's left
// write before its right one, all LinkLeaf writes after all MakeOctNodes
// writes). The GPU reproduces it without ordering threads:
//
//   emit      one thread per radix node computes every write it would make
//             and records, per (slot, child), the largest sequence tag
//             (atomicMax), per slot the largest writer of corner/cell_size,
//             and ORs child_node_mask bits;
//   finalize  one thread per slot turns the winning tags back into values
//             (a tag names its radix node and step) and writes the 60-byte
//             node once, coalesced.
//
// Sequence tags (32-bit, larger = later), of the stage entries and of clouds above
// kSlotTagMaxPoints points:
//   MakeOctNodes step j of node i : ((i << 4) | j) + 1        (i < 2^27)
//   LinkLeafNodes side s of node i: 0x80000000 | (i << 1) | s
// Whole and batched builds take slot tags (octree.cuh), which name their values:
// no owner tag, a mask byte per slot, and a CTA emits a tile of radix nodes that
// bulk copies bring to shared memory.
#include <algorithm>

#include "octree.cuh"

namespace octgb {

size_t oct_tags_bytes(int cap) {
  const size_t c = cap > 0 ? (size_t)cap : 1;
  return align_up(c * 8 * 4, 256) + align_up(c * 4, 256) * 2;
}

OctTags oct_tags_carve(void* base, int cap) {
  const size_t c = cap > 0 ? (size_t)cap : 1;
  char* p = static_cast<char*>(base);
  OctTags t;
  t.child = reinterpret_cast<uint32_t*>(p);
  p += align_up(c * 8 * 4, 256);
  t.owner = reinterpret_cast<uint32_t*>(p);
  p += align_up(c * 4, 256);
  t.mask = reinterpret_cast<uint32_t*>(p);
  t.cap = cap;
  return t;
}

__global__ void __launch_bounds__(256) oct_zero_kernel(OctArgs a, OctTags t,
                                                       uint32_t* __restrict__ status) {
  chain_enter();
  const Sizes z = read_sizes(a);
  if (!z.fits) {
    if (blockIdx.x == 0 && threadIdx.x == 0) raise_status(status, kStatusCapacity);
    return;
  }
  if (z.n_oct > 0)
    clear_tag_range(t, 0, (size_t)z.n_oct - 1, blockIdx.x * blockDim.x + threadIdx.x,
                    gridDim.x * blockDim.x);
}

__global__ void __launch_bounds__(256, 8) oct_emit_kernel(int mode, OctArgs a, OctTags t,
                                                       uint32_t* __restrict__ status,
                                                       bool report_capacity) {
  chain_enter();
  const Sizes z = read_sizes(a);
  if (!z.fits) {
    if (report_capacity && blockIdx.x == 0 && threadIdx.x == 0) raise_status(status, kStatusCapacity);
    return;
  }
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < z.n_brt; i += stride)
    emit_node(mode, i, a, t, z, status);
}

__global__ void __launch_bounds__(kFinThreads, 8) oct_finalize_kernel(int mode, OctArgs a, OctTags t) {
  chain_enter();
  __shared__ __align__(16) int s_nodes[kFinThreads * kNodeWords];
  const Sizes z = read_sizes(a);
  if (!z.fits || z.n_brt < 1) return;
  const int root_level = a.prefix_n[0] / 3;
  const bool fresh = mode & kOctFresh;
  for (int blk = blockIdx.x * kFinThreads; blk < z.n_oct; blk += gridDim.x * kFinThreads) {
    const int p = blk + threadIdx.x;
    if (p < z.n_oct) finalize_slot(fresh, p, a, t, root_level, s_nodes + threadIdx.x * kNodeWords);
    store_node_block(s_nodes, a.nodes + blk, min(kFinThreads, z.n_oct - blk));
  }
  if (threadIdx.x == 0) bulk_wait_all();
}

// The same stages with slot tags (whole builds).
__global__ void __launch_bounds__(kEmitThreads, 8)
    slot_emit_kernel(OctArgs a, SlotTags t, uint32_t* __restrict__ status) {
  chain_enter();
  __shared__ EmitSmem M;
  const Sizes z = read_sizes(a);
  if (!z.fits) {
    if (blockIdx.x == 0 && threadIdx.x == 0) raise_status(status, kStatusCapacity);
    return;
  }
  const int lo = (int)blockIdx.x * kEmitTile;
  if (lo >= z.n_brt) return;
  const int n = min(kEmitTile, z.n_brt - lo);
  if (threadIdx.x == 0) mbar_init(&M.bar, 1);
  bool ok;
  const uint32_t shift = load_emit_tile(M, a, 0u, (uint32_t)lo, (uint32_t)n,
                                        (uint32_t)a.n_brt_host, 0u, status, ok);
  if (!ok) return;
  emit_tile(M, a, t, (uint32_t)lo, (uint32_t)n, shift, z.n_brt, z.n_oct);
}

__global__ void __launch_bounds__(kFinThreads, 8) slot_finalize_kernel(OctArgs a, SlotTags t) {
  chain_enter();
  __shared__ __align__(16) int s_nodes[kFinThreads * kNodeWords];
  const Sizes z = read_sizes(a);
  if (!z.fits || z.n_brt < 1) return;
  const int root_level = a.prefix_n[0] / 3;
  for (int blk = blockIdx.x * kFinThreads; blk < z.n_oct; blk += gridDim.x * kFinThreads) {
    const int p = blk + threadIdx.x;
    if (p < z.n_oct) finalize_slots(p, a, t, z.n_brt, root_level, s_nodes + threadIdx.x * kNodeWords);
    store_node_block(s_nodes, a.nodes + blk, min(kFinThreads, z.n_oct - blk));
  }
  if (threadIdx.x == 0) bulk_wait_all();
}

cudaError_t launch_octree(int mode, const OctArgs& a, const OctTags& t, uint32_t* status,
                          cudaStream_t s, Recorder* rec, bool tags_clear, bool slots) {
  cudaError_t e;
  if (!tags_clear) {
    const int zgrid = device_sm_count() * 8;
    e = launch_chained(oct_zero_kernel, dim3(zgrid), dim3(256), 0, s, a, t, status);
    if (e != cudaSuccess) return e;
    mark(rec, s);
  }
  int nb = a.d_unique ? a.n_brt_host : a.n_brt_host;
  int egrid = (nb + 255) / 256;
  if (egrid < 1) egrid = 1;
  if (slots)
    e = launch_chained(slot_emit_kernel, dim3((std::max(nb, 1) + kEmitTile - 1) / kEmitTile),
                       dim3(kEmitThreads), 0, s, a, slot_tags(t, 0, a.cap), status);
  else
    e = launch_chained(oct_emit_kernel, dim3(egrid), dim3(256), 0, s, mode, a, t, status,
                       tags_clear);
  if (e != cudaSuccess) return e;
  mark(rec, s);
  // One wave at 8 CTAs per SM, each walking the 256-slot blocks: the node
  // count is known only on the device, and a grid sized by the capacity would
  // leave its CTAs past the last node to start, wait and exit in the tail.
  int fgrid = (a.cap + kFinThreads - 1) / kFinThreads;
  fgrid = std::min(fgrid, device_sm_count() * 8);
  if (fgrid < 1) fgrid = 1;
  if (slots)
    e = launch_chained(slot_finalize_kernel, dim3(fgrid), dim3(kFinThreads), 0, s, a,
                       slot_tags(t, 0, a.cap));
  else
    e = launch_chained(oct_finalize_kernel, dim3(fgrid), dim3(kFinThreads), 0, s, mode, a, t);
  if (e == cudaSuccess) mark(rec, s);
  return e;
}

__global__ void publish_counts_kernel(const int* d_unique, const int* d_max_slot,
                                      const uint32_t* status, int* out) {
  chain_enter();
  const int u = *d_unique;
  const int b = max(u - 1, 0);
  out[0] = u;
  out[1] = b;
  out[2] = b >= 1 ? *d_max_slot + 1 : 0;
  out[3] = status ? (int)*status : 0;
}

cudaError_t launch_publish_counts(const int* d_unique, const int* d_max_slot,
                                  const uint32_t* status, int* out, cudaStream_t s) {
  return launch_chained(publish_counts_kernel, dim3(1), dim3(1), 0, s, d_unique, d_max_slot, status,
                        out);
}

}  // namespace octgb

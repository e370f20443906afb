// Four-wide form of a hierarchy for the main traversal: wide nodes over sibling pairs and the
// primitives of each leaf regrouped two by two (layout.h). Derived on the device from the pair
// nodes and leaf-ordered records whenever those change (upload, refit, per-frame rebuild), so every
// way of building the hierarchy ends here and the launches can be captured in a graph.
//
// Leaf pairs are packed without gaps: a leaf of c primitives takes the next ceil(c / 2). Where a
// record goes is a running sum over the records before it, whatever the size of their leaves: a
// record opens a pair when it starts a leaf or follows a full pair of its leaf. The scan therefore
// runs over the maps (records placed, last pair half full) -> (the same, one record later), which
// compose; a thread per leaf instead took 4 ms more on an upload with one leaf of 100,000
// coincident spheres (coincident centroids are never split).
#include <cuda_runtime.h>
#include <math_constants.h>

#include "wide_build.h"

namespace tcb {
namespace {

constexpr int kBlock = 256;
constexpr int kPer = int(kWideChunk) / kBlock;

__device__ __forceinline__ uint32_t tag_of(const PrimRecord* prims, uint32_t k) {
  return __float_as_uint(prims[k].a[3]);
}
__device__ __forceinline__ bool starts_leaf(const PrimRecord* prims, uint32_t k) {
  return k == 0 || (tag_of(prims, k - 1) & kTagLast) != 0u;
}

// State before a record: pairs opened << 1 | whether the last one has room. A Step maps the low bit
// to (pairs opened << 1 | low bit after), so applying it is an addition.
struct Step {
  uint32_t full, half;  // from a full last pair, from a half full one
};
__device__ __forceinline__ uint32_t apply(uint32_t state, Step s) {
  return (state & ~1u) + ((state & 1u) ? s.half : s.full);
}
__device__ __forceinline__ Step compose(Step a, Step b) { return Step{apply(a.full, b), apply(a.half, b)}; }
__device__ __forceinline__ Step identity() { return Step{0u, 1u}; }
__device__ __forceinline__ Step step_of(const PrimRecord* prims, uint32_t k, uint32_t n) {
  if (k >= n) return identity();
  return starts_leaf(prims, k) ? Step{3u, 3u} : Step{3u, 0u};
}

// Composition of the steps of the threads before this one; `total` gets the whole block's.
__device__ __forceinline__ Step block_exclusive(Step v, Step* sh, Step& total) {
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  Step incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const Step u{__shfl_up_sync(0xffffffffu, incl.full, o), __shfl_up_sync(0xffffffffu, incl.half, o)};
    if (lane >= unsigned(o)) incl = compose(u, incl);
  }
  if (lane == 31u) sh[warp] = incl;
  Step excl{__shfl_up_sync(0xffffffffu, incl.full, 1), __shfl_up_sync(0xffffffffu, incl.half, 1)};
  if (lane == 0u) excl = identity();
  __syncthreads();
  Step before = identity(), all = identity();
  for (unsigned w = 0; w < blockDim.x / 32; ++w) {
    if (w == warp) before = all;
    all = compose(all, sh[w]);
  }
  __syncthreads();
  total = all;
  return compose(before, excl);
}

// Each chunk's step; a thread owns kPer consecutive records.
__global__ void __launch_bounds__(kBlock) leaf_steps_kernel(const PrimRecord* __restrict__ prims, uint32_t n,
                                                            Step* __restrict__ steps) {
  __shared__ Step sh[kBlock / 32];
  const uint32_t k0 = blockIdx.x * kWideChunk + threadIdx.x * kPer;
  Step v = identity();
  for (int i = 0; i < kPer; ++i) v = compose(v, step_of(prims, k0 + i, n));
  Step total;
  block_exclusive(v, sh, total);
  if (threadIdx.x == 0) steps[blockIdx.x] = total;
}

// Chunk steps into the states the chunks start from (in `full`).
__global__ void __launch_bounds__(1024) leaf_scan_kernel(Step* __restrict__ steps, uint32_t chunks) {
  __shared__ Step sh[32];
  uint32_t run = 0;
  for (uint32_t base = 0; base < chunks; base += 1024) {
    const uint32_t i = base + threadIdx.x;
    const Step v = i < chunks ? steps[i] : identity();
    Step total;
    const Step before = block_exclusive(v, sh, total);
    if (i < chunks) steps[i].full = apply(run, before);
    run = apply(run, total);
  }
}

// lanes[k] = leaf pair of record k << 1 | its place there.
__global__ void __launch_bounds__(kBlock) leaf_lanes_kernel(const PrimRecord* __restrict__ prims, uint32_t n,
                                                            const Step* __restrict__ steps,
                                                            uint32_t* __restrict__ lanes) {
  __shared__ Step sh[kBlock / 32];
  const uint32_t k0 = blockIdx.x * kWideChunk + threadIdx.x * kPer;
  Step own[kPer], v = identity();
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    own[i] = step_of(prims, k0 + i, n);
    v = compose(v, own[i]);
  }
  Step total;
  uint32_t state = apply(steps[blockIdx.x].full, block_exclusive(v, sh, total));
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    if (k0 + i >= n) break;
    const uint32_t after = apply(state, own[i]);
    // The pair opened last is the record's; it is the second one there unless it opened it.
    lanes[k0 + i] = (((after >> 1) - 1u) << 1) | (after >> 1 == state >> 1 ? 1u : 0u);
    state = after;
  }
}

__device__ __forceinline__ uint32_t sphere_flag(uint32_t tag, uint32_t place) {
  return (tag & kTagTriangle) ? 0u : (place ? kPairSphere1 : kPairSphere0);
}

// Record k into its leaf pair; a pair's first record writes the pair's words and, when it has no
// second, that one's zeros.
__device__ __forceinline__ void write_record(const PrimRecord* __restrict__ prims, uint32_t k, uint32_t n,
                                             const uint32_t* __restrict__ lanes, LeafPair* __restrict__ leaves) {
  const PrimRecord r = prims[k];
  const uint32_t lane = lanes[k], place = lane & 1u, tag = __float_as_uint(r.a[3]);
  LeafPair& p = leaves[lane >> 1];
  write_lane(p, place, r);
  if (place) return;
  uint32_t flags = sphere_flag(tag, 0u);
  if ((tag & kTagLast) || k + 1 >= n) {
    flags |= kPairLast;
    write_lane(p, 1u, PrimRecord{});
  } else {
    const uint32_t next = tag_of(prims, k + 1);
    flags |= sphere_flag(next, 1u) | ((next & kTagLast) ? kPairLast : 0u);
  }
  p.first = k;
  p.flags = flags;
}

// Half of a wide node: planes and links of what child `half` of pair p leads to.
__device__ __forceinline__ void write_half(const PairNode* __restrict__ pairs, uint32_t p, uint32_t half,
                                           const uint32_t* __restrict__ lanes, WideNode* __restrict__ nodes) {
  ChildRec g[2];
  wide_children(pairs, pairs[p].child[half], g);
  write_planes(nodes[p], p, half, g);
  uint2 links;
  uint32_t* l = &links.x;
#pragma unroll
  for (int k = 0; k < 2; ++k)
    l[k] = (g[k].link & kLeafBit) && g[k].count ? kLeafBit | (lanes[g[k].link & ~kLeafBit] >> 1) : g[k].link;
  *reinterpret_cast<uint2*>(&nodes[p].quad[6u ^ (p & 7u)][2 * half]) = links;
}

// One thread per record, then one per half of a wide node.
__global__ void __launch_bounds__(kBlock) wide_write_kernel(const PairNode* __restrict__ pairs, uint32_t pair_count,
                                                            const PrimRecord* __restrict__ prims, uint32_t n,
                                                            const WideForm wide) {
  const uint64_t i = uint64_t(blockIdx.x) * kBlock + threadIdx.x;
  if (i < n) {
    write_record(prims, uint32_t(i), n, wide.lanes, wide.leaves);
  } else {
    const uint64_t h = i - n;
    if (h < 2 * uint64_t(pair_count)) write_half(pairs, uint32_t(h >> 1), uint32_t(h & 1u), wide.lanes, wide.nodes);
  }
}

}  // namespace

cudaError_t launch_wide_write(const PairNode* pairs, uint32_t pair_count, const PrimRecord* prims, uint32_t prim_count,
                              const WideForm& wide, cudaStream_t stream) {
  if (prim_count == 0) return cudaSuccess;
  const uint64_t threads = uint64_t(prim_count) + 2 * uint64_t(pair_count);
  wide_write_kernel<<<unsigned((threads + kBlock - 1) / kBlock), kBlock, 0, stream>>>(pairs, pair_count, prims,
                                                                                      prim_count, wide);
  return cudaGetLastError();
}

cudaError_t launch_wide_build(const PairNode* pairs, uint32_t pair_count, const PrimRecord* prims, uint32_t prim_count,
                              const WideForm& wide, cudaStream_t stream) {
  if (prim_count == 0) return cudaSuccess;
  const uint32_t chunks = (prim_count + kWideChunk - 1) / kWideChunk;
  Step* steps = reinterpret_cast<Step*>(wide.lanes + wide_lane_words(prim_count));
  leaf_steps_kernel<<<chunks, kBlock, 0, stream>>>(prims, prim_count, steps);
  leaf_scan_kernel<<<1, 1024, 0, stream>>>(steps, chunks);
  leaf_lanes_kernel<<<chunks, kBlock, 0, stream>>>(prims, prim_count, steps, wide.lanes);
  return launch_wide_write(pairs, pair_count, prims, prim_count, wide, stream);
}

}  // namespace tcb

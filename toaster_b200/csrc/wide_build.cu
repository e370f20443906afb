// Four-wide form of a hierarchy for the main traversal: wide nodes over sibling pairs and the
// primitives of each leaf regrouped two by two (layout.h). Derived on the device from the pair
// nodes and leaf-ordered records whenever those change (upload, refit, per-frame rebuild), so every
// way of building the hierarchy ends here and the launches can be captured in a graph.
//
// Leaf pairs are packed without gaps: leaf j starts at the sum of ceil(count / 2) over the leaves
// before it, from a two-level scan over the records (per-chunk sums, their scan, then each leaf's
// first record finds its place and writes its leaf).
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

// Pairs that record k adds: ceil(leaf size / 2) at a leaf's first record, else 0.
__device__ __forceinline__ uint32_t pairs_at(const PrimRecord* prims, uint32_t k, uint32_t n) {
  if (k >= n || (k > 0 && !(tag_of(prims, k - 1) & kTagLast))) return 0u;
  uint32_t c = 1;
  while (!(tag_of(prims, k + c - 1) & kTagLast) && k + c < n) ++c;
  return (c + 1) / 2;
}

// Exclusive sum of one value per thread over the block; `total` gets the block's sum.
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t* sh, uint32_t& total) {
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= unsigned(o)) incl += u;
  }
  if (lane == 31u) sh[warp] = incl;
  __syncthreads();
  uint32_t before = 0, all = 0;
  for (unsigned w = 0; w < blockDim.x / 32; ++w) {
    if (w < warp) before += sh[w];
    all += sh[w];
  }
  __syncthreads();
  total = all;
  return before + incl - v;
}

// Chunk sums; each thread owns kPer consecutive records.
__global__ void __launch_bounds__(kBlock) leaf_sums_kernel(const PrimRecord* __restrict__ prims, uint32_t n,
                                                           uint32_t* __restrict__ sums) {
  __shared__ uint32_t sh[kBlock / 32];
  const uint32_t k0 = blockIdx.x * kWideChunk + threadIdx.x * kPer;
  uint32_t v = 0;
  for (int i = 0; i < kPer; ++i) v += pairs_at(prims, k0 + i, n);
  uint32_t total;
  block_exclusive(v, sh, total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(1024) leaf_scan_kernel(uint32_t* __restrict__ sums, uint32_t chunks) {
  __shared__ uint32_t sh[32];
  uint32_t run = 0;
  for (uint32_t base = 0; base < chunks; base += 1024) {
    const uint32_t i = base + threadIdx.x;
    const uint32_t v = i < chunks ? sums[i] : 0u;
    uint32_t total;
    const uint32_t before = block_exclusive(v, sh, total);
    if (i < chunks) sums[i] = run + before;
    run += total;
  }
}

__device__ void write_leaf(const PrimRecord* __restrict__ prims, uint32_t k, uint32_t n, LeafPair* __restrict__ out) {
  for (;;) {
    LeafPair p{};
    p.first = k;
    bool last = false;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      if (last) break;
      const PrimRecord r = prims[k];
      const uint32_t tag = __float_as_uint(r.a[3]);
      p.nv0x[i] = -r.a[0];
      p.nv0y[i] = -r.a[1];
      p.nv0z[i] = -r.a[2];
      p.e1x[i] = r.b[0];
      p.e1y[i] = r.b[1];
      if (tag & kTagTriangle) {
        p.e1z[i] = r.b[2];
        p.e2x[i] = r.c[0];
        p.ne2y[i] = -r.c[1];
        p.ne2z[i] = -r.c[2];
      } else {
        p.flags |= i ? kPairSphere1 : kPairSphere0;
      }
      ++k;
      last = (tag & kTagLast) != 0u || k >= n;
    }
    if (last) p.flags |= kPairLast;
    *out++ = p;
    if (last) return;
  }
}

// slot[k] = first leaf pair of the leaf that starts at record k (other entries unused).
__global__ void __launch_bounds__(kBlock) leaf_write_kernel(const PrimRecord* __restrict__ prims, uint32_t n,
                                                            const uint32_t* __restrict__ sums,
                                                            uint32_t* __restrict__ slot,
                                                            LeafPair* __restrict__ leaves) {
  __shared__ uint32_t sh[kBlock / 32];
  const uint32_t k0 = blockIdx.x * kWideChunk + threadIdx.x * kPer;
  uint32_t need[kPer], v = 0;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    need[i] = pairs_at(prims, k0 + i, n);
    v += need[i];
  }
  uint32_t total;
  uint32_t at = sums[blockIdx.x] + block_exclusive(v, sh, total);
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    if (!need[i]) continue;
    slot[k0 + i] = at;
    write_leaf(prims, k0 + i, n, leaves + at);
    at += need[i];
  }
}

// One thread per half of a wide node.
__global__ void __launch_bounds__(kBlock) wide_nodes_kernel(const PairNode* __restrict__ pairs, uint32_t n,
                                                            const uint32_t* __restrict__ slot,
                                                            WideNode* __restrict__ nodes) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t p = i >> 1, half = i & 1u;
  if (p >= n) return;
  const ChildRec c = pairs[p].child[half];
  ChildRec g[2];
  if (c.link & kLeafBit) {
    g[0] = c;
    g[1] = ChildRec{CUDART_INF_F, CUDART_INF_F, CUDART_INF_F, kLeafBit, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, 0u};
  } else {
    g[0] = pairs[c.link].child[0];
    g[1] = pairs[c.link].child[1];
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint32_t link = (g[k].link & kLeafBit) && g[k].count ? kLeafBit | slot[g[k].link & ~kLeafBit] : g[k].link;
    const float f[6] = {g[k].min_x, g[k].max_x, g[k].min_y, g[k].max_y, g[k].min_z, g[k].max_z};
    const uint32_t j = 2 * half + k;
#pragma unroll
    for (uint32_t q = 0; q < 6; ++q) nodes[p].quad[q ^ (p & 7u)][j] = __float_as_uint(f[q]);
    nodes[p].quad[6u ^ (p & 7u)][j] = link;
  }
}

}  // namespace

cudaError_t launch_wide_build(const PairNode* pairs, uint32_t pair_count, const PrimRecord* prims,
                              uint32_t prim_count, uint32_t* scan, WideNode* nodes, LeafPair* leaves,
                              cudaStream_t stream) {
  if (prim_count == 0) return cudaSuccess;
  const uint32_t chunks = (prim_count + kWideChunk - 1) / kWideChunk;
  uint32_t* slot = scan;
  uint32_t* sums = scan + prim_count;
  leaf_sums_kernel<<<chunks, kBlock, 0, stream>>>(prims, prim_count, sums);
  leaf_scan_kernel<<<1, 1024, 0, stream>>>(sums, chunks);
  leaf_write_kernel<<<chunks, kBlock, 0, stream>>>(prims, prim_count, sums, slot, leaves);
  if (pair_count)
    wide_nodes_kernel<<<unsigned((2 * uint64_t(pair_count) + kBlock - 1) / kBlock), kBlock, 0, stream>>>(
        pairs, pair_count, slot, nodes);
  return cudaGetLastError();
}

}  // namespace tcb

// Four-wide form of an uploaded hierarchy (wide_build.cu).
#ifndef TOASTER_B200_WIDE_BUILD_H
#define TOASTER_B200_WIDE_BUILD_H

#include <cuda_runtime.h>
#include <math_constants.h>
#include <stddef.h>
#include <stdint.h>

#include "layout.h"

namespace tcb {

constexpr uint32_t kWideChunk = 1024;  // primitive records per block of the leaf scan

// Leaf pairs of `prims` primitives whose hierarchy has `pairs` interior nodes: a leaf of c
// primitives takes ceil(c / 2), at most (c + 1) / 2, and there are pairs + 1 leaves.
inline size_t max_leaf_pairs(size_t prims, size_t pairs) { return (prims + pairs + 1) / 2; }

// The form's device memory. nodes: one per pair (at least one); leaves: max_leaf_pairs; lanes:
// wide_scan_words words, the leaf pair and place of every primitive record (wide_lane_words) followed
// by the scan's scratch. Null nodes: no form.
struct WideForm {
  WideNode* nodes = nullptr;
  LeafPair* leaves = nullptr;
  uint32_t* lanes = nullptr;
};
inline size_t wide_lane_words(size_t prims) { return (prims + 1) & ~size_t(1); }
inline size_t wide_scan_words(size_t prims) {
  return wide_lane_words(prims) + 2 * ((prims + kWideChunk - 1) / kWideChunk);
}

// Writes the whole form of a hierarchy; four launches on `stream`.
cudaError_t launch_wide_build(const PairNode* pairs, uint32_t pair_count, const PrimRecord* prims, uint32_t prim_count,
                              const WideForm& wide, cudaStream_t stream);
// The same for a hierarchy of the shape the form was last built for (its lanes stand); one launch.
cudaError_t launch_wide_write(const PairNode* pairs, uint32_t pair_count, const PrimRecord* prims, uint32_t prim_count,
                              const WideForm& wide, cudaStream_t stream);

#ifdef __CUDACC__
// A primitive record as place 0 or 1 of a leaf pair (a sphere's unused words are zero).
__device__ __forceinline__ void write_lane(LeafPair& p, uint32_t place, const PrimRecord& r) {
  p.nv0x[place] = -r.a[0];
  p.nv0y[place] = -r.a[1];
  p.nv0z[place] = -r.a[2];
  p.e1x[place] = r.b[0];
  p.e1y[place] = r.b[1];
  p.e1z[place] = r.b[2];
  p.e2x[place] = r.c[0];
  p.ne2y[place] = -r.c[1];
  p.ne2z[place] = -r.c[2];
}

// What child c of a pair contributes to the pair's wide node: its children, or itself and an empty
// box when it is a leaf.
__device__ __forceinline__ void wide_children(const PairNode* pairs, const ChildRec& c, ChildRec (&g)[2]) {
  if (c.link & kLeafBit) {
    g[0] = c;
    g[1] = ChildRec{CUDART_INF_F,  CUDART_INF_F,  CUDART_INF_F,  kLeafBit,
                    -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, 0u};
  } else {
    g[0] = pairs[c.link].child[0];
    g[1] = pairs[c.link].child[1];
  }
}
__device__ __forceinline__ void write_planes(WideNode& node, uint32_t p, uint32_t half, const ChildRec (&g)[2]) {
  auto put = [&](uint32_t q, float a, float b) {
    *reinterpret_cast<float2*>(&node.quad[q ^ (p & 7u)][2 * half]) = make_float2(a, b);
  };
  put(0, g[0].min_x, g[1].min_x);
  put(1, g[0].max_x, g[1].max_x);
  put(2, g[0].min_y, g[1].min_y);
  put(3, g[0].max_y, g[1].max_y);
  put(4, g[0].min_z, g[1].min_z);
  put(5, g[0].max_z, g[1].max_z);
}
#endif

}  // namespace tcb

#endif

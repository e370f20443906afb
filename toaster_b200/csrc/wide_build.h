// Four-wide form of an uploaded hierarchy (wide_build.cu).
#ifndef TOASTER_B200_WIDE_BUILD_H
#define TOASTER_B200_WIDE_BUILD_H

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "layout.h"

namespace tcb {

constexpr uint32_t kWideChunk = 1024;  // primitive records per block of the leaf scan

// Leaf pairs of `prims` primitives whose hierarchy has `pairs` interior nodes: a leaf of c
// primitives takes ceil(c / 2), at most (c + 1) / 2, and there are pairs + 1 leaves.
inline size_t max_leaf_pairs(size_t prims, size_t pairs) { return (prims + pairs + 1) / 2; }
inline size_t wide_scan_words(size_t prims) { return prims + (prims + kWideChunk - 1) / kWideChunk; }

// Writes the wide nodes (one per pair) and leaf pairs of a hierarchy; `scan` is scratch of
// wide_scan_words(prim_count) words. Enqueues four launches on `stream`.
cudaError_t launch_wide_build(const PairNode* pairs, uint32_t pair_count, const PrimRecord* prims,
                              uint32_t prim_count, uint32_t* scan, WideNode* nodes, LeafPair* leaves,
                              cudaStream_t stream);

}  // namespace tcb

#endif

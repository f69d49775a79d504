// Making the four-wide device form of a compact SBVH (tt_wide_build.cu); internal to libtt.so.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "tt_traverse.cuh"
#include "tt_wide.h"

namespace tt {

struct WideBVH {
    void *base = nullptr;  // one allocation: nodes, then pairs (the caller frees it)
    const char *nodes = nullptr, *pairs = nullptr;
    size_t top_bytes = 0;  // the top levels, laid out first
    uint32_t flags = 0;    // BvhView::wide_flags
};

// Makes the four-wide form of the device arrays of `two` (num_nodes and num_verts float4s). out.nodes
// stays nullptr when the tree must stay two-wide: not a tree with every node reachable from the root, a
// box or vertex outside the bounds of tt_wide.h, an inverted box, a child's box that sticks out
// of its parent's, a leaf that is not closed, shares a triangle with another or is longer than
// kLeafTriangles, a stack need above kWideStack, or no device memory for it. Works on the legacy stream
// and waits for it.
cudaError_t build_wide(const BvhView &two, uint32_t num_nodes, uint32_t num_verts, size_t top_bytes, int num_sms,
                       WideBVH &out);

}  // namespace tt

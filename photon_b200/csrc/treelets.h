// The order of a scene's BVH2 nodes on the device: treelets of up to eight nodes, each one after another in
// memory, so that a group of eight lanes reads a treelet's nodes at once (group_walk.cuh). Every other walk
// follows the same nodes by their links.
#pragma once

#include <cuda_runtime.h>

namespace ptw {

constexpr int kTreelet = 8;
constexpr int kTreeletBlock = 512;  // nodes of a tree that one block orders

// The ints of scratch that a tree takes.
inline size_t treelet_work(int num_nodes) { return 4 * size_t(num_nodes) + 4; }

// Writes the tree of `nodes` in treelet order to `ordered` (the root stays node 0) and the size of the root's
// treelet to *root_size, all on the device, in stream order. Up to kTreeletBlock nodes the two may be one array and
// `work` null; else they are apart and `work` has treelet_work ints. In the new order the count word of an inner
// child, which is 0 or less, says more:
//   -1 .. -8     the child starts another treelet, of that many nodes;
//   -16 * mask   it belongs to its parent's treelet; the mask has a bit per way out below it, a leaf or another
//                treelet: bit k for side 0 of the treelet's node k, 8 + k for side 1. Parents precede children.
// `levels`: the tree's (bvh_levels), at least 1.
void order_by_treelets(const float4* nodes, float4* ordered, int* work, int num_nodes, int levels, int* root_size, cudaStream_t stream);

}  // namespace ptw

// The order of a scene's BVH2 nodes on the device: treelets of up to eight nodes, each one after another in
// memory, so that a group of eight lanes reads a treelet's nodes at once (group_walk.cuh). Every other walk
// follows the same nodes by their links.
#pragma once

#include <cuda_runtime.h>

namespace ptw {

constexpr int kTreelet = 8;

template <typename T>
struct DeviceBuffer;

// Puts the device-resident tree into treelet order (the root stays node 0) and returns the size of the root's
// treelet, or 0, with the nodes as they were, where there is no memory for the second copy that this takes
// meanwhile. In the new order the count word of an inner child, which is 0 or less, says more:
//   -1 .. -8     the child starts another treelet, of that many nodes;
//   -16 * mask   it belongs to its parent's treelet; the mask has a bit per way out below it, a leaf or another
//                treelet: bit k for side 0 of the treelet's node k, 8 + k for side 1. Parents precede children.
// `levels`: bvh_levels of the tree, at least 1. `word`: an int of device scratch. Synchronises the stream.
int order_by_treelets(DeviceBuffer<float4>& nodes, int num_nodes, int levels, int* word, cudaStream_t stream);

}  // namespace ptw

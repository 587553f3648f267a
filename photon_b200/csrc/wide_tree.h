// The 8-wide tree of the group walk (group_walk.cuh): a collapse of the scene's BVH2, made on the device at
// upload.
#pragma once

#include <cuda_runtime.h>

namespace ptw {

constexpr int kWide = 8;

template <typename T>
struct DeviceBuffer;

// Fills `wide` (16 float4 per node) with the collapse of an order-free BVH2. Per child two float4 with the BVH2's own box: (low, index) (high, count), where
// count > 0 is a leaf of that many triangles from index on, 0 an inner child whose node index is, and -1
// an unused slot. A node's children are its BVH2 node's, the largest inner ones opened until there are
// eight. `depth`: the BVH2's levels. Synchronises the stream.
void wide_tree_build(const float4* nodes, int num_nodes, int depth, DeviceBuffer<float4>& wide, cudaStream_t stream);

}  // namespace ptw

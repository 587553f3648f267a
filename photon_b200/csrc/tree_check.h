// Whether a scene's BVH may be walked out of Photon's order (DevScene::order_free).
#pragma once

#include <cuda_runtime.h>

namespace ptw {

constexpr int kOrderFreeDepth = 60;  // levels of the tree: Photon's 64-entry stack then never drops a node

// Whether every box of the device-resident tree is finite, ordered and inside its parent's and every leaf's triangles
// lie inside its box (to rounding): *bad, on the device and in stream order, becomes 0 then and 1 otherwise. False, with
// nothing done, where a node has two parents, the tree is more than kOrderFreeDepth levels deep (`levels`: bvh_levels of
// it) or its nodes do not fit the list walk's entries.
bool check_order_free(const float4* nodes, int num_nodes, const float4* tris, int levels, int* bad, cudaStream_t stream);

}  // namespace ptw

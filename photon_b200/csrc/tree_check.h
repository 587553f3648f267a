// Whether a scene's BVH may be walked out of Photon's order (DevScene::order_free).
#pragma once

#include <cuda_runtime.h>

namespace ptw {

constexpr int kOrderFreeDepth = 60;  // levels of the tree: Photon's 64-entry stack then never drops a node

// True when every box of the device-resident tree is finite, ordered and inside its parent's, every leaf's
// triangles lie inside its box (to rounding), no node has two parents and the tree is at most kOrderFreeDepth
// levels deep (`levels`: bvh_levels of it), and its nodes fit the list walk's entries. `word`: an int of device
// scratch. Synchronises the stream.
bool tree_is_order_free(const float4* nodes, int num_nodes, const float4* tris, int levels, int* word, cudaStream_t stream);

}  // namespace ptw

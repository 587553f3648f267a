// The check behind DevScene::order_free: one pass over the nodes, a thread per child. A tree that a
// builder makes passes; a hand-made tree whose boxes are not nested, or do not hold their triangles, is
// walked in Photon's order, on which its hits then depend.
#include "tree_check.h"

#include "device_scene.h"
#include "pt_math.cuh"

namespace ptw {

namespace {

struct Side {
    V3 lo, hi;
    int index, count;
    __device__ bool used() const { return count > 0 || index >= 0; }
};

__device__ __forceinline__ Side side_of(const float4* __restrict__ nodes, int node, int k) {
    const float4 a = nodes[4 * size_t(node) + 2 * k], b = nodes[4 * size_t(node) + 2 * k + 1];
    return Side{xyz(a), xyz(b), __float_as_int(a.w), __float_as_int(b.w)};
}

__device__ __forceinline__ bool inside(V3 p, V3 lo, V3 hi, V3 slack) {
    return p.x >= lo.x - slack.x && p.x <= hi.x + slack.x && p.y >= lo.y - slack.y && p.y <= hi.y + slack.y && p.z >= lo.z - slack.z &&
           p.z <= hi.z + slack.z;
}

__global__ void __launch_bounds__(256) k_check_tree(const float4* __restrict__ nodes, int num_nodes, const float4* __restrict__ tris,
                                                    int* __restrict__ bad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * num_nodes) return;
    const Side s = side_of(nodes, i >> 1, i & 1);
    if (!s.used()) return;
    bool ok = is_finite(s.lo) && is_finite(s.hi) && inside(s.lo, s.lo, s.hi, v3(0)) && inside(s.hi, s.lo, s.hi, v3(0));
    if (s.count > 0) {
        for (int t = s.index; ok && t < s.index + s.count; t++) {
            const float4* g = tris + kTriStride * size_t(t);
            const V3 v0 = xyz(g[0]), e1 = xyz(g[1]), e2 = xyz(g[2]);
            // v1 and v2 are v0 + e1 and v0 + e2 up to the rounding of the edge and of this sum.
            const auto size = [](float a, float b, float c) { return 1e-6f * (fabsf(a) + fabsf(b) + fabsf(c)); };
            const V3 slack{size(v0.x, e1.x, e2.x), size(v0.y, e1.y, e2.y), size(v0.z, e1.z, e2.z)};
            ok = inside(v0, s.lo, s.hi, slack) && inside(v0 + e1, s.lo, s.hi, slack) && inside(v0 + e2, s.lo, s.hi, slack);
        }
    } else {
        for (int k = 0; ok && k < 2; k++) {
            const Side c = side_of(nodes, s.index, k);
            if (c.used()) ok = inside(c.lo, s.lo, s.hi, v3(0)) && inside(c.hi, s.lo, s.hi, v3(0));
        }
    }
    if (!ok) *bad = 1;
}

}  // namespace

bool check_order_free(const float4* nodes, int num_nodes, const float4* tris, int levels, int* bad, cudaStream_t stream) {
    // A list entry keeps 2 * node + side in 27 bits.
    if (levels < 1 || levels > kOrderFreeDepth || num_nodes < 1 || num_nodes >= (1 << 26)) return false;
    PTW_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), stream));
    k_check_tree<<<(2 * num_nodes + 255) / 256, 256, 0, stream>>>(nodes, num_nodes, tris, bad);
    PTW_CUDA(cudaGetLastError());
    return true;
}

}  // namespace ptw

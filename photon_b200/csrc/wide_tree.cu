// The collapse of wide_tree.h, level by level, a thread per node. Opening the child of largest area first
// visits 13.7 nodes per incoherent ray of the 262K scene where the BVH2 walk visits 38.4 (the collapse of
// least summed area: 12.8).
#include "wide_tree.h"

#include <algorithm>

#include "device_scene.h"
#include "pt_math.cuh"

namespace ptw {

namespace {

struct Side {
    float4 lo, hi;  // with the index and the count
    __device__ int index() const { return __float_as_int(lo.w); }
    __device__ int count() const { return __float_as_int(hi.w); }
    __device__ bool inner() const { return count() <= 0 && index() >= 0; }
    __device__ bool used() const { return count() > 0 || index() >= 0; }
    __device__ float half_area() const {
        const float x = hi.x - lo.x, y = hi.y - lo.y, z = hi.z - lo.z;
        return x * y + y * z + z * x;
    }
};

struct Levels {
    int begin, end;  // the level's nodes
    int count;       // nodes so far
};

__global__ void k_next_level(Levels* st) {
    st->begin = st->end;
    st->end = st->count;
}

// (wide: null only counts.)
__global__ void __launch_bounds__(128) k_collapse(const float4* __restrict__ nodes, float4* __restrict__ wide, int* __restrict__ source,
                                                  Levels* __restrict__ st) {
    for (int n = st->begin + int(blockIdx.x * blockDim.x + threadIdx.x); n < st->end; n += int(gridDim.x * blockDim.x)) {
        Side kid[kWide];
        int kids = 0;
        auto add = [&](int node) {
            for (int k = 0; k < 2; k++) {
                const Side s{nodes[4 * size_t(node) + 2 * k], nodes[4 * size_t(node) + 2 * k + 1]};
                if (s.used()) kid[kids++] = s;
            }
        };
        add(source[n]);
        while (kids < kWide) {
            int open = -1;
            float best = -1.0f;
            for (int k = 0; k < kids; k++)
                if (kid[k].inner() && kid[k].half_area() > best) {
                    best = kid[k].half_area();
                    open = k;
                }
            if (open < 0) break;
            const int from = kid[open].index();
            kid[open] = kid[--kids];
            add(from);
        }
        int inner = 0;
        for (int k = 0; k < kids; k++) inner += kid[k].inner() ? 1 : 0;
        int next = inner ? atomicAdd(&st->count, inner) : 0;
        for (int k = 0; k < kWide; k++) {
            float4 lo = make_float4(0, 0, 0, 0), hi = make_float4(0, 0, 0, __int_as_float(-1));
            if (k < kids) {
                lo = kid[k].lo;
                hi = kid[k].hi;
                if (kid[k].inner()) {
                    source[next] = kid[k].index();
                    lo.w = __int_as_float(next++);
                    hi.w = __int_as_float(0);
                }
            }
            if (wide) {
                wide[2 * kWide * size_t(n) + 2 * k] = lo;
                wide[2 * kWide * size_t(n) + 2 * k + 1] = hi;
            }
        }
    }
}

}  // namespace

// Two passes over the levels: the first counts the nodes, so that the tree is built where it stays and needs no
// room for the most there can be (256 bytes per BVH2 node: 540 MB for 4.19M triangles, whose tree takes 200).
// Both passes of that scene take 0.8 ms of its upload's 400.
void wide_tree_build(const float4* nodes, int num_nodes, int depth, DeviceBuffer<float4>& wide, cudaStream_t stream) {
    DeviceBuffer<Levels> st;
    DeviceBuffer<int> source;
    st.allocate(1);
    source.allocate(size_t(num_nodes));
    const int blocks = std::min((num_nodes + 127) / 128, 148 * 16);  // bound by dependent loads: all the warps an SM holds
    auto pass = [&](float4* out) {
        Levels h{0, 0, 1};  // the first level: the root, whose BVH2 node is 0
        PTW_CUDA(cudaMemcpyAsync(st.ptr, &h, sizeof(h), cudaMemcpyHostToDevice, stream));
        PTW_CUDA(cudaMemsetAsync(source.ptr, 0, sizeof(int), stream));
        for (int level = 0; level < depth; level++) {  // a level of the collapse covers at least one of the BVH2
            k_next_level<<<1, 1, 0, stream>>>(st.ptr);
            k_collapse<<<blocks, 128, 0, stream>>>(nodes, out, source.ptr, st.ptr);
        }
        PTW_CUDA(cudaGetLastError());
        PTW_CUDA(cudaMemcpyAsync(&h, st.ptr, sizeof(h), cudaMemcpyDeviceToHost, stream));
        PTW_CUDA(cudaStreamSynchronize(stream));
        return h.count;
    };
    wide.allocate(size_t(pass(nullptr)) * 2 * kWide);
    pass(wide.ptr);
}

}  // namespace ptw

// The treelet order of treelets.h. A thread per treelet takes the root of a subtree and opens its largest inner
// child until it has eight nodes; the children left start the treelets of the next level. The links are
// written once every node has its place.
#include "treelets.h"

#include <algorithm>

#include "device_scene.h"
#include "pt_math.cuh"

namespace ptw {

namespace {

struct Side {
    float4 lo, hi;  // with the index and the count
    __device__ int index() const { return __float_as_int(lo.w); }
    __device__ int count() const { return __float_as_int(hi.w); }
    __device__ bool leaf() const { return count() > 0; }
    __device__ bool inner() const { return count() <= 0 && index() >= 0; }
    __device__ float half_area() const {
        const float x = hi.x - lo.x, y = hi.y - lo.y, z = hi.z - lo.z;
        return x * y + y * z + z * x;
    }
};
__device__ __forceinline__ Side side_of(const float4* nodes, int node, int k) {
    return Side{nodes[4 * size_t(node) + 2 * k], nodes[4 * size_t(node) + 2 * k + 1]};
}

// Scratch, one entry per node. (Treelets are at most as many as nodes.)
struct Places {
    int* place;  // node -> its place
    int* node;   // place -> the node there
    int* size;   // node -> nodes of the treelet it starts, 0 inside one (cleared before)
    int* root;   // treelet -> the node it starts with
};
struct Levels {
    int begin, end;  // the level's treelets
    int treelets;    // so far
    int nodes;       // with a place, so far
};

__device__ void choose_treelet(const float4* nodes, const Places& p, Levels* st, int t) {
    int member[kTreelet], members = 1, way[kTreelet + 1], ways = 0;
    float area[kTreelet + 1];
    auto add = [&](int node) {
        for (int k = 0; k < 2; k++) {
            const Side s = side_of(nodes, node, k);
            if (!s.inner()) continue;
            way[ways] = s.index();
            area[ways++] = s.half_area();
        }
    };
    const int root = p.root[t];
    member[0] = root;
    add(root);
    while (members < kTreelet && ways > 0) {
        int open = 0;
        for (int k = 1; k < ways; k++)
            if (area[k] > area[open]) open = k;
        const int node = way[open];
        way[open] = way[--ways];
        area[open] = area[ways];
        member[members++] = node;
        add(node);
    }
    const int base = atomicAdd(&st->nodes, members);
    for (int k = 0; k < members; k++) {
        p.place[member[k]] = base + k;
        p.node[base + k] = member[k];
    }
    p.size[root] = members;
    if (ways == 0) return;
    const int next = atomicAdd(&st->treelets, ways);
    for (int k = 0; k < ways; k++) p.root[next + k] = way[k];
}

__device__ void write_treelet(const float4* nodes, float4* out, const Places& p, int t) {
    const int root = p.root[t], base = p.place[root], members = p.size[root];
    uint32_t below[kTreelet];
    for (int j = members - 1; j >= 0; j--) {
        below[j] = 0;
        for (int k = 0; k < 2; k++) {
            Side s = side_of(nodes, p.node[base + j], k);
            if (s.leaf()) {
                below[j] |= 1u << (8 * k + j);
            } else if (s.inner()) {
                const int child = s.index(), size = p.size[child];
                uint32_t mask = 1u << (8 * k + j);
                if (size == 0) mask = below[p.place[child] - base];
                below[j] |= mask;
                s.lo.w = __int_as_float(p.place[child]);
                s.hi.w = __int_as_float(size ? -size : -16 * int(mask));
            } else {
                s.hi.w = __int_as_float(0);
            }
            out[4 * size_t(base + j) + 2 * k] = s.lo;
            out[4 * size_t(base + j) + 2 * k + 1] = s.hi;
        }
    }
}

__global__ void k_next_level(Places p, Levels* st, bool first) {
    if (first) {
        p.root[0] = 0;
        *st = Levels{0, 1, 1, 0};
    } else {
        st->begin = st->end;
        st->end = st->treelets;
    }
}

__global__ void __launch_bounds__(128) k_choose(const float4* __restrict__ nodes, Places p, Levels* st) {
    const int step = int(gridDim.x * blockDim.x);
    for (int t = st->begin + int(blockIdx.x * blockDim.x + threadIdx.x); t < st->end; t += step) choose_treelet(nodes, p, st, t);
}

__global__ void __launch_bounds__(128) k_write(const float4* __restrict__ nodes, float4* __restrict__ out, Places p, const Levels* st,
                                                int* __restrict__ root_size) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *root_size = p.size[0];
    const int step = int(gridDim.x * blockDim.x);
    for (int t = int(blockIdx.x * blockDim.x + threadIdx.x); t < st->treelets; t += step) write_treelet(nodes, out, p, t);
}

// A small tree, by one block in its shared memory (nodes may be ordered).
__global__ void __launch_bounds__(128) k_order_block(const float4* nodes, float4* ordered, int n, int* root_size) {
    __shared__ float4 s_nodes[4 * kTreeletBlock];
    __shared__ int s_places[4][kTreeletBlock];
    __shared__ Levels st;
    const Places p{s_places[0], s_places[1], s_places[2], s_places[3]};
    for (int k = threadIdx.x; k < 4 * n; k += blockDim.x) s_nodes[k] = nodes[k];
    for (int k = threadIdx.x; k < n; k += blockDim.x) p.size[k] = 0;
    if (threadIdx.x == 0) {
        p.root[0] = 0;
        st = Levels{0, 1, 1, 0};
    }
    __syncthreads();
    while (st.begin < st.end) {
        for (int t = st.begin + int(threadIdx.x); t < st.end; t += blockDim.x) choose_treelet(s_nodes, p, &st, t);
        __syncthreads();
        if (threadIdx.x == 0) {
            st.begin = st.end;
            st.end = st.treelets;
        }
        __syncthreads();
    }
    for (int t = threadIdx.x; t < st.treelets; t += blockDim.x) write_treelet(s_nodes, ordered, p, t);
    // (Places left over belong to nodes that the root does not reach: both sides unused.)
    const float none = __int_as_float(-1);
    for (int k = 4 * st.nodes + int(threadIdx.x); k < 4 * n; k += blockDim.x) ordered[k] = make_float4(none, none, none, none);
    if (threadIdx.x == 0) *root_size = p.size[0];
}

}  // namespace

void order_by_treelets(const float4* nodes, float4* ordered, int* work, int num_nodes, int levels, int* root_size, cudaStream_t stream) {
    if (num_nodes <= kTreeletBlock) {
        k_order_block<<<1, 128, 0, stream>>>(nodes, ordered, num_nodes, root_size);
        PTW_CUDA(cudaGetLastError());
        return;
    }
    const size_t n = size_t(num_nodes);
    const Places p{work, work + n, work + 2 * n, work + 3 * n};
    Levels* st = reinterpret_cast<Levels*>(work + 4 * n);
    PTW_CUDA(cudaMemsetAsync(p.size, 0, n * sizeof(int), stream));
    const int blocks = std::min((num_nodes + 127) / 128, 148 * 16);  // bound by dependent loads: all the warps an SM holds
    for (int level = 0; level < levels; level++) {  // a level of treelets covers at least one of the tree
        k_next_level<<<1, 1, 0, stream>>>(p, st, level == 0);
        k_choose<<<blocks, 128, 0, stream>>>(nodes, p, st);
    }
    // (Nodes that the root does not reach leave places over: both sides unused.)
    PTW_CUDA(cudaMemsetAsync(ordered, 0xff, 4 * n * sizeof(float4), stream));
    k_write<<<blocks, 128, 0, stream>>>(nodes, ordered, p, st, root_size);
    PTW_CUDA(cudaGetLastError());
}

}  // namespace ptw

// Device memory helpers and the device-resident scene (host side).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <vector>

#include "photon_wavefront.h"
#include "pt_error.h"
#include "pt_types.h"

namespace ptw {

#define PTW_CUDA(x)                                                                                   \
    do {                                                                                              \
        cudaError_t e_ = (x);                                                                         \
        if (e_ != cudaSuccess)                                                                        \
            throw ::ptw::Error{PT_ERR_CUDA, std::string("CUDA error: ") + cudaGetErrorString(e_) + " (" #x ")"}; \
    } while (0)

// An owning device allocation (counts bytes against an optional budget).
template <typename T>
struct DeviceBuffer {
    T* ptr = nullptr;
    size_t count = 0;
    DeviceBuffer() = default;
    DeviceBuffer(const DeviceBuffer&) = delete;
    DeviceBuffer& operator=(const DeviceBuffer&) = delete;
    DeviceBuffer(DeviceBuffer&& o) noexcept : ptr(o.ptr), count(o.count) {
        o.ptr = nullptr;
        o.count = 0;
    }
    DeviceBuffer& operator=(DeviceBuffer&& o) noexcept {
        if (this != &o) {
            release();
            ptr = o.ptr;
            count = o.count;
            o.ptr = nullptr;
            o.count = 0;
        }
        return *this;
    }
    ~DeviceBuffer() { release(); }
    void release() {
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        count = 0;
    }
    void allocate(size_t n) {
        if (!try_allocate(n)) throw Error{PT_ERR_CUDA, "CUDA error: out of memory (cudaMalloc)"};
    }
    // False, with nothing held and no error left behind for a later call to find, where there is no memory.
    bool try_allocate(size_t n) {
        if (n == count && ptr) return true;
        release();
        if (n == 0) return true;
        const cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&ptr), n * sizeof(T));
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            ptr = nullptr;
            return false;
        }
        PTW_CUDA(e);
        count = n;
        return true;
    }
    // Grows (never shrinks) to at least n elements; returns true when the allocation changed.
    bool reserve(size_t n) {
        if (n <= count && ptr) return false;
        allocate(n);
        return true;
    }
    void upload(const T* src, size_t n, cudaStream_t s = 0) {
        allocate(n);
        if (n) PTW_CUDA(cudaMemcpyAsync(ptr, src, n * sizeof(T), cudaMemcpyHostToDevice, s));
    }
    void zero(cudaStream_t s = 0) {
        if (ptr) PTW_CUDA(cudaMemsetAsync(ptr, 0, count * sizeof(T), s));
    }
    size_t bytes() const { return count * sizeof(T); }
};

// A scene copied to the device and re-laid for 128-bit loads (see DevScene in pt_scene.cuh).
class DeviceScene {
public:
    // Validates and uploads; throws Error. update_lights_only re-uploads the arrays that
    // GpuRenderer::update_lights touches (triangles, materials, light tables, environment).
    void upload(const pt_scene_desc& d, cudaStream_t stream, bool update_lights_only = false);
    const DevScene& view() const { return view_; }
    const DevScene* device_view() const { return d_view_.ptr; }
    bool ready() const { return ready_; }
    size_t device_bytes() const;
    float extent() const { return extent_; }
    // Bytes a scene will occupy on the device (for admission before upload).
    static size_t estimate_bytes(const pt_scene_desc& d);
    // pt_rebuild_lights: new materials, punctual lights and environment; the light tables are built
    // on the device (light_build.cu).
    void rebuild_lights(const pt_light_update& u, cudaStream_t stream);

private:
    DeviceBuffer<float4> nodes4_;
    DeviceBuffer<float4> nodes_, tris_, normals_, tangents_, materials_, alias_, punctual_, env_texels_;
    DeviceBuffer<int4> tri_idx_, textures_;
    DeviceBuffer<float2> uvs_;
    DeviceBuffer<uint32_t> texels_;
    DeviceBuffer<uint8_t> shade_keys_, light_work_;  // light_work_: rebuild_lights' scratch, up to kKeptScratch
    DeviceBuffer<float> srgb_lut_, env_marginal_, env_conditional_, env_row_sin_;
    DeviceBuffer<int2> emissive_;
    DeviceBuffer<DevScene> d_view_;
    DevScene view_{};
    bool ready_ = false;
    float extent_ = 1.0f;
    int32_t num_vertices_ = 0;
    int32_t num_materials_ = 0;
    int tree_levels_ = 0;   // bvh_levels of the uploaded tree
    bool in_treelets_ = false;
    int root_treelet_ = 0;  // the size of its root's treelet, 0 if it keeps the order it came in
    void upload_nodes(const pt_scene_desc& d, cudaStream_t s);
    void upload_shade_keys(const pt_material* materials, int32_t n, cudaStream_t s);
    float bounds_[6] = {0, 0, 0, 0, 0, 0};  // the scene box (lo xyz, hi xyz), for the light-group weights
};

// Checks a scene description for internal consistency; throws Error(PT_ERR_INVALID). Returns bvh_levels of its tree
// (0 with lights_only).
int validate_scene(const pt_scene_desc& d, bool lights_only);

// The levels of a BVH (255 and more: 255), or 0 where two parents name one node, which is let through: the walks in
// Photon's order take such a graph as it is, but what counts on a tree's depth or on its number of nodes does not.
// Throws Error(PT_ERR_INVALID) where a child does not follow its parent or an index is out of range.
int bvh_levels(const pt_bvh_node* nodes, int32_t n, int32_t num_tris);

}  // namespace ptw

// Rays walked by groups of eight lanes, four rays per warp in lockstep, for the last paths of a render, whose
// time is the latency of the longest ray: each lane tests one child of an 8-wide node and one triangle at a
// time, so a ray takes about a third of the dependent node reads of the BVH2 walk and its leaves' triangles
// are tested together. The four groups step together (every exchange is one of the whole warp): groups
// left to themselves run one after another, at a quarter of the rate.
//
// The answers are Photon's (see walk_queue_list in wavefront.cu for why another order gives the same ones):
// the 8-wide tree's boxes are BVH2 boxes, tested by Photon's arithmetic. This walk's order of nodes is not
// Photon's, so it prunes later, at (1 + 2^-8) of the least distance; a ray with two nearly equal least
// distances, with a triangle accepted clearly ahead of its own box, an any-hit ray that enters a leaf at
// exactly its tmax, and one whose stack runs full are walked again in Photon's order.
#pragma once

#include "pt_traverse.cuh"
#include "wide_tree.h"

namespace ptw {

constexpr uint32_t kWarp = 0xffffffffu;
constexpr int kGroupStack = 40;  // a group's stack entries in shared memory
constexpr float kGroupPrune = 1.0f + 1.0f / 256.0f;
constexpr float kGroupTie = 1.0f + 1.0f / 16384.0f;

// The least of a group's values, in all its lanes.
PT_HD uint32_t group_min(uint32_t v) {
    v = min(v, __shfl_xor_sync(kWarp, v, 1));
    v = min(v, __shfl_xor_sync(kWarp, v, 2));
    return min(v, __shfl_xor_sync(kWarp, v, 4));
}

// traverse() of each group's ray (`on`: the group has one; the same in its eight lanes, as s, o, d and tmax
// are): every lane of the group gets the answer. The whole warp calls it. stack: the group's, kGroupStack
// entries of a node and its box entry's bits.
template <bool AnyHit>
PT_HD bool group_walk(bool on, uint2* stack, const DevScene& s, V3 o, V3 d, float tmax, Hit& hit) {
    const uint32_t gl = threadIdx.x & (kWide - 1), shift = threadIdx.x & 24u;  // lane in the group; its first lane
    auto any = [&](bool b) { return ((__ballot_sync(kWarp, b) >> shift) & 0xffu) != 0; };
    const RaySlab rs = ray_slab(o, V3{safe_inv(d.x), safe_inv(d.y), safe_inv(d.z)});
    const uint32_t none = 0x7f7fffffu;  // above every distance's bits
    float limit = tmax, best = kInf, second = __uint_as_float(none), bu = 0.0f, bv = 0.0f;
    int tri = -1, node = 0, sp = 0;
    bool run = on, doubt = false, found = false;
    while (__any_sync(kWarp, run)) {
        float near = kInf;
        int count = -1, index = 0;
        if (run) {
            float4 lo, hi;
            ldg_pair(s.wide + 2 * kWide * size_t(node) + 2 * gl, lo, hi);
            near = box_entry3(lo, hi, rs, limit);
            count = __float_as_int(hi.w);
            index = __float_as_int(lo.w);
        }
        const bool in = near != kInf, inner = in && count == 0 && near < limit, leaf = in && count > 0;
        if (__any_sync(kWarp, leaf)) {
            if (AnyHit && any(leaf && !(near < limit))) doubt = true;
            // The leaves' triangles, eight per group at a time: lane p takes pair p of its group's list.
            const int own = leaf ? count : 0;
            int incl = own;
#pragma unroll
            for (int k = 1; k < kWide; k <<= 1) {
                const int x = __shfl_up_sync(kWarp, incl, k, kWide);
                if (int(gl) >= k) incl += x;
            }
            const int total = __shfl_sync(kWarp, incl, kWide - 1, kWide);
            for (int base = 0; __any_sync(kWarp, base < total); base += kWide) {
                const int p = base + int(gl);
                int j = 0;
#pragma unroll
                for (int k = kWide / 2; k > 0; k >>= 1)
                    if (__shfl_sync(kWarp, incl, j + k - 1, kWide) <= p) j += k;
                const int i = __shfl_sync(kWarp, index - (incl - own), j, kWide) + p;
                const float entry = __shfl_sync(kWarp, near, j, kWide);
                float t = 0.0f, u = 0.0f, v = 0.0f;
                bool ok = false;
                if (p < total) {
                    const float4* rec = s.tris + kTriStride * size_t(i);
                    float4 g0, g1;
                    ldg_pair(rec, g0, g1);
                    const float4 g2 = __ldg(rec + 2);
                    ok = tri_intersect(g0, g1, g2, o, d, limit, t, u, v) &&
                         !((__float_as_int(g1.w) & 1) && alpha_passes(s, rec, __float_as_int(g0.w), u, v));
                }
                if (AnyHit) {
                    if (any(ok)) found = true;
                    continue;
                }
                if (!__any_sync(kWarp, ok)) continue;
                if (any(ok && t < entry * (1.0f - 1.0f / 16384.0f))) doubt = true;
                const uint32_t bits = ok ? __float_as_uint(t) : none, least = group_min(bits);
                const int w = (__ffs(int((__ballot_sync(kWarp, bits == least) >> shift) & 0xffu)) - 1) & (kWide - 1);  // the winner
                const uint32_t next = group_min(int(gl) == w ? none : bits);
                const float tl = __uint_as_float(least);
                second = fminf(second, fminf(__uint_as_float(next), fmaxf(tl, best)));
                const int wi = __shfl_sync(kWarp, i, w, kWide);
                const float wu = __shfl_sync(kWarp, u, w, kWide), wv = __shfl_sync(kWarp, v, w, kWide);
                if (tl < best) {
                    best = tl;
                    tri = wi;
                    bu = wu;
                    bv = wv;
                    limit = fminf(best * kGroupPrune, tmax);
                }
            }
        }
        // The nearest inner child next, the others onto the stack, farthest first.
        const int n = __popc((__ballot_sync(kWarp, inner) >> shift) & 0xffu);
        const uint32_t key = inner ? (__float_as_uint(near) & 0x7ffffff8u) | gl : ~0u;
        int rank = 0;
        if (__any_sync(kWarp, n > 1)) {
#pragma unroll
            for (int k = 0; k < kWide; k++) rank += __shfl_sync(kWarp, key, k, kWide) < key ? 1 : 0;
        }
        const uint32_t first = (__ballot_sync(kWarp, inner && rank == 0) >> shift) & 0xffu;
        const int next_node = __shfl_sync(kWarp, index, (__ffs(int(first)) - 1) & (kWide - 1), kWide);
        if (run) {
            if (found) {
                run = false;
            } else if (n > 0) {
                node = next_node;
                if (n > 1) {
                    if (sp + n - 1 > kGroupStack) {
                        doubt = true;
                        run = false;
                    } else {
                        if (inner && rank > 0) stack[sp + n - 1 - rank] = make_uint2(uint32_t(index), __float_as_uint(near));
                        sp += n - 1;
                    }
                }
            } else {
                node = -1;
                while (sp > 0 && node < 0) {
                    const uint2 e = stack[--sp];
                    if (__uint_as_float(e.y) < limit) node = int(e.x);
                }
                run = node >= 0;
            }
        }
        __syncwarp();
    }
    if (doubt || (!AnyHit && tri >= 0 && second <= best * kGroupTie)) {
        int in_order[kSmemStack];
        TraversalCounters tc{0, 0, 0};
        found = traverse<AnyHit, false>(s, o, d, tmax, hit, in_order, 1, &tc);
    } else if (!AnyHit && tri >= 0) {
        hit.t = best;
        hit.tri = tri;
        hit.u = bu;
        hit.v = bv;
        found = true;
    }
    __syncwarp();
    return found;
}

}  // namespace ptw

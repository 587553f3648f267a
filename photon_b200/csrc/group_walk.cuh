// Rays walked by groups of eight lanes, four rays per warp in lockstep, for the last paths of a render, whose
// time is the latency of the longest ray: each lane visits one node of a treelet of up to eight (treelets.h)
// and tests one triangle at a time, so a ray takes about a third of the dependent node reads of the BVH2 walk
// and its leaves' triangles are tested together. The four groups step together (every exchange is one of the
// whole warp): groups left to themselves run one after another, at a quarter of the rate.
//
// The answers are Photon's, for the reasons given for the list walk (walk_queue_list in wavefront.cu), because
// this walk too takes nodes and leaves in Photon's order and prunes later than Photon does. The ways out of a
// treelet that the ray enters, leaves and other treelets, go onto the group's stack in that order: at each
// node a leaf child before an inner one, else the nearer child first, side 0 on a tie. A leaf's triangles are
// tested once all that comes before it has been, and nothing that comes after it has lowered the limit.
// (Tested as soon as they are met, the nearest child first, they let the walk prune a triangle that Photon
// reaches before them and accepts: one seen edge-on, whose distance is rounding, can be further ahead of its
// box than any margin.) A ray with two nearly equal least distances, with a triangle accepted clearly ahead of
// its own box, an any-hit ray that enters a leaf at exactly its tmax, and one whose stack runs full are walked
// again, by Photon's walk.
#pragma once

#include "pt_traverse.cuh"
#include "treelets.h"

namespace ptw {

constexpr uint32_t kWarp = 0xffffffffu;
constexpr int kGroupStack = 48;  // a group's stack entries in shared memory

// traverse() of each group's ray (`on`: the group has one; the same in its eight lanes, as s, o, d and tmax
// are): every lane of the group gets the answer. The whole warp calls it. stack: the group's, kGroupStack
// entries: first triangle or node; count (of triangles, or less the nodes of the treelet); the bits of the box's
// entry and of what is pruned by.
template <bool AnyHit>
PT_HD bool group_walk(bool on, uint4* stack, const DevScene& s, V3 o, V3 d, float tmax, Hit& hit) {
    const int gl = int(threadIdx.x & (kTreelet - 1)), shift = int(threadIdx.x & 24u);  // lane in the group; its first lane
    auto group = [&](bool b) { return (__ballot_sync(kWarp, b) >> shift) & 0xffu; };
    const RaySlab rs = ray_slab(o, V3{safe_inv(d.x), safe_inv(d.y), safe_inv(d.z)});
    float limit = tmax, best = kInf, second = kInf;    // the group's
    float mine = kInf, bu = 0.0f, bv = 0.0f;           // the nearest this lane has found itself
    int tri = -1, sp = on ? 1 : 0;
    bool doubt = false, found = false;
    if (on && gl == 0) stack[0] = make_uint4(0u, uint32_t(-s.root_treelet), 0u, 0u);  // the root, entered at 0
    __syncwarp();
    while (__any_sync(kWarp, sp > 0)) {
        // The leaves on top of the stack, one per lane, and the treelet below them.
        uint4 e = make_uint4(0u, 0u, 0u, 0u);
        if (gl < sp) e = stack[sp - 1 - gl];
        const float near = __uint_as_float(e.z), prune = __uint_as_float(e.w);
        const uint32_t inner = group(gl < sp && int(e.y) < 0 && prune < limit);
        const int at = inner ? __ffs(int(inner)) - 1 : kTreelet - 1;
        const int first = __shfl_sync(kWarp, int(e.x), at, kTreelet), nodes = -__shfl_sync(kWarp, int(e.y), at, kTreelet);
        const int size = inner ? nodes : 0;
        const bool leaf = gl < sp && gl <= at && int(e.y) > 0 && prune <= limit;
        sp -= min(sp, at + 1);
        float4 n0{}, n1{}, n2{}, n3{};
        if (gl < size) {
            ldg_pair(s.nodes + 4 * size_t(first + gl), n0, n1);
            ldg_pair(s.nodes + 4 * size_t(first + gl) + 2, n2, n3);
        }
        if (__any_sync(kWarp, leaf)) {
            // The leaves' triangles, eight per group at a time: lane p takes pair p of its group's list.
            // (Exchanges that do not wait for one another, here and below, rather than fewer in a chain.)
            const int own = leaf ? int(e.y) : 0;
            for (int base = 0, total = 1; __any_sync(kWarp, base < total); base += kTreelet) {
                const int p = base + gl;
                int j = 0, at0 = 0;
                total = 0;
#pragma unroll
                for (int k = 0; k < kTreelet; k++) {
                    if (total <= p) {
                        j = k;
                        at0 = total;
                    }
                    total += __shfl_sync(kWarp, own, k, kTreelet);
                }
                const int i = __shfl_sync(kWarp, int(e.x), j, kTreelet) + p - at0;
                const float entry = __shfl_sync(kWarp, near, j, kTreelet);
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
                    if (group(ok)) found = true;
                    continue;
                }
                if (!__any_sync(kWarp, ok)) continue;
                doubt = doubt || (ok && t < entry * kAhead);
                // The least and the second least of the group.
                float least = ok ? t : kInf, next = kInf;
#pragma unroll
                for (int k = 1; k < kTreelet; k <<= 1) {
                    const float a = __shfl_xor_sync(kWarp, least, k), b = __shfl_xor_sync(kWarp, next, k);
                    next = fminf(fmaxf(least, a), fminf(next, b));
                    least = fminf(least, a);
                }
                second = fminf(second, fminf(next, fmaxf(least, best)));
                if (least < best) {
                    best = least;
                    limit = fminf(best * kPrune, tmax);
                }
                if (ok && t == best) {  // (this lane's; no other's, unless they tie)
                    mine = t;
                    tri = i;
                    bu = u;
                    bv = v;
                }
            }
        }
        __syncwarp();  // (the stack's entries have been read)
        if (__any_sync(kWarp, size > 0)) {
            // This lane's node: its children's entries, and which of them are ways out that the ray enters.
            const int c0 = __float_as_int(n1.w), i0 = __float_as_int(n0.w), c1 = __float_as_int(n3.w), i1 = __float_as_int(n2.w);
            const float t0 = gl < size ? box_entry3(n0, n1, rs, limit) : kInf, t1 = gl < size ? box_entry3(n2, n3, rs, limit) : kInf;
            const bool out0 = t0 != kInf && (c0 > 0 || (c0 < 0 && c0 >= -kTreelet && t0 < limit));
            const bool out1 = t1 != kInf && (c1 > 0 || (c1 < 0 && c1 >= -kTreelet && t1 < limit));
            if (AnyHit && group((out0 && !(t0 < limit)) || (out1 && !(t1 < limit)))) doubt = true;
            const uint32_t ways = group(out0) | group(out1) << 8;
            const int n = __popc(ways);
            // A way's rank: for every node above it of whose children it lies below the later, the ways below the earlier.
            int rank0 = 0, rank1 = 0;
            if (__any_sync(kWarp, n > 1)) {
                const uint32_t side0 = c0 > 0 || c0 >= -kTreelet ? 1u << gl : uint32_t(-c0) >> 4;
                const uint32_t side1 = c1 > 0 || c1 >= -kTreelet ? 0x100u << gl : uint32_t(-c1) >> 4;
                const bool swap = c0 > 0 || c1 > 0 ? c0 <= 0 : t0 > t1;
                const uint32_t order = gl < size ? ((swap ? side1 : side0) & ways) | (swap ? side0 : side1) << 16 : 0u;
#pragma unroll
                for (int k = 0; k < kTreelet; k++) {
                    const uint32_t above = __shfl_sync(kWarp, order, k, kTreelet);
                    const int before = __popc(above & 0xffffu);
                    if ((above >> (16 + gl)) & 1u) rank0 += before;
                    if ((above >> (24 + gl)) & 1u) rank1 += before;
                }
            }
            if (sp + n > kGroupStack) {
                doubt = true;
                sp = 0;
            } else {
                // (Photon tests the boxes of two leaves of one node before either's triangles: the second is not
                // pruned for what the first has.)
                const float prune1 = c0 > 0 && c1 > 0 ? fminf(t0, t1) : t1;
                if (out0) stack[sp + n - 1 - rank0] = make_uint4(uint32_t(i0), uint32_t(c0), __float_as_uint(t0), __float_as_uint(t0));
                if (out1) stack[sp + n - 1 - rank1] = make_uint4(uint32_t(i1), uint32_t(c1), __float_as_uint(t1), __float_as_uint(prune1));
                sp += n;
            }
        }
        if (found) sp = 0;
        __syncwarp();
    }
    const bool again = group(doubt) || (!AnyHit && best < kInf && second <= best * kNearTie);
    if (!AnyHit) {
        const int w = (__ffs(int(group(mine == best))) - 1) & (kTreelet - 1);
        hit.tri = __shfl_sync(kWarp, tri, w, kTreelet);
        hit.u = __shfl_sync(kWarp, bu, w, kTreelet);
        hit.v = __shfl_sync(kWarp, bv, w, kTreelet);
        hit.t = best;
        found = best < kInf;
    }
    if (again) {
        int in_order[kSmemStack];
        TraversalCounters tc{0, 0, 0};
        hit = Hit{kInf, -1, 0.0f, 0.0f};
        found = traverse<AnyHit, false>(s, o, d, tmax, hit, in_order, 1, &tc);
    }
    __syncwarp();
    return found;
}

}  // namespace ptw

/*
 * b2g_walk.cuh — a warp's walk of the broadphase hierarchy for one box.
 *
 * Up to 32 pending nodes are taken a round, so a walk costs about one dependent fetch for each level of the
 * hierarchy, where one thread pays one for each node it visits.
 */
#ifndef B2G_WALK_CUH
#define B2G_WALK_CUH

#include <climits>

#include "b2g_internal.h"

namespace b2g {

constexpr int kPendMax = 512;    /* pending nodes of a walk */
constexpr int kPendWide = 384;   /* above so many a round pops one node, a depth-first walk that adds at
                                    most one pending node for each level below it */

__device__ __forceinline__ bool aabb_overlap(const float4 a, const float4 b) {
    /* b2_test_overlap, src/b2_collision.rs:355-368 (closed boxes) */
    if (b.x - a.z > 0.0f || b.y - a.w > 0.0f) return false;
    if (a.x - b.z > 0.0f || a.y - b.w > 0.0f) return false;
    return true;
}

/* The leaves of world wd whose boxes overlap q: found(ok, leaf) is called by the whole warp, ok in the lanes
 * that have one. pend: kPendMax words of shared memory for this warp. */
template <typename Found>
__device__ __forceinline__ void walk_box(const DevWorld& w, float4 q, uint32_t wd, int* pend, Found found) {
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;
    int top = 0;
    for (int h = 0; h < 2; ++h) {
        const int root = w.bp_world_root[wd + (h ? (uint32_t)w.num_worlds : 0u)];
        if (root == INT_MIN) continue;
        if (root < 0) found(lane == 0 && aabb_overlap(w.bp_leaf[~root], q), ~root);
        else if (lane == 0) pend[top] = root;
        top += root >= 0 ? 1 : 0;
    }
    __syncwarp();
    while (top > 0) {
        const int take = min(top, top <= kPendWide ? 32 : 1);
        const bool mine = lane < take;
        const int node = mine ? pend[top - 1 - lane] : 0;
        top -= take;
        __syncwarp();
        int kids[2] = {0, 0};
        bool hit[2] = {false, false};
        if (mine) {
            const int2 ch = w.bp_node_child[node];
            kids[0] = ch.x;
            kids[1] = ch.y;
            hit[0] = aabb_overlap(w.bp_node_b0[node], q);
            hit[1] = aabb_overlap(w.bp_node_b1[node], q);
        }
        for (int c = 0; c < 2; ++c) {
            const bool leaf = hit[c] && kids[c] < 0, inner = hit[c] && kids[c] >= 0;
            if (__any_sync(full, leaf)) found(leaf, ~kids[c]);
            const unsigned in = __ballot_sync(full, inner);
            const int at = top + __popc(in & below);
            if (inner && at < kPendMax) pend[at] = kids[c];
            if (inner && at >= kPendMax) atomicOr((unsigned*)&w.cnt[CNT_STATUS], ST_STACK_OVERFLOW);
            top = min(top + __popc(in), kPendMax);
        }
        __syncwarp();
    }
}

}  // namespace b2g

#endif

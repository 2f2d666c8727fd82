// leaf.cuh — leaves of grid nodes, tested by the whole warp (triangle scenes).
//
// Lane by lane, a leaf phase takes as many turns as the longest leaf has
// records, each a dependent load of 48 bytes, with the lanes that hold
// shorter leaves or none idle: on the rays of a 1M sphere (4.3 records per
// leaf, 4 to 6 turns per phase) 9 of 32 lanes tested a record.  Here the
// (ray, record) pairs of all leaves are dealt over the 32 lanes, so a phase
// takes a turn per 32 records and consecutive lanes read consecutive records.
// And since a phase no longer needs many lanes at leaves to be worth it, the
// node phase ends once kLeafLanes wait.
//
// The origin, direction and interval that a pair needs lie in shared memory,
// written when a lane takes a ray: two loads where shuffles took eight, and
// seven registers less, without which the closest-hit kernel spills at the 64
// that keep 32 warps on an SM (4M incoherent rays: 2,166 us; with shuffles at
// 72 registers 2,481).  Lane by lane before, and here, in us: 1M sphere at
// 1080p, primaries 411 and 388, bounces 317 and 307, shadow rays 307 and 248;
// 4M incoherent rays 2,207 and 2,166; 1M occlusion rays 384 and 356.
#pragma once

#include <cstddef>

#include "grid.cuh"
#include "share.cuh"

namespace igxrt {

// Lanes waiting (at a leaf, or done) that end the node phase: 14, 20 and never
// (the rule of phase_break alone) gave 388, 397 and 403 us on the sphere's
// primaries, 2,166, 2,205 and 2,239 on the incoherent rays, 248, 248 and 252
// on the shadow rays.
constexpr uint32_t kLeafLanes = 14;

// A warp's part of shared memory, after the block's stacks.
struct WarpLeaves {
    float4 org_tmin[32], dir_tmax[32];  // per lane: the ray it traces
    uint2 leaf[32];                     // per leaf of a phase: {first record - first pair, lane}
    float4 found[32];                   // closest hit, per pair of a turn: {t, u, v, prim}

    __device__ __forceinline__ void put(uint32_t lane, const RayState& r) {
        org_tmin[lane] = make_float4(r.ox, r.oy, r.oz, r.tmin);
        dir_tmax[lane] = make_float4(r.dx, r.dy, r.dz, r.tmax_eff);
    }
};
// Any hit has no use for `found`.
IGXRT_HD constexpr uint32_t leaf_bytes(bool any) {
    return (uint32_t)(any ? sizeof(WarpLeaves) - sizeof(WarpLeaves::found) : sizeof(WarpLeaves));
}
static_assert(offsetof(WarpLeaves, found) == leaf_bytes(true) && leaf_bytes(true) % 16 == 0, "found comes last");

// A helper in the tail takes its victim's ray in shared memory too (share.cuh).
struct SharedRay {
    static constexpr bool kRayInShared = true;
    WarpLeaves* w;
    uint32_t lane;
    __device__ __forceinline__ void take(uint32_t src) {
        const float4 o = w->org_tmin[src], d = w->dir_tmax[src];
        __syncwarp();
        w->org_tmin[lane] = o;
        w->dir_tmax[lane] = d;
        __syncwarp();
    }
};

// All lanes of the warp call this together; the working lanes with a leaf in
// `next` are its owners.  A found pair of an any-hit query decides it
// (`occluded`); those of a closest-hit query are put in shared memory, where
// their owner takes the best by (t, prim) as in test_record.  Owners that go
// on take their next reference from their stack.
template <bool ANY>
__device__ __forceinline__ void warp_leaf_phase(const float4* __restrict__ prims, bool working, uint32_t lane,
                                                uint32_t lower, WarpLeaves& w, int32_t& next, uint32_t prev,
                                                BestHit& best, TraversalStack& st, bool& occluded) {
    constexpr uint32_t FULL = 0xffffffffu;
    const bool at_leaf = working && next < 0;
    const uint32_t leaves = __ballot_sync(FULL, at_leaf);
    if (leaves == 0)
        return;
    // this lane's pairs are [begin, begin + more + 1), by lane
    const uint32_t more = at_leaf ? (uint32_t)next & 15u : 0u;
    const uint32_t rank = __popc(leaves & lower);
    uint32_t begin = rank, total = __popc(leaves);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t b = __ballot_sync(FULL, (more >> k) & 1u);
        begin += (uint32_t)__popc(b & lower) << k;
        total += (uint32_t)__popc(b) << k;
    }
    if (at_leaf)
        w.leaf[rank] = make_uint2((((uint32_t)next & ~kGridLeaf) >> 4) - begin, lane);
    __syncwarp();
    uint32_t started = 0;  // leaves begun in earlier turns
    for (uint32_t base = 0; base < total; base += 32) {
        const uint32_t rel = begin - base;  // wraps for leaves of earlier turns
        const uint32_t starts = __reduce_or_sync(FULL, at_leaf && rel < 32u ? 1u << rel : 0u);
        const uint32_t leaf = started + __popc(starts & (lower | (1u << lane))) - 1u;
        started += __popc(starts);
        const uint32_t pair = base + lane;
        uint2 e = make_uint2(0u, lane);
        if (pair < total)
            e = w.leaf[leaf];
        // the owner's best t (closest) or excluded object (any hit); a closest
        // hit's excluded object is the owner's to reject
        const float limit = ANY ? 0.f : __shfl_sync(FULL, best.t, e.y);
        const uint32_t skip = ANY ? __shfl_sync(FULL, prev, e.y) : IGXRT_NO_RAY_HIT;
        bool found = false;
        if (pair < total) {
            const float4* p = prims + 3 * (size_t)(e.x + pair);
            const float4 v0 = __ldg(p), v1 = __ldg(p + 1), v2 = __ldg(p + 2);
            const float4 o = w.org_tmin[e.y], d = w.dir_tmax[e.y];
            RayState q;  // as far as the tests read it
            q.ox = o.x, q.oy = o.y, q.oz = o.z, q.tmin = o.w;
            q.dx = d.x, q.dy = d.y, q.dz = d.z, q.tmax_eff = d.w;
            q.prev = skip;
            if (ANY) {
                BestHit unused;
                found = test_record(v0, v1, v2, q, unused, true);
            } else {
                float t, u, v;
                if (tri_test(q, v0, v1, v2, t, u, v) && t <= limit && !(t <= q.tmin)) {
                    found = true;
                    w.found[lane] = make_float4(t, u, v, v0.w);
                }
            }
        }
        const uint32_t hits = __ballot_sync(FULL, found);
        if (hits == 0)
            continue;
        // this lane's pairs of the turn
        const int32_t from = max((int32_t)rel, 0), to = min((int32_t)rel + (int32_t)more + 1, 32);
        uint32_t mine = at_leaf && to > from ? hits & ((0xffffffffu >> (32 - (to - from))) << from) : 0u;
        if (ANY) {
            occluded = occluded || mine != 0u;
            continue;
        }
        __syncwarp();
        while (mine) {
            const float4 c = w.found[__ffs(mine) - 1];
            mine &= mine - 1;
            const uint32_t prim = __float_as_uint(c.w);
            if (prim != prev && (c.x < best.t || (c.x == best.t && prim < best.prim))) {
                best.t = c.x;
                best.u = c.y;
                best.v = c.z;
                best.prim = prim;
            }
        }
        // a helper's limit may be its owner's, below its own best
        best.tcull = fminf(best.tcull, cull_limit(best.t));
        __syncwarp();
    }
    __syncwarp();  // the list is free again
    if (at_leaf && !occluded)
        next = st.pop_split(best.tcull);
}

}  // namespace igxrt

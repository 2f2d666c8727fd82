// leaf.cuh — any-hit leaves of grid nodes, tested by the whole warp.
//
// Lane by lane, a leaf phase takes as many turns as the longest leaf has
// records, each a dependent load of 48 bytes, with the lanes that hold
// shorter leaves or none idle: on the shadow rays of a 1M sphere (4.3 records
// per leaf, 6 turns per phase) 9 of 32 lanes tested a record.  Here the
// (ray, record) pairs of all leaves are dealt over the 32 lanes, so a phase
// takes a turn per 32 records and consecutive lanes read consecutive records.
// And since a phase no longer needs many lanes at leaves to be worth it, the
// node phase ends once kLeafLanes wait.  373K shadow rays on the 1M sphere:
// 307 -> 258 us; 1M occlusion rays over 262K random triangles: 387 -> 379 us.
//
// Closest-hit kernels keep the lane-by-lane loop: the owners' best hits then
// go through shared memory and the phase needs 72 registers without the
// any-hit kernel's slack: 4M incoherent rays 2,377 -> 2,481 us (1M sphere
// primaries 432 -> 418 us), a mixed scene's 1M rays 689 -> 736 us.
#pragma once

#include "grid.cuh"

namespace igxrt {

// Lanes waiting (at a leaf, or done) that end the node phase: 10, 14, 20 and
// never (the rule of phase_break alone) gave 262, 262, 264 and 270 us on the
// sphere's shadow rays and 387, 383, 391 and 393 us on the occlusion rays.
constexpr uint32_t kLeafLanes = 14;

// Shared memory of the phase: one {first record - first pair, lane} per leaf,
// 32 per warp.
constexpr uint32_t kLeafEntryBytes = 8;

// All lanes of the warp call this together; the working lanes with a leaf in
// `next` are its owners.  Sets `occluded` where a record decides the owner's
// query, else takes the owner's next reference from its stack.  A helper
// applies the owner's interval and excluded object, so a found pair is an
// occluder as in process_grid_leaf.
__device__ __forceinline__ void any_leaf_phase(const float4* __restrict__ prims, bool working, uint32_t lane,
                                               uint32_t lower, uint2* list, int32_t& next, const RayState& r,
                                               const BestHit& best, TraversalStack& st, bool& occluded) {
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
        list[rank] = make_uint2((((uint32_t)next & ~kGridLeaf) >> 4) - begin, lane);
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
            e = list[leaf];
        RayState q;  // the owner's ray, as far as test_record reads it
        q.ox = __shfl_sync(FULL, r.ox, e.y);
        q.oy = __shfl_sync(FULL, r.oy, e.y);
        q.oz = __shfl_sync(FULL, r.oz, e.y);
        q.dx = __shfl_sync(FULL, r.dx, e.y);
        q.dy = __shfl_sync(FULL, r.dy, e.y);
        q.dz = __shfl_sync(FULL, r.dz, e.y);
        q.tmin = __shfl_sync(FULL, r.tmin, e.y);
        q.tmax_eff = __shfl_sync(FULL, r.tmax_eff, e.y);
        q.prev = __shfl_sync(FULL, r.prev, e.y);
        bool found = false;
        if (pair < total) {
            const float4* p = prims + 3 * (size_t)(e.x + pair);
            BestHit unused;
            found = test_record<true>(__ldg(p), __ldg(p + 1), __ldg(p + 2), q, unused);
        }
        const uint32_t hits = __ballot_sync(FULL, found);
        const int32_t from = max((int32_t)rel, 0), to = min((int32_t)rel + (int32_t)more + 1, 32);
        if (at_leaf && to > from)
            occluded = occluded || ((hits >> from) & (0xffffffffu >> (32 - (to - from)))) != 0u;
    }
    __syncwarp();  // the list is free again
    if (at_leaf && !occluded)
        next = st.pop_live(best.tcull);
}

}  // namespace igxrt

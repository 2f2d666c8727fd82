// lbvh.cu — BVH build on the GPU for geometry that changes every frame.
//
// The reference uploads its scene every frame (test/scene/niels_scene.cpp:
// 61-70) and traces it with a linear loop; the host SAH builder takes about a
// second per million triangles, so a per-frame scene needs a device build.
// This is a linear BVH (Morton order, then the radix tree over the keys, built
// bottom-up together with its boxes after Apetrei 2014, "Fast and Simple
// Agglomerative LBVH Construction"), emitted in the same node formats, records
// and padding rule as the host builder so that the traversal kernels, the
// refit and the read-back work on it unchanged:
//   1. scan: object bounds, max |coordinate|, scene and centroid boxes, the
//      non-finite check (shared with the refit);
//   2. keys: 30-bit Morton code of the centroid in the centroid box, above the
//      object id (so keys are unique), sorted with CUB's radix sort;
//   3. climb: one thread per object writes its record and climbs from its
//      leaf; a node joins its neighbour across the boundary whose keys differ
//      in the lower bit, and at each parent the first arriving child's thread
//      stops and the second goes on with the union of both (nothing waits);
//   4. leaves: a subtree of at most `max_leaf_size` objects becomes one leaf
//      (its objects are contiguous in key order, so records stay in leaf
//      order); the remaining internal nodes are compacted by a prefix sum and
//      written as BVH2 nodes with padded boxes;
//   5. BVH4: collapsed top down one level per launch, opening the child of
//      largest area until four slots are used (the host's choice); the levels
//      carry the traversal-stack bounds and the depth along the paths.
// The scene is then allocated exactly, the arrays are copied into it and its
// grid nodes are written.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <vector>

#include "geometry.cuh"

using namespace igxrt;

namespace {

// State words after the scan's (which use 0..13).
constexpr int kWordNodes2 = 16, kWordRoot = 17, kWordLeaves = 18, kWordStack4 = 19, kWordDepth = 20,
              kWordMalformed = 21;
constexpr int kWordSah = 32;       // double (words 32, 33)
constexpr int kWordLevels = 64;    // frontier sizes of the BVH4 levels
constexpr int kMaxLevels = 64;     // > key bits: no path is longer
// Levels launched over the whole GPU.  A tree over scattered objects has
// about log4 of its leaves, 10 at 300K objects; an empty level costs 1.2 us,
// and one block takes whatever levels are left (bvh4_rest_kernel).
constexpr int kWideLevels = 20;
// Largest scene whose BVH4 levels all run in that block, where a level costs no
// launch but has one SM: whole builds of 4,000 / 8,000 / 16,000 / 32,000 /
// 64,000 triangles take 247 / 248 / 256 / 263 / 280 us with launched levels
// and 204 / 218 / 242 / 279 / 390 in the block.
constexpr uint32_t kOneBlock = 16384;
constexpr int kStateWords = kWordLevels + kMaxLevels + 1;
constexpr uint32_t kDefaultLeaf = 4;

struct BuildArgs {
    SceneObjects obj;
    uint32_t n;       // objects in the tree
    uint32_t leaf;    // largest subtree emitted as one leaf
    uint32_t idbits;  // low key bits holding the object id
    uint32_t* state;
    const uint64_t* keys;  // sorted
    // Internal node p splits its keys between positions p and p + 1.  Four
    // float4 per node: the left child {lo, ref}{hi, first key position}, the
    // right child {lo, ref}{hi, last key position}; ref >= 0 is an internal
    // node, < 0 ~key position
    float4* slots;
    uint32_t* arrive;      // per internal node
    uint32_t* live;        // per internal node: 1 if it becomes a BVH2 node
    uint32_t* map;         // exclusive prefix sum of `live`
    igxrt_bvh2_node* nodes2;
    igxrt_bvh4_node* nodes4;
    uint32_t* parents2;
    uint32_t* parents4;
    igxrt_prim_record* prims;
    uint2* frontier[2];    // one level's {BVH2 node, stack entries above it | depth << 16}
};

__device__ __forceinline__ float key_float(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

__device__ __forceinline__ uint32_t object_of(const BuildArgs& a, uint32_t pos) {
    return (uint32_t)(a.keys[pos] & ((1ull << a.idbits) - 1));
}

__device__ __forceinline__ uint32_t spread10(uint32_t v) {  // 10 bits -> every third bit
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

__global__ void __launch_bounds__(kScanBlock) build_scan_kernel(BuildArgs a) {
    scan_objects<true>(a.obj, a.state);
}

// Every key is written, also when the scan found a non-finite value (the
// build is rejected afterwards): the object id in the low bits keeps the keys
// distinct, which is all the radix tree needs to be well formed.
__global__ void morton_kernel(BuildArgs a, uint64_t* keys) {
    const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= a.n)
        return;
    if (id + 1 < a.n)
        a.arrive[id] = 0;  // the climb's counters
    const Box b = object_box<false>(a.obj, id);
    uint32_t code = 0;
    for (int k = 0; k < 3; ++k) {
        const float lo = key_float(~a.state[kWordCenLo + k]);
        const float hi = key_float(a.state[kWordCenHi + k]);
        const float c = __fmul_rn(__fadd_rn(b.lo[k], b.hi[k]), 0.5f);
        const float ext = hi - lo;
        float u = ext > 0.f ? (c - lo) / ext : 0.f;
        u = fminf(fmaxf(u, 0.f), 1.f);  // a NaN becomes 0
        const uint32_t q = min((uint32_t)(u * 1024.f), 1023u);
        code |= spread10(q) << (2 - k);
    }
    keys[id] = ((uint64_t)code << a.idbits) | id;
}

__device__ __forceinline__ Box slot_box(const float4& lo, const float4& hi) {
    return {{lo.x, lo.y, lo.z}, {hi.x, hi.y, hi.z}};
}

// Records in key order (leaf_end is set when the leaves are emitted), and the
// tree with its boxes.  A climber's step is a release of the 32 bytes it hands
// to its parent, the arrival, and one load of its sibling's 32 bytes; its own
// box stays in registers.  For 300K random triangles this pass takes 69 us (cold),
// where records, radix tree and boxes as three kernels took 22 + 20 + 51 us.
__global__ void climb_kernel(BuildArgs a) {
    const uint32_t pos = blockIdx.x * blockDim.x + threadIdx.x;
    if (pos >= a.n)
        return;
    const uint32_t id = object_of(a, pos);
    igxrt_prim_record rec{};
    fill_record(a.obj, id, rec);
    const uint32_t type = id < a.obj.nt ? kPrimTriangle : (id < a.obj.nt + a.obj.ns ? kPrimSphere : kPrimCube);
    float4* out = reinterpret_cast<float4*>(a.prims + pos);
    out[0] = make_float4(rec.p0[0], rec.p0[1], rec.p0[2], __uint_as_float(id));
    out[1] = make_float4(rec.e1[0], rec.e1[1], rec.e1[2], 0.f);
    out[2] = make_float4(rec.e2[0], rec.e2[1], rec.e2[2], __uint_as_float(type));
    Box box = object_box<false>(a.obj, id);
    uint32_t first = pos, last = pos;
    int32_t ref = ~(int32_t)pos;
    for (int steps = 0; first != 0 || last != a.n - 1; ++steps) {
        if (steps >= kMaxLevels) {  // deeper than the key bits allow: malformed
            atomicOr(a.state + kWordMalformed, 1u);
            return;
        }
        // the keys are unique, so the two boundaries' differences never tie
        const uint64_t below = first > 0 ? a.keys[first - 1] ^ a.keys[first] : ~0ull;
        const uint64_t above = last < a.n - 1 ? a.keys[last] ^ a.keys[last + 1] : ~0ull;
        const bool left = above < below;  // the left child of the node that splits at `last`
        const uint32_t p = left ? last : first - 1;
        float4* own = a.slots + 4 * (size_t)p + (left ? 0 : 2);
        own[0] = make_float4(box.lo[0], box.lo[1], box.lo[2], __int_as_float(ref));
        own[1] = make_float4(box.hi[0], box.hi[1], box.hi[2], __uint_as_float(left ? first : last));
        if (arrive_at(a.arrive + p) == 0)
            return;  // the sibling's thread goes on
        const float4* other = a.slots + 4 * (size_t)p + (left ? 2 : 0);
        const float4 lo = __ldcg(other), hi = __ldcg(other + 1);
        Box sibling = slot_box(lo, hi);
        if (left) {
            box.grow(sibling);
            last = __float_as_uint(hi.w);
        } else {
            sibling.grow(box);
            box = sibling;
            first = __float_as_uint(hi.w);
        }
        a.live[p] = last - first + 1 > a.leaf ? 1u : 0u;
        ref = (int32_t)p;
    }
    if (a.n > 1)
        a.state[kWordRoot] = (uint32_t)ref;
}

// The BVH2 node of a live internal node: the prefix sum's place, with the
// root's and the first one's exchanged (traversals start at node 0).
__device__ __forceinline__ uint32_t node2_of(const BuildArgs& a, uint32_t i, uint32_t root) {
    const uint32_t m = a.map[i];
    return i == root ? 0u : (m == 0u ? a.map[root] : m);
}

// BVH2 nodes from the live internal nodes.  Sums the SAH cost (areas relative
// to the root box; node cost 1, object cost 1, as the host builder's default),
// one double atomic per block of a grid of at most a few rounds.
__global__ void __launch_bounds__(256) emit2_kernel(BuildArgs a) {
    if (a.state[kWordMalformed])
        return;  // slots may be unwritten
    double sah = 0.0;
    uint32_t leaves = 0;
    const uint32_t root = a.state[kWordRoot];
    const float4* rs = a.slots + 4 * (size_t)root;
    Box rb = slot_box(rs[0], rs[1]);
    rb.grow(slot_box(rs[2], rs[3]));
    const float root_area = rb.half_area();
    const float inv_root = root_area > 0.f ? 1.f / root_area : 0.f;
    const float pad = box_pad(a.state);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n - 1; i += gridDim.x * blockDim.x) {
        if (!a.live[i])
            continue;
        const uint32_t node = node2_of(a, i, root);
        const float4* s = a.slots + 4 * (size_t)i;
        igxrt_bvh2_node* o = a.nodes2 + node;
        int32_t refs[2];
        Box both;
        both.reset();
        for (int c = 0; c < 2; ++c) {
            const float4 lo = s[2 * c], hi = s[2 * c + 1];
            Box b = slot_box(lo, hi);
            both.grow(b);
            const float rel = root_area > 0.f ? b.half_area() * inv_root : 1.f;
            const int32_t ref = __float_as_int(lo.w);
            b.pad(pad);
            NodeOps<IGXRT_LAYOUT_BVH2>::put(o, c, b);
            if (ref >= 0 && a.live[ref]) {
                const uint32_t child = node2_of(a, (uint32_t)ref, root);
                refs[c] = (int32_t)child;
                a.parents2[child] = node;
            } else {
                const uint32_t bound = __float_as_uint(hi.w);
                const uint32_t first = c == 0 ? bound : i + 1, last = c == 0 ? i : bound;
                refs[c] = ~(int32_t)first;
                a.prims[last].leaf_end = 1;
                sah += (double)rel * (last - first + 1);
                ++leaves;
            }
        }
        sah += root_area > 0.f ? (double)both.half_area() * inv_root : 1.0;
        reinterpret_cast<int4*>(o)[3] = make_int4(refs[0], refs[1], 0, 0);
        if (i == root) {
            a.parents2[0] = kNoParent;
            a.state[kWordNodes2] = a.map[a.n - 2] + a.live[a.n - 2];
            // the first BVH4 level: the root
            a.frontier[0][0] = make_uint2(0, 0);
            a.state[kWordLevels] = 1;
            a.parents4[0] = kNoParent;
        }
    }
    __shared__ double block_sah[8];
    __shared__ uint32_t block_leaves[8];
    leaves = __reduce_add_sync(0xffffffffu, leaves);
    for (int off = 16; off > 0; off >>= 1)
        sah += __shfl_down_sync(0xffffffffu, sah, off);
    if ((threadIdx.x & 31) == 0) {
        block_sah[threadIdx.x / 32] = sah;
        block_leaves[threadIdx.x / 32] = leaves;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) {
            sah += block_sah[w];
            leaves += block_leaves[w];
        }
        if (leaves) {
            atomicAdd(a.state + kWordLeaves, leaves);
            atomicAdd(reinterpret_cast<double*>(a.state + kWordSah), sah);
        }
    }
}

// Scenes of at most `leaf` objects: one root node with the whole scene in
// slot 0 (the host builder's layout for a one-leaf tree).
__global__ void emit_single_leaf_kernel(BuildArgs a) {
    const float pad = box_pad(a.state);
    Box b;
    if (a.n == 1) {
        b = object_box<false>(a.obj, object_of(a, 0));
    } else {
        const float4* s = a.slots + 4 * (size_t)a.state[kWordRoot];
        b = slot_box(s[0], s[1]);
        b.grow(slot_box(s[2], s[3]));
    }
    b.pad(pad);
    Box e;
    for (int k = 0; k < 3; ++k)
        e.lo[k] = e.hi[k] = INFINITY;
    NodeOps<IGXRT_LAYOUT_BVH2>::put(a.nodes2, 0, b);
    NodeOps<IGXRT_LAYOUT_BVH2>::put(a.nodes2, 1, e);
    reinterpret_cast<int4*>(a.nodes2)[3] = make_int4(~0, 0, 0, 0);
    a.parents2[0] = kNoParent;
    igxrt_bvh4_node q{};
    for (int c = 0; c < 4; ++c) {
        NodeOps<IGXRT_LAYOUT_BVH4>::put(&q, c, c == 0 ? b : e);
        q.child[c] = c == 0 ? ~0 : 0;
    }
    a.nodes4[0] = q;
    a.parents4[0] = kNoParent;
    a.prims[a.n - 1].leaf_end = 1;
    a.state[kWordNodes2] = 1;
    a.state[kWordLevels] = 1;
    a.state[kWordLeaves] = 1;
    a.state[kWordDepth] = 1;
    *reinterpret_cast<double*>(a.state + kWordSah) = (double)a.n;
}

// One BVH4 level: each frontier BVH2 node becomes a BVH4 node whose slots are
// its descendants, opened largest-area-first until four slots are used.  The
// level's nodes follow the earlier levels' in frontier order, so a node's
// place and its parent's need no counter of their own: a warp takes places in
// the next level for all its children with one atomic (two atomics per child
// before, and two climbs over the finished trees, 40 + 32 us, for the stack
// bounds and the depth).  Along a path the
// frontier carries the stack entries a traversal may hold on arrival (each
// node above pushes its used slots minus one) and the BVH2 depth; every BVH2
// node is opened by exactly one BVH4 node, so the maxima cover the tree.
// Called by whole warps with the same arguments.  Returns the level's size.
__device__ uint32_t emit4_level(const BuildArgs& a, int level, uint32_t thread, uint32_t threads) {
    const uint32_t lane = threadIdx.x & 31u, lower = (1u << lane) - 1u;
    const uint32_t* counts = a.state + kWordLevels;
    const uint32_t count = __ldcg(counts + level);
    if (count == 0)
        return 0;
    uint32_t base = (int)lane < level ? __ldcg(counts + lane) : 0u;
    if ((int)lane + 32 < level)
        base += __ldcg(counts + lane + 32);
    base = __reduce_add_sync(0xffffffffu, base);  // nodes of the earlier levels
    const uint2* in = a.frontier[level & 1];
    uint2* out = a.frontier[(level + 1) & 1];
    uint32_t deepest = 0, stack = 0;
    for (uint32_t t0 = thread & ~31u; t0 < count; t0 += threads) {
        const uint32_t t = t0 + lane;
        const bool mine = t < count;
        Box box[4];
        int32_t ref[4];
        uint32_t depth[4];  // of the BVH2 node that holds the slot
        int used = 0;
        uint32_t kids = 0, above = 0;
        if (mine) {
            const uint2 job = __ldcg(in + t);
            float area[4];
            using Ops2 = NodeOps<IGXRT_LAYOUT_BVH2>;
            float f[Ops2::kFloats];
            Ops2::load(a.nodes2 + job.x, f);
#pragma unroll
            for (int c = 0; c < 2; ++c) {  // the trees of this path have no empty BVH2 slot
                Ops2::get(f, c, box[c]);
                ref[c] = Ops2::child(f, c);
                area[c] = box[c].half_area();
                depth[c] = (job.y >> 16) + 1u;
            }
            used = 2;
            // the opened slot's first child takes its place, the second the
            // next free slot: every index is fixed, so the slots stay in
            // registers
#pragma unroll
            for (int free = 2; free < 4; ++free) {
                if (used < free)
                    break;
                int pick = -1;
                int32_t open = 0;
                uint32_t d = 0;
                float best = -1.f;
#pragma unroll
                for (int s = 0; s < free; ++s)
                    if (ref[s] >= 0 && area[s] > best) {
                        best = area[s];
                        pick = s;
                        open = ref[s];
                        d = depth[s] + 1u;
                    }
                if (pick < 0)
                    break;
                Ops2::load(a.nodes2 + open, f);
                Box b;
                Ops2::get(f, 0, b);
#pragma unroll
                for (int s = 0; s < free; ++s)
                    if (s == pick) {
                        box[s] = b;
                        ref[s] = Ops2::child(f, 0);
                        area[s] = b.half_area();
                        depth[s] = d;
                    }
                Ops2::get(f, 1, box[free]);
                ref[free] = Ops2::child(f, 1);
                area[free] = box[free].half_area();
                depth[free] = d;
                used = free + 1;
            }
            above = (job.y & 0xffffu) + (uint32_t)used - 1u;
            stack = max(stack, above);
#pragma unroll
            for (int s = 0; s < 4; ++s)
                if (s < used) {
                    kids += ref[s] >= 0 ? 1u : 0u;
                    deepest = max(deepest, depth[s]);
                }
        }
        uint32_t place = 0, total = 0;
        for (int k = 0; k < 3; ++k) {  // kids <= 4
            const uint32_t b = __ballot_sync(0xffffffffu, (kids >> k) & 1u);
            place += (uint32_t)__popc(b & lower) << k;
            total += (uint32_t)__popc(b) << k;
        }
        uint32_t taken = 0;
        if (lane == 0 && total)
            taken = atomicAdd(a.state + kWordLevels + level + 1, total);
        place += __shfl_sync(0xffffffffu, taken, 0);
        if (!mine)
            continue;
        Box b[4];
        int32_t child[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            child[s] = 0;
            if (s < used) {
                b[s] = box[s];
                child[s] = ref[s];
                if (ref[s] >= 0) {
                    child[s] = (int32_t)(base + count + place);
                    a.parents4[child[s]] = base + t;
                    out[place++] = make_uint2((uint32_t)ref[s], above | depth[s] << 16);
                }
            } else {
                for (int k = 0; k < 3; ++k)
                    b[s].lo[k] = b[s].hi[k] = INFINITY;
            }
        }
        float4* node = reinterpret_cast<float4*>(a.nodes4 + base + t);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            node[2 * k] = make_float4(b[0].lo[k], b[1].lo[k], b[2].lo[k], b[3].lo[k]);
            node[2 * k + 1] = make_float4(b[0].hi[k], b[1].hi[k], b[2].hi[k], b[3].hi[k]);
        }
        reinterpret_cast<int4*>(node)[6] = make_int4(child[0], child[1], child[2], child[3]);
        reinterpret_cast<int4*>(node)[7] = make_int4(0, 0, 0, 0);
    }
    stack = __reduce_max_sync(0xffffffffu, stack);
    deepest = __reduce_max_sync(0xffffffffu, deepest);
    if (lane == 0) {  // the words soon hold the maxima: most warps only read them
        if (stack > __ldcg(a.state + kWordStack4))
            atomicMax(a.state + kWordStack4, stack);
        if (deepest > __ldcg(a.state + kWordDepth))
            atomicMax(a.state + kWordDepth, deepest);
    }
    return count;
}

// The wide levels, chained by programmatic dependent launch: the next level's
// blocks are scheduled as soon as this one starts, and its
// griddepcontrol.wait returns once this grid has finished and its writes are
// visible, so an empty level costs no launch gap.
__global__ void __launch_bounds__(256) emit4_level_kernel(BuildArgs a, int level) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
    // consecutive warps of jobs go to consecutive blocks: a level of a few
    // thousand nodes, each some forty 16-byte accesses to lines of its own,
    // spreads over all SMs instead of filling the first blocks'
    const uint32_t warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    emit4_level(a, level, warp * 32u + (threadIdx.x & 31u), gridDim.x * blockDim.x);
}

// The levels from `first` on, one block: empty but for deep trees, whose last
// levels are mostly narrow, and all levels of small scenes, where a level in
// the block costs 3 us and a launch 5.5 (kOneBlock).
__global__ void __launch_bounds__(1024) bvh4_rest_kernel(BuildArgs a, int first) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int level = first; level < kMaxLevels; ++level) {
        if (emit4_level(a, level, threadIdx.x, blockDim.x) == 0)
            return;
        __syncthreads();
    }
}

// The finished arrays, from the build's scratch (and the caller's triangles and
// planes) into the scene: up to kCopies segments of whole 4-byte words in one
// launch, 16 bytes at a time where both ends are aligned.  Seven copies in a
// row took a launch gap each.
constexpr int kCopies = 7;
struct CopyList {
    const uint32_t* src[kCopies];
    uint32_t* dst[kCopies];
    uint64_t words[kCopies];
};

__global__ void __launch_bounds__(256) copy_kernel(CopyList c) {
    const uint64_t first = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, step = gridDim.x * (uint64_t)blockDim.x;
    for (int k = 0; k < kCopies; ++k) {
        const bool wide = (((uintptr_t)c.src[k] | (uintptr_t)c.dst[k]) & 15u) == 0;
        const uint64_t quads = wide ? c.words[k] / 4 : 0;
        for (uint64_t i = first; i < quads; i += step)
            reinterpret_cast<uint4*>(c.dst[k])[i] = __ldcs(reinterpret_cast<const uint4*>(c.src[k]) + i);
        for (uint64_t i = 4 * quads + first; i < c.words[k]; i += step)
            c.dst[k][i] = __ldcs(c.src[k] + i);
    }
}

// Build scratch, given back in stream order.
struct Scratch {
    void* mem = nullptr;
    bool pooled = false;
    cudaStream_t stream = nullptr;
    ~Scratch() {
        if (mem && pooled)
            cudaFreeAsync(mem, stream);
        else if (mem)
            cudaFree(mem);
    }
};

}  // namespace

extern "C" {

igxrt_status igxrt_scene_create_gpu(igxrt_context* ctx, const igxrt_scene_desc* desc,
                                    const igxrt_build_options* opts, uint32_t flags, void* stream,
                                    igxrt_scene** out) {
    if (!ctx || !out)
        return IGXRT_ERROR_INVALID_ARGUMENT;
    *out = nullptr;
    if (!desc)
        return fail(ctx, IGXRT_ERROR_INVALID_ARGUMENT, "desc is NULL");
    if (flags & ~IGXRT_TRACE_HOST_MEMORY)
        return fail(ctx, IGXRT_ERROR_INVALID_ARGUMENT, format("unknown flags 0x%x", flags));
    const uint32_t leaf = (opts && opts->max_leaf_size) ? opts->max_leaf_size : kDefaultLeaf;
    if (leaf > 16)
        return fail(ctx, IGXRT_ERROR_INVALID_ARGUMENT, format("max_leaf_size %u outside 1..16", leaf));
    DeviceGuard guard(ctx->device);
    if (!guard.ok())
        return fail(ctx, IGXRT_ERROR_CUDA, "cannot select the context's device");
    cudaStream_t s = static_cast<cudaStream_t>(stream);

    BuildArgs a{};
    igxrt_status st = stage_scene_desc(ctx, desc, flags, s, a.obj);
    if (st != IGXRT_OK)
        return st;
    const uint32_t n = a.obj.count();
    a.n = n;
    a.leaf = leaf;
    a.idbits = 1;
    while (a.idbits < 31 && (1u << a.idbits) < n)
        ++a.idbits;
    const size_t ni = std::max<size_t>(n, 2) - 1;  // internal nodes (at least one slot)
    const size_t nl = std::max<size_t>(n, 1);

    // CUB scratch sizes
    size_t sort_bytes = 0, scan_bytes = 0;
    cub::DoubleBuffer<uint64_t> keys_db(nullptr, nullptr);
    cudaError_t e = cub::DeviceRadixSort::SortKeys(nullptr, sort_bytes, keys_db, (int)nl, (int)a.idbits,
                                                    30 + (int)a.idbits, s);
    if (e == cudaSuccess)
        e = cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                          (int)ni, s);
    if (e != cudaSuccess)
        return cuda_fail(ctx, e, "build scratch sizes");

    // one scratch allocation, 256-byte aligned parts
    std::vector<size_t> sizes = {
        kStateWords * 4, 2 * nl * 8, 4 * ni * sizeof(float4), ni * 4, ni * 4, ni * 4,
        ni * sizeof(igxrt_bvh2_node), ni * sizeof(igxrt_bvh4_node), ni * 4, ni * 4,
        nl * sizeof(igxrt_prim_record), 2 * ni * 8, std::max(sort_bytes, scan_bytes)};
    std::vector<size_t> offs(sizes.size());
    size_t total = 0;
    for (size_t k = 0; k < sizes.size(); ++k) {
        offs[k] = total;
        total += round_up(std::max<size_t>(sizes[k], 1), 256);
    }
    Scratch scratch;
    scratch.stream = s;
    e = pool_alloc(ctx, &scratch.mem, total, s, scratch.pooled);
    if (e != cudaSuccess)
        return cuda_fail(ctx, e, "build scratch");
    char* base = static_cast<char*>(scratch.mem);
    int part = 0;
    auto next = [&](auto* ptr) { return reinterpret_cast<decltype(ptr)>(base + offs[part++]); };
    a.state = next((uint32_t*)nullptr);
    uint64_t* keys0 = next((uint64_t*)nullptr);
    uint64_t* keys1 = keys0 + nl;
    a.slots = next((float4*)nullptr);
    a.arrive = next((uint32_t*)nullptr);
    a.live = next((uint32_t*)nullptr);
    a.map = next((uint32_t*)nullptr);
    a.nodes2 = next((igxrt_bvh2_node*)nullptr);
    a.nodes4 = next((igxrt_bvh4_node*)nullptr);
    a.parents2 = next((uint32_t*)nullptr);
    a.parents4 = next((uint32_t*)nullptr);
    a.prims = next((igxrt_prim_record*)nullptr);
    a.frontier[0] = next((uint2*)nullptr);
    a.frontier[1] = a.frontier[0] + ni;
    void* cub_temp = base + offs[part++];

    const uint32_t threads = 256;
    auto blocks = [threads](size_t count) { return (uint32_t)std::max<size_t>((count + threads - 1) / threads, 1); };
    e = cudaMemsetAsync(a.state, 0, kStateWords * 4, s);
    if (e != cudaSuccess)
        return cuda_fail(ctx, e, "build state reset");
    const uint32_t scan_grid = std::min<uint32_t>(blocks(std::max<size_t>({(size_t)n, 4 * (size_t)a.obj.np, 1})),
                                                  (uint32_t)std::max(ctx->sm_count, 1) * 4);
    build_scan_kernel<<<scan_grid, kScanBlock, 0, s>>>(a);
    if (n) {
        morton_kernel<<<blocks(n), threads, 0, s>>>(a, keys0);
        keys_db = cub::DoubleBuffer<uint64_t>(keys0, keys1);
        // by the code bits alone: the keys go in by ascending id and the sort
        // is stable (four passes instead of seven at 300K objects, -33 us)
        e = cub::DeviceRadixSort::SortKeys(cub_temp, sort_bytes, keys_db, (int)n, (int)a.idbits,
                                           30 + (int)a.idbits, s);
        if (e != cudaSuccess)
            return cuda_fail(ctx, e, "key sort");
        a.keys = keys_db.Current();
        climb_kernel<<<blocks(n), threads, 0, s>>>(a);
    }
    const bool single = n >= 1 && n <= leaf;
    if (single) {
        emit_single_leaf_kernel<<<1, 1, 0, s>>>(a);
    } else if (n > 1) {
        e = cub::DeviceScan::ExclusiveSum(cub_temp, scan_bytes, a.live, a.map, (int)(n - 1), s);
        if (e != cudaSuccess)
            return cuda_fail(ctx, e, "node compaction");
        emit2_kernel<<<std::min<uint32_t>(blocks(n - 1), (uint32_t)std::max(ctx->sm_count, 1) * 8), threads, 0, s>>>(a);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((uint32_t)std::max(ctx->sm_count, 1) * 4);
        cfg.blockDim = dim3(threads);
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        const int wide = n <= kOneBlock ? 0 : kWideLevels;
        for (int level = 0; level < wide && e == cudaSuccess; ++level)
            e = cudaLaunchKernelEx(&cfg, emit4_level_kernel, a, level);
        cfg.gridDim = dim3(1);
        cfg.blockDim = dim3(1024);
        if (e == cudaSuccess)
            e = cudaLaunchKernelEx(&cfg, bvh4_rest_kernel, a, wide);
        if (e != cudaSuccess)
            return cuda_fail(ctx, e, "BVH4 level launch");
    }
    e = cudaGetLastError();
    uint32_t w[kStateWords];
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(w, a.state, sizeof(w), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(s);
    if (e != cudaSuccess)
        return cuda_fail(ctx, e, "GPU build");
    if (w[kWordBad])
        return fail(ctx, IGXRT_ERROR_INVALID_ARGUMENT, non_finite_message(w[kWordBad], n));
    if (w[kWordMalformed])
        return fail(ctx, IGXRT_ERROR_INVALID_BVH, "GPU build: malformed radix tree");
    const uint32_t n2 = n ? w[kWordNodes2] : 0;
    uint32_t n4 = 0;
    for (int level = 0; level <= kMaxLevels; ++level)
        n4 += w[kWordLevels + level];
    if (w[kWordLevels + kMaxLevels] != 0)
        return fail(ctx, IGXRT_ERROR_INVALID_BVH, "GPU build: BVH4 deeper than the level limit");
    if (n2 > ni || n4 > ni)
        return fail(ctx, IGXRT_ERROR_INVALID_BVH, "GPU build: node count out of range");

    igxrt_bvh_info info{};
    info.triangle_count = a.obj.nt;
    info.sphere_count = a.obj.ns;
    info.cube_count = a.obj.nc;
    info.plane_count = a.obj.np;
    info.bvh2_nodes = n2;
    info.bvh4_nodes = n4;
    info.leaf_count = n ? w[kWordLeaves] : 0;
    info.max_depth = n ? w[kWordDepth] : 0;
    info.max_leaf_size = leaf;
    double sah;
    memcpy(&sah, &w[kWordSah], 8);
    info.sah_cost = n ? (float)sah : 0.f;
    float maxabs;
    memcpy(&maxabs, &w[kWordMaxAbs], 4);
    info.pad_abs = std::max(maxabs * 0x1p-18f, 1e-30f);
    for (int k = 0; k < 3; ++k) {
        info.bounds[k] = n ? key_to_float(~w[kWordLo + k]) : 0.f;
        info.bounds[3 + k] = n ? key_to_float(w[kWordHi + k]) : 0.f;
    }
    // a BVH2 node pushes one entry, the root of a one-leaf tree none
    info.max_stack[IGXRT_LAYOUT_BVH2] = n && !single ? w[kWordDepth] : 0;
    info.max_stack[IGXRT_LAYOUT_BVH4] = n ? w[kWordStack4] : 0;
    info.device_bytes = sizeof(igxrt_bvh2_node) * (uint64_t)n2 + sizeof(igxrt_bvh4_node) * (uint64_t)n4 +
                        sizeof(igxrt_prim_record) * (uint64_t)n + sizeof(igxrt_triangle) * (uint64_t)a.obj.nt +
                        16 * (uint64_t)a.obj.np;
    for (int l = 0; l < IGXRT_LAYOUT_COUNT; ++l)
        if (info.max_stack[l] > kStackCapacity)
            return fail(ctx, IGXRT_ERROR_INVALID_BVH,
                        format("layout %d needs a %u-entry stack (limit %u)", l, info.max_stack[l],
                               kStackCapacity));

    igxrt_scene* scene = nullptr;
    if ((st = allocate_scene(ctx, info, n2, n4, 0, scene, true, s)) != IGXRT_OK)
        return st;
    CopyList copies{};
    int parts = 0;
    auto copy = [&](const void* dst, const void* src, size_t bytes) {
        copies.src[parts] = static_cast<const uint32_t*>(src);
        copies.dst[parts] = static_cast<uint32_t*>(const_cast<void*>(dst));
        copies.words[parts++] = bytes / 4;
    };
    copy(scene->nodes[IGXRT_LAYOUT_BVH2], a.nodes2, sizeof(igxrt_bvh2_node) * (size_t)n2);
    copy(scene->nodes[IGXRT_LAYOUT_BVH4], a.nodes4, sizeof(igxrt_bvh4_node) * (size_t)n4);
    copy(scene->parents[IGXRT_LAYOUT_BVH2], a.parents2, 4 * (size_t)n2);
    copy(scene->parents[IGXRT_LAYOUT_BVH4], a.parents4, 4 * (size_t)n4);
    copy(scene->prims, a.prims, sizeof(igxrt_prim_record) * (size_t)n);
    copy(scene->tris, a.obj.tris, sizeof(igxrt_triangle) * (size_t)a.obj.nt);
    copy(scene->planes, a.obj.planes, 16 * (size_t)a.obj.np);
    copy_kernel<<<std::min<uint32_t>(blocks(std::max<size_t>(3 * (size_t)n, 1)), (uint32_t)std::max(ctx->sm_count, 1) * 8),
                  threads, 0, s>>>(copies);
    if (e == cudaSuccess)
        e = cudaGetLastError();
    if (e == cudaSuccess)
        e = cudaMemsetAsync(scene->refit_words, 0, kRefitStateWords * sizeof(uint32_t), s);
    if (e == cudaSuccess)
        e = write_grid_nodes(ctx, scene, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(w, scene->refit_words, kRefitStateWords * sizeof(uint32_t), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
        igxrt_scene_destroy(scene);
        return cuda_fail(ctx, e, "GPU build copy");
    }
    scene->grid_ok = grid_usable(w);
    *out = scene;
    return IGXRT_OK;
}

}  // extern "C"

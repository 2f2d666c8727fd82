// grid_write.cuh — the pass that writes a scene's grid nodes (grid.cuh) from
// its BVH4 nodes, shared by scene creation (grid.cu) and the refit (refit.cu).
#pragma once

#include "geometry.cuh"
#include "grid.cuh"

namespace igxrt {

constexpr uint32_t kGridBlock = 128;


struct GridAxis {
    float scale, origin, inv;  // inv: 1 / scale, for estimates only
};

// Grid of one axis over [lo, hi]: value 2^15 lies at or below lo and 131070
// (word 65535) at or above hi.  The scale is at least the coordinates' own
// rounding step, finer words would not separate planes any further.
__device__ __forceinline__ GridAxis grid_axis(float lo, float hi) {
    GridAxis g;
    g.scale = fmaxf(__fdiv_ru(__fsub_ru(hi, lo), 98300.f), fmaxf(fabsf(lo), fabsf(hi)) * 0x1p-24f);
    for (int i = 0; i < 16; ++i) {
        g.origin = __fmaf_rd(-32768.f, g.scale, lo);
        if (__fmaf_rn(131070.f, g.scale, g.origin) >= hi && __fmaf_rn(32768.f, g.scale, g.origin) <= lo)
            break;
        g.scale = __fmul_ru(g.scale, 1.000001f);
    }
    // a range near the end of the floats: launches go to the exact nodes
    // (grid_usable), and a captured batch that kept these finds the axis out
    // of its box tests (to_grid) instead of boxes at infinity
    if (!isfinite(g.scale) || !isfinite(g.origin))
        g.scale = __int_as_float(0x7fffffff);
    g.inv = 1.f / g.scale;
    return g;
}

__device__ __forceinline__ float decode(const GridAxis& g, uint32_t q) {
    return __fmaf_rn(grid_value(q), g.scale, g.origin);
}

__device__ __forceinline__ uint32_t estimate(const GridAxis& g, float x) {
    const float v = fminf(fmaxf((x - g.origin) * g.inv, 32768.f), 131070.f);  // NaN: 32768
    return (__float_as_uint(v) - kGridTop) >> 8;
}

// The largest word whose plane is at most lo, the smallest whose plane is at
// least hi (planes rise with the word; the estimate is a step or two away).
__device__ __forceinline__ uint32_t quantize(const GridAxis& g, float lo, float hi) {
    uint32_t a = estimate(g, lo), b = estimate(g, hi);
    while (a > 0 && decode(g, a) > lo)
        --a;
    while (a < 65535u && decode(g, a + 1) <= lo)
        ++a;
    while (b < 65535u && decode(g, b) < hi)
        ++b;
    while (b > 0 && decode(g, b - 1) >= hi)
        --b;
    return a | (b << 16);
}

// A thread per slot, so that a warp reads eight whole nodes and writes eight,
// and a thread quantizes six planes.  For the 210,616 nodes of a 1M sphere (40
// MB read and written, 6 us at the copy rate) a refit's pass takes 18.7 us
// from cold caches; a thread per node, with 24 planes and its own copy of the
// grid, took 25.6, and a block per 128 slots, with its two atomics on the same
// words, 22.2.  The grid spans the root's boxes, which three threads of every
// block read (in L2) instead of waiting for a kernel before this one.
// The blocks of kGridBlock threads that call it are `block` of `blocks`.
// REFIT: the child words stay as they are (a refit keeps the topology).
// `words`: kGridWord* of the scene's refit words, zeroed before the launch.
template <bool REFIT>
__device__ __forceinline__ void write_grid(const igxrt_bvh4_node* nodes, uint32_t count,
                                           const igxrt_prim_record* prims, float4* out, float4* grid,
                                           uint32_t* words, uint32_t block, uint32_t blocks) {
    __shared__ GridAxis g[3];
    if (threadIdx.x < 3) {
        const int k = (int)threadIdx.x;
        const float* f = reinterpret_cast<const float*>(nodes) + 8 * k;  // lo[4], hi[4] of this axis
        float lo = INFINITY, hi = -INFINITY;
        for (int c = 0; c < 4; ++c) {
            const float a = __ldcg(f + c), b = __ldcg(f + 4 + c);
            if (a == INFINITY && b == INFINITY)
                continue;  // absent
            lo = fminf(lo, a);
            hi = fmaxf(hi, b);
        }
        g[k] = grid_axis(lo, hi);
        if (block == 0) {
            reinterpret_cast<float*>(grid)[k] = g[k].scale;
            reinterpret_cast<float*>(grid + 1)[k] = g[k].origin;
        }
    }
    __syncthreads();
    float growth = 0.f;
    uint32_t slots = 0;
    for (uint64_t i = block * (uint64_t)kGridBlock + threadIdx.x; i < 4 * (uint64_t)count;
         i += blocks * (uint64_t)kGridBlock) {
        const float* f = reinterpret_cast<const float*>(nodes + (i >> 2)) + (i & 3u);
        const Box b = {{__ldcg(f), __ldcg(f + 8), __ldcg(f + 16)}, {__ldcg(f + 4), __ldcg(f + 12), __ldcg(f + 20)}};
        const int32_t ref = __ldg(reinterpret_cast<const int32_t*>(f) + 24);
        uint32_t w[3] = {0xffffu, 0xffffu, 0xffffu}, child = kGridLeaf;  // absent
        if (!(b.lo[0] == INFINITY && b.hi[0] == INFINITY)) {
            if (REFIT) {
                child = __float_as_uint(out[i].w);
            } else if (ref >= 0) {
                child = (uint32_t)ref;
            } else {
                const uint32_t first = ~(uint32_t)ref;
                uint32_t more = 0;
                while (!prims[first + more].leaf_end)  // at most 16 records
                    ++more;
                child = kGridLeaf | (first << 4) | (more & 15u);
            }
            Box q;
            for (int k = 0; k < 3; ++k) {
                w[k] = quantize(g[k], b.lo[k], b.hi[k]);
                q.lo[k] = decode(g[k], w[k] & 0xffffu);
                q.hi[k] = decode(g[k], w[k] >> 16);
                if (!(q.lo[k] <= b.lo[k] && q.hi[k] >= b.hi[k]))  // an overflowing grid
                    atomicOr(words + kGridWordUnfit, 1u);
            }
            growth += __fdividef(q.half_area(), b.half_area());
            ++slots;
        }
        out[i] = make_float4(__uint_as_float(w[0]), __uint_as_float(w[1]), __uint_as_float(w[2]),
                             __uint_as_float(child));
    }
    __shared__ float block_growth[4];
    __shared__ uint32_t block_slots[4];
    slots = __reduce_add_sync(0xffffffffu, slots);
    for (int off = 16; off > 0; off >>= 1)
        growth += __shfl_down_sync(0xffffffffu, growth, off);
    if ((threadIdx.x & 31) == 0) {
        block_growth[threadIdx.x / 32] = growth;
        block_slots[threadIdx.x / 32] = slots;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicAdd(words + kGridWordSlots, block_slots[0] + block_slots[1] + block_slots[2] + block_slots[3]);
        atomicAdd(reinterpret_cast<double*>(words + kGridWordGrowth),
                  (double)block_growth[0] + block_growth[1] + block_growth[2] + block_growth[3]);
    }
}

// Blocks of the pass over n4 nodes: two rounds at most, each ends in two
// atomics on the same words.
inline uint32_t grid_write_blocks(const igxrt_context* ctx, uint32_t n4) {
    const uint64_t all = (4 * (uint64_t)n4 + kGridBlock - 1) / kGridBlock;
    const uint64_t most = 16 * (uint64_t)(ctx->sm_count > 0 ? ctx->sm_count : 1);
    return (uint32_t)(all < most ? all : most);
}

}  // namespace igxrt

// grid.cuh — the engine's own form of the BVH4 nodes: 64 bytes, child boxes
// as 16-bit words on a grid over the scene.
//
// What bounds the traversal kernels is their L1 wavefronts and instructions
// per ray: lanes visit different nodes, every 256-bit load of a lane is a
// wavefront of its own, and a BVH2 visit takes two of them for one level of
// the tree.  A grid node is two loads for two levels: half the wavefronts,
// half the visits in a ray's chain of dependent loads, and half the bytes per
// tree in L1 and L2.
//
// A word q stands for the plane value(q) * scale + origin of its axis, where
// value(q) is the float whose top byte is 0x47 and whose middle bytes are q:
// one byte permute decodes it.  These floats run from 2^15 to 2^17, in steps
// of 1 below 2^16 and of 2 above, in the order of q.  Boxes are quantized
// outward from the exact padded boxes (grid.cu), so a ray that enters the
// exact box enters this one.  With the scale and origin folded into the ray
// (to_grid) a slab distance is one fused multiply-add, and the permute's
// selector picks the near and the far plane by the direction's sign, where
// the exact layouts sort the two distances with a min and a max.
//
// Node, 16 words: per slot {x, y, z, child}; an axis word is lo | hi << 16.
// child >= 0 is a grid node; a leaf is kGridLeaf | first record << 4 |
// (records - 1).  An absent child has inverted words (lo 65535, hi 0), which
// no axis in the test lets pass, and refers to record 0 alone: where all three
// axes are out of the test (to_grid) it is a record the linear loop tests too.
#pragma once

#include "traverse.cuh"

namespace igxrt {

constexpr uint32_t kGridLeaf = 0x80000000u;
constexpr uint32_t kGridTop = 0x47000000u;  // value(0), 2^15

__device__ __forceinline__ float grid_value(uint32_t q) { return __uint_as_float(kGridTop | (q << 8)); }

// The plane of an axis word that `sel` picks: kPickLo, or kPickLo ^ kPickSwap
// for the hi half (bytes 7 and 4 of the permute's operands are kGridTop's
// first and last).
constexpr uint32_t kPickLo = 0x7104u, kPickSwap = 0x0220u;
__device__ __forceinline__ float grid_plane(float word, uint32_t sel) {
    return __uint_as_float(__byte_perm(__float_as_uint(word), kGridTop, sel));
}
__device__ __forceinline__ uint32_t grid_near(float step) {
    return kPickLo ^ ((uint32_t)(__float_as_int(step) >> 31) & kPickSwap);
}

// What an axis' plane distances are widened by at either end, in units of the
// origin's distance along it.  The folded origin is rounded to 2^-24 of that
// distance three times (1/dir, its product with the origin, the sum with the
// grid's), and the triangle test's own rounding moves a hit point by as much.
// The boxes' padding covers that up to some 60 scene sizes; from farther out
// rays at edges missed boxes of triangles that they hit: of 200,000 such hits
// 15 at 200 scene sizes and 700 at 1,000 (over the exact nodes, which have the
// same limit, 180 and 1,550), and none with this.  Within 10 scene sizes it is
// less than half a word's step, and the multiply-adds cost at most 0.4%.
constexpr float kGridSlack = 0x1p-22f;

// The intercept of the far planes, from that of the near ones (to_grid), made
// anew at every visit: kept in registers of the ray, the three cost the closest-hit
// kernels more (the 1M sphere's step 905 us, 868 so).
__device__ __forceinline__ float grid_far(float oi) { return __fmaf_rn(fabsf(oi), -2.f * kGridSlack, oi); }

// Folds the scene's grid ({scale}, {origin}) into the ray's slab terms: the
// distance to a plane word of axis a is then fmaf(value, ia, -oia), with oia
// widened for the near planes and grid_far(oia) for the far ones.  An axis
// whose step leaves the range in which that arithmetic is as precise as the
// exact layouts' (a direction beyond 2^90 or so, or an axis-parallel ray in a
// scene beyond 2^40) is taken out of the test: its distances are NaN, which
// the slab test's min and max pass over, so more boxes are entered, never
// fewer.  tmin_box stays finite for the same reason.
__device__ __forceinline__ void to_grid(RayState& r, const float4* __restrict__ grid) {
    const float4 s = __ldg(grid), o = __ldg(grid + 1);
    const auto axis = [](float& i, float& oi, float scale, float origin) {
        const float step = __fmul_rn(scale, i);
        oi = __fmaf_rn(-origin, i, oi);
        oi = __fmaf_rn(fabsf(oi), kGridSlack, oi);
        i = fabsf(step) >= 0x1p-108f && fabsf(step) <= 0x1p108f ? step : __int_as_float(0x7fffffff);
    };
    axis(r.ix, r.oix, s.x, o.x);
    axis(r.iy, r.oiy, s.y, o.y);
    axis(r.iz, r.oiz, s.z, o.z);
    r.tmin_box = fmaxf(r.tmin_box, -3.4028235e38f);
}

template <bool MIXED>
__device__ __forceinline__ bool grid_box_test(const RayState& r, float ofx, float ofy, float ofz, uint32_t sx, uint32_t sy, uint32_t sz, float x,
                                              float y, float z, float tcull, float& tn) {
    const float nx = __fmaf_rn(grid_plane(x, sx), r.ix, -r.oix);
    const float fx = __fmaf_rn(grid_plane(x, sx ^ kPickSwap), r.ix, -ofx);
    const float ny = __fmaf_rn(grid_plane(y, sy), r.iy, -r.oiy);
    const float fy = __fmaf_rn(grid_plane(y, sy ^ kPickSwap), r.iy, -ofy);
    const float nz = __fmaf_rn(grid_plane(z, sz), r.iz, -r.oiz);
    const float fz = __fmaf_rn(grid_plane(z, sz ^ kPickSwap), r.iz, -ofz);
    if (MIXED) {
        // the bounds by FLT_MAX count only when all three axes are out of the test
        const float tnear = fmaxf(fmaxf(nx, ny), fmaxf(nz, -3.4028235e38f));
        const float tslab = fminf(fminf(fx, fy), fminf(fz, 3.4028235e38f));
        tn = tnear;
        return tslab >= r.tmin_box && tnear <= fminf(tslab, tcull);
    }
    return slab_test<false>(r, nx, fx, ny, fy, nz, fz, tcull, tn);
}

// Compare-exchange by entry distance, the child along with it.  The distances
// are compared as signed words: negative ones come out in reverse among
// themselves, which only changes the order of visits.
__device__ __forceinline__ void grid_order(int32_t& ta, int32_t& tb, int32_t& ca, int32_t& cb) {
    const bool swap = tb < ta;
    const int32_t t = swap ? tb : ta, c = swap ? cb : ca;
    tb = swap ? ta : tb;
    cb = swap ? ca : cb;
    ta = t;
    ca = c;
}

// One grid node visit: descend into the nearest hit child, push the others,
// farthest first.  Returns the next reference as visit_node does.
template <bool MIXED>
__device__ __forceinline__ int32_t visit_grid(const float4* __restrict__ nodes, int32_t node, const RayState& r,
                                              float tcull, TraversalStack& st, bool& overflow) {
    constexpr int32_t kMiss = 0x7fffffff;  // above every distance that passes the test (at most the finite tcull)
    const float4* n = nodes + 4 * (size_t)node;
    float4 s[4];
    ldg256(n, s[0], s[1]);
    ldg256(n + 2, s[2], s[3]);
    const uint32_t sx = grid_near(r.ix), sy = grid_near(r.iy), sz = grid_near(r.iz);
    const float ofx = grid_far(r.oix), ofy = grid_far(r.oiy), ofz = grid_far(r.oiz);
    int32_t t[4], c[4];
    uint32_t m = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float tn;
        const bool hit = grid_box_test<MIXED>(r, ofx, ofy, ofz, sx, sy, sz, s[k].x, s[k].y, s[k].z, tcull, tn);
        m += hit ? 1u : 0u;
        t[k] = hit ? __float_as_int(tn) : kMiss;
        c[k] = __float_as_int(s[k].w);
    }
    if (m == 0)
        return st.pop_live(tcull);
    grid_order(t[0], t[1], c[0], c[1]);
    grid_order(t[2], t[3], c[2], c[3]);
    grid_order(t[0], t[2], c[0], c[2]);
    grid_order(t[1], t[3], c[1], c[3]);
    grid_order(t[1], t[2], c[1], c[2]);
    if (st.sp + 3u <= st.sh_depth) {
        // one check and one address for the visit's pushes, as predicated
        // stores: with a check per push and branches around them, 4M
        // incoherent rays took 2,379 us instead of 2,202
        const uint32_t row = st.stride * kStackEntryBytes;
        const uint32_t top = (uint32_t)__cvta_generic_to_shared(st.sh) + (st.sp + m - 2u) * row;
        asm volatile(
            "{\n\t.reg .pred two, three, four;\n\t"
            "setp.gt.u32 two, %0, 1;\n\tsetp.gt.u32 three, %0, 2;\n\tsetp.gt.u32 four, %0, 3;\n\t"
            "@two st.shared.v2.b32 [%1], {%4, %5};\n\t"
            "@three st.shared.v2.b32 [%2], {%6, %7};\n\t"
            "@four st.shared.v2.b32 [%3], {%8, %9};\n\t}" ::"r"(m),
            "r"(top), "r"(top - row), "r"(top - 2u * row), "r"(c[1]), "r"(t[1]), "r"(c[2]), "r"(t[2]), "r"(c[3]),
            "r"(t[3])
            : "memory");
        st.sp += m - 1u;
        return c[0];
    }
    if (st.sp + m - 1 > kStackCapacityDevice) {
        overflow = true;
        return kRefDone;
    }
    if (m > 3)
        st.push(c[3], __int_as_float(t[3]));
    if (m > 2)
        st.push(c[2], __int_as_float(t[2]));
    if (m > 1)
        st.push(c[1], __int_as_float(t[1]));
    return c[0];
}

// The leaf `ref` of a grid node.  Returns true when an any-hit query is decided.
// `any` may differ between lanes (the batch kernel): one loop for both kinds of
// query, since a loop for each made the batch kernel 8% slower (328 us, 304 so).
template <bool MIXED>
__device__ __forceinline__ bool process_grid_leaf(const float4* __restrict__ prims, int32_t ref, const RayState& r,
                                                  BestHit& best, bool any) {
    uint32_t i = ((uint32_t)ref & ~kGridLeaf) >> 4;
    const float4* p = prims + 3 * (size_t)i;
    for (int32_t more = ref & 15;; --more, ++i, p += 3) {
        const float4 v0 = __ldg(p), v1 = __ldg(p + 1), v2 = __ldg(p + 2);
        if ((MIXED ? test_record_mixed(v0, v1, v2, i, r, best, any) : test_record(v0, v1, v2, r, best, any)) && any)
            return true;
        if (more == 0)
            return false;
    }
}

}  // namespace igxrt

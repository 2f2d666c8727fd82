// grid.cu — writes a scene's grid nodes (grid.cuh) at its creation, and the
// rule that decides whether launches use them.
#include <cstring>

#include "grid_write.cuh"

namespace igxrt {

namespace {

__global__ void __launch_bounds__(kGridBlock) grid_nodes_kernel(const igxrt_bvh4_node* nodes, uint32_t count,
                                                                const igxrt_prim_record* prims, float4* out,
                                                                float4* grid, uint32_t* words) {
    write_grid<false>(nodes, count, prims, out, grid, words, blockIdx.x, gridDim.x);
}

}  // namespace

cudaError_t write_grid_nodes(const igxrt_context* ctx, const igxrt_scene* s, cudaStream_t stream) {
    const uint32_t n4 = s->node_count[IGXRT_LAYOUT_BVH4];
    if (!n4 || !s->grid_fits)
        return cudaSuccess;
    grid_nodes_kernel<<<grid_write_blocks(ctx, n4), kGridBlock, 0, stream>>>(
        static_cast<const igxrt_bvh4_node*>(s->nodes[IGXRT_LAYOUT_BVH4]), n4, s->prims, s->grid_nodes, s->grid,
        s->refit_words);
    return cudaGetLastError();
}

// The rule that decides whether launches use the grid nodes: they were written
// (grid_fits), and the slots' surface areas grew by the quantization to at
// most kGridGrowth times on average (a ray visits boxes about in proportion
// to their area).  The mean over the slots, not over the area: a scene whose
// detail is smaller than the grid's steps, however small a part of its area,
// has slots that grew by orders of magnitude and stays on the exact layouts.
bool grid_usable(const uint32_t* words) {
    double growth;
    memcpy(&growth, words + kGridWordGrowth, sizeof(growth));
    return words[kGridWordSlots] && !words[kGridWordUnfit] && growth <= kGridGrowth * words[kGridWordSlots];
}

}  // namespace igxrt

extern "C" {

uint32_t igxrt_internal_uses_grid(const igxrt_scene* scene) { return igxrt::use_grid(*scene, IGXRT_LAYOUT_BVH2); }

void igxrt_internal_set_grid_records(igxrt_context* ctx, uint64_t records) { ctx->grid_records = records; }

}  // extern "C"

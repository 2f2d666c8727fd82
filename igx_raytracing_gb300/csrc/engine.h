// engine.h — host-side engine objects shared by the C ABI translation units.
#pragma once

#include <cuda_runtime.h>

#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "internal.h"

namespace igxrt {
// Ring of item tables used by igxrt_trace_batch.
constexpr uint32_t kBatchSlots = 16;
constexpr uint32_t kBatchSlotItems = 4096;

// A device memory pool and what keeps it: its context, and every scene whose
// memory it holds (the runtime does not survive a free into a destroyed
// pool), so the last of them destroys it.
struct MemoryPool {
    cudaMemPool_t pool = nullptr;
    int device = 0;
    ~MemoryPool();
};
}  // namespace igxrt

struct igxrt_context {
    int device = 0;
    int sm_count = 0;
    std::string device_name;
    std::string last_error;
    // igxrt_trace_batch item tables and the events guarding their reuse.
    void* d_batch = nullptr;
    cudaEvent_t batch_events[igxrt::kBatchSlots] = {};
    uint32_t next_batch_slot = 0;
    // Device words: kQueueSlots work-queue counters, the error word, then one
    // exit counter per queue slot (see launch_trace).
    uint32_t* d_words = nullptr;
    uint32_t next_slot = 0;
    igxrt_launch_params params{};
    // Staging for IGXRT_TRACE_HOST_MEMORY calls on host memory the kernels
    // cannot address (grown on demand).
    void* d_stage = nullptr;
    size_t stage_bytes = 0;
    // Device memory of GPU builds: their scratch and the scenes they make come
    // from this pool and go back to it, so a frame that rebuilds its scene
    // maps no memory (cudaMalloc and cudaFree of both took 260 of the 1,135 us of a
    // 300K-triangle frame).  Idle memory beyond kPoolKeep returns to the device
    // at the next synchronisation, the rest when the context and the last
    // scene are gone.  Null where the device has no pools.
    std::shared_ptr<igxrt::MemoryPool> pool;
    // Largest scene, in records, that gets grid nodes (2^27, the leaf
    // references' field; tests lower it: igxrt_internal_set_grid_records).
    uint64_t grid_records = 1ull << 27;
    // The device loads and stores pageable host memory through the host's
    // page tables (cudaDevAttrPageableMemoryAccessUsesHostPageTables).
    bool pageable_access = false;
};

struct igxrt_scene {
    int device = 0;
    igxrt_bvh_info info{};
    void* d_mem = nullptr;
    std::shared_ptr<igxrt::MemoryPool> pool;  // d_mem's, if it came from one
    const void* nodes[IGXRT_LAYOUT_COUNT] = {nullptr, nullptr, nullptr};
    uint32_t node_count[IGXRT_LAYOUT_COUNT] = {0, 0, 0};
    const igxrt_prim_record* prims = nullptr;
    const igxrt_triangle* tris = nullptr;
    // mixed scenes: spheres and cubes are in the tree, planes are not
    bool mixed = false;
    const float* planes = nullptr;  // 4 floats per plane
    uint32_t plane_count = 0;
    uint32_t plane_base = 0;        // object id of the first plane
    // refit: the parent of every node per layout (kNoParent at the root), and
    // kRefitStateWords state words followed by one arrival counter per node
    // of BVH2, then of BVH4 (zeroed before each refit)
    const uint32_t* parents[IGXRT_LAYOUT_COUNT] = {nullptr, nullptr, nullptr};
    uint32_t* refit_words = nullptr;
    // the grid form of the BVH4 nodes (grid.cuh: 64 bytes per node, {scale},
    // {origin} of the grid), written at creation and by every refit; launches
    // that ask for BVH2 or BVH4 trace it while grid_ok (grid_usable) holds
    float4* grid_nodes = nullptr;
    float4* grid = nullptr;
    bool grid_ok = false;
    // every record fits a grid leaf's reference: the scene's size, so a refit
    // does not change it
    bool grid_fits = false;
    // BVH8 slots' sources in the BVH2 layout (8 per BVH8 node), for the refit
    const uint32_t* src8 = nullptr;
    // GPU refit scratch, two float4 per record ({box lo, leaf_end}, {box hi,
    // 0}), written by the record pass and read by the node climb; allocated
    // at the scene's first GPU refit, freed with the scene
    float4* refit_boxes = nullptr;

    // A layout can be traced when the tree has it; an empty scene has none
    // and traces as all misses in every layout.
    bool has_layout(uint32_t layout) const {
        return layout < IGXRT_LAYOUT_COUNT &&
               (node_count[layout] > 0 || info.triangle_count + info.sphere_count + info.cube_count == 0);
    }
};

namespace igxrt {

constexpr uint32_t kQueueSlots = 4096;
constexpr uint32_t kNoParent = 0xffffffffu;
// State words before the refit's arrival counters: the scan's (geometry.cuh:
// kWord*), then what the grid kernel found (grid.cu).
constexpr uint32_t kRefitStateWords = 12;
constexpr uint32_t kGridWordSlots = 8, kGridWordUnfit = 9, kGridWordGrowth = 10;  // growth: a double
constexpr double kGridGrowth = 1.5;
// Node layout of the launches that trace the grid nodes (internal: callers
// name IGXRT_LAYOUT_*).
constexpr uint32_t kLayoutGrid = IGXRT_LAYOUT_COUNT;

inline size_t round_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Idle bytes a context's pool keeps.
constexpr uint64_t kPoolKeep = 1ull << 30;

// cudaMalloc, which gets the pool's idle memory too where it would fail.
cudaError_t device_alloc(igxrt_context* ctx, void** ptr, size_t bytes);
// Memory from the context's pool, ordered on `stream`; from device_alloc where
// there is no pool or it cannot serve the size (`pooled` says which).
cudaError_t pool_alloc(igxrt_context* ctx, void** ptr, size_t bytes, cudaStream_t stream, bool& pooled);

// One device allocation for a scene of `info`'s primitive counts and n2 / n4
// / n8 nodes; every pointer of the scene is set, the contents are unwritten.
// `pool`: from the context's pool, usable on `stream`.
igxrt_status allocate_scene(igxrt_context* ctx, const igxrt_bvh_info& info, uint32_t n2, uint32_t n4,
                            uint32_t n8, igxrt_scene*& out, bool pool = false, cudaStream_t stream = nullptr);

// Queues the kernel that writes a new scene's grid nodes and folds its findings
// into the refit words kGridWord* (zeroed before); a refit writes them itself
// (refit.cu).  grid_usable judges the words once they are on the host.
// Scenes without grid_fits get none, at creation and at every refit alike:
// the words stay zero, which grid_usable refuses.
cudaError_t write_grid_nodes(const igxrt_context* ctx, const igxrt_scene* scene, cudaStream_t stream);
bool grid_usable(const uint32_t* words);
// Launches over a scene with grid nodes use them in place of the two layouts
// of exact boxes, whichever of the two the caller names: both find the same
// hits, and the grid nodes were the faster at every size measured (a 1M
// sphere's primaries 471 us over BVH2 and 388 so, 4M incoherent rays over 2M
// triangles 3,003 and 2,160 us).  BVH8 stays as named.
inline bool use_grid(const igxrt_scene& s, uint32_t layout) { return s.grid_ok && layout != IGXRT_LAYOUT_BVH8; }
// A scene without nodes takes part in any launch.
inline bool grid_or_empty(const igxrt_scene& s, uint32_t layout) {
    return use_grid(s, layout) || (layout != IGXRT_LAYOUT_BVH8 && s.node_count[layout] == 0);
}

// Parent links of both layouts, computed on the host at scene creation and
// stored after the scene's other buffers (see refit.cu).
void node_parents(const igxrt_bvh& bvh, std::vector<uint32_t>& parents2,
                  std::vector<uint32_t>& parents4);

// Camera rays as a traversal launch's ray source: ray i is the primary ray
// of pixel (i mod width, i / width) (igxrt_trace_gbuffer's first step).
struct CameraSource {
    igxrt_camera cam;
    float inv_w, inv_h;
};

// One traversal launch over `count` rays of one scene (device pointers).
struct TraceRequest {
    const igxrt_scene* scene;
    const igxrt_ray* rays;
    const uint32_t* prev;
    uint32_t count;
    uint32_t mode;  // 0 closest, 1 any
    igxrt_hit* hits;
    uint32_t* occluded;
    uint32_t* node_fetches;  // non-null: instrumented kernel
    uint32_t* prim_fetches;
    // non-null: the number of rays is this device word (written by an earlier
    // kernel on the stream), at most `count`, which sizes the launch
    const uint32_t* count_dev = nullptr;
    // IGXRT_TRACE_INDEPENDENT: the kernel need not wait for the kernel
    // queued before it on the stream
    bool independent = false;
    // non-null: the rays are this camera's, one per pixel (closest hit on a
    // triangle scene; `rays` and `prev` unused)
    const CameraSource* camera = nullptr;
    // instrumented launches: over the grid nodes (the scene must use them)
    // instead of the named layout's
    bool grid_fetches = false;
};

// Records `msg` as the context's last error and returns `st`.
igxrt_status fail(igxrt_context* ctx, igxrt_status st, const std::string& msg);
igxrt_status cuda_fail(igxrt_context* ctx, cudaError_t e, const char* what);

// Checks the launch parameters and fills defaults.
igxrt_status resolve_params(igxrt_context* ctx, const igxrt_launch_params& in,
                            igxrt_launch_params& out);

// Queues the traversal kernel (with its queue reset) on `stream`.
igxrt_status launch_trace(igxrt_context* ctx, const TraceRequest& req,
                          const igxrt_launch_params& params, cudaStream_t stream);

// Same launch, with the work-queue counter and error word supplied by the
// caller (device addresses); the counter is not reset here.
igxrt_status launch_trace_words(igxrt_context* ctx, const TraceRequest& req,
                                const igxrt_launch_params& params, cudaStream_t stream,
                                uint32_t* queue, uint32_t* status);

// Device descriptor of one batch item (see batch.cu).
struct BatchItemDev {
    const float4* nodes;
    const float4* prims;
    const igxrt_ray* rays;
    const uint32_t* prev;
    void* out;
    const float4* planes;   // mixed scenes: the planes outside the tree (else NULL)
    const float4* grid;     // the scene's grid (launches over grid nodes)
    uint32_t count;
    uint32_t mode;
    uint32_t node_count;
    uint32_t packet_begin;  // first packet of this item in the batch's packet space
    uint32_t plane_count;
    uint32_t plane_base;    // object id of the scene's first plane
};

// Node layout of one launch over all items: kLayoutGrid when every item's
// scene allows it (grid_or_empty), else the named one.
uint32_t batch_layout(const igxrt_batch_item* items, uint32_t count, uint32_t layout);
// Fills the device table of `count` items; `mixed` is set when an item's
// scene holds spheres, cubes or planes (the batch then runs the mixed kernel,
// which traces triangle-only items as well), `layout` to the nodes the table
// points at (batch_layout).
igxrt_status build_batch_table(igxrt_context* ctx, const igxrt_batch_item* items, uint32_t count,
                               const igxrt_launch_params& p, std::vector<BatchItemDev>& table,
                               uint32_t& total_packets, uint64_t& total_rays, bool& mixed,
                               uint32_t& layout);
// One item table entry for rays [first, first + count) of a scene (the
// server's request slices); `rays`, `prev` and `out` already point at the
// slice's first element.
void batch_item_for(const igxrt_scene* scene, uint32_t layout, const igxrt_ray* rays,
                    const uint32_t* prev, void* out, uint32_t count, uint32_t mode, BatchItemDev& d);
// `times` (optional, device memory): the earliest CTA start and the latest
// warp exit of the launch, %globaltimer nanoseconds, folded in by atomicMin /
// atomicMax (the caller sets them to ~0 and 0 first).
igxrt_status launch_batch(igxrt_context* ctx, const BatchItemDev* d_table, uint32_t count,
                          uint32_t total_packets, uint64_t total_rays, const igxrt_launch_params& p,
                          uint32_t* queue, cudaStream_t stream, bool mixed, uint32_t layout,
                          unsigned long long* times = nullptr);

// Next work-queue counter of the context (a ring of kQueueSlots words); the
// slot's exit counter is exit_word(slot).
uint32_t* take_queue_slot(igxrt_context* ctx);
inline uint32_t* exit_word(uint32_t* queue_slot) { return queue_slot + kQueueSlots + 1; }
uint32_t* status_word(igxrt_context* ctx);

// Opts a kernel into more than 48 KB of dynamic shared memory when `smem`
// needs it (the traversal stacks of deep shared stacks and large blocks).
inline cudaError_t allow_smem(const void* kernel, size_t smem) {
    if (smem <= 48 * 1024)
        return cudaSuccess;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

// Scene belongs to the context's device.
igxrt_status check_scene(igxrt_context* ctx, const igxrt_scene* scene);
// Grows the context's staging buffer for host-memory calls to `bytes`.
igxrt_status grow_stage(igxrt_context* ctx, size_t bytes);
// Reads and clears the context's kernel error word (synchronous).
igxrt_status read_status(igxrt_context* ctx);

// True when a kernel may dereference p: device, managed or mapped pinned
// memory (NULL counts as accessible).  Pageable host memory is not.
bool device_accessible(const void* p);

// True when the context's kernels may load and store p in place for a
// host-memory call: device or managed memory, pinned host memory mapped at
// the same address, or any host memory when the device reads pageable memory
// through the host's page tables (Grace over NVLink-C2C).  NULL counts.
bool host_direct(const igxrt_context* ctx, const void* p);

// Flags of a trace-like call: IGXRT_TRACE_HOST_MEMORY, IGXRT_TRACE_STAGED
// only together with it, and the bits of `extra` the call also takes.
igxrt_status check_trace_flags(igxrt_context* ctx, uint32_t flags, uint32_t extra = 0);

// Makes ctx->device current for the lifetime of the guard.
class DeviceGuard {
   public:
    explicit DeviceGuard(int device);
    ~DeviceGuard();
    bool ok() const { return ok_; }

   private:
    int prev_ = -1;
    bool ok_ = false;
};

}  // namespace igxrt

// Entry points for the tests and the benchmark, in no public header: which nodes the scene's
// BVH2 and BVH4 launches trace now (1: grid nodes, 0: exact), and a context's
// limit on the records of a scene with grid nodes, for scenes created after
// the call (0: every scene stays on the exact nodes for its life).
extern "C" {
uint32_t igxrt_internal_uses_grid(const igxrt_scene* scene);
void igxrt_internal_set_grid_records(igxrt_context* ctx, uint64_t records);
// igxrt_count_fetches for the launches that trace grid nodes (host arrays).
igxrt_status igxrt_internal_count_grid_fetches(igxrt_context* ctx, const igxrt_scene* scene, const igxrt_ray* rays,
                                               const uint32_t* prev_hit, uint32_t count, uint32_t mode,
                                               uint32_t* node_fetches, uint32_t* prim_fetches);
// The nodes of a batch's latest launch (1: grid nodes).
uint32_t igxrt_internal_batch_uses_grid(const igxrt_batch* batch);
}

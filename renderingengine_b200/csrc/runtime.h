// Internal runtime helpers shared by the C-ABI translation units: error
// reporting, CUDA checks and the scene object.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

#include "re_b200.h"
#include "sah_builder.h"

namespace re {

re_status set_error(re_status code, const std::string& message);
re_status clear_error();

#define RE_CUDA_TRY(expr)                                                             \
    do {                                                                              \
        cudaError_t re_err_ = (expr);                                                 \
        if (re_err_ != cudaSuccess) {                                                 \
            return ::re::set_error(re_err_ == cudaErrorMemoryAllocation               \
                                       ? RE_OUT_OF_MEMORY                             \
                                       : RE_CUDA_ERROR,                               \
                                   std::string(#expr) + ": " +                        \
                                       cudaGetErrorString(re_err_));                  \
        }                                                                             \
    } while (0)

// Device attribute record per leaf-ordered triangle (64 B): the data only the
// final hit needs (shading normals and the canonical identity tuple).
struct alignas(16) DeviceAttr {
    float n0[4];   // n0.xyz, w unused
    float n1[4];
    float n2[4];
    uint32_t ids[4];  // instance, primitive, geometry, material
};
static_assert(sizeof(DeviceAttr) == 64, "attribute record is 64 bytes");

// Scratch buffer that grows on demand and is reused between calls.
//
// A pooled buffer comes from the device's scene pool (scene.cu) in place of
// cudaMalloc.  It is ready on every stream when reserve returns, as with
// cudaMalloc; unlike cudaFree, release does not wait: no work in flight may use
// the buffer any more.
struct DeviceBuffer {
    void* ptr = nullptr;
    size_t bytes = 0;
    int device = 0;
    bool pooled = false;
    cudaError_t reserve(size_t n);
    // Pooled and empty only: ready on `stream` alone, in its order, without a
    // wait or a retry.
    cudaError_t reserve_on(size_t n, cudaStream_t stream);
    void release();
    DeviceBuffer() = default;
    explicit DeviceBuffer(bool from_pool) : pooled(from_pool) {}
    ~DeviceBuffer() { release(); }
};

// Pooled scratch of a build, used on the legacy default stream alone.
struct BuildBuffer : DeviceBuffer {
    BuildBuffer() : DeviceBuffer(true) {}
    ~BuildBuffer() {
        if (ptr != nullptr) cudaStreamSynchronize(cudaStreamLegacy);
    }
};

// What the scene pool of `device` holds unused goes back to the device.
void trim_scene_pool(int device);
// The scene pool's stream, which waits for no other: for copies of a finished
// scene's buffers beside whatever the caller's streams do.
cudaError_t scene_pool_stream(int device, cudaStream_t* out);

// Makes a device current for a scope.
struct DeviceScope {
    int before = 0, device;
    explicit DeviceScope(int d) : device(d) {
        cudaGetDevice(&before);
        if (before != device) cudaSetDevice(device);
    }
    ~DeviceScope() {
        if (before != device) cudaSetDevice(before);
    }
};

// For a scope, this thread's calls are not held against another thread's stream
// capture, whatever its mode.
struct RelaxedCaptureScope {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCaptureScope() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCaptureScope() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

}  // namespace re

struct re_scene;

namespace re {
// GPU LBVH build of a scene from host records (validated by the caller):
// uploads them and builds as below.
re_status build_lbvh_on_device(re_scene* sc, const re_canonical_triangle* tris);
// GPU LBVH build (Morton codes, radix sort, Karras hierarchy) from
// CanonicalTraversalTriangle records in device memory, with the leaf-ordered
// triangle and attribute records and the four-wide nodes.  `check` validates
// them on the device; traversal IDs must then be a permutation of 0 ..
// triangle_count - 1.
re_status build_lbvh_from_device_records(re_scene* sc, const re_canonical_triangle* d_tris, bool check);
// Four-wide nodes from the scene's child-pair nodes, made on the device in
// `scratch` (wide_scratch_bytes of the child-pair node count).
size_t wide_scratch_bytes(uint32_t interior);
re_status build_wide_on_device(re_scene* sc, void* scratch, uint32_t* max_depth);
// Queues making the quad nodes of the scene's child pairs (traverse.cuh,
// trace_quad) on `stream`; false, with nothing left behind, when that fails.
bool make_quad_nodes(re_scene* sc, cudaStream_t stream);
// Fills sc->flat's nodes and leaf order when the tree was built on the device.
re_status host_flat(const re_scene* sc);
// Child-pair device nodes of sc->flat.
re_status upload_scene_nodes(re_scene* sc);
// Leaf-ordered device triangle and attribute records from host records.
re_status upload_scene_triangles(re_scene* sc, const re_canonical_triangle* src_in_leaf_order_or_null,
                                 const re_canonical_triangle* src, const std::vector<uint32_t>& leaf_order);

// Renderer services for the render server (wavefront.cu).
// Film mean of paths [offset, offset + n) into pinned host memory, queued on
// `s` without synchronising.
re_status renderer_copy_mean_async(re_renderer* r, uint32_t offset, uint32_t n, void* host_dst, cudaStream_t s);
// Adds the sample last rendered into paths [src, src + n) to the film of paths
// [dst, dst + n), queued on `s`.
re_status renderer_add_sample_async(re_renderer* r, uint32_t dst, uint32_t src, uint32_t n, cudaStream_t s);
// Allocates the ReSTIR state now (so a budget can account for it).
re_status renderer_reserve_restir(re_renderer* r);
// Device bytes held by the renderer (path pool, tables, ReSTIR state).
uint64_t renderer_device_bytes(const re_renderer* r);
// Running totals since creation: launches' path rays and shadow rays.
re_status renderer_ray_totals(re_renderer* r, uint64_t* path_rays, uint64_t* shadow_rays);
}  // namespace re

struct re_scene {
    int device = 0;
    uint64_t fingerprint = 0;
    uint32_t generation = 0;
    uint32_t triangle_count = 0;
    uint32_t build_kind = 0;
    // Flattened tree: depth and leaf count, and the host copy of its nodes and
    // leaf order (for a tree built on the device, made by host_flat when they
    // are asked for; guarded by flat_mutex).
    re::FlatBvh flat;
    std::mutex flat_mutex;
    uint32_t flat_node_count = 0;
    float root_lo[3] = {}, root_hi[3] = {};
    // The tree is this library's own (its child boxes lie in their parents'),
    // not the caller's flattened nodes.
    bool own_tree = true;
    bool loose = false;  // some child box sticks out of its parent's
    re::DeviceLayout layout_meta;   // node_original / root flag (nodes freed after upload)
    // Resident device buffers.
    re::DeviceBuffer nodes{true};         // DeviceNode[]
    re::DeviceBuffer tris{true};          // DeviceTriangle[]
    re::DeviceBuffer attrs{true};         // DeviceAttr[]
    re::DeviceBuffer leaf_order{true};    // source index per leaf (trees built on the device)
    uint32_t device_node_count = 0;
    double build_ms = 0.0;
    double lbvh_gpu_ms = 0.0;    // device time of the GPU LBVH passes
    double lbvh_total_ms = 0.0;
    // Per-scene staging for host-memory trace batches and the work counter of
    // the persistent traversal kernels.
    re::DeviceBuffer stage_rays{true};
    re::DeviceBuffer stage_hits{true};
    re::DeviceBuffer work_counter;
    // Quad nodes of trace batches, made on the stream of the batch that is the
    // first to walk them.
    enum QuadState { kQuadNone, kQuadQueued, kQuadReady };  // queued: there behind quad_event
    re::DeviceBuffer quad_nodes{true};
    cudaEvent_t quad_event = nullptr;
    std::mutex quad_mutex;
    std::atomic<int> quad_state{kQuadNone};
    std::atomic<uint64_t> quad_owed{0};  // rays of batches without them since the last attempt
    re::DeviceBuffer counters;
    // Four-wide nodes over the same triangles (re::WideNode): made with the
    // scene for this library's own trees, else on first use by a renderer
    // tuned for them.
    re::DeviceBuffer wide_nodes{true};
    uint32_t wide_node_count = 0;
    uint32_t wide_stack_bound = 0;
    // Eight-wide nodes, plain (re::Wide8Node) and compressed (re::Wide8QNode),
    // built on first use by a renderer tuned for them.
    re::DeviceBuffer eight_nodes, eight_qnodes;
    uint32_t eight_node_count = 0;
    uint32_t eight_stack_bound = 0;
    // Alpha masks: per leaf-ordered triangle texture coordinates + material
    // (2 x float4, made when any triangle is alpha-masked), and the tables
    // of re_scene_set_alpha_masks with their device AlphaView.
    bool alpha_masked = false;
    re::DeviceBuffer alpha_tc, alpha_materials, alpha_atlas, alpha_view;
    // Copy streams of chunked host-memory trace batches (created on first use).
    cudaStream_t copy_in = nullptr, copy_out = nullptr;
    ~re_scene();  // waits for the device's work in flight, as cudaFree does
};

namespace re {
// Builds and uploads the scene's four-wide nodes if it has none yet.
re_status ensure_wide_layout(re_scene* sc);
// Builds and uploads the scene's eight-wide nodes (plain and compressed).
re_status ensure_eight_layout(re_scene* sc);
}  // namespace re

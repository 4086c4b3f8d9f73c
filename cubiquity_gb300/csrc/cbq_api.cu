// Device-side C ABI: DAG upload, traversal launches (plain and persistent).
#include "cbq_flat.cuh"
#include "cbq_hostcopy.hpp"
#include "cbq_internal.hpp"
#include "cbq_stage.cuh"
#include "cbq_traverse.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <exception>
#include <new>
#include <vector>

using namespace cbq;

namespace {

constexpr int kFlatBlockDefault = 128;  // GB300, terrain-4096: 64, 128 and 256 threads within 1-3%
constexpr uint32_t kRefillDefault = 16;
constexpr uint32_t kStepsDefault = 8;
// One thread per ray: a warp walks until all its lanes have stopped, so a check for idle lanes
// only costs (camera rays of spheres-256, 1 Mi: every 16 iterations 64.0 us, every 32 63.3).
constexpr uint32_t kStepsPlain = 32;
// An image of up to this many rays takes one thread per ray: its warps stay full to the end, so
// refilling them gains less than the counter's zeroing and the refills cost (about 8 us a call).
// Larger ones gain from refills.  us, one thread per ray / refilled: spheres 0.26 Mi 26 / 33, 1 Mi
// 63 / 70, terrain 1 Mi 85 / 92, city with LOD 1 Mi 105 / 108, 2 Mi 152 / 149, terrain 2.25 Mi
// 187 / 186, 4 Mi 345 / 329.
constexpr uint64_t kPlainImageRays = 3ull << 19;

bool use_flat(const cbq_dag* dag)
{
    return dag->cfg.kernel != CBQ_KERNEL_NESTED || dag->layout == CBQ_DAG_LAYOUT_COMPACT;
}

int flat_block(const cbq_dag* dag) { return dag->cfg.block > 0 ? dag->cfg.block : kFlatBlockDefault; }

FlatLaunch flat_launch(const cbq_dag* dag, bool persistent, uint64_t* counter, uint32_t refill)
{
    FlatLaunch fl;
    fl.persistent = persistent;
    fl.counter = counter;
    fl.block = flat_block(dag);
    fl.refill_min = refill ? refill : dag->cfg.refill_min;
    fl.local_stack = dag->cfg.stack == CBQ_STACK_LOCAL;
    fl.steps = (uint32_t)dag->cfg.steps;
    // Either alone takes the other's default; neither leaves both to the kernel (WarpRefill).
    if (fl.steps && !fl.refill_min) fl.refill_min = kRefillDefault;
    if (!fl.steps) fl.steps = persistent ? kStepsDefault : kStepsPlain;
    return fl;
}

// Rays per warp where a launch without a shape of the caller's is spread (spread_warp_rays) or
// takes one thread per ray (kPlainImageRays), else 0.
uint32_t spread_rays(const cbq_dag* dag, uint64_t n, const cbq_query* query)
{
    if (own_shape(dag->cfg)) return 0u;
    const uint32_t spread = spread_warp_rays(n, dag->device);
    return !spread && query && query->image_width && n <= kPlainImageRays ? 32u : spread;
}

constexpr uint64_t kTaggedMaxNodes = 1ull << 24;  // a tagged reference holds 24 bits of node index
constexpr int kPlainBlock = 128;
constexpr int kPersistBlock = 256;
constexpr uint32_t kDefaultChunk = 64;

dev::DagParams make_dag_params(const cbq_dag* dag)
{
    dev::DagParams p;
    p.nodes = dag->d_nodes;
    p.occupied = 0u;
    p.top = (const uint4*)dag->d_top;
    for (int i = 0; i < 8; i++) {
        if (dag->sd_ref[i] != 0u) p.occupied |= 1u << i;
        p.sd[i].lx = dag->subdags[i].lower_bound[0];
        p.sd[i].ly = dag->subdags[i].lower_bound[1];
        p.sd[i].lz = dag->subdags[i].lower_bound[2];
        p.sd[i].height = dag->subdags[i].node_height;
        p.sd[i].node = dag->sd_ref[i];
        p.sd[i].top = dag->top_index[i];
        p.sd[i].pad[0] = p.sd[i].pad[1] = 0;
    }
    return p;
}

dev::QueryParams make_query(const cbq_query* q)
{
    dev::QueryParams p;
    p.compute_surface = q ? q->compute_surface : 1;
    p.max_footprint = q ? q->max_footprint : CBQ_MAX_FOOTPRINT_DISABLED;
    p.footprint_tmax = footprint_exit_max(p.max_footprint);
    p.flags = q ? q->flags : 0u;
    p.image_width = q ? q->image_width : 0u;  // checked against each launch's ray count by launch_flat
    return p;
}

dev::HitsOut make_hits(const cbq_hits* h)
{
    dev::HitsOut o;
    o.hit = h->hit;
    o.distance = h->distance;
    o.material = h->material;
    o.position = h->position;
    o.normal = h->normal;
    o.voxel = h->voxel;
    o.status = h->status;
    return o;
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

// Copies `bytes` per ray of a chunk between the host array (every ray of the
// call) and the device array (the chunk's rays from c.start).
bool copy_chunk(void* host, void* dev, size_t bytes, const HostChunk& c, cudaMemcpyKind kind, uint64_t max_pitch,
                cudaStream_t s)
{
    const bool in = kind == cudaMemcpyHostToDevice;
    return for_each_copy(c, bytes, max_pitch, [&](const HostCopy& x) {
        char *h = (char*)host + x.host, *d = (char*)dev + x.dev;
        if (x.rows == 1)
            return (in ? cudaMemcpyAsync(d, h, x.width, kind, s) : cudaMemcpyAsync(h, d, x.width, kind, s)) == cudaSuccess;
        return (in ? cudaMemcpy2DAsync(d, x.width, h, x.pitch, x.width, x.rows, kind, s)
                   : cudaMemcpy2DAsync(h, x.pitch, d, x.width, x.width, x.rows, kind, s)) == cudaSuccess;
    });
}

// The copies of a call in one chunk with page-locked buffers: one kernel each way.
struct HostOut {
    StageOut row[kHitFields];
};
__global__ void __launch_bounds__(kStageBlock) cbq_k_host_in(const __grid_constant__ StageIn in)
{
    dev::stage_in(in, (uint64_t)blockIdx.x * kStageBlock + threadIdx.x, (uint64_t)gridDim.x * kStageBlock);
}
// Row y of the grid copies out.row[y].
__global__ void __launch_bounds__(kStageBlock) cbq_k_host_out(const __grid_constant__ HostOut out)
{
    dev::stage_out(out.row[blockIdx.y], (uint64_t)blockIdx.x * kStageBlock + threadIdx.x,
                   (uint64_t)gridDim.x * kStageBlock);
}

// Whether all of a call's host buffers are page-locked (or managed): copies from and to them
// are asynchronous.
bool page_locked(const float* o, const float* d, uint64_t n, const cbq_hits& h)
{
    const struct {
        const void* p;
        uint64_t width;
    } buffers[] = {{o, 16},          {d, 16},       {h.hit, 1},    {h.distance, 4}, {h.material, 4},
                   {h.position, 12}, {h.normal, 12}, {h.voxel, 12}, {h.status, 1}};
    for (const auto& b : buffers)
        if (b.p && !device_alias(b.p, n * b.width)) return false;
    return true;
}

// The two copies of a call of n rays, where all its buffers are page-locked (and the rays
// 16-byte aligned); false otherwise.
bool host_staging(const float* o, const float* d, uint64_t n, const cbq_hits& h, float* d_o, float* d_d,
                  const cbq_hits& dh, StageIn* in, HostOut* out, int* rows)
{
    if (!aligned16(o) || !aligned16(d)) return false;
    const void *ao = device_alias(o, n * 16), *ad = ao ? device_alias(d, n * 16) : nullptr;
    if (!ad) return false;
    *in = StageIn{(const float4*)ao, (const float4*)ad, (float4*)d_o, (float4*)d_d, n, 0};
    struct Field {
        void* host;
        const void* dev;
        uint64_t width;
    };
    const Field fields[kHitFields] = {{h.hit, dh.hit, 1},           {h.distance, dh.distance, 4},
                                      {h.material, dh.material, 4}, {h.position, dh.position, 12},
                                      {h.normal, dh.normal, 12},    {h.voxel, dh.voxel, 12},
                                      {h.status, dh.status, 1}};
    *rows = 0;
    for (const Field& f : fields) {
        if (!f.host) continue;
        char* host = (char*)device_alias(f.host, n * f.width);
        if (!host) return false;
        out->row[(*rows)++] = StageOut{(const char*)f.dev, host, n * f.width};
    }
    return true;
}

// A zeroed work counter of the persistent form for the next launch on `stream`
// (from the stream's ring, allocated on first use), or nullptr where none can be
// had: the id query fails, or the stream is being captured (no allocation inside
// a capture).  The launch is queued while `lk` is held.  A memset
// before every launch took 2 us of the stream (1.5 M shadow rays 123.4 us,
// without 121.4; city camera with LOD 150.5, 148.7).
uint64_t* stream_counter(const cbq_dag* cdag, cudaStream_t stream, std::unique_lock<std::mutex>& lk)
{
    cbq_dag* dag = const_cast<cbq_dag*>(cdag);
    // Only the capture query is legal while a capture is under way: ask it first.
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    if (capture != cudaStreamCaptureStatusNone) return nullptr;
    unsigned long long id = 0;
    if (cudaStreamGetId(stream, &id) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return dag->stream_counters.take(
        id,
        [] {
            void* p = nullptr;
            if (cudaMalloc(&p, CounterRings::kSize * sizeof(uint64_t)) == cudaSuccess) return (uint64_t*)p;
            cudaGetLastError();
            return (uint64_t*)nullptr;
        },
        [&](uint64_t* ring) {
            if (cudaMemsetAsync(ring, 0, CounterRings::kSize * sizeof(uint64_t), stream) == cudaSuccess) return true;
            cudaGetLastError();
            return false;
        },
        lk);
}

cbq_status check_rays(const cbq_rays* rays)
{
    if (!rays || !rays->origin_tmax || !rays->direction) return CBQ_ERR_INVALID_ARGUMENT;
    if (!aligned16(rays->origin_tmax) || !aligned16(rays->direction)) return CBQ_ERR_INVALID_ARGUMENT;
    return CBQ_OK;
}

}  // namespace

// ---------------------------------------------------------------------------
// Kernels
// ---------------------------------------------------------------------------

// One ray per thread, stack in local memory.
__global__ void __launch_bounds__(kPlainBlock) cbq_k_intersect_plain(dev::DagParams dag,
                                                                     const float4* __restrict__ orig,
                                                                     const float4* __restrict__ dir, uint64_t n,
                                                                     dev::QueryParams q, dev::HitsOut out,
                                                                     uint32_t* __restrict__ fetch_out)
{
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    dev::LocalStack stack;
    uint32_t fetches = 0;
    const dev::RayResult r = dev::intersect_volume(dag, __ldg(orig + i), __ldg(dir + i), q, stack, &fetches);
    dev::write_result(out, i, r);
    if (fetch_out) fetch_out[i] = fetches;
}

// Persistent warps: each warp takes `chunk` rays at a time from an atomic
// counter; the descent stack lives in shared memory (one column per thread).
__global__ void __launch_bounds__(kPersistBlock) cbq_k_intersect_persistent(
    dev::DagParams dag, const float4* __restrict__ orig, const float4* __restrict__ dir, uint64_t n,
    dev::QueryParams q, dev::HitsOut out, unsigned long long* __restrict__ counter, uint32_t chunk)
{
    extern __shared__ uint32_t smem_stack[];
    dev::SharedStack stack;
    stack.init(smem_stack + threadIdx.x, blockDim.x);
    const unsigned lane = threadIdx.x & 31u;
    for (;;) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(counter, (unsigned long long)chunk);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= n) break;
        const uint64_t end = min((uint64_t)base + chunk, n);
        for (uint64_t i = base + lane; i < end; i += 32) {
            const dev::RayResult r = dev::intersect_volume(dag, __ldg(orig + i), __ldg(dir + i), q, stack,
                                                           (uint32_t*)nullptr);
            dev::write_result(out, i, r);
        }
    }
}

// The tagged store (dev::Store::kTagged) of a reference node array: one word per
// thread; a word that refers to an internal node reads that node's 32 bytes for
// its occupancy mask.  The material slots stay as they are.
__global__ void __launch_bounds__(256) cbq_k_tag_nodes(const uint4* __restrict__ nodes, uint64_t words,
                                                       uint32_t* __restrict__ tagged)
{
    const uint32_t* w = (const uint32_t*)nodes;
    for (uint64_t i = (uint64_t)blockIdx.x * 256u + threadIdx.x; i < words; i += (uint64_t)gridDim.x * 256u) {
        uint32_t c = __ldg(w + i);
        if (c >= dev::kMaterialCount) {
            const uint4 a = __ldg(nodes + 2ull * c), b = __ldg(nodes + 2ull * c + 1u);
            const uint32_t mask = (a.x ? 1u : 0u) | (a.y ? 2u : 0u) | (a.z ? 4u : 0u) | (a.w ? 8u : 0u) |
                                  (b.x ? 16u : 0u) | (b.y ? 32u : 0u) | (b.z ? 64u : 0u) | (b.w ? 128u : 0u);
            c = (c << 8) | mask;
        }
        tagged[i] = c;
    }
}

// The table of upper cells of the SubDAG with root reference `root`: one cell per thread.
template <dev::Store S>
__global__ void __launch_bounds__(256) cbq_k_top_table(const uint32_t* __restrict__ nodes, uint32_t root,
                                                       uint4* __restrict__ table)
{
    const uint32_t cell = blockIdx.x * 256u + threadIdx.x;
    uint32_t path[dev::kTopLevels] = {0u, 0u, 0u, 0u, 0u};
    uint32_t ref = root, count = 0u, loads = 0u;
#pragma unroll
    for (int d = 0; d < dev::kTopLevels; d++) {
        const int b = dev::kTopLevels - 1 - d;
        const uint32_t slot = ((cell >> b) & 1u) | (((cell >> (b + 5)) & 1u) << 1) | (((cell >> (b + 10)) & 1u) << 2);
        const uint32_t child = (int)count == d ? dev::child_of<S>(nodes, ref, slot, loads) : 0u;
        if (child >= dev::kMaterialCount) {
            path[d] = ref = child;
            count++;
        }
    }
    table[2u * cell] = make_uint4(path[0], path[1], path[2], path[3]);
    table[2u * cell + 1u] = make_uint4(path[4], count, ref, 0u);
}

namespace {

// Numbers the tables of a DAG whose walk store carries masks; returns how many there are.
uint32_t number_top_tables(cbq_dag* dag)
{
    uint32_t tables = 0;
    for (int k = 0; k < 8; k++) {
        const cbq_subdag& s = dag->subdags[k];
        const bool has = s.node_index >= dev::kMaterialCount && s.node_height > dev::kTopLevels;
        dag->top_index[k] = has ? ++tables : 0u;
    }
    return tables;
}

// Queues the kernels that fill them.
cbq_status build_top_tables(const cbq_dag* dag)
{
    for (int k = 0; k < 8; k++) {
        if (!dag->top_index[k]) continue;
        uint4* table = (uint4*)dag->d_top + 2ull * (dag->top_index[k] - 1u) * dev::kTopCells;
        if (dag->layout == CBQ_DAG_LAYOUT_COMPACT)
            cbq_k_top_table<dev::Store::kCompact><<<dev::kTopCells / 256u, 256, 0, cudaStreamLegacy>>>(
                dag->walk_nodes(), dag->walk_root(k), table);
        else
            cbq_k_top_table<dev::Store::kTagged><<<dev::kTopCells / 256u, 256, 0, cudaStreamLegacy>>>(
                dag->walk_nodes(), dag->walk_root(k), table);
    }
    return cudaGetLastError() == cudaSuccess ? CBQ_OK : CBQ_ERR_CUDA;
}

cbq_status preload_nested_persistent()
{
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, cbq_k_intersect_persistent) == cudaSuccess) return CBQ_OK;
    cudaGetLastError();
    return CBQ_ERR_CUDA;
}

}  // namespace

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------

extern "C" {

cbq_status cbq_dag_create(const uint32_t* host_nodes, uint64_t node_count, uint32_t root, cbq_dag** out)
{
    return cbq_dag_create_ex(host_nodes, node_count, root, CBQ_DAG_LAYOUT_REFERENCE, out);
}

cbq_status cbq_dag_create_ex(const uint32_t* host_nodes, uint64_t node_count, uint32_t root, uint32_t layout,
                             cbq_dag** out)
{
    if (!out || layout > CBQ_DAG_LAYOUT_COMPACT) return CBQ_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    cbq_status st = validate_nodes(host_nodes, node_count, root);
    if (st != CBQ_OK) return st;
    cbq_dag* dag = new (std::nothrow) cbq_dag();
    if (!dag) return CBQ_ERR_OUT_OF_MEMORY;
    st = find_subdags(host_nodes, node_count, root, dag->subdags);
    if (st == CBQ_OK) st = validate_heights(host_nodes, node_count, dag->subdags);
    if (st != CBQ_OK) { delete dag; return st; }
    dag->node_count = node_count;
    dag->flat_ok = float_positions_exact(dag);
    dag->root = root;
    dag->max_height = 0;
    for (int i = 0; i < 8; i++)
        if (dag->subdags[i].node_index > 0) dag->max_height = std::max(dag->max_height, dag->subdags[i].node_height);
    if (cudaGetDevice(&dag->device) != cudaSuccess) { delete dag; return CBQ_ERR_CUDA; }
    // Materialise cbq_intersect_host_noalloc's fixed array, and load the persistent
    // kernels it launches, on this device now, while allocating is expected, so that
    // the no-allocation entry point never does (CUDA loads both lazily).
    if (noalloc_prepare(dag->device) != CBQ_OK || preload_persistent_kernels() != CBQ_OK ||
        preload_nested_persistent() != CBQ_OK)
        cbq::log(CBQ_LOG_WARNING, "device %d: the no-allocation staging array could not be prepared", dag->device);
    for (int i = 0; i < 8; i++) dag->sd_ref[i] = dag->subdags[i].node_index;
    const uint32_t* src = host_nodes;
    size_t bytes = (size_t)node_count * 32u;
    std::vector<uint32_t> compact;
    if (layout == CBQ_DAG_LAYOUT_COMPACT) {
        uint32_t refs[8];
        const cbq_status cst = dag->flat_ok ? build_compact(host_nodes, node_count, dag->subdags, compact, refs)
                                            : CBQ_ERR_INVALID_ARGUMENT;
        if (cst == CBQ_OK) {
            dag->layout = CBQ_DAG_LAYOUT_COMPACT;
            std::memcpy(dag->sd_ref, refs, sizeof(refs));
            src = compact.data();
            bytes = compact.size() * sizeof(uint32_t);
        } else {
            cbq::log(CBQ_LOG_WARNING, "compact layout unavailable (%s): using the reference layout",
                     dag->flat_ok ? "store beyond 128 MB" : "coordinates beyond 2^21");
        }
    }
    dag->device_bytes = bytes;
    const bool tag = dag->flat_ok && dag->layout == CBQ_DAG_LAYOUT_REFERENCE && node_count <= kTaggedMaxNodes;
    // One allocation: the node array, its tagged copy and the tables of upper cells (a cudaMalloc
    // takes 70 us).
    const bool masks = tag || dag->layout == CBQ_DAG_LAYOUT_COMPACT;
    const size_t part = (bytes + 255u) & ~(size_t)255u;
    const size_t top_bytes = masks ? (size_t)number_top_tables(dag) * dev::kTopCells * 32u : 0u;
    const size_t total = masks ? part + (tag ? part : 0u) + top_bytes : bytes;
    bool whole = false;
    dag->d_nodes = (uint32_t*)allocate_store(total, bytes, [](uint64_t n) {
        void* p = nullptr;
        if (cudaMalloc(&p, n) == cudaSuccess) return p;
        cudaGetLastError();
        return (void*)nullptr;
    }, &whole);
    if (!dag->d_nodes) {
        delete dag;
        return CBQ_ERR_OUT_OF_MEMORY;
    }
    if (!whole)
        for (uint32_t& t : dag->top_index) t = 0u;
    cudaError_t e = cudaMemcpy(dag->d_nodes, src, bytes, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && whole && tag) {
        dag->d_tagged = dag->d_nodes + part / 4u;
        const uint64_t words = node_count * 8u;
        cbq_k_tag_nodes<<<(unsigned)std::min<uint64_t>((words + 255) / 256, 1u << 20), 256, 0, cudaStreamLegacy>>>(
            (const uint4*)dag->d_nodes, words, dag->d_tagged);
        e = cudaGetLastError();
        for (int i = 0; i < 8; i++) {
            const uint32_t r = dag->subdags[i].node_index;
            uint32_t mask = 0;
            for (int k = 0; k < 8; k++) mask |= host_nodes[(uint64_t)r * 8 + k] != 0u ? 1u << k : 0u;
            dag->tagged_ref[i] = r == 0u ? 0u : (r << 8) | mask;
        }
    }
    if (e == cudaSuccess && whole && top_bytes != 0u) {
        dag->d_top = dag->d_nodes + (total - top_bytes) / 4u;
        if (build_top_tables(dag) != CBQ_OK) e = cudaErrorUnknown;
    }
    if (e != cudaSuccess || cudaStreamSynchronize(cudaStreamLegacy) != cudaSuccess) {
        cudaFree(dag->d_nodes);
        delete dag;
        return CBQ_ERR_CUDA;
    }
    cbq::log(CBQ_LOG_INFO,
             "DAG uploaded to device %d: %llu nodes, %s layout (%.1f MB), root %u, max sub-DAG height %d, %s kernel",
             dag->device, (unsigned long long)node_count,
             dag->layout == CBQ_DAG_LAYOUT_COMPACT ? "compact" : "reference", bytes / 1e6, root, dag->max_height,
             dag->flat_ok ? "flat (float positions)" : "flat (integer positions: coordinates beyond 2^21 or 2^29 nodes)");
    *out = dag;
    return CBQ_OK;
}

cbq_status cbq_dag_destroy(cbq_dag* dag)
{
    if (!dag) return CBQ_ERR_INVALID_ARGUMENT;
    cudaFree(dag->d_nodes);
    dag->stream_counters.release([](uint64_t* ring) { cudaFree(ring); });
    pt_workspace_release(dag->pt);
    for (auto& hs : dag->stages) {
        if (hs->d_stage) cudaFree(hs->d_stage);
        for (cudaStream_t& st : hs->pipe)
            if (st) cudaStreamDestroy(st);
        for (cudaEvent_t& ev : hs->pipe_ev)
            if (ev) cudaEventDestroy(ev);
    }
    delete dag;
    return CBQ_OK;
}

cbq_status cbq_dag_get_info(const cbq_dag* dag, cbq_dag_info* info)
{
    if (!dag || !info) return CBQ_ERR_INVALID_ARGUMENT;
    info->node_count = dag->node_count;
    info->bytes = dag->node_count * 32u;
    info->root = dag->root;
    info->max_subdag_height = dag->max_height;
    std::memcpy(info->subdags, dag->subdags, sizeof(dag->subdags));
    info->device_nodes = dag->d_nodes;
    info->layout = dag->layout;
    info->device_bytes = dag->device_bytes;
    return CBQ_OK;
}

cbq_status cbq_dag_set_l2_persistence(const cbq_dag* dag, cbq_stream_t stream, float fraction)
{
    if (!dag || fraction < 0.0f || fraction > 1.0f) return CBQ_ERR_INVALID_ARGUMENT;
    cudaStreamAttrValue attr;
    std::memset(&attr, 0, sizeof(attr));
    if (fraction > 0.0f) {
        int max_window = 0, max_persist = 0;
        cudaDeviceGetAttribute(&max_window, cudaDevAttrMaxAccessPolicyWindowSize, dag->device);
        cudaDeviceGetAttribute(&max_persist, cudaDevAttrMaxPersistingL2CacheSize, dag->device);
        if (max_window <= 0 || max_persist <= 0) return CBQ_OK;  // not supported: leave caching as is
        const size_t want = (size_t)((double)max_persist * fraction);
        if (cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, want) != cudaSuccess) return CBQ_ERR_CUDA;
        const size_t window = std::min<size_t>(dag->device_bytes, (size_t)max_window);
        attr.accessPolicyWindow.base_ptr = (void*)dag->walk_nodes();
        attr.accessPolicyWindow.num_bytes = window;
        attr.accessPolicyWindow.hitRatio = (float)std::min(1.0, (double)want / (double)window);
        attr.accessPolicyWindow.hitProp = cudaAccessPropertyPersisting;
        attr.accessPolicyWindow.missProp = cudaAccessPropertyStreaming;
    }
    if (cudaStreamSetAttribute((cudaStream_t)stream, cudaStreamAttributeAccessPolicyWindow, &attr) != cudaSuccess)
        return CBQ_ERR_CUDA;
    if (fraction == 0.0f) {
        // Give the set-aside back to normal caching, and demote lines already marked
        // persisting (both settings belong to this process's context).
        if (cudaDeviceSetLimit(cudaLimitPersistingL2CacheSize, 0) != cudaSuccess ||
            cudaCtxResetPersistingL2Cache() != cudaSuccess)
            return CBQ_ERR_CUDA;
    }
    return CBQ_OK;
}

cbq_status cbq_intersect(const cbq_dag* dag, const cbq_rays* rays, uint64_t n, const cbq_query* query,
                         const cbq_hits* hits, cbq_stream_t stream)
{
    if (!dag || !hits) return CBQ_ERR_INVALID_ARGUMENT;
    if (!rays) return CBQ_ERR_INVALID_ARGUMENT;
    if (n == 0) return CBQ_OK;  // an empty batch may carry NULL buffers
    cbq_status st = check_rays(rays);
    if (st != CBQ_OK) return st;
    if (use_flat(dag)) {
        // The DAG's form: persistent (the default, with this stream's work counter) or plain.
        const uint32_t spread = spread_rays(dag, n, query);
        std::unique_lock<std::mutex> queueing;
        uint64_t* counter = dag->cfg.form != CBQ_FORM_PLAIN && !spread
                                ? stream_counter(dag, (cudaStream_t)stream, queueing) : nullptr;
        FlatLaunch fl = counter ? flat_launch(dag, true, counter, 0u) : flat_launch(dag, false, nullptr, 0u);
        fl.counter_zeroed = counter != nullptr;
        if (spread) fl.warp_rays = spread;
        return launch_flat(dag, make_dag_params(dag), make_query(query), make_hits(hits),
                           (const float4*)rays->origin_tmax, (const float4*)rays->direction, n, nullptr, fl,
                           (cudaStream_t)stream);
    }
    const uint64_t blocks = (n + kPlainBlock - 1) / kPlainBlock;
    if (blocks > 0x7fffffffull) return CBQ_ERR_INVALID_ARGUMENT;
    cbq_k_intersect_plain<<<(unsigned)blocks, kPlainBlock, 0, (cudaStream_t)stream>>>(
        make_dag_params(dag), (const float4*)rays->origin_tmax, (const float4*)rays->direction, n,
        make_query(query), make_hits(hits), nullptr);
    return cudaGetLastError() == cudaSuccess ? CBQ_OK : CBQ_ERR_CUDA;
}

cbq_status cbq_dag_set_launch_config(cbq_dag* dag, const cbq_launch_config* cfg)
{
    if (!dag || !cfg) return CBQ_ERR_INVALID_ARGUMENT;
    if (cfg->kernel < CBQ_KERNEL_AUTO || cfg->kernel > CBQ_KERNEL_FLAT) return CBQ_ERR_INVALID_ARGUMENT;
    if (cfg->block < 0 || cfg->block > 256 || (cfg->block % 32) != 0) return CBQ_ERR_INVALID_ARGUMENT;
    if (cfg->refill_min > 32) return CBQ_ERR_INVALID_ARGUMENT;
    if (cfg->stack != CBQ_STACK_SHARED && cfg->stack != CBQ_STACK_LOCAL) return CBQ_ERR_INVALID_ARGUMENT;
    if (cfg->form < CBQ_FORM_PLAIN || cfg->form > CBQ_FORM_SORTED) return CBQ_ERR_INVALID_ARGUMENT;
    if (cfg->steps < 0 || cfg->steps > 32) return CBQ_ERR_INVALID_ARGUMENT;
    if (cfg->registers != 0 && cfg->registers != 56) return CBQ_ERR_INVALID_ARGUMENT;
    if (cfg->kernel == CBQ_KERNEL_NESTED && dag->layout == CBQ_DAG_LAYOUT_COMPACT) return CBQ_ERR_INVALID_ARGUMENT;
    dag->cfg = *cfg;
    return CBQ_OK;
}

uint64_t cbq_scratch_bytes(uint64_t n) { return 256 + 4 * n; }

cbq_status cbq_intersect_auto(const cbq_dag* dag, const cbq_rays* rays, uint64_t n, const cbq_query* query,
                              const cbq_hits* hits, void* scratch, uint64_t scratch_bytes, cbq_stream_t stream)
{
    if (!dag || !hits || !rays) return CBQ_ERR_INVALID_ARGUMENT;
    if (n == 0) return CBQ_OK;
    if (!scratch || scratch_bytes < cbq_scratch_bytes(n) || ((uintptr_t)scratch & 15u))
        return CBQ_ERR_INVALID_ARGUMENT;
    cbq_status st = check_rays(rays);
    if (st != CBQ_OK) return st;
    // Scratch: [0, 8) work counter | [64, 128) octant counts and cursors | [256, 256 + 4n) permutation
    uint64_t* counter = (uint64_t*)scratch;
    uint32_t* counts = (uint32_t*)((char*)scratch + 64);
    uint32_t* perm = (uint32_t*)((char*)scratch + 256);
    if (dag->cfg.form == CBQ_FORM_PLAIN) return cbq_intersect(dag, rays, n, query, hits, stream);
    if (dag->cfg.form == CBQ_FORM_PERSISTENT || !use_flat(dag))
        return cbq_intersect_persistent(dag, rays, n, query, hits, counter, 0u, stream);
    st = launch_octant_sort((const float4*)rays->direction, n, counts, perm, dag->device, (cudaStream_t)stream);
    if (st != CBQ_OK) return st;
    FlatLaunch fl = flat_launch(dag, true, counter, 0u);
    fl.perm = perm;
    return launch_flat(dag, make_dag_params(dag), make_query(query), make_hits(hits),
                       (const float4*)rays->origin_tmax, (const float4*)rays->direction, n, nullptr, fl,
                       (cudaStream_t)stream);
}

cbq_status cbq_autotune(cbq_dag* dag, const cbq_rays* rays, uint64_t n, const cbq_query* query,
                        const cbq_hits* hits, void* scratch, uint64_t scratch_bytes, int32_t repetitions,
                        cbq_launch_config* best, float* best_ms, cbq_stream_t stream)
{
    if (!dag || repetitions <= 0 || n == 0) return CBQ_ERR_INVALID_ARGUMENT;
    if (!scratch || scratch_bytes < cbq_scratch_bytes(n)) return CBQ_ERR_INVALID_ARGUMENT;
    cudaEvent_t e0, e1;
    if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess) return CBQ_ERR_CUDA;
    const cbq_launch_config saved = dag->cfg;
    cbq_launch_config winner = saved;
    float win_ms = 1e30f;
    cbq_status st = CBQ_OK;
    for_each_tuned_config(saved, [&](const cbq_launch_config& c) {
        dag->cfg = c;
        st = cbq_intersect_auto(dag, rays, n, query, hits, scratch, scratch_bytes, stream);  // warm-up
        if (st != CBQ_OK) return false;
        cudaEventRecord(e0, (cudaStream_t)stream);
        for (int r = 0; r < repetitions && st == CBQ_OK; r++)
            st = cbq_intersect_auto(dag, rays, n, query, hits, scratch, scratch_bytes, stream);
        cudaEventRecord(e1, (cudaStream_t)stream);
        if (st != CBQ_OK || cudaEventSynchronize(e1) != cudaSuccess) {
            st = CBQ_ERR_CUDA;
            return false;
        }
        float ms = 0;
        cudaEventElapsedTime(&ms, e0, e1);
        ms /= (float)repetitions;
        if (ms < win_ms) {
            win_ms = ms;
            winner = c;
        }
        return true;
    });
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    dag->cfg = st == CBQ_OK ? winner : saved;
    if (st == CBQ_OK)
        cbq::log(CBQ_LOG_INFO,
                 "autotune over %llu rays: form %d, block %d, refill %u, stack %s, steps %d: %.3f ms",
                 (unsigned long long)n, winner.form, winner.block, winner.refill_min,
                 winner.stack == CBQ_STACK_LOCAL ? "local" : "shared", winner.steps, win_ms);
    if (best) *best = dag->cfg;
    if (best_ms) *best_ms = st == CBQ_OK ? win_ms : 0.0f;
    return st;
}

cbq_status cbq_dag_get_launch_config(const cbq_dag* dag, cbq_launch_config* cfg)
{
    if (!dag || !cfg) return CBQ_ERR_INVALID_ARGUMENT;
    *cfg = dag->cfg;
    if (cfg->kernel == CBQ_KERNEL_AUTO) cfg->kernel = CBQ_KERNEL_FLAT;
    if (cfg->block == 0) cfg->block = use_flat(dag) ? kFlatBlockDefault : kPlainBlock;
    if (cfg->chunk == 0) cfg->chunk = kDefaultChunk;
    // refill_min and steps stay 0 where they are automatic: no fixed value gives the same launches.
    return CBQ_OK;
}

cbq_status cbq_count_fetches(const cbq_dag* dag, const cbq_rays* rays, uint64_t n, const cbq_query* query,
                             uint32_t* fetches, cbq_stream_t stream)
{
    if (!dag || !fetches) return CBQ_ERR_INVALID_ARGUMENT;
    if (!rays) return CBQ_ERR_INVALID_ARGUMENT;
    if (n == 0) return CBQ_OK;  // an empty batch may carry NULL buffers
    cbq_status st = check_rays(rays);
    if (st != CBQ_OK) return st;
    dev::HitsOut none;
    std::memset(&none, 0, sizeof(none));
    if (use_flat(dag))
        return launch_flat(dag, make_dag_params(dag), make_query(query), none, (const float4*)rays->origin_tmax,
                           (const float4*)rays->direction, n, fetches, flat_launch(dag, false, nullptr, 0u),
                           (cudaStream_t)stream);
    const uint64_t blocks = (n + kPlainBlock - 1) / kPlainBlock;
    cbq_k_intersect_plain<<<(unsigned)blocks, kPlainBlock, 0, (cudaStream_t)stream>>>(
        make_dag_params(dag), (const float4*)rays->origin_tmax, (const float4*)rays->direction, n,
        make_query(query), none, fetches);
    return cudaGetLastError() == cudaSuccess ? CBQ_OK : CBQ_ERR_CUDA;
}

cbq_status cbq_intersect_persistent(const cbq_dag* dag, const cbq_rays* rays, uint64_t n, const cbq_query* query,
                                    const cbq_hits* hits, uint64_t* work_counter, uint32_t chunk,
                                    cbq_stream_t stream)
{
    if (!dag || !hits || !work_counter) return CBQ_ERR_INVALID_ARGUMENT;
    if (!rays) return CBQ_ERR_INVALID_ARGUMENT;
    if (n == 0) return CBQ_OK;  // an empty batch may carry NULL buffers
    cbq_status st = check_rays(rays);
    if (st != CBQ_OK) return st;
    if (use_flat(dag)) {
        const uint32_t spread = chunk == 0 ? spread_rays(dag, n, query) : 0u;
        FlatLaunch fl = flat_launch(dag, !spread, spread ? nullptr : work_counter, std::min<uint32_t>(chunk, 32u));
        if (spread) fl.warp_rays = spread;
        return launch_flat(dag, make_dag_params(dag), make_query(query), make_hits(hits),
                           (const float4*)rays->origin_tmax, (const float4*)rays->direction, n, nullptr, fl,
                           (cudaStream_t)stream);
    }
    if (chunk == 0) chunk = dag->cfg.chunk ? dag->cfg.chunk : kDefaultChunk;
    const int stack_h = std::max(1, (int)dag->max_height);
    const size_t smem = (size_t)stack_h * kPersistBlock * sizeof(uint32_t);
    int sms = 0, per_sm = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dag->device) != cudaSuccess) return CBQ_ERR_CUDA;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cbq_k_intersect_persistent, kPersistBlock, smem) !=
        cudaSuccess)
        return CBQ_ERR_CUDA;
    per_sm = std::max(per_sm, 1);
    if (cudaMemsetAsync(work_counter, 0, sizeof(uint64_t), (cudaStream_t)stream) != cudaSuccess) return CBQ_ERR_CUDA;
    cbq_k_intersect_persistent<<<sms * per_sm, kPersistBlock, smem, (cudaStream_t)stream>>>(
        make_dag_params(dag), (const float4*)rays->origin_tmax, (const float4*)rays->direction, n,
        make_query(query), make_hits(hits), (unsigned long long*)work_counter, chunk);
    return cudaGetLastError() == cudaSuccess ? CBQ_OK : CBQ_ERR_CUDA;
}

}  // extern "C"

namespace cbq {

bool takes_device_count(const cbq_dag* dag)
{
    return use_flat(dag) && dag->cfg.stack == CBQ_STACK_SHARED && dag->cfg.form == CBQ_FORM_PERSISTENT;
}

cbq_status intersect_device_count(const cbq_dag* dag, const cbq_rays* rays, uint64_t most, const uint32_t* n_dev,
                                  const cbq_query* query, const cbq_hits* hits, uint64_t* zeroed_counter,
                                  cbq_stream_t stream)
{
    const cbq_status st = check_rays(rays);
    if (st != CBQ_OK || most == 0) return st;
    FlatLaunch fl = flat_launch(dag, true, zeroed_counter, 0u);
    fl.n_dev = n_dev;
    return launch_flat(dag, make_dag_params(dag), make_query(query), make_hits(hits),
                       (const float4*)rays->origin_tmax, (const float4*)rays->direction, most, nullptr, fl,
                       (cudaStream_t)stream);
}

}  // namespace cbq

namespace {

// Takes a staging set of `dag` for one call, locked: a free one, else a new
// one while fewer than kHostStagesMax exist, else the first (waiting for it).
std::unique_lock<std::mutex> take_stage(cbq_dag* dag, HostStage** out)
{
    std::unique_lock<std::mutex> pool(dag->stages_lock);
    for (auto& hs : dag->stages) {
        std::unique_lock<std::mutex> lk(hs->lock, std::try_to_lock);
        if (lk.owns_lock()) {
            *out = hs.get();
            return lk;
        }
    }
    if ((int)dag->stages.size() < kHostStagesMax) {
        HostStage* hs = new (std::nothrow) HostStage();
        if (hs) {
            try {
                dag->stages.emplace_back(hs);
            } catch (const std::exception&) {  // nothing may throw across the C ABI
                delete hs;
                hs = nullptr;
            }
        }
        if (hs) {
            *out = hs;
            return std::unique_lock<std::mutex>(hs->lock);
        }
        if (dag->stages.empty()) {
            *out = nullptr;
            return std::unique_lock<std::mutex>();
        }
    }
    HostStage* hs = dag->stages.front().get();
    pool.unlock();
    *out = hs;
    return std::unique_lock<std::mutex>(hs->lock);
}

}  // namespace

extern "C" cbq_status cbq_intersect_host(const cbq_dag* cdag, const float* host_origin_tmax,
                                         const float* host_direction, uint64_t n, const cbq_query* query,
                                         const cbq_hits* host_hits)
{
    if (!cdag || !host_origin_tmax || !host_direction || !host_hits) return CBQ_ERR_INVALID_ARGUMENT;
    if (n == 0) return CBQ_OK;
    cbq_dag* dag = const_cast<cbq_dag*>(cdag);
    HostStage* hs = nullptr;
    std::unique_lock<std::mutex> lock = take_stage(dag, &hs);
    if (!hs) return CBQ_ERR_OUT_OF_MEMORY;
    // Staging: rays (32 B), hit fields (46 B) per ray, then one work counter per chunk.
    const size_t per_ray = 32 + 1 + 4 + 4 + 12 + 12 + 12 + 1;
    const size_t tail = 256 + kHostChunksMax * 64;
    if (n > hs->capacity) {
        if (hs->d_stage) cudaFree(hs->d_stage);
        hs->d_stage = nullptr;
        hs->capacity = 0;
        if (cudaMalloc(&hs->d_stage, (size_t)n * per_ray + tail) != cudaSuccess) {
            cudaGetLastError();
            return CBQ_ERR_OUT_OF_MEMORY;
        }
        hs->capacity = n;
    }
    if (!hs->pipe[0]) {  // created all together, or not at all
        bool ok = true;
        for (int k = 0; k < 4 && ok; k++)
            ok = cudaStreamCreateWithFlags(&hs->pipe[k], cudaStreamNonBlocking) == cudaSuccess;
        for (uint64_t k = 0; k < 2 * kHostChunksMax && ok; k++)
            ok = cudaEventCreateWithFlags(&hs->pipe_ev[k], cudaEventDisableTiming) == cudaSuccess;
        if (!ok) {
            cudaGetLastError();
            for (cudaStream_t& st : hs->pipe)
                if (st) { cudaStreamDestroy(st); st = nullptr; }
            for (cudaEvent_t& ev : hs->pipe_ev)
                if (ev) { cudaEventDestroy(ev); ev = nullptr; }
            return CBQ_ERR_CUDA;
        }
    }
    char* p = (char*)hs->d_stage;
    float* d_o = (float*)p;
    p += n * 16;
    float* d_d = (float*)p;
    p += n * 16;
    cbq_hits dh;
    dh.position = (float*)p; p += n * 12;
    dh.normal = (float*)p; p += n * 12;
    dh.voxel = (int32_t*)p; p += n * 12;
    dh.distance = (float*)p; p += n * 4;
    dh.material = (uint32_t*)p; p += n * 4;
    dh.hit = (uint8_t*)p; p += n;
    dh.status = (uint8_t*)p;
    p += n;
    // Work counters, one 64-byte line per chunk.
    uint64_t* d_counters = (uint64_t*)(((uintptr_t)p + 255u) & ~(uintptr_t)255u);
    cudaStream_t s_in = hs->pipe[0], s_out = hs->pipe[1];
    // Every queued copy and launch ends before the call returns (the staging buffers are reused).
    auto drain = [&](cbq_status st) {
        bool ok = true;
        for (cudaStream_t s : hs->pipe) ok = cudaStreamSynchronize(s) == cudaSuccess && ok;
        return ok ? st : CBQ_ERR_CUDA;
    };
    // Chunks pipeline the copies with the traversal: while chunk k is traversed, chunk k + 1 is
    // copied in and chunk k - 1 copied out.  Consecutive chunks are traversed on alternating
    // streams, so the next chunk's blocks fill the SMs while the previous launch drains (a
    // persistent launch ends with a tail of few busy warps).  Events order each chunk's copy in,
    // traversal and copy out.  The copies out take longest, so the first chunks are the smallest:
    // the copies out then begin early and the larger chunks are traversed under them.  us per
    // call of 300 Ki / 1 Mi / 4 Mi bounce rays: chunks of 1:2:3:4 238 / 494 / 1,399; up to 8 equal
    // ones of 256 Ki rays or more 259 / 528 / 1,498, up to 8 of 1:2:3:4:4:.. 235 / 507 / 1,450.
    // Pageable buffers take one chunk: their copies block the calling thread, so nothing overlaps
    // and every chunk adds nine copies (300 K / 1 M bounce rays 434 -> 310 us, 1,015 -> 637).
    HostChunk plan[kHostChunksMax];
    const bool overlaps = host_chunks(n) > 1 && page_locked(host_origin_tmax, host_direction, n, *host_hits);
    const uint64_t chunks = plan_host_chunks(n, overlaps, plan);
    StageIn stage_rays;
    HostOut stage_hits;
    int stage_rows = 0;
    if (chunks == 1 && host_staging(host_origin_tmax, host_direction, n, *host_hits, d_o, d_d, dh, &stage_rays,
                                    &stage_hits, &stage_rows)) {
        // One chunk of page-locked buffers: a copy kernel in, the traversal and a copy kernel out
        // in a row on one stream.
        cudaStream_t s = hs->pipe[2];
        cbq_k_host_in<<<stage_blocks(2 * n), kStageBlock, 0, s>>>(stage_rays);
        if (cudaGetLastError() != cudaSuccess) return drain(CBQ_ERR_CUDA);
        cbq_rays rays{d_o, d_d};
        cbq_hits launch = dh;
        if (!host_hits->hit) launch.hit = nullptr;
        if (!host_hits->distance) launch.distance = nullptr;
        if (!host_hits->material) launch.material = nullptr;
        if (!host_hits->position) launch.position = nullptr;
        if (!host_hits->normal) launch.normal = nullptr;
        if (!host_hits->voxel) launch.voxel = nullptr;
        if (!host_hits->status) launch.status = nullptr;
        const cbq_status st = cbq_intersect_persistent(dag, &rays, n, query, &launch, d_counters, 0u, (cbq_stream_t)s);
        if (st != CBQ_OK) return drain(st);
        if (stage_rows != 0) {
            cbq_k_host_out<<<dim3(stage_blocks(n * 12 / 16), stage_rows), kStageBlock, 0, s>>>(stage_hits);
            if (cudaGetLastError() != cudaSuccess) return drain(CBQ_ERR_CUDA);
        }
        return cudaStreamSynchronize(s) == cudaSuccess ? CBQ_OK : CBQ_ERR_CUDA;
    }
    int max_pitch = 0;
    if (cudaDeviceGetAttribute(&max_pitch, cudaDevAttrMaxPitch, dag->device) != cudaSuccess) return CBQ_ERR_CUDA;
    for (uint64_t k = 0; k < chunks; k++) {
        const HostChunk& hc = plan[k];
        const uint64_t a = hc.start, m = hc.rays();
        if (m == 0) continue;
        cudaStream_t s_run = hs->pipe[2 + (k & 1)];
        cudaEvent_t copied = hs->pipe_ev[2 * k], traversed = hs->pipe_ev[2 * k + 1];
        if (!copy_chunk((void*)host_origin_tmax, d_o, 16, hc, cudaMemcpyHostToDevice, max_pitch, s_in) ||
            !copy_chunk((void*)host_direction, d_d, 16, hc, cudaMemcpyHostToDevice, max_pitch, s_in) ||
            cudaEventRecord(copied, s_in) != cudaSuccess || cudaStreamWaitEvent(s_run, copied, 0) != cudaSuccess)
            return drain(CBQ_ERR_CUDA);
        cbq_hits launch;
        launch.hit = host_hits->hit ? dh.hit + a : nullptr;
        launch.distance = host_hits->distance ? dh.distance + a : nullptr;
        launch.material = host_hits->material ? dh.material + a : nullptr;
        launch.position = host_hits->position ? dh.position + 3 * a : nullptr;
        launch.normal = host_hits->normal ? dh.normal + 3 * a : nullptr;
        launch.voxel = host_hits->voxel ? dh.voxel + 3 * a : nullptr;
        launch.status = host_hits->status ? dh.status + a : nullptr;
        cbq_rays rays{d_o + 4 * a, d_d + 4 * a};
        // Persistent form; each chunk's counter is private to this call (its staging set is held).
        cbq_status st = cbq_intersect_persistent(dag, &rays, m, query, &launch, d_counters + 8 * k, 0u,
                                                 (cbq_stream_t)s_run);
        if (st != CBQ_OK) return drain(st);
        if (cudaEventRecord(traversed, s_run) != cudaSuccess || cudaStreamWaitEvent(s_out, traversed, 0) != cudaSuccess)
            return drain(CBQ_ERR_CUDA);
        struct Copy {
            void* host;
            void* dev;
            size_t width;
        };
        const Copy copies[] = {{host_hits->hit, dh.hit, 1},           {host_hits->distance, dh.distance, 4},
                               {host_hits->material, dh.material, 4}, {host_hits->position, dh.position, 12},
                               {host_hits->normal, dh.normal, 12},    {host_hits->voxel, dh.voxel, 12},
                               {host_hits->status, dh.status, 1}};
        for (const Copy& c : copies) {
            if (!c.host) continue;
            if (!copy_chunk(c.host, c.dev, c.width, hc, cudaMemcpyDeviceToHost, max_pitch, s_out)) return drain(CBQ_ERR_CUDA);
        }
    }
    return drain(CBQ_OK);
}

// Wavefront pathtracer on top of the traversal (cbq_pathtrace).
//
// Restates the reference's CPU pathtracer (pathtracing_demo.cpp:81-190:
// traceSingleRayRecurse / gatherLighting) as GPU waves.  Per pass (as many
// samples per pixel as fit in kPtRaysPerPass paths, traced together):
//   camera rays -> [extension traversal -> shade -> shadow traversal -> add]
//   repeated for depth 0..bounces
// Shading follows the reference: a hit multiplies the path throughput by the
// material's colour and gathers direct light from a sun shadow ray (offset
// 0.001 along the normal, pathtracing_demo.cpp:83-97) and a sky shadow ray in
// the direction normalize(normal + random point in the unit sphere) (:99-114);
// the bounce ray starts 0.01 along the normal (:166) in the same kind of
// direction; a miss returns the background colour.  Materials may also emit.
// All traversals use the library's traversal with the LOD footprint given
// (the demo uses 0.0035, pathtracing_demo.h:84), computeSurfaceProperties on
// extension rays and off on shadow rays, exactly as the reference calls it.
// Random numbers come from a counter-based hash of (seed, pixel, sample,
// depth, purpose), so a frame is reproducible.
#include "cbq_internal.hpp"

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstring>
#include <exception>
#include <vector>

namespace {

struct PathState {
    uint32_t pixel, sample;
    float tr, tg, tb;  // throughput
};

// Paths traced together in one pass: the samples of a pass share each wave's
// launches (fewer, larger launches).
constexpr uint64_t kPtRaysPerPass = 1ull << 24;

struct Frame {
    int width, height;
    uint32_t sample, samples;  // the pass's first sample and its sample count
    uint64_t seed;
    float ex, ey, ez;              // eye
    float fx, fy, fz;              // forward
    float rx, ry, rz;              // right
    float ux, uy, uz;              // up
    float tan_half, aspect;
};

struct Shading {
    float max_footprint;
    float sun[3], sun_colour[3], sky_colour[3], background[3];
    float albedo[256][3];
    float emission[256][3];
};

__device__ __forceinline__ uint64_t mix64(uint64_t x)
{
    x ^= x >> 30;
    x *= 0xbf58476d1ce4e5b9ull;
    x ^= x >> 27;
    x *= 0x94d049bb133111ebull;
    x ^= x >> 31;
    return x;
}

__device__ __forceinline__ uint64_t rng_key(uint64_t seed, uint32_t pixel, uint32_t sample, uint32_t depth,
                                            uint32_t purpose)
{
    return mix64(seed ^ mix64(((uint64_t)pixel << 32) | ((uint64_t)sample << 8) | (depth << 4) | purpose));
}

__device__ __forceinline__ float u01(uint64_t& h)
{
    h = mix64(h + 0x9e3779b97f4a7c15ull);
    return (float)(h >> 40) * (1.0f / 16777216.0f);
}

// A point uniformly inside the unit sphere: direction from two uniforms
// (sincospif), radius from the cube root of a third.
__device__ __forceinline__ float3 in_unit_sphere(uint64_t h)
{
    const float z = 1.0f - 2.0f * u01(h);
    const float r = sqrtf(fmaxf(0.0f, 1.0f - z * z));
    float s, c;
    sincospif(2.0f * u01(h), &s, &c);
    const float rad = cbrtf(u01(h));
    return make_float3(r * c * rad, r * s * rad, z * rad);
}

__device__ __forceinline__ float3 normalize3(float3 v)
{
    const float l = sqrtf(v.x * v.x + v.y * v.y + v.z * v.z);
    return l > 0.0f ? make_float3(v.x / l, v.y / l, v.z / l) : make_float3(0.0f, 0.0f, 1.0f);
}

// Path i of a pass: pixel i % npix of sample f.sample + i / npix.
__global__ void cbq_k_pt_camera(Frame f, float4* __restrict__ o, float4* __restrict__ d, PathState* __restrict__ st)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t npix = (uint32_t)f.width * (uint32_t)f.height;
    if (i >= npix * f.samples) return;
    const uint32_t pixel = i % npix, sample = f.sample + i / npix;
    const uint32_t px = pixel % (uint32_t)f.width, py = pixel / (uint32_t)f.width;
    uint64_t h = rng_key(f.seed, pixel, sample, 0, 0);
    const float jx = u01(h), jy = u01(h);
    const float sx = (((px + jx) / f.width) * 2.0f - 1.0f) * f.aspect * f.tan_half;
    const float sy = (1.0f - ((py + jy) / f.height) * 2.0f) * f.tan_half;
    const float3 dir = normalize3(make_float3(f.fx + f.rx * sx + f.ux * sy, f.fy + f.ry * sx + f.uy * sy,
                                              f.fz + f.rz * sx + f.uz * sy));
    o[i] = make_float4(f.ex, f.ey, f.ez, __int_as_float(0x7f800000));
    d[i] = make_float4(dir.x, dir.y, dir.z, 0.0f);
    st[i] = PathState{pixel, sample, 1.0f, 1.0f, 1.0f};
}

// Contributions are never negative and the image starts at +0, so adding a zero
// changes nothing: black contributions (most materials emit nothing) are skipped.
__device__ __forceinline__ void add_pixel(float* image, uint32_t pixel, float r, float g, float b)
{
    if (r == 0.0f && g == 0.0f && b == 0.0f) return;
    atomicAdd(image + 3 * (size_t)pixel, r);
    atomicAdd(image + 3 * (size_t)pixel + 1, g);
    atomicAdd(image + 3 * (size_t)pixel + 2, b);
}

// Reserves the warp's slots in both compacted arrays with one 64-bit atomic
// (all 32 lanes call it): two shadow rays per hit in the low word of `counts`
// (the shadow count), one bounce ray per continuing path in the high word (the
// bounce count).  A lane's shadow rays are slots s0 and s0 + 1.  One atomic
// round trip per warp instead of three in a row: the kernel waits on memory.
__device__ __forceinline__ void reserve_slots(unsigned long long* counts, bool hit, bool cont, uint32_t& s0,
                                              uint32_t& b)
{
    const unsigned hm = __ballot_sync(0xffffffffu, hit), cm = __ballot_sync(0xffffffffu, cont);
    const unsigned lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    unsigned long long base = 0;
    if (lane == 0 && (hm | cm))
        base = atomicAdd(counts, 2ull * (unsigned)__popc(hm) | ((unsigned long long)(unsigned)__popc(cm) << 32));
    base = __shfl_sync(0xffffffffu, base, 0);
    s0 = (uint32_t)base + 2u * (uint32_t)__popc(hm & below);
    b = (uint32_t)(base >> 32) + (uint32_t)__popc(cm & below);
}

__global__ void cbq_k_pt_shade(const Shading* __restrict__ sh, uint32_t n, const uint32_t* __restrict__ n_dev,
                               uint32_t depth, uint64_t seed, int last, const PathState* __restrict__ st,
                               const uint8_t* __restrict__ hit, const uint32_t* __restrict__ material,
                               const float* __restrict__ position, const float* __restrict__ normal,
                               float* __restrict__ image, float4* __restrict__ so, float4* __restrict__ sd,
                               float4* __restrict__ sw, unsigned long long* __restrict__ counts,
                               float4* __restrict__ no, float4* __restrict__ nd, PathState* __restrict__ nst,
                               uint32_t* __restrict__ seen)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (n_dev) n = __ldg(n_dev);  // the count of an earlier wave's shading; n otherwise
    if (seen && i == 0) *seen = n;
    const bool live = i < n;
    PathState p{0u, 0u, 0.0f, 0.0f, 0.0f};
    bool h = false;
    if (live) {
        p = st[i];
        h = hit[i] != 0;
        if (!h) add_pixel(image, p.pixel, p.tr * sh->background[0], p.tg * sh->background[1], p.tb * sh->background[2]);
    }
    float3 pos = make_float3(0.0f, 0.0f, 0.0f), nrm = make_float3(0.0f, 0.0f, 0.0f);
    float tr = 0.0f, tg = 0.0f, tb = 0.0f;
    uint64_t key = 0;
    if (h) {
        const uint32_t m = material[i] & 255u;
        pos = make_float3(position[3 * i], position[3 * i + 1], position[3 * i + 2]);
        nrm = make_float3(normal[3 * i], normal[3 * i + 1], normal[3 * i + 2]);
        add_pixel(image, p.pixel, p.tr * sh->emission[m][0], p.tg * sh->emission[m][1], p.tb * sh->emission[m][2]);
        tr = p.tr * sh->albedo[m][0];
        tg = p.tg * sh->albedo[m][1];
        tb = p.tb * sh->albedo[m][2];
        key = rng_key(seed, p.pixel, p.sample, depth + 1, 0);
    }
    // Two shadow rays per hit (sun and sky) and a bounce ray per continuing path.
    const bool cont = h && !last;
    uint32_t s0 = 0, b = 0;
    reserve_slots(counts, h, cont, s0, b);
    const uint32_t s1 = s0 + 1u;
    if (h) {
        const float3 off = make_float3(nrm.x * 0.001f, nrm.y * 0.001f, nrm.z * 0.001f);
        const float3 org = make_float3(pos.x + off.x, pos.y + off.y, pos.z + off.z);
        const float sdot = fmaxf(sh->sun[0] * nrm.x + sh->sun[1] * nrm.y + sh->sun[2] * nrm.z, 0.0f);
        so[s0] = make_float4(org.x, org.y, org.z, __int_as_float(0x7f800000));
        sd[s0] = make_float4(sh->sun[0], sh->sun[1], sh->sun[2], 0.0f);
        sw[s0] = make_float4(tr * sh->sun_colour[0] * sdot, tg * sh->sun_colour[1] * sdot, tb * sh->sun_colour[2] * sdot,
                             __uint_as_float(p.pixel));
        const float3 q = in_unit_sphere(mix64(key ^ 1u));
        const float3 sky = normalize3(make_float3(nrm.x + q.x, nrm.y + q.y, nrm.z + q.z));
        so[s1] = make_float4(org.x, org.y, org.z, __int_as_float(0x7f800000));
        sd[s1] = make_float4(sky.x, sky.y, sky.z, 0.0f);
        sw[s1] = make_float4(tr * sh->sky_colour[0], tg * sh->sky_colour[1], tb * sh->sky_colour[2],
                             __uint_as_float(p.pixel));
    }
    // The bounce ray.
    if (cont) {
        const float3 q = in_unit_sphere(mix64(key ^ 2u));
        const float3 dir = normalize3(make_float3(nrm.x + q.x, nrm.y + q.y, nrm.z + q.z));
        no[b] = make_float4(pos.x + nrm.x * 0.01f, pos.y + nrm.y * 0.01f, pos.z + nrm.z * 0.01f,
                            __int_as_float(0x7f800000));
        nd[b] = make_float4(dir.x, dir.y, dir.z, 0.0f);
        nst[b] = PathState{p.pixel, p.sample, tr, tg, tb};
    }
}

__global__ void cbq_k_pt_shadow_add(uint32_t n, const uint32_t* __restrict__ n_dev, const uint8_t* __restrict__ hit,
                                    const float4* __restrict__ sw, float* __restrict__ image)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (n_dev) n = __ldg(n_dev);
    if (i >= n || hit[i]) return;
    const float4 w = sw[i];
    add_pixel(image, __float_as_uint(w.w), w.x, w.y, w.z);
}

__global__ void cbq_k_pt_scale(float* image, size_t count, float scale)
{
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) image[i] *= scale;
}

std::atomic<uint64_t> g_kept{0};  // bytes of the workspaces kept between frames

void release_memory(cbq::PtWorkspace& w)
{
    if (w.base) cudaFree(w.base);
    w.base = nullptr;
    w.bytes = 0;
    g_kept -= w.kept;
    w.kept = 0;
}

// After a frame: keeps the memory of `w` for the next, or gives it back.
void keep_or_release(cbq::PtWorkspace& w)
{
    const uint64_t more = w.bytes - w.kept;  // a kept workspace only grows
    uint64_t total = g_kept.load();
    while (total + more <= cbq::kPtKeptBytes && !g_kept.compare_exchange_weak(total, total + more)) {
    }
    if (total + more <= cbq::kPtKeptBytes)
        w.kept = w.bytes;
    else
        release_memory(w);
}

template <typename F>
void for_each_event(cbq::PtWorkspace& w, F f)
{
    f(w.begin);
    for (cudaEvent_t& ev : w.shaded) f(ev);
    for (cudaEvent_t& ev : w.traced) f(ev);
}

// Streams, events, at least `bytes` of device memory and, for a frame that looks at
// its waves' counts, the host memory for them in `w`.
cbq_status prepare_workspace(cbq::PtWorkspace& w, uint64_t bytes, bool look)
{
    if (!w.wave) {
        int low = 0, high = 0;
        bool ok = cudaDeviceGetStreamPriorityRange(&low, &high) == cudaSuccess &&
                  cudaStreamCreateWithPriority(&w.wave, cudaStreamNonBlocking, high) == cudaSuccess &&
                  cudaStreamCreateWithPriority(&w.shadow, cudaStreamNonBlocking, low) == cudaSuccess;
        for_each_event(w, [&](cudaEvent_t& ev) {
            ok = ok && cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) == cudaSuccess;
        });
        if (!ok) {
            cudaGetLastError();
            return CBQ_ERR_CUDA;
        }
    }
    if (look && !w.seen && cudaMallocHost((void**)&w.seen, cbq::kPtAhead * sizeof(uint32_t)) != cudaSuccess) {
        cudaGetLastError();
        w.seen = nullptr;
        return CBQ_ERR_OUT_OF_MEMORY;
    }
    if (w.bytes >= bytes) return CBQ_OK;
    release_memory(w);
    if (cudaMalloc((void**)&w.base, bytes) != cudaSuccess) {
        cudaGetLastError();
        w.base = nullptr;
        return CBQ_ERR_OUT_OF_MEMORY;
    }
    w.bytes = bytes;
    return CBQ_OK;
}

template <typename T>
T* carve(char*& p, size_t count)
{
    T* r = (T*)p;
    p += (count * sizeof(T) + 255) & ~(size_t)255;
    return r;
}

}  // namespace

void cbq::pt_workspace_release(PtWorkspace& w)
{
    release_memory(w);
    for (cudaStream_t* q : {&w.wave, &w.shadow}) {
        if (*q) cudaStreamDestroy(*q);
        *q = nullptr;
    }
    for_each_event(w, [](cudaEvent_t& ev) {
        if (ev) cudaEventDestroy(ev);
        ev = nullptr;
    });
    if (w.seen) cudaFreeHost(w.seen);
    w.seen = nullptr;
}

extern "C" cbq_status cbq_copy_to_host(void* host_dst, const void* device_src, uint64_t bytes)
{
    if (bytes == 0) return CBQ_OK;
    if (!host_dst || !device_src) return CBQ_ERR_INVALID_ARGUMENT;
    return cudaMemcpy(host_dst, device_src, bytes, cudaMemcpyDeviceToHost) == cudaSuccess ? CBQ_OK : CBQ_ERR_CUDA;
}

extern "C" cbq_status cbq_pathtrace(const cbq_dag* dag, const cbq_pt_config* cfg, float* device_image,
                                    cbq_pt_wave_fn on_wave, void* user, cbq_pt_stats* stats, cbq_stream_t cstream)
{
    if (!dag || !cfg || !device_image || !cfg->materials) return CBQ_ERR_INVALID_ARGUMENT;
    if (cfg->width <= 0 || cfg->height <= 0 || cfg->samples_per_pixel <= 0 || cfg->bounces < 0 ||
        cfg->bounces > 64)
        return CBQ_ERR_INVALID_ARGUMENT;
    const uint64_t npix = (uint64_t)cfg->width * (uint64_t)cfg->height;
    if (npix > (1u << 30)) return CBQ_ERR_INVALID_ARGUMENT;
    cudaStream_t s = (cudaStream_t)cstream;
    const auto t_start = std::chrono::steady_clock::now();

    // Camera basis (z up), as cbq_gen_pinhole_rays.
    double f[3] = {cfg->target[0] - cfg->eye[0], cfg->target[1] - cfg->eye[1], cfg->target[2] - cfg->eye[2]};
    const double fl = std::sqrt(f[0] * f[0] + f[1] * f[1] + f[2] * f[2]);
    if (!(fl > 0)) return CBQ_ERR_INVALID_ARGUMENT;
    for (double& v : f) v /= fl;
    double r[3] = {f[1], -f[0], 0.0};
    const double rl = std::sqrt(r[0] * r[0] + r[1] * r[1]);
    if (!(rl > 0)) return CBQ_ERR_INVALID_ARGUMENT;
    r[0] /= rl;
    r[1] /= rl;
    const double u[3] = {r[1] * f[2] - r[2] * f[1], r[2] * f[0] - r[0] * f[2], r[0] * f[1] - r[1] * f[0]};

    Shading host_sh;
    host_sh.max_footprint = cfg->max_footprint;
    for (int a = 0; a < 3; a++) {
        host_sh.sun[a] = cfg->sun_direction[a];
        host_sh.sun_colour[a] = cfg->sun_colour[a];
        host_sh.sky_colour[a] = cfg->sky_colour[a];
        host_sh.background[a] = cfg->background[a];
    }
    for (int m = 0; m < 256; m++)
        for (int a = 0; a < 3; a++) {
            host_sh.albedo[m][a] = cfg->materials[m].albedo[a];
            host_sh.emission[m][a] = cfg->materials[m].emission[a];
        }

    // Without a wave callback the host waits for nothing until the frame is done: a wave's ray
    // count stays on the device (the shading that compacts the next wave's rays leaves it
    // there), and shadow waves run on a stream of their own beside the next extension wave,
    // each filling the SMs that the other's last rays leave.
    const bool ahead = !on_wave && cbq::takes_device_count(dag);
    // Buffers for one pass: two extension sets (ping-pong) and one shadow set (260 bytes a path),
    // or two where a depth's shadow wave may still run while the next depth is shaded (358): in
    // frames whose workspace is kept.  ms, one set / two: city-2048, 4 bounces, 1920x1080 1.69 /
    // 1.58, 640x360 0.53 / 0.48; with 2 samples, where the workspace is allocated for the frame,
    // 3.63 / 3.80, 16 samples 23.0 / 23.6 (their waves fill the chip by themselves).
    const uint64_t per_pass = std::max<uint64_t>(
        1, std::min<uint64_t>((uint64_t)cfg->samples_per_pixel, kPtRaysPerPass / npix));
    const size_t ext = npix * per_pass, sha = 2 * ext;
    const size_t passes = ((size_t)cfg->samples_per_pixel + per_pass - 1) / per_pass;
    const size_t waves = passes * ((size_t)cfg->bounces + 1);
    const size_t per_ext = 2 * 16 + sizeof(PathState) + 1 + 4 + 12 + 12;
    const size_t control = waves * (8 + 2 * 8);  // per wave: shadow and next count, two work counters
    const auto frame_bytes = [&](int sets) {
        return 2 * ext * per_ext + sets * sha * (16 * 3 + 1) + control + sizeof(Shading) + 40 * 256;  // + carve padding
    };
    const int sets = ahead && frame_bytes(2) <= cbq::kPtKeptBytes ? 2 : 1;
    const size_t bytes = frame_bytes(sets);

    // The DAG's workspace, or one of this frame's own where another frame has it.
    cbq_dag* owner = const_cast<cbq_dag*>(dag);
    std::unique_lock<std::mutex> lock(owner->pt_lock, std::try_to_lock);
    cbq::PtWorkspace own;
    cbq::PtWorkspace& ws = lock.owns_lock() ? owner->pt : own;
    // The paths of a frame of many bounces may all have ended long before the last, so each
    // shading (ahead) also leaves its wave's count in host memory, and the host looks at it kPtAhead waves
    // later, which keeps the device busy: smaller grids, and no more waves once one had no rays.
    // One sphere, 64 bounces: 640x360 1,030 -> 295 us, 2048x2048, 10 samples 25.2 -> 8.7 ms.
    const bool look = ahead && cfg->bounces >= cbq::kPtAhead;
    cbq_status st = prepare_workspace(ws, bytes, look);
    if (st != CBQ_OK) {
        cbq::pt_workspace_release(ws);
        return st;
    }
    char* p = ws.base;
    Shading* d_sh = carve<Shading>(p, 1);
    uint64_t* counts = carve<uint64_t>(p, 3 * waves);  // per wave: [shadow count, next count], extension and shadow work
    struct Ext {
        float4 *o, *d;
        PathState* st;
        uint8_t* hit;
        uint32_t* material;
        float *position, *normal;
    } e[2];
    struct Sha {
        float4 *o, *d, *w;
        uint8_t* hit;
    } s2[2];
    for (int k = 0; k < 2; k++) {
        e[k].o = carve<float4>(p, ext);
        e[k].d = carve<float4>(p, ext);
        e[k].st = carve<PathState>(p, ext);
        e[k].hit = carve<uint8_t>(p, ext);
        e[k].material = carve<uint32_t>(p, ext);
        e[k].position = carve<float>(p, 3 * ext);
        e[k].normal = carve<float>(p, 3 * ext);
    }
    for (int k = 0; k < sets; k++) {
        s2[k].o = carve<float4>(p, sha);
        s2[k].d = carve<float4>(p, sha);
        s2[k].w = carve<float4>(p, sha);
        s2[k].hit = carve<uint8_t>(p, sha);
    }
    if ((size_t)(p - ws.base) > bytes) return CBQ_ERR_INVALID_ARGUMENT;

    const cudaStream_t sw = ahead ? (cudaStream_t)ws.wave : s;
    const cudaStream_t ss = ahead ? (cudaStream_t)ws.shadow : s;
    uint64_t ext_rays = 0, shadow_rays = 0, launches = 0;
    auto fail = [&](cbq_status code) {
        st = code;
        cudaGetLastError();
    };
    auto ok = [](cudaError_t e) { return e == cudaSuccess; };
    if (!ok(cudaMemcpyAsync(d_sh, &host_sh, sizeof(Shading), cudaMemcpyHostToDevice, s)) ||
        !ok(cudaMemsetAsync(counts, 0, 3 * waves * sizeof(uint64_t), s)) ||
        !ok(cudaMemsetAsync(device_image, 0, npix * 3 * sizeof(float), s)))
        fail(CBQ_ERR_CUDA);
    if (st == CBQ_OK && ahead &&
        (!ok(cudaEventRecord(ws.begin, s)) || !ok(cudaStreamWaitEvent(sw, ws.begin, 0)) ||
         !ok(cudaStreamWaitEvent(ss, ws.begin, 0))))
        fail(CBQ_ERR_CUDA);

    const cbq_query qext{1, cfg->max_footprint, 0u, 0u};
    const cbq_query qsh{0, cfg->max_footprint, 0u, 0u};
    // The camera wave's paths are the pass's samples' images stacked in row-major
    // order: the traversal may deal them to warps in image tiles.
    const cbq_query qcam{1, cfg->max_footprint, 0u, (uint32_t)cfg->width};
    size_t wave = 0;  // over the frame's passes and depths
    bool set_used[2] = {false, false};
    for (int sample = 0; sample < cfg->samples_per_pixel && st == CBQ_OK; sample += (int)per_pass) {
        const uint32_t samples = (uint32_t)std::min<uint64_t>(per_pass, (uint64_t)(cfg->samples_per_pixel - sample));
        Frame fr;
        fr.width = cfg->width;
        fr.height = cfg->height;
        fr.sample = (uint32_t)sample;
        fr.samples = samples;
        fr.seed = cfg->seed;
        fr.ex = (float)cfg->eye[0];
        fr.ey = (float)cfg->eye[1];
        fr.ez = (float)cfg->eye[2];
        fr.fx = (float)f[0]; fr.fy = (float)f[1]; fr.fz = (float)f[2];
        fr.rx = (float)r[0]; fr.ry = (float)r[1]; fr.rz = (float)r[2];
        fr.ux = (float)u[0]; fr.uy = (float)u[1]; fr.uz = (float)u[2];
        fr.tan_half = (float)cfg->tan_half_fov;
        fr.aspect = (float)cfg->width / (float)cfg->height;
        const uint32_t paths = (uint32_t)(npix * samples);
        cbq_k_pt_camera<<<(paths + 255) / 256, 256, 0, sw>>>(fr, e[0].o, e[0].d, e[0].st);
        launches++;
        uint32_t n = paths;                  // this wave's rays, or (ahead, depth > 0) at most that
        const uint32_t* n_dev = nullptr;     // ... and their count on the device
        int cur = 0;
        ext_rays += paths;
        for (int depth = 0; depth <= cfg->bounces && n > 0 && st == CBQ_OK; depth++, wave++) {
            const int slot = (int)(wave % cbq::kPtAhead);
            if (look && depth >= cbq::kPtAhead) {  // paths only end: no later wave has more rays
                if (!ok(cudaEventSynchronize(ws.shaded[slot]))) { fail(CBQ_ERR_CUDA); break; }
                n = std::min(n, ws.seen[slot]);
                if (n == 0) break;
            }
            Ext& E = e[cur];
            Ext& N = e[cur ^ 1];
            const int set = (int)(wave % (size_t)sets);
            Sha& S = s2[set];
            uint32_t* count = (uint32_t*)(counts + wave);                 // [0] shadow rays, [1] next extension rays
            uint64_t* work = counts + waves + 2 * wave;                   // extension and shadow work counters
            cbq_rays rays{(const float*)E.o, (const float*)E.d};
            cbq_hits hits{E.hit, nullptr, E.material, E.position, E.normal, nullptr, nullptr};
            const cbq_query* qe = depth == 0 ? &qcam : &qext;
            cbq_status ts = n_dev ? cbq::intersect_device_count(dag, &rays, n, n_dev, qe, &hits, work, (cbq_stream_t)sw)
                                  : cbq_intersect_persistent(dag, &rays, n, qe, &hits, work, 0u, (cbq_stream_t)sw);
            if (ts != CBQ_OK) { fail(ts); break; }
            launches++;
            if (on_wave) {
                if (!ok(cudaStreamSynchronize(s))) { fail(CBQ_ERR_CUDA); break; }
                on_wave(user, 0, depth, sample, (const float*)E.o, (const float*)E.d, n, &hits, qe);
            }
            if (ahead && set_used[set] && !ok(cudaStreamWaitEvent(sw, ws.traced[set], 0))) { fail(CBQ_ERR_CUDA); break; }
            const int last = depth == cfg->bounces;
            cbq_k_pt_shade<<<(n + 255) / 256, 256, 0, sw>>>(d_sh, n, n_dev, (uint32_t)depth, cfg->seed, last, E.st, E.hit,
                                                            E.material, E.position, E.normal, device_image, S.o, S.d,
                                                            S.w, (unsigned long long*)count, N.o, N.d, N.st,
                                                            look ? ws.seen + slot : nullptr);
            launches++;
            uint32_t ns = 2u * n, next = n;
            if (!ahead) {
                uint32_t h_counts[2] = {0, 0};
                if (!ok(cudaMemcpyAsync(h_counts, count, sizeof(h_counts), cudaMemcpyDeviceToHost, s)) ||
                    !ok(cudaStreamSynchronize(s))) {
                    fail(CBQ_ERR_CUDA);
                    break;
                }
                ns = h_counts[0];
                next = h_counts[1];
                shadow_rays += ns;
                ext_rays += next;
            } else if (!ok(cudaEventRecord(ws.shaded[slot], sw)) || !ok(cudaStreamWaitEvent(ss, ws.shaded[slot], 0))) {
                fail(CBQ_ERR_CUDA);
                break;
            }
            if (ns > 0) {
                cbq_rays srays{(const float*)S.o, (const float*)S.d};
                cbq_hits shits{S.hit, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
                ts = ahead ? cbq::intersect_device_count(dag, &srays, ns, count, &qsh, &shits, work + 1, (cbq_stream_t)ss)
                           : cbq_intersect_persistent(dag, &srays, ns, &qsh, &shits, work + 1, 0u, (cbq_stream_t)ss);
                if (ts != CBQ_OK) { fail(ts); break; }
                launches++;
                if (on_wave) {
                    if (!ok(cudaStreamSynchronize(s))) { fail(CBQ_ERR_CUDA); break; }
                    on_wave(user, 1, depth, sample, (const float*)S.o, (const float*)S.d, ns, &shits, &qsh);
                }
                cbq_k_pt_shadow_add<<<(ns + 255) / 256, 256, 0, ss>>>(ns, ahead ? count : nullptr, S.hit, S.w,
                                                                      device_image);
                launches++;
            }
            if (ahead) {
                if (!ok(cudaEventRecord(ws.traced[set], ss))) { fail(CBQ_ERR_CUDA); break; }
                set_used[set] = true;
                n_dev = count + 1;
            }
            n = next;
            cur ^= 1;
        }
    }
    if (ahead) {  // both streams' work ends before the caller's goes on, errors or not
        for (cudaStream_t q : {sw, ss})
            if (!ok(cudaEventRecord(ws.begin, q)) || !ok(cudaStreamWaitEvent(s, ws.begin, 0))) fail(CBQ_ERR_CUDA);
    }
    std::vector<uint64_t> h_counts;
    if (st == CBQ_OK) {
        const size_t cnt = npix * 3;
        cbq_k_pt_scale<<<(unsigned)((cnt + 255) / 256), 256, 0, s>>>(device_image, cnt,
                                                                     1.0f / (float)cfg->samples_per_pixel);
        launches++;
        if (ahead) {
            try {
                h_counts.resize(waves);
            } catch (const std::exception&) {  // nothing may throw across the C ABI
                fail(CBQ_ERR_OUT_OF_MEMORY);
            }
            if (st == CBQ_OK &&
                !ok(cudaMemcpyAsync(h_counts.data(), counts, waves * sizeof(uint64_t), cudaMemcpyDeviceToHost, s)))
                fail(CBQ_ERR_CUDA);
        }
    }
    // The workspace is this frame's until everything on it is done.
    if (!ok(cudaStreamSynchronize(s))) fail(CBQ_ERR_CUDA);
    if (ahead && st != CBQ_OK) {
        cudaStreamSynchronize(sw);
        cudaStreamSynchronize(ss);
        cudaGetLastError();
    }
    for (size_t w = 0; w < h_counts.size() && st == CBQ_OK; w++) {
        shadow_rays += (uint32_t)h_counts[w];
        ext_rays += h_counts[w] >> 32;
    }
    if (!lock.owns_lock()) cbq::pt_workspace_release(own);
    else keep_or_release(ws);
    if (stats) {
        stats->extension_rays = ext_rays;
        stats->shadow_rays = shadow_rays;
        stats->kernel_launches = launches;
        stats->milliseconds =
            std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_start).count();
    }
    return st;
}

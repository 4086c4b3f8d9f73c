// Flat ("while-while") form of the ESVO traversal for sm_103a.
//
// The reference's control flow (raytracing.cpp:397-478 around :213-371) is two
// nested loops with early exits: an octant walk, and inside it the ESVO
// descend/advance/pop loop.  Run per thread as written, the lanes of a warp
// leave those loops at different times and drift apart (measured: 1.8-2.8
// active lanes per instruction).  Here the traversal is a per-lane state
// machine driven by a single loop, and the warp reconverges at the top of every
// iteration.  Two walks take the ESVO steps: the ordered walk
// (lane_walk_ordered), for rays on which the reference's decisions follow from
// the order of the slab distances, and the reference's own steps (lane_walk)
// for all others.  In the persistent form, lanes whose ray is done pull new
// rays from a global counter (warp-aggregated).
//
// Floating-point operations are those of cbq_traverse.cuh / the reference, in
// the same order (compile with -fmad=false).  Child positions are carried as
// floats updated by exact float additions; the host only selects this form
// when every SubDAG's reflected coordinates lie within +-2^21, where
// (float)(a + b) == (float)a + (float)b and p + 1.5 * 2^23 is exact with a
// fixed exponent, so the integer bits the pop's XOR/MSB logic needs are the
// low bits of that sum's bit pattern (no float/int conversion).
#pragma once

#include "../../include/cubiquity_gb300.h"
#include "cbq_traverse.cuh"

namespace cbq {
namespace dev {

// Float positions p with |p| <= 2^21: the bit pattern of p + kPosBias is
// 0x4B400000 + p (two's complement), exactly, so its low 22 bits are p's.
constexpr float kPosBias = 12582912.0f;  // 1.5 * 2^23

// From kLaneMiss on: finished within a step batch (a miss; a hit at child
// `node` of the current child position; a miss that got stuck or reached the
// fetch cap), completed after it.
enum : uint32_t {
    kLaneIdle = 0u, kLaneEnter = 1u, kLaneNext = 2u, kLaneWalk = 3u,
    kLaneMiss = 4u, kLaneHit = 5u, kLaneStuck = 6u, kLaneLimit = 7u
};

// Two single-precision operations, each rounded, in one instruction.
__device__ __forceinline__ float2 add2(float2 a, float2 b)
{
    float2 r;
    asm("{ .reg .b64 x, y, z; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; add.rn.f32x2 z, x, y; mov.b64 {%0, %1}, z; }"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b)
{
    float2 r;
    asm("{ .reg .b64 x, y, z; mov.b64 x, {%2, %3}; mov.b64 y, {%4, %5}; mul.rn.f32x2 z, x, y; mov.b64 {%0, %1}, z; }"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}

// What a lane keeps of its ray and walk.  Registers decide how many warps an SM
// holds: the ray itself, the octant distances and a finished ray's results are
// read or computed again where they are needed (56 registers a thread, 36 warps
// an SM, instead of 64 and 32).  Held to 48 registers the walk spills and was
// slower (bounce rays 562 against 549 us, camera rays 362 against 345).
struct Lane {
    float rox, roy, roz;         // reflected origin
    float ix, iy, iz;            // 1 / |dir|
    uint32_t sign, oct, moves;   // octant (reflected) and how many octant transitions led to it
    // ESVO walk state
    uint32_t node, cid;          // ordered walk: `cid` is the child slot (child id ^ sign)
    int32_t cns;                 // child size (integer-position form)
    float fx, fy, fz, fcns;      // child position and size as exact floats (float-position form)
    int32_t px, py, pz;          // child position as wrapping i32 (integer-position form)
    int h;                       // height of `node`; ordered walk: its stack address
    uint32_t limit;              // size of the SubDAG
    float last_exit;             // ordered walk: the entry distance of the child cell
    uint32_t fetches, mode;      // ordered walk: `fetches` is an upper bound
    bool fast;                   // float positions: the ordered walk applies; integer positions: no slab
                                 // distance can be NaN or -0, so min/max need no NaN ordering
    uint32_t loads;              // node loads made (fetches minus skipped empty children)
    uint32_t job;                // batch kernel: index of the lane's job
    uint64_t ray;                // ray index within its job
    const uint32_t* nodes;       // batch kernel: the job's node store
};

// Where a lane's volume, rays and outputs are.  The lane functions below are
// templates over this "source" so that the single-volume kernel and the
// multi-volume batch kernel share the same arithmetic.  STORE is how
// they refer to nodes; COUNT_LOADS is the fetch-count pass (cbq_count_fetches),
// which writes per ray the node loads (child probes in the reference layout,
// fewer in the compact one) to fetch_out.  It is a separate instantiation, so
// the traversal kernels carry no counting code (measured: 1-2% faster).
template <Store STORE, bool COUNT_LOADS = false, bool INT_POS = false, bool LOD = false>
struct FlatCtxT {
    static constexpr Store kStore = STORE;
    // INT_POS: child positions as wrapping i32 converted to float where a slab
    // plane is needed (the reference's own arithmetic, any coordinates, 64-bit
    // node offsets); otherwise exact floats (coordinates within +-2^21, fewer
    // than 2^29 nodes).
    static constexpr bool kIntPos = INT_POS;
    // LOD: the query may stop at a footprint (max_footprint >= 0); without it
    // the ordered walk leaves the test out.
    static constexpr bool kLod = LOD;
    // The fetch-count pass takes the reference form only: the ordered walk does not count.
    static constexpr bool kOrdered = !COUNT_LOADS && !INT_POS;
    DagParams dag;
    QueryParams q;
    HitsOut out;
    const float4* __restrict__ orig;
    const float4* __restrict__ dir;
    uint32_t* __restrict__ fetch_out;

    __device__ __forceinline__ const QueryParams& query(const Lane&) const { return q; }
    __device__ __forceinline__ const uint32_t* nodes(const Lane&) const { return dag.nodes; }
    // Ray of work item g: g itself, or with an image width (q.image_width, a
    // multiple of 4 dividing the launch into whole 8-row bands) the pixel of
    // tile g / 32 (tiles of 4 x 8 pixels, a band's tiles left to right) at
    // place g % 32 (row-major in the tile): a bijection of [0, n).
    __device__ __forceinline__ uint64_t ray_slot(uint64_t g) const
    {
        const uint32_t w = q.image_width;
        if (w == 0u) return g;
        const uint32_t t = (uint32_t)(g >> 5), k = (uint32_t)g & 31u;
        const uint32_t per_band = w >> 2;
        const uint32_t band = t / per_band, col = t - band * per_band;
        return (uint64_t)(band * 8u + (k >> 2)) * w + col * 4u + (k & 3u);
    }
    __device__ __forceinline__ uint32_t occupied(const Lane&) const { return dag.occupied; }
    __device__ __forceinline__ const uint4* top(const Lane&) const { return dag.top; }
    __device__ __forceinline__ const SubDag& subdag(const Lane&, uint32_t k) const { return dag.sd[k]; }
    // A ray is read where its walk starts and again where it ends in a hit (flush_held), crosses
    // octants by the quotients or starts again; streaming loads (evict-first) leave L2 to the node
    // store, at up to 32 bytes of DRAM traffic for a hit's second read.
    __device__ __forceinline__ float4 ray_origin(const Lane&, uint64_t i) const { return __ldcs(orig + i); }
    __device__ __forceinline__ float4 ray_direction(const Lane&, uint64_t i) const { return __ldcs(dir + i); }
    __device__ __forceinline__ void write(const Lane& L, const RayResult& r) const
    {
        write_result(out, L.ray, r);
        if constexpr (COUNT_LOADS) fetch_out[L.ray] = STORE == Store::kCompact ? L.loads : L.fetches;
    }
};

__device__ __forceinline__ uint32_t first_child_f(const Lane& L, float entry, float fcx, float fcy, float fcz)
{
    const float mx = (fcx - L.rox) * L.ix;
    const float my = (fcy - L.roy) * L.iy;
    const float mz = (fcz - L.roz) * L.iz;
    uint32_t id = (mx < entry ? 1u : 0u) | (my < entry ? 2u : 0u) | (mz < entry ? 4u : 0u);
    if (entry <= 0.0f) {
        id |= (L.rox >= fcx ? 1u : 0u) | (L.roy >= fcy ? 2u : 0u) | (L.roz >= fcz ? 4u : 0u);
    }
    return id;
}

// The same with each axis's bit also returned as a predicate, for callers that
// move the child position by it (cheaper than unpacking the id again).
__device__ __forceinline__ uint32_t first_child_p(const Lane& L, float entry, float fcx, float fcy, float fcz,
                                                  bool& bx, bool& by, bool& bz)
{
    bx = ((fcx - L.rox) * L.ix) < entry;
    by = ((fcy - L.roy) * L.iy) < entry;
    bz = ((fcz - L.roz) * L.iz) < entry;
    if (entry <= 0.0f) {
        bx = bx || L.rox >= fcx;
        by = by || L.roy >= fcy;
        bz = bz || L.roz >= fcz;
    }
    return (uint32_t)bx | ((uint32_t)by << 1) | ((uint32_t)bz << 2);
}

// Rays of the ordered walk (lane_walk_ordered): reflected origin within
// +-2^21, every |dir| component within [2^-60, 2^60].  With planes that are
// integers within +-2^21 (float_positions_exact) the slab distances along one
// axis are then strictly increasing in the plane: the rounded differences of
// planes one apart stay at least 0.75 apart below 2^22, more than the
// rounding of the product can close, and a non-zero difference is at least
// 2^-25, so no product underflows or overflows.
constexpr float kOrderedOrigin = 2097152.0f;                                     // 2^21
constexpr float kOrderedDirMin = 8.673617379884035e-19f, kOrderedDirMax = 1.152921504606847e18f;  // 2^-60, 2^60

// Integer positions: the wider range in which only the rules of lane_begin and
// lane_next hold (the octants around the origin without divisions, min/max
// without NaN).  1 Mi rays on terrain-1024 moved to 2^30: camera 174 -> 162 us,
// bounce 200 -> 190.
constexpr float kIntOrigin = 4294967296.0f;  // 2^32

template <bool INT = false>
__device__ __forceinline__ bool ordered_axis(float rd, float ro)
{
    return rd >= kOrderedDirMin && rd <= kOrderedDirMax && fabsf(ro) <= (INT ? kIntOrigin : kOrderedOrigin);
}

// Rays parallel to one or two of the axes (a component of exactly 0) are
// ordered too where the origin lies on no plane of those axes (not an integer):
// there 1/|dir| is infinite, a plane behind the origin lies at -inf and one
// ahead at +inf, never NaN.  Such an axis never bounds a cell's distances,
// since the other axes' are finite, and of two halves the walk takes the one
// that holds the origin, as the reference does.  1 Mi rays on terrain-1024: an
// orthographic view along an axis 161 -> 92 us, bounce rays with one in sixteen
// parallel to a plane 221 -> 136.
constexpr uint32_t kParallelMoves = 16u;  // such a ray's mark in Lane::moves
__device__ __forceinline__ bool parallel_axis(float rd, float ro)
{
    return rd == 0.0f && truncf(ro) != ro && fabsf(ro) <= kOrderedOrigin;
}

// The walk over the octants around the origin (raytracing.cpp:424-434,
// :469-475).  A lane keeps only its octant and the transitions made: the
// distances are computed again where a transition is due, which most rays
// never need.
struct OctantWalk {
    float dx, dy, dz;  // distToOrigin
    uint32_t oct;
    __device__ __forceinline__ void begin(const Lane& L, float4 d)
    {
        oct = 0u;
        dx = (-L.rox) / fabsf(d.x);
        dy = (-L.roy) / fabsf(d.y);
        dz = (-L.roz) / fabsf(d.z);
        if (dx < 0.0f) { oct += 1u; dx = __fadd_rn(dx, FLT_MAX); }
        if (dy < 0.0f) { oct += 2u; dy = __fadd_rn(dy, FLT_MAX); }
        if (dz < 0.0f) { oct += 4u; dz = __fadd_rn(dz, FLT_MAX); }
    }
    // One transition; false where the octant stays the same (NaN distances).
    __device__ __forceinline__ bool next()
    {
        const float md = min3_ref(dx, dy, dz);
        const uint32_t before = oct;
        if (dx <= md) { oct += 1u; dx = __fadd_rn(dx, FLT_MAX); }
        if (dy <= md) { oct += 2u; dy = __fadd_rn(dy, FLT_MAX); }
        if (dz <= md) { oct += 4u; dz = __fadd_rn(dz, FLT_MAX); }
        return oct != before;
    }
};

// Per-ray set-up: intersectVolume up to the octant loop (raytracing.cpp:409-434).
// `ordered` false: by the reference form, whatever the ray.
// Returns the ray's direction.
template <typename Src>
__device__ __forceinline__ float4 lane_begin(Lane& L, const Src& c, uint64_t i, bool ordered = true)
{
    L.ray = i;
    const float4 o = c.ray_origin(L, i);
    const float4 d = c.ray_direction(L, i);
    const uint32_t sbx = d.x < 0.0f, sby = d.y < 0.0f, sbz = d.z < 0.0f;
    L.sign = sbx | (sby << 1) | (sbz << 2);
    const float sx = sbx ? -1.0f : 1.0f, sy = sby ? -1.0f : 1.0f, sz = sbz ? -1.0f : 1.0f;
    L.rox = __fmul_rn(__fadd_rn(o.x, 0.5f), sx);
    L.roy = __fmul_rn(__fadd_rn(o.y, 0.5f), sy);
    L.roz = __fmul_rn(__fadd_rn(o.z, 0.5f), sz);
    const float rdx = fabsf(d.x), rdy = fabsf(d.y), rdz = fabsf(d.z);
    // 1 / |dir|: the correctly rounded reciprocal, the same value as the IEEE division.
    L.ix = __frcp_rn(rdx);
    L.iy = __frcp_rn(rdy);
    L.iz = __frcp_rn(rdz);
    // Integer positions: the range in which a slab distance
    // (plane - o') * (1/|dir|) is never NaN, and never -0 (planes are floats of
    // integers, so plane - o' is +0 when they are equal, and a difference of at
    // least 2^-25 does not underflow): for such rays fminf/fmaxf give the bits of
    // the reference's std::min/std::max compositions.
    L.fast = (Src::kOrdered || Src::kIntPos) && ordered && ordered_axis<Src::kIntPos>(rdx, L.rox) &&
             ordered_axis<Src::kIntPos>(rdy, L.roy) && ordered_axis<Src::kIntPos>(rdz, L.roz);
    L.moves = 0u;
    if (Src::kOrdered && ordered && !L.fast) {
        const bool px = parallel_axis(rdx, L.rox), py = parallel_axis(rdy, L.roy), pz = parallel_axis(rdz, L.roz);
        L.fast = (px || ordered_axis(rdx, L.rox)) && (py || ordered_axis(rdy, L.roy)) &&
                 (pz || ordered_axis(rdz, L.roz)) && !(px && py && pz);
        L.moves = kParallelMoves;
    }
    // The octant of the origin: distToOrigin = -o' / |dir| below 0
    // (raytracing.cpp:424-434), which is o' > 0 for a ray within the range.
    if (L.fast) {
        L.oct = (L.rox > 0.0f ? 1u : 0u) | (L.roy > 0.0f ? 2u : 0u) | (L.roz > 0.0f ? 4u : 0u);
    } else {
        OctantWalk w;
        w.begin(L, d);
        L.oct = w.oct;
    }
    L.fetches = 0u;
    L.loads = 0u;
    L.mode = ((c.occupied(L) >> ((L.oct ^ L.sign) & 7u)) & 1u) ? kLaneEnter : kLaneNext;
    return d;
}

// Completes a finished ray with the reference's operations and frees the lane:
// the entry distance max3(childT0) (raytracing.cpp:270-271), the material
// (findNearestMaterial, :310) and the normal vec3(equal(tChildEntry, childT0))
// * -rayDirSign (:317-318), the position (:440).  The step loop only records
// how a ray ended; this runs after the step batch for all the warp's lanes
// that finished in it at once: finishes are spread over the steps, so
// completing each at once ran this code at a few active lanes.  Misses and
// hits share one pass over the result stores.  The ray is read again here:
// eight registers less through the walk.
template <typename Src>
__device__ __forceinline__ void flush_held(Lane& L, const Src& c)
{
    if (L.mode < kLaneMiss) return;
    RayResult r;
    r.hit = false;
    r.distance = 0.0f;
    r.material = 0u;
    r.px = r.py = r.pz = 0.0f;
    r.nx = r.ny = r.nz = 0.0f;
    r.status = L.mode == kLaneStuck ? kRayStuck : L.mode == kLaneLimit ? kRayIterLimit : kRayOk;
    if (L.mode == kLaneHit) {
        constexpr bool INT = Src::kIntPos;
        const float4 o = c.ray_origin(L, L.ray), d = c.ray_direction(L, L.ray);
        if (!INT && L.fast) {
            L.fx -= kPosBias;
            L.fy -= kPosBias;
            L.fz -= kPosBias;
        }
        const float c0x = ((INT ? (float)L.px : L.fx) - L.rox) * L.ix;
        const float c0y = ((INT ? (float)L.py : L.fy) - L.roy) * L.iy;
        const float c0z = ((INT ? (float)L.pz : L.fz) - L.roz) * L.iz;
        const float tce = max3_ref(c0x, c0y, c0z);
        uint32_t material = 0u;
        if (c.query(L).compute_surface)
            material = nearest_material<Src::kStore, INT>(c.nodes(L), L.node, L.sign, L.fetches, r.status, L.loads);
        if (r.status == kRayOk && !((c.query(L).flags & 1u) && !(tce <= o.w))) {
            r.hit = true;
            r.distance = tce;
            r.material = material;
            if (c.query(L).compute_surface) {
                r.nx = __fmul_rn(tce == c0x ? 1.0f : 0.0f, (L.sign & 1u) ? 1.0f : -1.0f);
                r.ny = __fmul_rn(tce == c0y ? 1.0f : 0.0f, (L.sign & 2u) ? 1.0f : -1.0f);
                r.nz = __fmul_rn(tce == c0z ? 1.0f : 0.0f, (L.sign & 4u) ? 1.0f : -1.0f);
            }
            r.px = __fadd_rn(o.x, __fmul_rn(d.x, tce));
            r.py = __fadd_rn(o.y, __fmul_rn(d.y, tce));
            r.pz = __fadd_rn(o.z, __fmul_rn(d.z, tce));
        }
    }
    c.write(L, r);
    L.mode = kLaneIdle;
}

// The SubDAGs (bits by octant index) of the octants a ray can still come to
// from octant `oct` (reflected): the octant walk only ever raises bits of it.
__device__ __forceinline__ uint32_t octants_ahead(uint32_t oct, uint32_t sign)
{
    uint32_t m = 0xffu;
    if (oct & 1u) m &= (sign & 1u) ? 0x55u : 0xaau;
    if (oct & 2u) m &= (sign & 2u) ? 0x33u : 0xccu;
    if (oct & 4u) m &= (sign & 4u) ? 0x0fu : 0xf0u;
    return m & ~(1u << (oct ^ sign));
}

// On to the next octant with a SubDAG (raytracing.cpp:469-475), or the end.
template <typename Src>
__device__ __forceinline__ void lane_next(Lane& L, const Src& c)
{
    const uint32_t occupied = c.occupied(L);
    // (A ray parallel to an axis takes the reference's own transitions: a distance of -inf
    // plus FLT_MAX stays -inf, and is crossed again.)
    if (L.fast && L.moves < kParallelMoves) {
        const uint32_t ahead = occupied & octants_ahead(L.oct, L.sign);
        if (ahead == 0u) {
            L.mode = kLaneMiss;
            return;
        }
        if ((ahead & (ahead - 1u)) == 0u) {
            // One octant with a SubDAG ahead.  The walk comes to it exactly when it crosses all
            // the planes between (`need`) before any other (`rest`).  Products with 1/|dir| are
            // within 2^-22 of the quotients that decide; only closer calls take the walk itself,
            // with its three divisions (camera rays 345 -> 334 us, spheres-256 72 -> 69.5).
            const uint32_t k = (31u - __clz(ahead)) ^ L.sign, need = k & ~L.oct, rest = ~k;
            const float tx = -L.rox * L.ix, ty = -L.roy * L.iy, tz = -L.roz * L.iz;
            const float last = fmaxf(fmaxf((need & 1u) ? tx : 0.0f, (need & 2u) ? ty : 0.0f), (need & 4u) ? tz : 0.0f);
            const float first = fminf(fminf((rest & 1u) ? tx : FLT_MAX, (rest & 2u) ? ty : FLT_MAX),
                                      (rest & 4u) ? tz : FLT_MAX);
            const float slack = first * 9.5367431640625e-07f;  // 2^-20
            if (last < first - slack) {
                L.oct = k;
                L.mode = kLaneEnter;
                return;
            }
            if (last > first + slack) {
                L.mode = kLaneMiss;
                return;
            }
        }
    }
    OctantWalk w;
    w.begin(L, c.ray_direction(L, L.ray));
    for (uint32_t k = 0; k < (L.moves & (kParallelMoves - 1u)); k++) w.next();
    do {
        if (!w.next()) {  // the reference would revisit this octant forever
            L.mode = kLaneStuck;
            return;
        }
        if (w.oct > 7u) {
            L.mode = kLaneMiss;
            return;
        }
        L.moves++;
    } while (((occupied >> (w.oct ^ L.sign)) & 1u) == 0u);
    L.oct = w.oct;
    L.mode = kLaneEnter;
}

// Whether a child exists, and the child (0 where it does not), in the ordered
// walk, whose references to plain nodes are word indices (node * 8).  Plain and
// tagged stores hold a 0 for an empty child, so it is loaded like any other: a
// test or a branch around the load costs more.
template <Store S>
__device__ __forceinline__ bool walk_occupied(const uint32_t* __restrict__ nodes, uint32_t ref, uint32_t slot)
{
    if constexpr (S == Store::kPlain)
        return __ldg(nodes + (ref | slot)) != 0u;
    else
        return ((ref >> slot) & 1u) != 0u;
}
template <Store S>
__device__ __forceinline__ uint32_t walk_child(const uint32_t* __restrict__ nodes, uint32_t ref, uint32_t slot)
{
    if constexpr (S == Store::kPlain) {
        return __ldg(nodes + (ref | slot));
    } else if constexpr (S == Store::kTagged) {
        uint32_t child;
        asm volatile("{ .reg .pred p; setp.ne.u32 p, %2, 0; mov.u32 %0, 0; @p ld.global.nc.u32 %0, [%1]; }"
                     : "=r"(child) : "l"(occupied_at<S>(nodes, ref, slot)), "r"((ref >> slot) & 1u));
        return child;
    } else {
        uint32_t child;
        asm volatile("{ .reg .pred p; setp.ne.u32 p, %2, 0; mov.u32 %0, 0; @p ld.global.nc.u32 %0, [%1]; }"
                     : "=r"(child) : "l"(occupied_at<S>(nodes, ref, slot)), "r"((ref >> slot) & 1u));
        return child;
    }
}

// An ordered ray enters SubDAG `s`, whose reflected corner is (px, py, pz) and
// whose size is ns.
//
// Origin inside (entry <= 0 < exit): descend to the cell that holds it here,
// with all of a refill's lanes in step.  Every cell on the way has entry <= 0 <
// tChildExit, so the first child is the one that holds the origin: its slot is a
// bit of each of the origin's voxel coordinates, and no distance is needed
// (terrain-4096 bounce rays make 8.1 of their 17.2 descents here; by distances
// and positions as in the walk the descent took a third more instructions:
// bounce rays 550 -> 536 us, 1.5 M shadow rays 134 -> 129, a path-traced frame
// 900 -> 878).  Origin outside: the slab test, and the first child by one
// compare per axis.
template <typename Src, typename Stack>
__device__ __forceinline__ void enter_ordered(Lane& L, const Src& c, Stack& stack, const SubDag& s, int32_t px,
                                              int32_t py, int32_t pz, uint32_t ns)
{
    constexpr Store S = Src::kStore;
    constexpr uint32_t kBiasBits = 0x4B400000u;  // of kPosBias
    const uint32_t mx = (uint32_t)(__float2int_rd(L.rox) - px), my = (uint32_t)(__float2int_rd(L.roy) - py),
                   mz = (uint32_t)(__float2int_rd(L.roz) - pz);
    L.node = S == Store::kPlain ? s.node * 8u : s.node;  // plain: the word index of its children
    // With LOD, a cell of size s that holds the origin has tChildExit <= s * min(1 / |dir|):
    // where that minimum is within footprint_tmax all of them are large.
    bool inside = (mx | my | mz) < ns && s.height > 0;
    if constexpr (Src::kLod) inside = inside && fminf(fminf(L.ix, L.iy), L.iz) <= c.query(L).footprint_tmax;
    if (inside) {
        const uint32_t* nodes = c.nodes(L);
        int l = s.height - 1;  // the cell's size is 1 << l
        uint32_t slot;
        L.h = (int)stack.at(s.height);
        stack.store((uint32_t)L.h, L.node);
        if (S != Store::kPlain && s.top != 0u) {
            // The first five levels at once, from the table: two loads instead of a
            // chain of five (bounce rays 536 -> 519 us, shadow rays 129 -> 124, the
            // compact store 152 -> 146).  Slots below the last node get the row's
            // empty entries: they are stored again before they are read.
            const uint32_t flip = ns - 1u;
            const int sh = s.height - kTopLevels;
            const uint32_t ux = (mx ^ ((L.sign & 1u) ? flip : 0u)) >> sh, uy = (my ^ ((L.sign & 2u) ? flip : 0u)) >> sh,
                           uz = (mz ^ ((L.sign & 4u) ? flip : 0u)) >> sh;
            const uint4* row = c.top(L) + 2u * ((s.top - 1u) * kTopCells + (ux | (uy << 5) | (uz << 10)));
            const uint4 a = __ldg(row), b = __ldg(row + 1);
            uint32_t at = stack.below((uint32_t)L.h);
            stack.store(at, a.x);
            stack.store(at = stack.below(at), a.y);
            stack.store(at = stack.below(at), a.z);
            stack.store(at = stack.below(at), a.w);
            stack.store(at = stack.below(at), b.x);
            if (b.y != 0u) L.node = b.z;
            l -= (int)b.y;
            L.h = (int)stack.at(l + 1);
        }
        for (;;) {
            const uint32_t m = 1u << l;
            slot = (((mx & m) + ((my & m) << 1) + ((mz & m) << 2)) >> l) ^ L.sign;
            if (!walk_occupied<S>(nodes, L.node, slot)) break;
            const uint32_t child = walk_child<S>(nodes, L.node, slot);
            if (child < kMaterialCount) break;  // fetched again by the walk
            L.node = S == Store::kPlain ? child * 8u : child;
            L.h = (int)stack.below((uint32_t)L.h);
            stack.store((uint32_t)L.h, L.node);
            l--;
        }
        const uint32_t keep = 0u - (1u << l);
        L.cid = slot;
        L.fcns = __uint_as_float((uint32_t)(127 + l) << 23);  // 2^l
        L.fx = __uint_as_float(kBiasBits + (uint32_t)px + (mx & keep));
        L.fy = __uint_as_float(kBiasBits + (uint32_t)py + (my & keep));
        L.fz = __uint_as_float(kBiasBits + (uint32_t)pz + (mz & keep));
        L.last_exit = 0.0f;  // an entry at or behind the origin
    } else {
        const float fpx = (float)px, fpy = (float)py, fpz = (float)pz, fns = (float)ns;
        const float entry = fmaxf(fmaxf((fpx - L.rox) * L.ix, (fpy - L.roy) * L.iy), (fpz - L.roz) * L.iz);
        const float exit_ = fminf(fminf(((fpx + fns) - L.rox) * L.ix, ((fpy + fns) - L.roy) * L.iy),
                                  ((fpz + fns) - L.roz) * L.iz);
        if (!(entry < exit_)) {
            L.mode = kLaneNext;
            return;
        }
        L.fcns = (float)(ns >> 1);
        const float te = fmaxf(entry, FLT_MIN);
        const float cx = fpx + L.fcns, cy = fpy + L.fcns, cz = fpz + L.fcns;
        const bool bx = (cx - L.rox) * L.ix < te, by = (cy - L.roy) * L.iy < te, bz = (cz - L.roz) * L.iz < te;
        L.cid = ((uint32_t)bx | ((uint32_t)by << 1) | ((uint32_t)bz << 2)) ^ L.sign;
        L.fx = (bx ? cx : fpx) + kPosBias;
        L.fy = (by ? cy : fpy) + kPosBias;
        L.fz = (bz ? cz : fpz) + kPosBias;
        L.last_exit = entry;
        L.h = (int)stack.at(s.height);
        if (s.height > 0) stack.store((uint32_t)L.h, L.node);
    }
    L.fetches += 64u;  // more than were made here
    L.mode = kLaneWalk;
}

// Enters the SubDAG of the current octant: the slab test and set-up at the top
// of intersectRayNodeESVO (raytracing.cpp:218-250, 443-460).
template <typename Src, typename Stack>
__device__ __forceinline__ void lane_enter(Lane& L, const Src& c, Stack& stack)
{
    const SubDag& s = c.subdag(L, L.oct ^ L.sign);
    if (s.node == 0u) {
        L.mode = kLaneNext;
        return;
    }
    const uint32_t sbx = L.sign & 1u, sby = (L.sign >> 1) & 1u, sbz = (L.sign >> 2) & 1u;
    const uint32_t ns = 1u << s.height;
    const int32_t px = (int32_t)((sbx ? 0u - (uint32_t)s.lx : (uint32_t)s.lx) - (sbx ? ns : 0u));
    const int32_t py = (int32_t)((sby ? 0u - (uint32_t)s.ly : (uint32_t)s.ly) - (sby ? ns : 0u));
    const int32_t pz = (int32_t)((sbz ? 0u - (uint32_t)s.lz : (uint32_t)s.lz) - (sbz ? ns : 0u));
    L.limit = ns;
    if constexpr (!Src::kIntPos) {
        if (L.fast) {
            enter_ordered(L, c, stack, s, px, py, pz, ns);
            return;
        }
    }
    const float fpx = (float)px, fpy = (float)py, fpz = (float)pz, fns = (float)ns;
    const float t0x = (fpx - L.rox) * L.ix;
    const float t0y = (fpy - L.roy) * L.iy;
    const float t0z = (fpz - L.roz) * L.iz;
    const float t1x = ((fpx + fns) - L.rox) * L.ix;
    const float t1y = ((fpy + fns) - L.roy) * L.iy;
    const float t1z = ((fpz + fns) - L.roz) * L.iz;
    const float entry = max3_ref(t0x, t0y, t0z);
    const float exit_ = min3_ref(t1x, t1y, t1z);
    if (!(entry < exit_)) {
        L.mode = kLaneNext;
        return;
    }
    L.node = s.node;
    L.mode = kLaneWalk;
    L.h = s.height;
    L.last_exit = exit_;
    if constexpr (Src::kIntPos) {
        L.cns = (int32_t)(ns >> 1);
        L.cid = first_child_f(L, entry, (float)wadd(px, L.cns), (float)wadd(py, L.cns), (float)wadd(pz, L.cns));
        L.px = wadd(px, (L.cid & 1u) ? L.cns : 0);
        L.py = wadd(py, (L.cid & 2u) ? L.cns : 0);
        L.pz = wadd(pz, (L.cid & 4u) ? L.cns : 0);
    } else {
        L.fcns = (float)(ns >> 1);
        L.cid = first_child_f(L, entry, fpx + L.fcns, fpy + L.fcns, fpz + L.fcns);
        L.fx = fpx + ((L.cid & 1u) ? L.fcns : 0.0f);
        L.fy = fpy + ((L.cid & 2u) ? L.fcns : 0.0f);
        L.fz = fpz + ((L.cid & 4u) ? L.fcns : 0.0f);
    }
    stack.clear(s.height);
}

// min3/max3 of slab distances: the reference's NaN-ordered forms, or (FAST,
// the lane's ray has Lane::fast) one fminf/fmaxf per pair, the same bits.
template <bool FAST>
__device__ __forceinline__ float slab_min3(float x, float y, float z)
{
    if constexpr (FAST) return fminf(fminf(x, y), z);
    else return min3_ref(x, y, z);
}
template <bool FAST>
__device__ __forceinline__ float slab_max3(float x, float y, float z)
{
    if constexpr (FAST) return fmaxf(fmaxf(x, y), z);
    else return max3_ref(x, y, z);
}

// The ordered walk: the ESVO loop (raytracing.cpp:253-367) for rays whose
// slab distances are strictly increasing along each axis (ordered_axis).  It
// takes the reference's decisions, cell by cell and fetch by fetch, with fewer
// operations:
//  - The entry distance E = max3(childT0) is carried (in last_exit) instead of
//    recomputed.  A descent at E > 0 keeps it: the entry axis's centre plane
//    lies beyond E, so its bit stays 0.  An advance makes it tChildExit, which
//    no entry distance of the child exceeds unless both are <= 0.
//  - findFirstChild is one compare per axis where E > 0.  Where E <= 0 < exit
//    the origin lies in the cell, and the first child is the one that holds it
//    (lane_enter).  Where both are <= 0 the SubDAG lies behind the origin; such
//    rays start again in the reference form at their first descent.
//  - A descent always stores its node.  The reference skips the store when
//    tChildExit equals the node's own exit; the child then shares the node's
//    exit plane, and a walk that leaves the child through it pops past the
//    node, so the slot is never read (after a pop it still holds the node).  No
//    slot is read before it is stored, so the stack needs no clearing.
//  - An advance inside a node is a pop to the node's own height: the stack
//    holds the current node too, so both are the same instructions.
//  - Positions stay biased by kPosBias (their bits are integers); the child
//    size is subtracted from the bias instead (sb), which is exact.
//  - max_footprint: see footprint_exit_max, one compare instead of a division
//    (which the compiler had moved out of its branch: 12 instructions a step).
//  - References carry their node's occupancy mask (Store), so that an empty
//    child costs no load: 18 loads per terrain-4096 bounce ray instead of 37
//    (bounce rays 592 -> 545 us; the compact store's 196 -> 156).  Loading empty
//    children too, without a test, was slower (575 us).
//  - Fetches are not counted: an upper bound decides when a ray may come near
//    the fetch cap.
//
// One iteration is an advance, if the child is empty, and then a descent, if
// the child reached is not.  Both sections run in nearly every iteration of an
// incoherent warp anyway, so one iteration takes a lane up to two steps for the
// price of one: 16.5 iterations per terrain-4096 bounce ray instead of 30.8
// steps.  The x and y planes are computed with packed instructions, and the
// axis bits move positions and form the child id through multiply-adds, off the
// integer pipe.  Bound by instruction issue (76% of issue slots, the ALU pipe
// 62%) and the latency of a dependent load (17 / 24 active lanes per
// instruction on incoherent / coherent rays).  4 Mi rays on terrain-4096, from
// the reference's steps: camera rays 607 -> 343 us, bounce rays 1,100 -> 545 us,
// and with enter_ordered's and lane_next's shortcuts 334 and 518 us.

// Up to `steps` iterations of a walking ordered lane.
template <typename Src, typename Stack>
__device__ __forceinline__ void lane_walk_ordered(Lane& L, const Src& c, Stack& stack, uint32_t steps)
{
    constexpr Store S = Src::kStore;
    // At most two fetches per iteration, and a hit's material within 512 more.
    // A ray that may come near the fetch cap starts again in the reference
    // form, which counts every fetch.
    L.fetches += 2u * steps;
    if (L.fetches + 512u >= kMaxFetches) {
        lane_begin(L, c, L.ray, false);
        return;
    }
    const float tmax1 = Src::kLod ? c.query(L).footprint_tmax : 0.0f;
    const float2 nro = make_float2(-L.rox, -L.roy), inv = make_float2(L.ix, L.iy);
    const uint32_t* nodes = c.nodes(L);
    float sb = L.fcns - kPosBias;
    uint32_t child;
    bool stopped;
    do {
        if (!walk_occupied<S>(nodes, L.node, L.cid)) {
            const float2 c1 = mul2(add2(add2(make_float2(L.fx, L.fy), make_float2(sb, sb)), nro), inv);
            const float c1z = ((L.fz + sb) - L.roz) * L.iz;
            const float tcx = fminf(fminf(c1.x, c1.y), c1z);
            L.last_exit = tcx;
            const float nx = __fmaf_rn(c1.x <= tcx ? 1.0f : 0.0f, L.fcns, L.fx);
            const float ny = __fmaf_rn(c1.y <= tcx ? 1.0f : 0.0f, L.fcns, L.fy);
            const float nz = __fmaf_rn(c1z <= tcx ? 1.0f : 0.0f, L.fcns, L.fz);
            const uint32_t cx = __float_as_uint(nx), cy = __float_as_uint(ny), cz = __float_as_uint(nz);
            const uint32_t diff = (cx ^ __float_as_uint(L.fx)) | (cy ^ __float_as_uint(L.fy)) |
                                  (cz ^ __float_as_uint(L.fz));
            const int msb = 31 - __clz(diff);
            const uint32_t m = 1u << msb;
            const uint32_t keep = 0u - m;
            L.cid = (((cx & m) + ((cy & m) << 1) + ((cz & m) << 2)) >> msb) ^ L.sign;
            L.h = (int)stack.at(msb + 1);
            // Outside the SubDAG: the empty node, and the loop's last iteration.
            const bool inside = diff < L.limit;
            L.node = stack.load_if((uint32_t)L.h, inside, 0u);
            if (!inside) steps = 1u;
            L.fcns = __uint_as_float((uint32_t)(127 + msb) << 23);  // 2^msb
            sb = L.fcns - kPosBias;
            L.fx = __uint_as_float(cx & keep);
            L.fy = __uint_as_float(cy & keep);
            L.fz = __uint_as_float(cz & keep);
        }
        // The value is opaque here, so that lanes that did not advance wait for
        // the others: the compiler otherwise sent them straight to their
        // descent, which then ran twice (1,086 instead of 960 us, bounce rays).
        // A loop whose condition the compiler can tell from `down` has the same
        // fault at its end (1,523 instead of 592 us): `steps` is all it tests.
        asm volatile("" : "+r"(L.node));
        child = walk_child<S>(nodes, L.node, L.cid);
        // hasLargeFootprint (raytracing.cpp:276).  Without LOD every child is
        // large whose exit is not behind the origin, which an entry beyond it
        // ensures.  Cells with an entry at or behind the origin are left to the
        // reference form (those that hold the origin were passed on entering).
        bool down = child >= kMaterialCount && L.last_exit > 0.0f;
        if constexpr (Src::kLod) {
            const float2 c1 = mul2(add2(add2(make_float2(L.fx, L.fy), make_float2(sb, sb)), nro), inv);
            const float tcx = fminf(fminf(c1.x, c1.y), ((L.fz + sb) - L.roz) * L.iz);
            down = down && tcx <= L.fcns * tmax1;
        }
        stopped = child != 0u && !down;
        if (down) {
            L.node = S == Store::kPlain ? child * 8u : child;
            L.h = (int)stack.below((uint32_t)L.h);
            stack.store((uint32_t)L.h, L.node);
            L.fcns *= 0.5f;
            sb = L.fcns - kPosBias;
            const float te = L.last_exit;
            const float2 mm = mul2(add2(add2(make_float2(L.fx, L.fy), make_float2(sb, sb)), nro), inv);
            const float mz = ((L.fz + sb) - L.roz) * L.iz;
            const float bx = mm.x < te ? 1.0f : 0.0f, by = mm.y < te ? 1.0f : 0.0f, bz = mz < te ? 1.0f : 0.0f;
            // The three bits as the low bits of a subnormal: 2^-149, 2^-148, 2^-147.
            L.cid = __float_as_uint(__fmaf_rn(bz, __uint_as_float(4u), __fmaf_rn(by, __uint_as_float(2u),
                                              bx * __uint_as_float(1u)))) ^ L.sign;
            L.fx = __fmaf_rn(bx, L.fcns, L.fx);
            L.fy = __fmaf_rn(by, L.fcns, L.fy);
            L.fz = __fmaf_rn(bz, L.fcns, L.fz);
        }
        steps = stopped ? 0u : steps - 1u;
    } while (steps != 0u);
    if (!stopped) {
        if (L.node == 0u) L.mode = kLaneNext;  // left the SubDAG
    } else if (child >= kMaterialCount && !(L.last_exit > 0.0f)) {
        lane_begin(L, c, L.ray, false);
    } else {
        L.node = child;  // a hit at this child
        L.mode = kLaneHit;
    }
}

// One iteration of the ESVO loop (raytracing.cpp:253-367).
template <bool FAST, typename Src, typename Stack>
__device__ __forceinline__ void lane_walk(Lane& L, const Src& c, Stack& stack)
{
    constexpr bool INT = Src::kIntPos;
    // Exit planes: vec3(childPos + childNodeSize) (raytracing.cpp:259-260).
    const float c1x = ((INT ? (float)wadd(L.px, L.cns) : L.fx + L.fcns) - L.rox) * L.ix;
    const float c1y = ((INT ? (float)wadd(L.py, L.cns) : L.fy + L.fcns) - L.roy) * L.iy;
    const float c1z = ((INT ? (float)wadd(L.pz, L.cns) : L.fz + L.fcns) - L.roz) * L.iz;
    const float tcx = slab_min3<FAST>(c1x, c1y, c1z);
    const uint32_t child = child_of<Src::kStore, INT>(c.nodes(L), L.node, L.cid ^ L.sign, L.loads);
    L.fetches++;
    if (child > 0u) {
        if (child >= kMaterialCount && large_footprint(INT ? (float)L.cns : L.fcns, tcx, c.query(L).max_footprint)) {
            const float c0x = ((INT ? (float)L.px : L.fx) - L.rox) * L.ix;
            const float c0y = ((INT ? (float)L.py : L.fy) - L.roy) * L.iy;
            const float c0z = ((INT ? (float)L.pz : L.fz) - L.roz) * L.iz;
            const float tce = slab_max3<FAST>(c0x, c0y, c0z);
            if (tcx < L.last_exit) stack.put(L.h, L.node);
            L.last_exit = tcx;
            L.h--;
            L.node = child;
            if constexpr (INT) {
                L.cns >>= 1;
                L.cid = first_child_f(L, tce, (float)wadd(L.px, L.cns), (float)wadd(L.py, L.cns),
                                      (float)wadd(L.pz, L.cns));
                if (L.cid & 1u) L.px = wadd(L.px, L.cns);
                if (L.cid & 2u) L.py = wadd(L.py, L.cns);
                if (L.cid & 4u) L.pz = wadd(L.pz, L.cns);
            } else {
                L.fcns *= 0.5f;
                const float mcx = L.fx + L.fcns, mcy = L.fy + L.fcns, mcz = L.fz + L.fcns;
                bool bx, by, bz;
                L.cid = first_child_p(L, tce, mcx, mcy, mcz, bx, by, bz);
                L.fx = bx ? mcx : L.fx;
                L.fy = by ? mcy : L.fy;
                L.fz = bz ? mcz : L.fz;
            }
        } else {  // a hit at this child: completed by flush_held
            L.node = child;
            L.mode = kLaneHit;
        }
        return;
    }
    const bool ax = c1x <= tcx, ay = c1y <= tcx, az = c1z <= tcx;
    const uint32_t flips = (uint32_t)ax | ((uint32_t)ay << 1) | ((uint32_t)az << 2);
    // With slab distances that cannot be NaN (FAST), tcx is one of the three
    // and that axis flips: only the reference's form can get stuck here.
    if (!FAST && !(ax || ay || az)) {
        L.mode = kLaneStuck;
        return;
    }
    L.cid ^= flips;
    float ofx = 0.0f, ofy = 0.0f, ofz = 0.0f;  // float positions before the advance
    if constexpr (INT) {
        if (ax) L.px = wadd(L.px, L.cns);
        if (ay) L.py = wadd(L.py, L.cns);
        if (az) L.pz = wadd(L.pz, L.cns);
    } else {
        ofx = L.fx;
        ofy = L.fy;
        ofz = L.fz;
        if (ax) L.fx += L.fcns;
        if (ay) L.fy += L.fcns;
        if (az) L.fz += L.fcns;
    }
    if ((L.cid & flips) != flips) {
        // The pop (raytracing.cpp:339-361) on integer positions: the wrapping
        // i32 ones, or the biased bit patterns of the float ones, whose low 22
        // bits are the integer's.  The highest differing bit is the same in
        // both below bit 21; at bit 21 or above (a sign change included) both
        // leave the SubDAG, whose height is at most 21.
        const uint32_t cx = INT ? (uint32_t)L.px : __float_as_uint(L.fx + kPosBias);
        const uint32_t cy = INT ? (uint32_t)L.py : __float_as_uint(L.fy + kPosBias);
        const uint32_t cz = INT ? (uint32_t)L.pz : __float_as_uint(L.fz + kPosBias);
        uint32_t diff;
        if constexpr (INT) {  // on a flipped axis the position before the advance was p - childSize
            const uint32_t cs = (uint32_t)L.cns;
            diff = (ax ? (cx ^ (cx - cs)) : 0u) | (ay ? (cy ^ (cy - cs)) : 0u) | (az ? (cz ^ (cz - cs)) : 0u);
        } else {  // before against after: an axis that did not move gives 0
            diff = (cx ^ __float_as_uint(ofx + kPosBias)) | (cy ^ __float_as_uint(ofy + kPosBias)) |
                   (cz ^ __float_as_uint(ofz + kPosBias));
        }
        const int msb = 31 - __clz(diff);
        if (diff >= L.limit) {  // left the sub-DAG: on to the next octant
            L.mode = kLaneNext;
            return;
        }
        L.h = msb + 1;
        L.node = stack.get(L.h);
        const uint32_t m = 1u << msb;
        const uint32_t keep = 0u - m;
        if constexpr (INT) {
            L.cid = ((cx >> msb) & 1u) | (((cy >> msb) & 1u) << 1) | (((cz >> msb) & 1u) << 2);
            L.px = (int32_t)(cx & keep);
            L.py = (int32_t)(cy & keep);
            L.pz = (int32_t)(cz & keep);
            L.cns = (int32_t)m;
        } else {
            // Bit msb (< 21) of each axis, gathered at msb..msb+2, then shifted down.
            L.cid = ((cx & m) + ((cy & m) << 1) + ((cz & m) << 2)) >> msb;
            L.fcns = __uint_as_float((uint32_t)(127 + msb) << 23);  // 2^msb
            L.fx = __uint_as_float(cx & keep) - kPosBias;
            L.fy = __uint_as_float(cy & keep) - kPosBias;
            L.fz = __uint_as_float(cz & keep) - kPosBias;
        }
        L.last_exit = 0.0f;
    }
}

// Up to `steps` ESVO steps.  The reference ends a ray when a step starts with
// the fetch budget spent (raytracing.cpp:253 with the cap): the steps here are
// bounded by the budget left, and a lane still walking with the budget spent
// ends exactly as that next step would have ended it.
template <bool FAST, typename Src, typename Stack>
__device__ __forceinline__ void lane_walk_steps(Lane& L, const Src& c, Stack& stack, uint32_t steps)
{
    if (L.mode != kLaneWalk) return;
    const uint32_t budget = kMaxFetches - L.fetches;  // > 0: a walking lane is below the cap
    // Every step makes one fetch, so the fetch count doubles as the step counter.
    const uint32_t end = L.fetches + (steps < budget ? steps : budget);
    while (L.fetches < end && L.mode == kLaneWalk) lane_walk<FAST>(L, c, stack);
    if (L.mode == kLaneWalk && L.fetches >= kMaxFetches) L.mode = kLaneLimit;
}

// Steps of the reference form between a warp's checks, at least: an incoherent
// warp's eight iterations are made for the ordered walk, whose iteration takes up
// to two steps.  With eight, 1 Mi incoherent rays from 2^24 voxels away 329 us,
// with sixteen 323.
constexpr uint32_t kReferenceSteps = 16u;

// The walk of a whole warp (all 32 lanes must call it), then the results of
// the rays that finished in it are written.  Float positions: ordered lanes walk
// until `idle_min` of the warp's lanes do not (checked every `steps`
// iterations), the others take up to `steps` steps of the reference form, or
// kReferenceSteps.
// Integer positions: the FAST min/max when every walking lane's ray allows it.
template <typename Src, typename Stack>
__device__ __forceinline__ void warp_walk_steps(Lane& L, const Src& c, Stack& stack, uint32_t steps,
                                                uint32_t idle_min)
{
    if constexpr (Src::kIntPos) {
        if (__all_sync(0xffffffffu, L.mode != kLaneWalk || L.fast))
            lane_walk_steps<true>(L, c, stack, steps);
        else
            lane_walk_steps<false>(L, c, stack, steps);
    } else {
        for (;;) {
            if (L.mode == kLaneWalk && L.fast) lane_walk_ordered(L, c, stack, steps);
            const uint32_t walking = __ballot_sync(0xffffffffu, L.mode == kLaneWalk && L.fast);
            if (walking == 0u || 32u - __popc(walking) >= idle_min) break;
        }
        if (L.mode == kLaneWalk && !L.fast)
            lane_walk_steps<false>(L, c, stack, steps < kReferenceSteps ? kReferenceSteps : steps);
        __syncwarp();
        if (L.mode == kLaneNext) lane_next(L, c);
    }
    flush_held(L, c);
}

// When a persistent warp refills: once `idle_min` lanes are idle, checked every
// `steps` walk iterations.  A warp of coherent rays keeps its lanes in step
// longest when nearly all of them start together, while one of incoherent rays
// loses more to idle lanes than a refill costs.  So without a shape from the
// caller (refill_min 0) each refill looks at its rays' directions: within a
// quarter of their size of the first one's, the warp waits for 24 idle lanes
// and checks every 32 iterations, else for 16 and every 8.  Both ways, us:
// terrain-4096 camera rays 331 / 365, bounce rays 569 / 545 (camera rays checked
// every 16 iterations 333).  Equal directions (sun rays from scattered surfaces)
// tell less: every 16 (1.5 M shadow rays of a frame in its pixels' order 136, every
// 32 138; the same rays shuffled 165 / 178).  The batch and
// server launches keep 16 and 8: their small volumes' camera rays gain nothing
// from waiting (12 volumes: 240 us, chosen by the rays 245).
struct WarpRefill {
    uint32_t idle_min, steps;
    bool automatic;
    __device__ __forceinline__ WarpRefill(uint32_t refill_min, uint32_t steps_)
        : idle_min(refill_min ? refill_min : 16u), steps(refill_min ? steps_ : 8u), automatic(refill_min == 0u)
    {
    }
    // After a refill (all 32 lanes call it): `fresh` lanes started rays of direction d.
    __device__ __forceinline__ void look(bool fresh, float4 d)
    {
        if (!automatic) return;
        const uint32_t mask = __ballot_sync(0xffffffffu, fresh);
        const int first = __ffs(mask) - 1;  // (of -1, lane 31: no lane is fresh, the vote holds)
        const float x = __shfl_sync(0xffffffffu, d.x, first), y = __shfl_sync(0xffffffffu, d.y, first),
                    z = __shfl_sync(0xffffffffu, d.z, first);
        const float near = 0.25f * fmaxf(fmaxf(fabsf(x), fabsf(y)), fabsf(z));
        const float off = fmaxf(fmaxf(fabsf(d.x - x), fabsf(d.y - y)), fabsf(d.z - z));
        const bool coherent = __all_sync(0xffffffffu, !fresh || off <= near);
        const bool beam = !__any_sync(0xffffffffu, fresh && off > 0.0f);
        idle_min = coherent ? 24u : 16u;
        steps = !coherent ? 8u : beam ? 16u : 32u;
    }
};

// Octant transitions until the lane walks a SubDAG or has finished.  Bounded:
// every kLaneNext raises `oct` (or finishes the ray), every kLaneEnter walks or
// moves on, so at most 16 transitions happen.
template <typename Src, typename Stack>
__device__ __forceinline__ void lane_settle(Lane& L, const Src& c, Stack& stack)
{
    while (L.mode == kLaneEnter || L.mode == kLaneNext) {
        if (L.mode == kLaneNext) lane_next(L, c);
        if (L.mode == kLaneEnter) lane_enter(L, c, stack);
    }
}

}  // namespace dev

// Launch shape of the single-volume flat kernel.
struct FlatLaunch {
    bool persistent = false;
    uint64_t* counter = nullptr;     // persistent: work counter (zeroed by the launch)
    bool counter_zeroed = false;     // ... unless it is already zero, in stream order
    int block = 64;
    uint32_t refill_min = 8;
    bool local_stack = false;        // descent stack in local memory instead of shared
    const uint32_t* perm = nullptr;  // octant-sorted order (from launch_octant_sort), or null
    uint32_t steps = 1;              // ESVO steps per outer loop iteration
    uint32_t warp_rays = 32;         // plain form: rays per warp
    // Counted launches (always persistent, shared stack, in order): the device's ray count, at
    // most the launch's n; the work counter is already zero, in stream order.
    const uint32_t* n_dev = nullptr;
};

// Rays per warp of a launch that the chip holds at once, 0 for a larger one.
// A warp runs an iteration's advance and descent for any of its lanes, and a
// small launch leaves most warp slots empty, so its rays are spread over all of
// them: the call takes as long as its slowest ray, and a ray that shares its
// warp with fewer others gets through its iterations sooner.  No work counter,
// no atomics.  us per call, refilled from a counter / spread: 1,000 collision
// rays 28.7 / 21.0, 12,000 33.4 / 28.4, 150,000 camera rays 37.7 / 32.1; one ray
// per lane is reached at 32 rays a warp, where the two are alike (150,000
// collision rays 46.6 / 43.4).  The server's launches run beside each other and
// are not spread.
constexpr int kSpreadWarpsPerSm = 32;
uint32_t spread_warp_rays(uint64_t n, int device);

}  // namespace cbq

struct cbq_dag;
namespace cbq {
cbq_status launch_flat(const cbq_dag* dag, const dev::DagParams& dp, const dev::QueryParams& q,
                       const dev::HitsOut& out, const float4* orig, const float4* dir, uint64_t n,
                       uint32_t* fetch_out, const FlatLaunch& fl, cudaStream_t stream);
// Groups ray indices by octant (direction sign bits) into perm[n]; counts16 is
// 16 uint32 of scratch (zeroed here).
cbq_status launch_octant_sort(const float4* dir, uint64_t n, uint32_t* counts16, uint32_t* perm, int device,
                              cudaStream_t stream);
bool float_positions_exact(const cbq_dag* dag);
// Loads every flat traversal kernel that cbq_intersect_host_noalloc can launch
// (persistent, or spread where the launch is small) on the current device.
cbq_status preload_persistent_kernels();
}  // namespace cbq

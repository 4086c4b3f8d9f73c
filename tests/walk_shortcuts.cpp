// Plain C++ restatement of two shortcuts of the ordered walk, each against the
// reference's own arithmetic:
//   octants: which SubDAG a ray comes to next, from signs and products with
//            1/|dir|, against the distances and transitions of raytracing.cpp:424-475
//   descent: the cell that holds an origin inside a SubDAG, from the bits of its
//            voxel coordinates, against findFirstChild's slab distances (:178-196)
// Both return the number of disagreements.  Compile with -ffp-contract=off.
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdint>

namespace {

struct Walk {  // the reference's octant walk, reflected
    float d[3];
    uint32_t oct = 0;
    Walk(const float* ro, const float* dir)
    {
        for (int a = 0; a < 3; a++) {
            d[a] = -ro[a] / std::fabs(dir[a]);
            if (d[a] < 0.0f) { oct += 1u << a; d[a] += FLT_MAX; }
        }
    }
    void next()
    {
        const float first = std::min(std::min(d[0], d[1]), d[2]);
        for (int a = 0; a < 3; a++)
            if (d[a] <= first) { oct += 1u << a; d[a] += FLT_MAX; }
    }
};

uint32_t ahead(uint32_t oct, uint32_t sign)
{
    uint32_t m = 0xffu;
    if (oct & 1u) m &= (sign & 1u) ? 0x55u : 0xaau;
    if (oct & 2u) m &= (sign & 2u) ? 0x33u : 0xccu;
    if (oct & 4u) m &= (sign & 4u) ? 0x0fu : 0xf0u;
    return m & ~(1u << (oct ^ sign));
}

// The next octant (reflected) with a SubDAG, 8 for none, 9 where only the walk can tell.
uint32_t shortcut(uint32_t oct, uint32_t sign, uint32_t occupied, const float* ro, const float* inv)
{
    const uint32_t m = occupied & ahead(oct, sign);
    if (m == 0u) return 8u;
    if (m & (m - 1u)) return 9u;
    uint32_t bit = 0;
    while (!((m >> bit) & 1u)) bit++;
    const uint32_t k = bit ^ sign, need = k & ~oct, rest = ~k;
    float last = 0.0f, first = FLT_MAX;
    for (int a = 0; a < 3; a++) {
        const float t = -ro[a] * inv[a];
        last = std::fmax(last, (need >> a) & 1u ? t : 0.0f);
        first = std::fmin(first, (rest >> a) & 1u ? t : FLT_MAX);
    }
    const float slack = first * 9.5367431640625e-07f;
    if (last < first - slack) return k;
    if (last > first + slack) return 8u;
    return 9u;
}

void reflect(const float* o, const float* dir, float* ro, float* inv, uint32_t& sign)
{
    sign = 0;
    for (int a = 0; a < 3; a++) {
        const bool neg = dir[a] < 0.0f;
        sign |= neg ? 1u << a : 0u;
        ro[a] = (o[a] + 0.5f) * (neg ? -1.0f : 1.0f);
        inv[a] = 1.0f / std::fabs(dir[a]);
    }
}

}  // namespace

// o, dir: n times three floats.  `decided` counts the calls that took no division.
extern "C" uint64_t octants_differ(uint64_t n, const float* o, const float* dir, uint64_t* decided)
{
    uint64_t bad = 0;
    *decided = 0;
    for (uint64_t i = 0; i < n; i++) {
        float ro[3], inv[3];
        uint32_t sign;
        reflect(o + 3 * i, dir + 3 * i, ro, inv, sign);
        const uint32_t start = (ro[0] > 0.0f ? 1u : 0u) | (ro[1] > 0.0f ? 2u : 0u) | (ro[2] > 0.0f ? 4u : 0u);
        if (Walk(ro, dir + 3 * i).oct != start) { bad++; continue; }
        for (uint32_t occupied = 0; occupied < 256u; occupied++) {
            // From every octant with a SubDAG that the walk comes to (and from the first).
            Walk w(ro, dir + 3 * i);
            while (w.oct <= 7u) {
                const uint32_t from = w.oct;
                do w.next(); while (w.oct <= 7u && !((occupied >> (w.oct ^ sign)) & 1u));
                const uint32_t got = shortcut(from, sign, occupied, ro, inv);
                if (got != 9u) {
                    ++*decided;
                    bad += got != (w.oct <= 7u ? w.oct : 8u);
                }
            }
        }
    }
    return bad;
}

// Origins inside the box of size 2^height whose reflected corner is `corner`, all levels down.
extern "C" uint64_t descents_differ(uint64_t n, const float* o, const float* dir, const int32_t* low, int height)
{
    uint64_t bad = 0;
    for (uint64_t i = 0; i < n; i++) {
        float ro[3], inv[3], at[3];
        uint32_t sign, v[3];
        reflect(o + 3 * i, dir + 3 * i, ro, inv, sign);
        const int32_t size = 1 << height;
        bool inside = true;
        for (int a = 0; a < 3; a++) {
            const int32_t p = (sign >> a) & 1u ? -low[a] - size : low[a];
            at[a] = (float)p;
            v[a] = (uint32_t)((int32_t)std::floor(ro[a]) - p);
            inside = inside && v[a] < (uint32_t)size;
        }
        float entry = -FLT_MAX, exit_ = FLT_MAX;
        for (int a = 0; a < 3; a++) {
            entry = std::fmax(entry, (at[a] - ro[a]) * inv[a]);
            exit_ = std::fmin(exit_, ((at[a] + (float)size) - ro[a]) * inv[a]);
        }
        if (inside != (entry <= 0.0f && 0.0f < exit_)) { bad++; continue; }
        if (!inside) continue;
        for (int l = height - 1; l >= 0; l--) {
            const float half = (float)(1 << l);
            float e = (at[0] - ro[0]) * inv[0];
            e = std::max(std::max(e, (at[1] - ro[1]) * inv[1]), (at[2] - ro[2]) * inv[2]);
            uint32_t want = 0, got = 0;
            for (int a = 0; a < 3; a++) {
                const float mid = at[a] + half;
                want |= (mid - ro[a]) * inv[a] < e || (e <= 0.0f && ro[a] >= mid) ? 1u << a : 0u;
                got |= ((v[a] >> l) & 1u) << a;
            }
            if (got != want) { bad++; break; }
            float t_exit = FLT_MAX;
            for (int a = 0; a < 3; a++) {
                at[a] += (got >> a) & 1u ? half : 0.0f;
                t_exit = std::fmin(t_exit, ((at[a] + half) - ro[a]) * inv[a]);
            }
            if (!(t_exit > 0.0f)) { bad++; break; }  // every cell on the way is left ahead of the origin
        }
    }
    return bad;
}

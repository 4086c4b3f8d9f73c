// Plain C++ restatement of the ordered walk's rules (the flat kernels' walk for
// rays with strictly increasing slab distances), without the reference's
// per-step forms: the entry distance is carried, findFirstChild is one compare
// per axis, every descent stores its node, positions are biased floats, the
// footprint test is a compare with a precomputed exit.  Compared with the
// oracle by test_ordered_walk.py.  Compile with -ffp-contract=off.
#include <cfloat>
#include <cmath>
#include <cstdint>
#include <cstring>

namespace {

constexpr float kBias = 12582912.0f;
constexpr uint32_t kCap = 1u << 17;

struct Sub {
    int32_t lo[3];
    int32_t height;
    uint32_t pad0, node, pad1, pad2;
};

uint32_t bits(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }
float flt(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }

struct Result { int hit; float distance; uint32_t node, fetches; int status; };  // status 3: handed over

Result trace(const uint32_t* nodes, const Sub* subs, const float* o4, const float* d4, float mf, float tmax1)
{
    Result r{0, 0.0f, 0u, 0u, 0};
    float ro[3], iv[3], dd[3];
    uint32_t sign = 0, oct = 0;
    for (int a = 0; a < 3; a++) {
        const bool neg = d4[a] < 0.0f;
        sign |= neg ? 1u << a : 0u;
        ro[a] = (o4[a] + 0.5f) * (neg ? -1.0f : 1.0f);
        iv[a] = 1.0f / std::fabs(d4[a]);
        oct |= ro[a] > 0.0f ? 1u << a : 0u;
    }
    uint32_t start = 0;
    for (int a = 0; a < 3; a++) {
        dd[a] = -ro[a] / std::fabs(d4[a]);
        if (dd[a] < 0.0f) { start += 1u << a; dd[a] += FLT_MAX; }
    }
    if (start != oct) { r.status = 9; return r; }  // the origin's octant from the sign of o' alone
    for (; oct <= 7u;) {
        const Sub& s = subs[oct ^ sign];
        bool entered = false;
        float x[3], t0[3], t1[3], size = 0.0f, entry = 0.0f, exit_ = 0.0f;
        const float ns = (float)(1u << s.height);
        if (s.node != 0u) {
            for (int a = 0; a < 3; a++) {
                const bool neg = (sign >> a) & 1u;
                const float p = neg ? -(float)s.lo[a] - ns : (float)s.lo[a];
                x[a] = p;
                t0[a] = (p - ro[a]) * iv[a];
                t1[a] = ((p + ns) - ro[a]) * iv[a];
            }
            entry = std::fmax(std::fmax(t0[0], t0[1]), t0[2]);
            exit_ = std::fmin(std::fmin(t1[0], t1[1]), t1[2]);
            entered = entry < exit_;
        }
        if (entered) {
            uint32_t stack[33], limit = 1u << s.height, node = s.node, cid = 0;
            int h = s.height;
            for (uint32_t& v : stack) v = 0xffffffffu;  // a slot read before it is stored: out of range, found below
            stack[h] = node;
            float te = std::fmax(entry, FLT_MIN);
            size = (float)(limit >> 1);
            for (int a = 0; a < 3; a++) {
                const bool b = ((x[a] + size) - ro[a]) * iv[a] < te;
                cid |= b ? 1u << a : 0u;
                x[a] = x[a] + kBias + (b ? size : 0.0f);
            }
            for (;;) {
                if (r.fetches + 2 > kCap) { r.status = 3; return r; }
                float c1[3], tc;
                const float sb = size - kBias;
                for (int a = 0; a < 3; a++) c1[a] = ((x[a] + sb) - ro[a]) * iv[a];
                tc = std::fmin(std::fmin(c1[0], c1[1]), c1[2]);
                const uint32_t child = nodes[8ull * node + (cid ^ sign)];
                r.fetches++;
                if (child == 0u) {
                    uint32_t n[3], diff = 0;
                    for (int a = 0; a < 3; a++) {
                        n[a] = bits(c1[a] <= tc ? x[a] + size : x[a]);
                        diff |= n[a] ^ bits(x[a]);
                    }
                    if (diff >= limit) break;
                    te = std::fmax(tc, FLT_MIN);
                    const int msb = 31 - __builtin_clz(diff);
                    h = msb + 1;
                    node = stack[h];
                    if (node == 0xffffffffu) { r.status = 8; return r; }
                    size = (float)(1u << msb);
                    cid = 0;
                    for (int a = 0; a < 3; a++) {
                        cid |= ((n[a] >> msb) & 1u) << a;
                        x[a] = flt(n[a] & (0u - (1u << msb)));
                    }
                    continue;
                }
                const bool large = tc >= 0.0f && tc <= size * tmax1;
                if (child >= 256u && !large && tc < 0.0f && mf < 0.0f) { r.status = 3; return r; }
                if (child < 256u || !large) {
                    float c0[3];
                    for (int a = 0; a < 3; a++) c0[a] = ((x[a] - kBias) - ro[a]) * iv[a];
                    r.hit = 1;
                    r.distance = std::fmax(std::fmax(c0[0], c0[1]), c0[2]);
                    r.node = child;
                    return r;
                }
                node = child;
                stack[--h] = node;
                size *= 0.5f;
                cid = 0;
                for (int a = 0; a < 3; a++) {
                    const bool b = ((x[a] + (size - kBias)) - ro[a]) * iv[a] < te;
                    cid |= b ? 1u << a : 0u;
                    if (b) x[a] += size;
                }
            }
        }
        const float md = std::fmin(std::fmin(dd[0], dd[1]), dd[2]);
        for (int a = 0; a < 3; a++)
            if (dd[a] <= md) { oct += 1u << a; dd[a] += FLT_MAX; }
    }
    return r;
}

}  // namespace

extern "C" void ordered_trace(const uint32_t* nodes, const void* subs, const float* o4, const float* d4, uint64_t n,
                              float mf, float tmax1, uint8_t* hit, float* distance, uint32_t* node,
                              uint32_t* fetches, uint8_t* status)
{
    for (uint64_t i = 0; i < n; i++) {
        const Result r = trace(nodes, (const Sub*)subs, o4 + 4 * i, d4 + 4 * i, mf, tmax1);
        hit[i] = (uint8_t)r.hit;
        distance[i] = r.distance;
        node[i] = r.node;
        fetches[i] = r.fetches;
        status[i] = (uint8_t)r.status;
    }
}

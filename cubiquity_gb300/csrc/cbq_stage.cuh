// Copies between page-locked host buffers and device staging by kernels: rays
// in, hit fields out (the request server and cbq_intersect_host).
//
// The copy engine takes one call of 2-5 us on the launching thread, and a few us
// of the stream's time, per array: two for the rays and up to seven for the hit
// fields of every request or chunk.  One kernel each way does them all.  They
// are bound by the host link; 16-byte accesses by whole warps on the host side,
// so that the link carries full lines.
#pragma once

#include "cbq_hostmem.hpp"

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

namespace cbq {

struct StageIn {
    const float4 *o, *d;   // host rays, 16-byte aligned
    float4 *dst_o, *dst_d;
    uint64_t count;
    uint64_t pad;
};
struct StageOut {
    const char* src;       // device, any alignment
    char* dst;             // host, any alignment
    uint64_t bytes;
};
constexpr int kStageBlock = 256;
constexpr int kHitFields = 7;

namespace dev {

// The rays of `s`, items `first`, `first + stride`, ...
__device__ __forceinline__ void stage_in(const StageIn& s, uint64_t first, uint64_t stride)
{
    for (uint64_t i = first; i < s.count; i += stride) {
        const float4 o = __ldcs(s.o + i), d = __ldcs(s.d + i);
        s.dst_o[i] = o;
        s.dst_d[i] = d;
    }
}

// The bytes of `s`: 16-byte stores to the host side, the source words shifted
// into place where the two sides' alignments differ; the unaligned ends byte by
// byte (by the first 16 items).  Reads the whole aligned words that the source
// lies in.
__device__ __forceinline__ void stage_out(const StageOut& s, uint64_t first, uint64_t stride)
{
    const uint64_t lead = (16u - ((uintptr_t)s.dst & 15u)) & 15u, head = lead < s.bytes ? lead : s.bytes;
    const uint64_t body = (s.bytes - head) / 16u, tail = head + body * 16u;
    if (first < head) s.dst[first] = s.src[first];
    if (first < s.bytes - tail) s.dst[tail + first] = s.src[tail + first];
    // From the aligned word that holds the first byte of the body.
    const char* from = s.src + head;
    const uint32_t off = (uint32_t)((uintptr_t)from & 3u), shift = off * 8u;
    const uint32_t* words = (const uint32_t*)(from - off);
    uint4* dst = (uint4*)(s.dst + head);
    for (uint64_t i = first; i < body; i += stride) {
        const uint32_t* w = words + 4 * i;
        uint4 v = make_uint4(__ldcs(w), __ldcs(w + 1), __ldcs(w + 2), __ldcs(w + 3));
        if (shift != 0u) {
            const uint32_t next = __ldcs(w + 4);
            v = make_uint4(__funnelshift_r(v.x, v.y, shift), __funnelshift_r(v.y, v.z, shift),
                           __funnelshift_r(v.z, v.w, shift), __funnelshift_r(v.w, next, shift));
        }
        dst[i] = v;
    }
}

}  // namespace dev

// Blocks per row for rows of up to `items` 16-byte accesses: two per thread,
// at most 64 (16,384 threads keep enough lines in flight for the host link).
inline unsigned stage_blocks(uint64_t items)
{
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(64, (items + 2 * kStageBlock - 1) / (2 * kStageBlock)));
}

}  // namespace cbq

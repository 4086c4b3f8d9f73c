// How a cbq_intersect_host call is cut into chunks, and the copies of a chunk.
// Host code only, no CUDA.
#pragma once

#include <cstdint>

namespace cbq {

// A call is split into at most kHostChunksMax chunks, the first of at least
// kHostChunkMin rays.
constexpr uint64_t kHostChunksMax = 4;
constexpr uint64_t kHostChunkMin = 1ull << 16;
// Blocks of the call that every chunk takes a part of.
constexpr uint64_t kHostBlocksPerChunk = 4;
constexpr unsigned kHostWeights[kHostChunksMax] = {1, 2, 3, 4};

// One chunk of a call.  The call's rays are cut into kHostBlocksPerChunk blocks
// of `pitch` consecutive rays, and every chunk takes `width` rays of each (its
// rows), from `offset` in the block: so every chunk samples the whole batch (a
// camera batch whose first rows are sky and whose middle rows are terrain), and
// the copies and traversals of consecutive chunks stay in proportion.  The rays
// after the last block go to the last chunk.  On the device a chunk's rays and
// hits are contiguous, from ray `start`; on the host its rows are those of a
// pitched array.
struct HostChunk {
    uint64_t start = 0, width = 0, offset = 0, pitch = 0, rows = 0;
    uint64_t tail = 0, tail_at = 0;  // rays after the last block, and the host index of the first
    uint64_t rays() const { return rows * width + tail; }
};

// Chunks of a call of n rays whose copies overlap the traversals.
inline uint64_t host_chunks(uint64_t n)
{
    uint64_t chunks = 1, sum = kHostWeights[0];
    while (chunks < kHostChunksMax && n >= kHostChunkMin * (sum + kHostWeights[chunks])) sum += kHostWeights[chunks++];
    return chunks;
}

// The chunks of a call of n rays (one chunk, of all rays in order, unless
// `overlaps`); returns how many there are.
inline uint64_t plan_host_chunks(uint64_t n, bool overlaps, HostChunk plan[kHostChunksMax])
{
    const uint64_t chunks = overlaps ? host_chunks(n) : 1, blocks = chunks == 1 ? 1 : kHostBlocksPerChunk;
    const uint64_t pitch = n / blocks;
    uint64_t offset = 0, start = 0, sum = 0;
    for (uint64_t k = 0; k < chunks; k++) sum += kHostWeights[k];
    for (uint64_t k = 0; k < chunks; k++) {
        HostChunk& c = plan[k];
        c = HostChunk();
        c.start = start;
        c.offset = offset;
        c.pitch = pitch;
        c.rows = blocks;
        c.width = k + 1 < chunks ? pitch * kHostWeights[k] / sum / 32 * 32 : pitch - offset;
        if (k + 1 == chunks) {
            c.tail_at = blocks * pitch;
            c.tail = n - c.tail_at;
        }
        offset += c.width;
        start += c.rays();
    }
    return chunks;
}

// One copy between a host array and a device array, byte offsets in both:
// `rows` rows of `width` bytes, `pitch` apart on the host and contiguous on the
// device; a plain copy where there is one row.
struct HostCopy {
    uint64_t host, dev, width, pitch, rows;
};

// The copies of a chunk of an array of `bytes` per ray, until f(copy) is false;
// returns whether it never was.  CUDA's pitched copies take pitches up to
// `max_pitch` (cudaDevAttrMaxPitch, 2^31 - 1): beyond it each row is a copy.
template <typename F>
bool for_each_copy(const HostChunk& c, uint64_t bytes, uint64_t max_pitch, F f)
{
    const uint64_t host = c.offset * bytes, dev = c.start * bytes, width = c.width * bytes, pitch = c.pitch * bytes;
    if (width != 0 && (c.rows == 1 || pitch <= max_pitch)) {
        if (!f(HostCopy{host, dev, width, pitch, c.rows})) return false;
    } else if (width != 0) {
        for (uint64_t r = 0; r < c.rows; r++)
            if (!f(HostCopy{host + r * pitch, dev + r * width, width, pitch, 1})) return false;
    }
    return c.tail == 0 || f(HostCopy{c.tail_at * bytes, dev + c.rows * width, c.tail * bytes, 0, 1});
}

}  // namespace cbq

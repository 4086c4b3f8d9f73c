// Prints the copies of a cbq_intersect_host call (cbq_hostcopy.hpp) for the rays
// "n overlaps" and bytes per ray given: chunk, host, dev, width, pitch, rows.
#include "../cubiquity_gb300/csrc/cbq_hostcopy.hpp"

#include <cstdio>
#include <cstdlib>

int main(int argc, char** argv)
{
    if (argc != 5) return 2;
    const uint64_t n = std::strtoull(argv[1], nullptr, 10), bytes = std::strtoull(argv[3], nullptr, 10);
    const uint64_t max_pitch = std::strtoull(argv[4], nullptr, 10);
    cbq::HostChunk plan[cbq::kHostChunksMax];
    const uint64_t chunks = cbq::plan_host_chunks(n, argv[2][0] == '1', plan);
    for (uint64_t k = 0; k < chunks; k++)
        cbq::for_each_copy(plan[k], bytes, max_pitch, [&](const cbq::HostCopy& c) {
            std::printf("%llu %llu %llu %llu %llu %llu\n", (unsigned long long)k, (unsigned long long)c.host,
                        (unsigned long long)c.dev, (unsigned long long)c.width, (unsigned long long)c.pitch,
                        (unsigned long long)c.rows);
            return true;
        });
    return 0;
}

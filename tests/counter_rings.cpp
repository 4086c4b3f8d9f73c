// The work counter rings (cbq_counters.hpp) over host memory.
#include "../cubiquity_gb300/csrc/cbq_counters.hpp"

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstring>
#include <set>
#include <thread>
#include <vector>

using Rings = cbq::CounterRings;
using Lock = std::unique_lock<std::mutex>;

static std::atomic<int> allocs{0}, zeros{0};
static uint64_t* alloc() { allocs++; return new uint64_t[Rings::kSize]; }
static bool zero(uint64_t* p) { zeros++; std::memset(p, 0, Rings::kSize * sizeof(uint64_t)); return true; }

#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

// Takes a counter of stream `id` in another thread; whether it had it within 5 s (200 ms if it should not).
static bool taken_elsewhere(Rings& rings, unsigned long long id, std::thread& t, bool expected)
{
    struct Shared { std::mutex m; std::condition_variable cv; bool done = false; };
    auto* s = new Shared;  // the thread may outlive this call
    t = std::thread([&rings, id, s] {
        Lock held;
        rings.take(id, alloc, zero, held);
        std::lock_guard<std::mutex> lk(s->m);
        s->done = true;
        s->cv.notify_all();
    });
    Lock lk(s->m);
    return s->cv.wait_for(lk, std::chrono::milliseconds(expected ? 5000 : 200), [s] { return s->done; });
}

int main()
{
    Rings rings;
    {
        std::set<uint64_t*> seen;
        for (uint32_t i = 0; i < 3 * Rings::kSize; i++) {
            Lock held;
            uint64_t* c = rings.take(7, alloc, zero, held);
            CHECK(c && held.owns_lock() && *c == 0);
            (*c)++;  // as its launch would
            seen.insert(c);
        }
        CHECK(seen.size() == Rings::kSize && allocs == 1 && zeros == 3);
    }
    {  // a launch in the making on stream 7 holds up stream 7 only
        Lock held;
        CHECK(rings.take(7, alloc, zero, held));
        std::thread other, same;
        CHECK(taken_elsewhere(rings, 8, other, true));
        CHECK(!taken_elsewhere(rings, 7, same, false));
        held.unlock();
        other.join();
        same.join();
    }
    {  // no memory, and a memset that cannot be queued: no counter, nothing held, and a later call tries again
        Lock held;
        CHECK(!rings.take(9, [] { return (uint64_t*)nullptr; }, zero, held) && !held.owns_lock());
        CHECK(!rings.take(9, alloc, [](uint64_t*) { return false; }, held) && !held.owns_lock());
        uint64_t* c = rings.take(9, alloc, zero, held);
        CHECK(c && *c == 0 && held.owns_lock());
    }
    {  // many threads on two streams: every counter is zero when it is taken
        std::atomic<int> bad{0};
        std::vector<std::thread> ts;
        for (int k = 0; k < 8; k++)
            ts.emplace_back([&, k] {
                for (int i = 0; i < 5000; i++) {
                    Lock held;
                    uint64_t* c = rings.take(20 + k % 2, alloc, zero, held);
                    if (!c || *c != 0) bad++;
                    else (*c)++;
                }
            });
        for (auto& t : ts) t.join();
        CHECK(bad == 0);
    }
    int freed = 0;
    rings.release([&](uint64_t* p) { freed++; delete[] p; });
    CHECK(freed == allocs);
    std::printf("ok\n");
    return 0;
}

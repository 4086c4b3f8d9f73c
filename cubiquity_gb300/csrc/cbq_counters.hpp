// Work counters of a DAG's persistent launches.  Host code only, no CUDA.
//
// Each launch takes the next counter of its stream's ring, which is zeroed as a
// whole, in stream order, when it has been used up: one memset in `kSize`
// launches.  (Stream ids are unique for the context's lifetime, so launches that
// share a ring are ordered by their stream.)  Taking a counter and queueing its
// launch happen under the ring's lock: another thread's memset of the ring must
// not come between them.  The lock is the stream's, so that a thread that waits
// for room in one stream's queue holds up no launch on another.
#pragma once

#include <cstdint>
#include <exception>
#include <map>
#include <mutex>

namespace cbq {

class CounterRings {
public:
    static constexpr uint32_t kSize = 256;

    // A zeroed counter for the next launch on stream `id`, to be queued while
    // `held` is locked; nullptr where there is none.  `alloc` gives a ring of kSize
    // counters or nullptr, `zero(ring)` queues its memset on the stream.
    template <typename Alloc, typename Zero>
    uint64_t* take(unsigned long long id, Alloc alloc, Zero zero, std::unique_lock<std::mutex>& held)
    {
        Ring* ring = nullptr;
        try {
            std::lock_guard<std::mutex> lk(lock_);
            ring = &rings_[id];  // stays where it is
        } catch (const std::exception&) {  // nothing may throw across the C ABI
            return nullptr;
        }
        std::unique_lock<std::mutex> lk(ring->lock);
        if (!ring->at) {
            ring->at = alloc();
            ring->used = kSize;
        }
        if (!ring->at) return nullptr;
        if (ring->used == kSize) {
            if (!zero(ring->at)) return nullptr;
            ring->used = 0;
        }
        held = std::move(lk);
        return ring->at + ring->used++;
    }
    // Every ring, for the owner's destruction.
    template <typename Free>
    void release(Free free)
    {
        for (auto& r : rings_)
            if (r.second.at) free(r.second.at);
        rings_.clear();
    }

private:
    struct Ring {
        std::mutex lock;
        uint64_t* at = nullptr;
        uint32_t used = 0;
    };
    std::mutex lock_;  // of the map
    std::map<unsigned long long, Ring> rings_;
};

}  // namespace cbq

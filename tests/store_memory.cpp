// allocate_store (cbq_internal.hpp) with less and less memory: prints the bytes
// allocated, whether that is all, and the warnings logged.
#include "../cubiquity_gb300/csrc/cbq_internal.hpp"

#include <cstdio>
#include <cstdlib>

static uint64_t room, got;
static int warnings;

int main()
{
    cbq_set_log_handler([](void*, int32_t level, const char*) { warnings += level == CBQ_LOG_WARNING; }, nullptr);
    for (uint64_t memory : {3000, 2999, 1000, 999}) {
        for (uint64_t whole : {3000, 1000}) {
            room = memory;
            got = 0;
            warnings = 0;
            bool is_whole = true;
            void* p = cbq::allocate_store(whole, 1000, [](uint64_t n) {
                if (n > room) return (void*)nullptr;
                got = n;
                return std::malloc(n);
            }, &is_whole);
            std::printf("%d %d %d %d %d %d\n", (int)memory, (int)whole, p ? 1 : 0, (int)got, is_whole ? 1 : 0, warnings);
            std::free(p);
        }
    }
    return 0;
}

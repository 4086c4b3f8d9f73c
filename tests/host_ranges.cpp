// Prints what cbq_hostmem.hpp says about host buffers; no kernel is launched and
// no buffer is copied.  Without an argument: the range rule alone (no GPU).
// With "device": registered, page-locked, managed and pageable memory, queried
// from the main thread and from a thread that has made no CUDA call before.
#include "../cubiquity_gb300/csrc/cbq_hostmem.hpp"

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>

static void rule(const char* name, bool got) { std::printf("%s %d\n", name, got ? 1 : 0); }

static void show(const char* name, const void* p, uint64_t bytes)
{
    cbq::HostRange main_thread = cbq::host_range(p, bytes), other;
    std::thread([&] { other = cbq::host_range(p, bytes); }).join();
    const bool same = main_thread.whole == other.whole && main_thread.device == other.device &&
                      main_thread.device == cbq::device_alias(p, bytes);
    std::printf("%s %d %d %d\n", name, main_thread.whole ? 1 : 0, main_thread.device ? 1 : 0, same ? 1 : 0);
}

int main(int argc, char** argv)
{
    using cbq::range_holds;
    if (argc < 2) {
        rule("all", range_holds(4096, 100, 4096, 100));
        rule("inside", range_holds(4100, 96, 4096, 100));
        rule("one_past", range_holds(4100, 97, 4096, 100));
        rule("longer", range_holds(4096, 101, 4096, 100));
        rule("before", range_holds(4095, 10, 4096, 100));
        rule("last_byte", range_holds(4195, 1, 4096, 100));
        rule("at_end", range_holds(4196, 1, 4096, 100));
        rule("empty_range", range_holds(4096, 1, 0, 0));
        rule("huge", range_holds(4096, ~0ull, 4096, 100));
        rule("wraps", range_holds(~(uintptr_t)0 - 10, 20, ~(uintptr_t)0 - 100, 101));
        return 0;
    }
    const size_t page = 65536;
    char* a = (char*)std::aligned_alloc(page, 16 * page);
    std::memset(a, 0, 16 * page);
    char *locked = nullptr, *managed = nullptr, *device = nullptr;
    if (cudaHostRegister(a + 2 * page, 3 * page, cudaHostRegisterDefault) != cudaSuccess ||
        cudaHostRegister(a + 5 * page, page, cudaHostRegisterDefault) != cudaSuccess ||
        cudaHostRegister(a + 8 * page + 100, 1000, cudaHostRegisterDefault) != cudaSuccess ||
        cudaHostAlloc((void**)&locked, 1000, cudaHostAllocDefault) != cudaSuccess ||
        cudaMallocManaged((void**)&managed, 1000) != cudaSuccess || cudaMalloc((void**)&device, 1000) != cudaSuccess)
        return 2;
    show("registered", a + 2 * page, 3 * page);
    show("registered_part", a + 2 * page + 17, 2 * page);
    show("registered_end", a + 5 * page - 1, 1);
    show("over_the_end_of_it", a + 8 * page + 100, 1001);
    show("all_but_its_first", a + 8 * page + 101, 999);
    show("before_it", a + 8 * page + 99, 4);
    show("two_registrations", a + 4 * page, 2 * page);
    show("starts_pageable", a + page, 2 * page);
    show("ends_pageable", a + 5 * page + 4, page);
    show("hole_between", a + 5 * page, 4 * page);
    show("pageable", a + 10 * page, page);
    show("locked", locked, 1000);
    show("locked_tail", locked + 999, 1);
    show("past_locked", locked + 8, 1000);
    show("managed", managed, 1000);
    show("past_managed", managed, 1001);
    show("device_memory", device, 1000);
    return 0;
}

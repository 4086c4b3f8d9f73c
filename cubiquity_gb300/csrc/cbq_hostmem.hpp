// What the GPU may do with a caller's host buffer.
//
// A buffer may start in page-locked memory and end outside it (part of an array
// registered with cudaHostRegister, a view across the end of a pinned pool), and
// cudaPointerGetAttributes tells about its first byte only.  Kernels take a
// buffer from the host only where all of it lies in one allocation or
// registration; any other is left to the copy calls, which look at the range
// themselves.  Host code only.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace cbq {

// Whether [p, p + bytes) lies within [start, start + size).
inline bool range_holds(uintptr_t p, uint64_t bytes, uintptr_t start, uint64_t size)
{
    return p >= start && bytes <= size && p - start <= size - bytes;
}

struct HostRange {
    bool whole = false;             // one CUDA allocation or registration holds the whole buffer
    const void* device = nullptr;   // where the GPU can use it directly, or nullptr
};

// A function of the driver, or nullptr.
template <typename F>
F driver_function(const char* name)
{
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPointByVersion(name, &f, 12000, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return (F)f;
}

// What the driver knows about the buffer [p, p + bytes): one query of five
// attributes (68 ns; cudaPointerGetAttributes, which has no range, 74 ns).
inline HostRange host_range(const void* p, uint64_t bytes)
{
    using Query = CUresult (*)(unsigned int, CUpointer_attribute*, void**, CUdeviceptr);
    using Current = CUresult (*)(CUcontext*);
    static const Query query = driver_function<Query>("cuPointerGetAttributes");
    static const Current current = driver_function<Current>("cuCtxGetCurrent");
    HostRange r;
    if (!query || !current) return r;
    unsigned int type = 0, managed = 0;  // (IS_MANAGED writes 32 bits)
    CUdeviceptr device = 0, start = 0;
    size_t size = 0;
    CUpointer_attribute what[] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED,
                                  CU_POINTER_ATTRIBUTE_DEVICE_POINTER, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                                  CU_POINTER_ATTRIBUTE_RANGE_SIZE};
    void* into[] = {&type, &managed, &device, &start, &size};
    // In a thread that has not used CUDA yet the driver gives no device address: the runtime
    // makes its device's context current.
    CUcontext context = nullptr;
    int index = 0;
    if (current(&context) != CUDA_SUCCESS ||
        (!context && (cudaGetDevice(&index) != cudaSuccess || cudaSetDevice(index) != cudaSuccess))) {
        cudaGetLastError();
        return r;
    }
    if (query(5, what, into, (CUdeviceptr)(uintptr_t)p) != CUDA_SUCCESS) return r;
    // Memory that CUDA does not know leaves the type at 0 and the range as it was.
    r.whole = type != 0 && range_holds((uintptr_t)p, bytes, (uintptr_t)start, size);
    if (!r.whole) return r;
    if (managed)
        r.device = p;
    else if (type == CU_MEMORYTYPE_HOST)
        r.device = (const void*)(uintptr_t)device;
    return r;
}

// The device address of host memory the GPU can use directly (page-locked and
// mapped, or managed) for all its `bytes`, or nullptr when it has to be copied.
inline const void* device_alias(const void* p, uint64_t bytes) { return host_range(p, bytes).device; }

}  // namespace cbq

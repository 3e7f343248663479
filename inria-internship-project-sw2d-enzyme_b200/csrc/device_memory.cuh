// device_memory.cuh — the library's device and pinned allocations.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace sw2d {

// sw2d_test_fail_allocations: requests of the calling thread that fail as on a full device, by asking
// CUDA for more than any device holds
struct AllocationFaults {
    int64_t skip = 0, count = 0, seen = 0;
};
inline AllocationFaults& allocation_faults()
{
    thread_local AllocationFaults f;
    return f;
}
constexpr size_t kNoDeviceHolds = (size_t)1 << 60;

inline size_t request_bytes(size_t bytes)
{
    AllocationFaults& f = allocation_faults();
    f.seen++;
    if (f.count <= 0) return bytes;
    if (f.skip > 0) {
        f.skip--;
        return bytes;
    }
    f.count--;
    return kNoDeviceHolds;
}

// The error of a request that failed goes to the caller and is not left behind as CUDA's last error,
// where the next launch's check would find it although the caller did without the memory.
inline cudaError_t taken(cudaError_t e)
{
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

template <class T>
cudaError_t device_malloc(T** p, size_t bytes)
{
    return taken(cudaMalloc(p, request_bytes(bytes)));
}

template <class T>
cudaError_t pinned_malloc(T** p, size_t bytes)
{
    return taken(cudaMallocHost(p, request_bytes(bytes)));
}

}  // namespace sw2d

// device_memory.cuh — the library's device and pinned allocations, and the device memory that a handle
// holds only to save time.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <vector>

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

// Device memory that a handle does without at the price of time (a gradient's kept steps and slopes).
// All holders on a device together take at most 1/32 of its memory, so that ensembles of handles leave
// each other and the caller room, and any allocation of the library on that device that finds none is
// given what the holders have idle (device_malloc).  A holder that lost its memory so may take it again.
class OptionalMemory {
public:
    // forget(owner) drops the owner's pointers into the memory; called with the pool's mutex held
    OptionalMemory(void* owner, void (*forget)(void*)) : owner_(owner), forget_(forget) {}
    OptionalMemory(const OptionalMemory&) = delete;
    OptionalMemory& operator=(const OptionalMemory&) = delete;
    ~OptionalMemory() { drop(); }

    // While one lives the memory stays: in every call that uses it or sets the owner's pointers
    struct Use {
        OptionalMemory& m;
        explicit Use(OptionalMemory& m_) : m(m_) { count(1); }
        ~Use() { count(-1); }
        Use(const Use&) = delete;
        Use& operator=(const Use&) = delete;
        void count(int n)
        {
            std::lock_guard<std::mutex> lock(pool().mu);
            m.uses_ += n;
        }
    };

    // bytes that may be had on the current device: at most free / part
    static size_t room(size_t part)
    {
        std::lock_guard<std::mutex> lock(pool().mu);
        size_t free_b = 0, share = 0;
        int device = 0;
        if (cudaGetDevice(&device) != cudaSuccess || !share_left(device, free_b, share)) return 0;
        return std::min(free_b / part, share);
    }

    // a buffer of `bytes` on the current device in place of what it held, or null
    void* take(size_t bytes)
    {
        std::lock_guard<std::mutex> lock(pool().mu);
        free_all();
        size_t free_b = 0, share = 0;
        if (cudaGetDevice(&device_) != cudaSuccess || !share_left(device_, free_b, share) || bytes > share) return nullptr;
        void* p = nullptr;
        if (taken(cudaMalloc(&p, request_bytes(bytes))) != cudaSuccess) return nullptr;
        pool().holders.push_back(this);
        buffer_ = p;
        bytes_ = bytes;
        lost_ = false;
        return p;
    }

    void drop()
    {
        std::lock_guard<std::mutex> lock(pool().mu);
        free_all();
        lost_ = false;
    }

    // an allocation that found no room has had it since the last take or drop
    bool lost() const
    {
        std::lock_guard<std::mutex> lock(pool().mu);
        return lost_;
    }

    size_t bytes() const
    {
        std::lock_guard<std::mutex> lock(pool().mu);
        return bytes_;
    }

    // frees what the holders on the current device have idle; whether that was anything
    static bool give_back()
    {
        std::lock_guard<std::mutex> lock(pool().mu);
        int device = 0;
        if (cudaGetDevice(&device) != cudaSuccess) return false;
        bool any = false;
        const std::vector<OptionalMemory*> all = pool().holders;
        for (OptionalMemory* m : all)
            if (m->device_ == device && !m->uses_) {
                m->free_all();
                m->lost_ = true;
                any = true;
            }
        return any;
    }

private:
    struct Pool {
        std::mutex mu;
        std::vector<OptionalMemory*> holders;
    };
    static Pool& pool()
    {
        static Pool* p = new Pool;  // outlives every holder
        return *p;
    }
    // what the holders on the (current) device may still take of its 1/32
    static bool share_left(int device, size_t& free_b, size_t& share)
    {
        size_t total_b = 0, held = 0;
        if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) return false;
        for (const OptionalMemory* m : pool().holders)
            if (m->device_ == device) held += m->bytes_;
        share = total_b / 32 - std::min(total_b / 32, held);
        return true;
    }
    void free_all()
    {
        auto& all = pool().holders;
        all.erase(std::remove(all.begin(), all.end(), this), all.end());
        if (!buffer_) return;
        cudaFree(buffer_);
        forget_(owner_);
        buffer_ = nullptr;
        bytes_ = 0;
    }

    void* owner_;
    void (*forget_)(void*);
    void* buffer_ = nullptr;
    size_t bytes_ = 0;
    int device_ = 0;
    int uses_ = 0;
    bool lost_ = false;
};

template <class T>
cudaError_t device_malloc(T** p, size_t bytes)
{
    const cudaError_t e = taken(cudaMalloc(p, request_bytes(bytes)));
    if (e != cudaErrorMemoryAllocation || !OptionalMemory::give_back()) return e;
    return taken(cudaMalloc(p, bytes));
}

template <class T>
cudaError_t pinned_malloc(T** p, size_t bytes)
{
    return taken(cudaMallocHost(p, request_bytes(bytes)));
}

}  // namespace sw2d

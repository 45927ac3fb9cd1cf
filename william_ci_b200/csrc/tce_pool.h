// tce_pool.h -- device memory of single calls (workspaces of tce_ao_to_kmo,
// tce_dfmp2, tce_dfmp2_energy).
//
// The buffers come from one stream-ordered pool per device, which all handles of
// the process share, and go back to it when the call ends, on every way out of
// it.  The pool keeps up to TCE_POOL_KEEP bytes for later calls while a handle
// lives: allocating and freeing some 100 MB takes longer than the calls' kernels
// (tce_ao_to_kmo of 20 cells: 3 of 4.4 ms; tce_dfmp2 of 96 cells: 6 of 10).  What
// it keeps goes back to the device when the last handle goes, and whenever an
// allocation of the library finds no memory.  Threads and streams: the allocator
// orders a buffer's next use behind its free.
// What the pool would not keep (a call's bytes past the limit, or no handle alive)
// is allocated and freed by itself: making the pool larger for one call takes
// twice as long as cudaMalloc (354 MB: 16 against 9 ms for the whole call).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <vector>

namespace tcehost {

constexpr size_t TCE_POOL_KEEP = 1000000000;   // bytes kept between calls, per device

// a member of every handle whose calls use the pool: the pool's count of handles
struct PoolUser {
    PoolUser();
    ~PoolUser();
    PoolUser(const PoolUser &) = delete;
    PoolUser &operator=(const PoolUser &) = delete;
};
// the unused memory of the current device's pool back to the device; false: there was no pool
bool pool_trim();
// cudaMalloc, once more after pool_trim when there is no memory; clears the error it returns
cudaError_t device_malloc(void **p, size_t bytes);

class CallMemory {
public:
    explicit CallMemory(cudaStream_t st) : st_(st) {}
    ~CallMemory();
    CallMemory(const CallMemory &) = delete;
    CallMemory &operator=(const CallMemory &) = delete;
    // n elements for use on the stream; false (and *p null) when there is no memory
    template <class T>
    bool get(T **p, size_t n)
    {
        *p = static_cast<T *>(take((n ? n : 1) * sizeof(T)));
        return *p != nullptr;
    }
    void drop(void *p);    // one buffer back before the call ends
    void drop_all();

private:
    void *take(size_t bytes);
    cudaStream_t st_;
    struct Buffer {
        void *p;
        bool pooled;
    };
    void give(const Buffer &b);
    size_t pooled_ = 0;        // bytes of this call from the pool
    std::vector<Buffer> mem_;
};

}  // namespace tcehost

// Scratch memory of one call: stream-ordered allocations from a pool the
// library keeps per device, for the buffers a construction, a training run or a
// ground truth allocates and gives up before it returns.
//
// Why a pool: cudaMalloc and cudaFree of the tens of buffers of such a call
// took 3 to 60 ms of it (250,000-vector construction: 27 pairs) and, on a busy
// host, up to a second, since each maps or unmaps memory and waits for the
// device; from the pool they take microseconds. The pool keeps at most
// kScratchKeep bytes between calls (what is above goes back to the driver at
// the next synchronisation) and all of it goes back when an index is closed or
// an allocation of an index fails. Allocation and release are ordered on the
// call's stream, so calls on several threads and streams share the pool safely;
// every call synchronises its stream before it returns.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>

namespace panns {

constexpr size_t kScratchKeep = 2ull << 30;

// From / to the current device's pool, ordered on `s`.
cudaError_t scratch_alloc(void **p, size_t bytes, cudaStream_t s);
void scratch_free(void *p, cudaStream_t s);
// Give the device's idle pool memory back to the driver.
void scratch_trim(int device);

// Let `kern` be launched with as much dynamic shared memory as a block can have.
// The limit is a property of the kernel, not of a launch: set to each launch's
// own size, one thread's launch could fail on the smaller size another thread has
// set in between.
cudaError_t allow_shared(const void *kern);

template <typename T>
struct Scratch {
    T *p = nullptr;
    size_t n = 0;
    cudaStream_t s = nullptr;
    Scratch() = default;
    Scratch(const Scratch &) = delete;
    Scratch &operator=(const Scratch &) = delete;
    ~Scratch() { release(); }
    void release() {
        if (p) scratch_free(p, s);
        p = nullptr;
        n = 0;
    }
    T *take() {  // the caller frees it (scratch_free)
        T *q = p;
        p = nullptr;
        n = 0;
        return q;
    }
    cudaError_t alloc(size_t count, cudaStream_t stream) {
        release();
        s = stream;
        void *q = nullptr;
        const cudaError_t e = scratch_alloc(&q, std::max<size_t>(count, 1) * sizeof(T), stream);
        if (e == cudaSuccess) {
            p = static_cast<T *>(q);
            n = count;
        }
        return e;
    }
};

}  // namespace panns

// Internal types shared by the graph construction units (graph_build.cu,
// nsg_build.cu) and the index code (panns_abi.cu).
#pragma once

#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <new>
#include <vector>

#include "dev_scratch.h"

namespace panns {

// Host words that every element is written to once: no zero fill, and pages
// that are never written are never touched.
struct HostWords {
    uint32_t *p = nullptr;
    size_t n = 0;
    HostWords() = default;
    HostWords(const HostWords &) = delete;
    HostWords &operator=(const HostWords &) = delete;
    ~HostWords() { free(p); }
    void resize(size_t count, size_t room = 0) {  // drops the contents; room: elements allocated, if more
        free(p);
        p = static_cast<uint32_t *>(malloc(((room > count ? room : count) + 1) * sizeof(uint32_t)));
        if (!p) throw std::bad_alloc();
        n = count;
    }
    void assign(const uint32_t *b, const uint32_t *e) {
        resize((size_t) (e - b));
        if (n) memcpy(p, b, n * sizeof(uint32_t));
    }
    uint32_t *begin() { return p; }
    uint32_t *data() { return p; }
    const uint32_t *data() const { return p; }
    size_t size() const { return n; }
    bool empty() const { return n == 0; }
    uint32_t &operator[](size_t i) { return p[i]; }
};

}  // namespace panns

// A built graph in CSR form, returned through the opaque panns_graph handle
// of include/panns_build.h. The k-NN lists (n x k, for callers that ask) are in
// host memory, or still in the scratch memory of the device that built them.
struct panns_graph {
    uint32_t n = 0, width = 0, entry = 0;
    std::vector<uint64_t> off;
    panns::HostWords nbrs;
    panns::HostWords knn;
    uint32_t *knn_dev = nullptr;
    int device = 0;
    // Calls on the lists in device memory go to the calling thread's own stream, in a
    // mode that a stream capture under way does not object to (the legacy stream
    // would become part of it), and leave the thread's device as it was.
    template <typename F>
    cudaError_t on_device(F call) const {
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        int before = 0;
        cudaGetDevice(&before);
        cudaError_t e = cudaSetDevice(device);
        if (e == cudaSuccess) e = call(cudaStreamPerThread);
        cudaSetDevice(before);
        cudaThreadExchangeStreamCaptureMode(&mode);
        return e;
    }
    cudaError_t copy_knn(uint32_t *out) const {
        return on_device([&](cudaStream_t s) {
            const cudaError_t e = cudaMemcpyAsync(out, knn_dev, (size_t) n * k * 4, cudaMemcpyDeviceToHost, s);
            return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
        });
    }
    ~panns_graph() {
        if (knn_dev) on_device([&](cudaStream_t s) { return cudaFreeAsync(knn_dev, s); });
    }
    uint32_t k = 0;
    uint32_t repaired = 0;
    // Cell-restricted construction only: each vertex's cell and each cell's
    // `probe` nearest cells (cells x probe).
    uint32_t cells = 0, probe = 0;
    std::vector<uint32_t> cell, near;
};

namespace panns {

// One output of glibc's rand() from the state panns_rand_seed set up
// (panns_abi.cu).
int32_t glibc_rand_next(int32_t *state);

}  // namespace panns

// Page-locked scratch of one call, from the pool of result buffers (hostmem.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>

namespace svdb {

void* host_result_alloc(size_t bytes);
void host_result_free(void* p);

// Copies on `s` may still be writing it when a call is left early, and the pool
// hands it to another thread at once: the stream is waited for first.
struct HostScratch {
    void* p;
    cudaStream_t s;
    HostScratch(size_t bytes, cudaStream_t stream) : p(host_result_alloc(bytes)), s(stream) {}
    HostScratch(const HostScratch&) = delete;
    HostScratch& operator=(const HostScratch&) = delete;
    ~HostScratch() {
        cudaStreamSynchronize(s);
        host_result_free(p);
    }
};

}  // namespace svdb

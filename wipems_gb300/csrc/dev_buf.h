// Device memory of an engine.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <string>

#include "fdtd_host.h"

namespace wipems {

// Device buffer.  With a stream the memory comes from the device's
// stream-ordered pool (cudaMallocAsync / cudaFreeAsync on that stream):
// unlike cudaMalloc / cudaFree, neither synchronises the device, so a
// server can create and destroy engines while other engines' work is in
// flight.  The stream must outlive the buffer.
template <class T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;  // elements held: 0 before, after a release and after a failed alloc
    cudaStream_t s = nullptr;
    ~DevBuf() { release(); }
    void release() {
        if (p) {
            if (s) cudaFreeAsync(p, s);
            else cudaFree(p);
        }
        p = nullptr;
        n = 0;
    }
    int alloc(size_t count, uint64_t& total, cudaStream_t stream = nullptr) {
        n = 0;
        s = stream;
        if (count == 0) return FDTD_OK;
        cudaError_t e = stream ? cudaMallocAsync(&p, count * sizeof(T), stream) : cudaMalloc(&p, count * sizeof(T));
        if (e == cudaSuccess && stream) e = cudaStreamSynchronize(stream);  // usable from any stream from here on
        if (e != cudaSuccess) {
            cudaGetLastError();  // reported here: not by the next launch's check
            p = nullptr;
            set_error(std::string(stream ? "cudaMallocAsync: " : "cudaMalloc: ") + cudaGetErrorString(e));
            return FDTD_ERR_NOMEM;
        }
        n = count;
        total += count * sizeof(T);
        return FDTD_OK;
    }
    // at least `count` elements (the old contents are lost)
    int grow(size_t count, uint64_t& total, cudaStream_t stream) {
        if (n >= count) return FDTD_OK;
        total -= n * sizeof(T);
        release();
        return alloc(count, total, stream);
    }
};

}  // namespace wipems

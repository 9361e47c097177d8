// Device buffers against a CUDA runtime of this file that runs out of memory
// on demand: no GPU.
#include <cstdio>
#include <cstdlib>
#include <set>

#include "dev_buf.h"

static size_t g_limit = 0, g_used = 0;
static std::set<void*> g_live;
static cudaError_t g_last = cudaSuccess;

extern "C" {
cudaError_t cudaMallocAsync(void** p, size_t bytes, cudaStream_t) {
    if (g_used + bytes > g_limit) return g_last = cudaErrorMemoryAllocation;
    *p = std::malloc(bytes ? bytes : 1);
    g_live.insert(*p);
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t bytes) { return cudaMallocAsync(p, bytes, nullptr); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
    if (!g_live.erase(p)) std::abort();
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) { return cudaFreeAsync(p, nullptr); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}
namespace wipems {
void set_error(const std::string&) {}
}

#define CHECK(x)                                              \
    do {                                                      \
        if (!(x)) {                                           \
            std::fprintf(stderr, "line %d: %s\n", __LINE__, #x); \
            return 1;                                         \
        }                                                     \
    } while (0)

int main() {
    using wipems::DevBuf;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(1);
    uint64_t total = 100;
    {
        DevBuf<float> b;
        g_limit = 64;
        CHECK(b.alloc(1000, total, st) == FDTD_ERR_NOMEM && !b.p && b.n == 0 && total == 100);
        CHECK(cudaGetLastError() == cudaSuccess);  // nothing left for the next launch's check
        // a second attempt must not take the first one's size for memory it has
        CHECK(b.grow(1000, total, st) == FDTD_ERR_NOMEM && !b.p && b.n == 0 && total == 100);
        g_limit = 1 << 20;
        CHECK(b.grow(1000, total, st) == FDTD_OK && b.p && b.n == 1000 && total == 4100);
        float* p = b.p;
        CHECK(b.grow(10, total, st) == FDTD_OK && b.p == p && b.n == 1000);
        g_limit = 64;
        CHECK(b.grow(2000, total, st) == FDTD_ERR_NOMEM && !b.p && b.n == 0 && total == 100);
        CHECK(b.grow(16, total, st) == FDTD_OK && b.n == 16 && total == 164);
        b.release();
        CHECK(!b.p && b.n == 0);
    }
    CHECK(g_live.empty());
    std::puts("ok");
    return 0;
}

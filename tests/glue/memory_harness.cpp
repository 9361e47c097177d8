// Device buffers against a CUDA runtime of this file that runs out of memory
// on demand: no GPU.
#include <cstdio>
#include <cstdlib>
#include <new>
#include <set>

#include <vector>

#include "readback.h"

static size_t g_limit = 0;  // of one allocation
static std::set<void*> g_live;
static cudaError_t g_last = cudaSuccess;

extern "C" {
cudaError_t cudaMallocAsync(void** p, size_t bytes, cudaStream_t) {
    if (bytes > g_limit) return g_last = cudaErrorMemoryAllocation;
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

static long g_news = -1;  // operator new calls before it throws (-1: never)
void* operator new(size_t n) {
    if (g_news == 0) throw std::bad_alloc();
    if (g_news > 0) --g_news;
    if (void* p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

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
    {  // the planes of a readback: all of them, fewer where memory is short, none
        using wipems::readback_planes;
        DevBuf<float> keep;
        total = 0;
        g_limit = 1 << 30;
        CHECK(readback_planes(20, 1000, keep, total, st) == 20 && keep.n == 20000 && total == 80000);
        CHECK(readback_planes(771, 257 * 257, keep, total, st) == 63 && keep.n == 63 * 257 * 257);
        CHECK(readback_planes(771, 257 * 257, keep, total, st) == 63 && total == 4 * keep.n);
        CHECK(readback_planes(30, (size_t)5 << 20, keep, total, st) == 1 && keep.n == (size_t)5 << 20);
        CHECK(readback_planes(771, 257 * 257, keep, total, st) == 79);  // what it has
        keep.release();
        total = 0;
        g_limit = 4 * 257 * 257 * 20;
        CHECK(readback_planes(771, 257 * 257, keep, total, st) == 15);
        keep.release();
        g_limit = 4 * 257 * 257;
        CHECK(readback_planes(771, 257 * 257, keep, total, st) == 1);
        g_limit = 1000;
        keep.release();
        CHECK(readback_planes(771, 257 * 257, keep, total, st) == 0 && !keep.p);
        CHECK(cudaGetLastError() == cudaSuccess);
    }
    CHECK(g_live.empty());
    for (int rot = 0; rot < 3; ++rot) {  // device axis a = operator axis (a + rot) % 3
        const uint32_t M[3] = {3, 5, 7}, N[3] = {M[rot], M[(1 + rot) % 3], M[(2 + rot) % 3]};
        std::vector<float> dev(105), out(105, -1.f);
        uint32_t d[3];
        for (d[0] = 0; d[0] < N[0]; ++d[0])
            for (d[1] = 0; d[1] < N[1]; ++d[1])
                for (d[2] = 0; d[2] < N[2]; ++d[2]) {
                    uint32_t o[3];
                    for (int a = 0; a < 3; ++a) o[(a + rot) % 3] = d[a];
                    dev[(d[0] * N[1] + d[1]) * N[2] + d[2]] = (float)((o[0] * M[1] + o[1]) * M[2] + o[2]);
                }
        wipems::turn_axes(dev.data(), M, rot, out.data());
        for (int k = 0; k < 105; ++k) CHECK(out[k] == (float)k);
    }
    for (long news : {0L, 1L, 2L, 5L, -1L}) {  // fresh pages are touched whatever the host's memory allows, nothing is thrown
        const size_t len = (size_t)16 << 20;
        char* m = static_cast<char*>(mmap(nullptr, len, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
        CHECK(m != MAP_FAILED && !wipems::pages_mapped(m + 3, len - 7));
        g_news = news;
        wipems::touch_pages(m + 3, len - 7);
        g_news = -1;
        CHECK(wipems::pages_mapped(m + 3, (size_t)1 << 19));  // the calling thread's share at least
        CHECK(news >= 0 || wipems::pages_mapped(m + 3, len - 7));
        munmap(m, len);
    }
    {  // a mapped array is touched within its bounds
        std::vector<char> dst((size_t)40 << 20, 1);
        wipems::touch_pages(dst.data() + 3, dst.size() - 7);
        CHECK(dst[2] == 1 && dst[3] == 0 && dst[dst.size() - 5] == 0 && dst[dst.size() - 4] == 1);
    }
    std::puts("ok");
    return 0;
}

// Host side of field readbacks: the pages they write to, the device scratch
// they get and the order of axes without one.
#pragma once

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <thread>

#include "dev_buf.h"

namespace wipems {

constexpr size_t kFreshBytes = (size_t)256 << 10;  // allocators give arrays above this fresh pages

// Whether the pages of a host array are there already, by a sample of them
// (a system call of 0.4 us each): an array that was written before, or memory
// that the allocator hands out again.
inline bool pages_mapped(const void* p, size_t bytes) {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    const int n = bytes < (size_t)4 << 20 ? 4 : 16;
    for (int k = 0; k < n; ++k) {
        const uintptr_t a = (uintptr_t)p + (bytes - 1) / (n - 1) * k;
        unsigned char there = 0;
        if (mincore((void*)(a / page * page), page, &there) != 0 || !(there & 1)) return false;
    }
    return true;
}

// Maps the pages of a large host destination before the device writes to it,
// a share per thread.  A fresh array's pages do not exist yet, and faulting
// them in one by one under the copy takes many times the copy: both fields of
// 257^3 lines (408 MB) took 335 ms to read, 6.4 ms with their pages mapped by
// 16 threads first.  Small arrays are touched by the calling thread alone, and
// mapped ones are left alone (touching those took 1.1 ms of the 4.1 ms that
// the same fields took into arrays written before).
inline void touch_pages(void* p, size_t bytes) noexcept {
    if (bytes < kFreshBytes || pages_mapped(p, bytes)) return;
    const size_t page = 4096;
    const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
    const unsigned nt = (unsigned)std::max<size_t>(1, std::min<size_t>(std::min(hw, 16u), bytes >> 21));
    auto part = [=](unsigned k) {
        volatile char* b = static_cast<volatile char*>(p);
        const size_t lo = bytes / nt * k, hi = k + 1 == nt ? bytes : bytes / nt * (k + 1);
        for (size_t o = lo; o < hi; o += page) b[o] = 0;
        if (hi > lo) b[hi - 1] = 0;
    };
    std::thread th[16];
    try {
        for (unsigned k = 1; k < nt; ++k) th[k] = std::thread(part, k);
    } catch (...) {  // fewer threads (or no memory for one): the copy maps the rest
    }
    part(0);
    for (std::thread& t : th)
        if (t.joinable()) t.join();
}

constexpr size_t kReadbackFloats = (size_t)32 << 20;  // scratch of a readback, at most (128 MB), and
constexpr size_t kReadbackKept = (size_t)4 << 20;     // what of it an engine keeps for the next one (16 MB)

// Planes (of `plane` floats each, at most `planes`) that a readback packs at
// a time, with a scratch for them: `keep` if that is small, else `once`, which
// the caller gives back.  Where memory is short fewer planes at a time, down
// to one; 0 if there is not even that.
inline uint32_t readback_planes(uint32_t planes, size_t plane, DevBuf<float>& keep, DevBuf<float>& once,
                                uint64_t& kept_bytes, cudaStream_t st, float** scratch) {
    uint64_t bytes = 0;  // of `once`: not the engine's
    for (uint32_t n = (uint32_t)std::min<size_t>(planes, std::max<size_t>(1, kReadbackFloats / plane)); n > 0; n /= 2) {
        const bool small = n * plane <= std::max(kReadbackKept, keep.n);
        if ((small ? keep.grow(n * plane, kept_bytes, st) : once.grow(n * plane, bytes, st)) != FDTD_OK) continue;
        *scratch = small ? keep.p : once.p;
        return n;
    }
    return 0;
}

// One component from device axes to the operator's (device axis a = operator
// axis (a + rot) % 3): s[N0][N1][N2] with N[a] = M[(a + rot) % 3], d[M0][M1][M2].
inline void turn_axes(const float* s, const uint32_t M[3], int rot, float* d) {
    uint32_t o[3];
    const size_t N1 = M[(1 + rot) % 3], N2 = M[(2 + rot) % 3];
    for (o[0] = 0; o[0] < M[0]; ++o[0])
        for (o[1] = 0; o[1] < M[1]; ++o[1])
            for (o[2] = 0; o[2] < M[2]; ++o[2])
                *d++ = s[(o[rot % 3] * N1 + o[(1 + rot) % 3]) * N2 + o[(2 + rot) % 3]];
}

}  // namespace wipems

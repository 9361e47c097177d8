// Host side of field readbacks: the pages they write to, the device scratch
// they get and the order of axes without one.
#pragma once

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <thread>

#include "dev_buf.h"

namespace wipems {

// Whether the pages of a host array are there already, by a sample of them: an
// array that was written before, or memory that the allocator hands out again.
inline bool pages_mapped(const void* p, size_t bytes) {
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    for (size_t k = 0; k < 16; ++k) {
        const uintptr_t a = (uintptr_t)p + (bytes - 1) / 15 * k;
        unsigned char there = 0;
        if (mincore((void*)(a / page * page), page, &there) != 0 || !(there & 1)) return false;
    }
    return true;
}

// Writes to every page of a large host destination before the device does, a
// share per thread.  A fresh array's pages do not exist yet, and faulting them
// in one by one under the copy takes many times the copy: both fields of 257^3
// lines (408 MB) took 335 ms to read, 6.4 ms with their pages mapped by 16
// threads first.  Pages that are mapped are touched all the same: where they
// come from memory that the program used for something else before, a copy
// into them took up to ten times as long without (193^3 lines 34 ms, 1.4
// touched).  That is quick, so fewer threads do it.  Under 4 MB it costs more
// than it saves (a dump of 0.8 MB 55 us, touched 63).  The contents are lost
// either way: the whole array is the destination.
inline void touch_pages(void* p, size_t bytes) noexcept {
    if (bytes < (size_t)4 << 20) return;
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
    const unsigned nt = (unsigned)std::max<size_t>(
        1, std::min<size_t>(std::min(hw, 16u), pages_mapped(p, bytes) ? bytes >> 26 : bytes >> 21));
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

constexpr size_t kReadbackFloats = (size_t)4 << 20;  // scratch of a readback (16 MB; a plane if that is more)

// Planes (of `plane` floats each, at most `planes`) that a readback packs at
// a time, in a scratch that the engine keeps (a larger one, allocated and
// freed by each call, took up to 100 ms where the memory pool had to grow).
// Where memory is short fewer planes at a time, down to one; 0 if there is not
// even that.
inline uint32_t readback_planes(uint32_t planes, size_t plane, DevBuf<float>& scratch, uint64_t& bytes, cudaStream_t st) {
    uint32_t n = (uint32_t)std::min<size_t>(planes, std::max<size_t>(1, std::max(kReadbackFloats, scratch.n) / plane));
    while (n > 0 && scratch.grow(n * plane, bytes, st) != FDTD_OK) n /= 2;
    return n;
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

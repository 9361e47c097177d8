// Launch side of the resident timesteps (kernels_resident.cuh): how a grid is
// cut into boxes, the buffers a run needs, and the launches of a run.
#include <cuda_runtime.h>

#include <algorithm>

#include "engine_state.h"
#include "kernels_resident.cuh"

namespace wipems {
namespace {

// Box capacities compiled: a small box leaves the L1 cache what it does not
// need (the tuple tables live there); UPML and Lorentz/Drude states and Mur
// nodes take their share of the largest.  Dispersive graded meshes, whose
// thousands of tuples miss L1 more often, gain too (41 x 46 x 51 lines with
// UPML 8.3 -> 4.7 us per step, 65 x 71 x 61 13.1 -> 9.5).
template <int NS, int FEAT, bool LATE = false>
const void* kernel_g(bool geo) {
    return geo ? (const void*)k_resident<NS, FEAT, true, LATE> : (const void*)k_resident<NS, FEAT, false, LATE>;
}
struct Variant {
    int ns;  // capacity (0 = no such variant)
    const void* kernel;
};
Variant variant_of(int nodes, int feat, bool geo, bool late) {
    constexpr int U = FEAT_UPML, A = FEAT_ADE;
    if (feat == 0 && !late) {
        if (nodes <= 1536) return {1536, kernel_g<1536, 0>(geo)};
        if (nodes <= 3072) return {3072, kernel_g<3072, 0>(geo)};
        return {7680, kernel_g<7680, 0>(geo)};
    }
    if (feat == U && !late) {
        if (nodes <= 1536) return {1536, kernel_g<1536, U>(geo)};
        if (nodes <= 3072) return {3072, kernel_g<3072, U>(geo)};
        return {4096, kernel_g<4096, U>(geo)};
    }
    if (feat == 0) {
        if (nodes <= 3072) return {3072, kernel_g<3072, 0, true>(geo)};
        return {5632, kernel_g<5632, 0, true>(geo)};
    }
    if (feat == U) return {3072, kernel_g<3072, U, true>(geo)};
    if (feat == A) return {3072, late ? kernel_g<3072, A, true>(geo) : kernel_g<3072, A>(geo)};
    if (feat == (A | RES_LOR))
        return {2048, late ? kernel_g<2048, A | RES_LOR, true>(geo) : kernel_g<2048, A | RES_LOR>(geo)};
    if ((feat & ~RES_LOR) == (A | U) && !late) return {2048, kernel_g<2048, A | U | RES_LOR>(geo)};
    return {0, nullptr};
}

constexpr size_t kSampleBytes = (size_t)16 << 20;  // of a run's energy segments
constexpr int kMaxRunSamples = 64;
constexpr int kMaxRunFd = 256;
constexpr uint32_t kMaxRun = 1024;  // timesteps of one launch
constexpr uint32_t kMaxTag = 1u << 30;  // the exchange words are cleared above it

}  // namespace

// The cut with the cheapest largest box: its 32-node tasks (eight or fewer
// take the same time), its rows at a cut (which wait for a neighbour), and a
// z cut's lone lanes.
bool resident_plan(const int cov[3], const bool mur[3], int blocks, int nodes, int p[3]) {
    const int segs = (cov[2] + 31) / 32;
    double best = 1e30;
    for (int pz = 1; pz <= std::min(segs, blocks); ++pz) {
        const int nzc = (segs + pz - 1) / pz;
        for (int py = 1; py <= std::min(cov[1], blocks / pz); ++py) {
            for (int px = 1; px <= std::min(cov[0], blocks / (pz * py)); ++px) {
                const int bx = (cov[0] + px - 1) / px, by = (cov[1] + py - 1) / py, bz = std::min(32 * nzc, cov[2]);
                const long long tasks = (long long)bx * by * nzc;
                if ((long long)bx * by * bz > nodes || tasks > RES_TASKS) continue;
                // a Mur face and the line next to it lie in one box, the face nodes fit
                if ((mur[0] && cov[0] / px < 2) || (mur[1] && cov[1] / py < 2) ||
                    (mur[2] && cov[2] - res_cut_z(cov[2], pz, pz - 1) < 2))
                    continue;
                auto faces = [&](int k, int q) { return mur[k] ? (q == 1 ? 2 : 1) : 0; };
                if (faces(0, px) * by * bz + faces(1, py) * bx * bz + faces(2, pz) * bx * by > RES_MUR) continue;
                const double cost = std::max(8.0, (double)tasks) + 0.25 * (bx + by) * nzc +
                                    (pz > 1 ? 0.1 * bx * by : 0.0) + 1e-3 * (px * py * pz);
                if (cost < best) {
                    best = cost;
                    p[0] = px;
                    p[1] = py;
                    p[2] = pz;
                }
            }
        }
    }
    return best < 1e30;
}

int plan_resident(fdtd_engine_s* e) {
    if (e->res_planned) return FDTD_OK;
    e->res_planned = true;
    int sms = 0, coop = 0, smem = 0;
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, e->device));
    CK(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, e->device));
    CK(cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, e->device));
    ResArgs& a = e->ra;
    const size_t entries = e->h_entries.size();
    // Mur faces change lines that the voltage update leaves out
    bool mur[3] = {false, false, false};
    for (int k = 0; k < e->mur.nface; ++k) mur[e->mur.f[k].ny] = true;
    for (int k = 0; k < 3; ++k) {
        a.ne[k] = e->ti.ne[k];
        a.cov[k] = e->mur.nface ? (int)e->N[k] : a.ne[k];
    }
    a.mur = e->mur;
    a.rlc = e->rlc;
    const bool late = e->mur.nface || e->rlc.count;
    int feat = e->feat | (e->LV.p || e->LI.p ? RES_LOR : 0);
    if ((feat & (FEAT_ADE | FEAT_UPML)) == (FEAT_ADE | FEAT_UPML)) feat |= RES_LOR;
    const int cap = variant_of(1 << 30, feat, e->geo_on, late).ns;
    if (!coop || cap == 0 || entries > RES_ENTRIES || e->rlc.count > RES_RLC ||
        !resident_plan(a.cov, mur, sms, cap, a.p))
        return FDTD_OK;
    const int segs = (a.cov[2] + 31) / 32, nzc = (segs + a.p[2] - 1) / a.p[2];
    const int bx = (a.cov[0] + a.p[0] - 1) / a.p[0], by = (a.cov[1] + a.p[1] - 1) / a.p[1],
              bz = std::min(32 * nzc, a.cov[2]);
    const Variant v = variant_of(bx * by * bz, feat, e->geo_on, late);
    const int need = res_smem(v.ns, feat, late);
    if (smem < need + 64) return FDTD_OK;
    e->res_smem = need;
    e->res_threads = 32 * std::min(RES_THREADS / 32, bx * by * nzc);
    e->res_kernel = v.kernel;
    CK(cudaFuncSetAttribute(e->res_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, need));
    int per_sm = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, e->res_kernel, e->res_threads, (size_t)need));
    if (per_sm < 1) return FDTD_OK;
    const long long wx = (long long)a.cov[1] * a.cov[2], wy = (long long)a.cov[0] * a.cov[2],
                    wz = (long long)a.cov[0] * a.cov[1];
    a.ll_pairs = ((a.p[0] - 1) * wx + (a.p[1] - 1) * wy + (a.p[2] - 1) * wz);
    a.interval = (int)e->interval;
    a.nentry = (int)entries;
    const bool fd = e->fd_interval && !e->h_freq.empty() && e->ps.nprobe;
    a.fd_interval = fd ? (int)e->fd_interval : 0;
    a.d_err = e->p_err();
    a.seg_stride = (long long)(e->N[0] - 1) * (e->N[1] - 1) * e->g.nzt;
    e->res_samples = (int)std::max<size_t>(1, std::min<size_t>(kMaxRunSamples, kSampleBytes / (8 * a.seg_stride)));
    e->res_fits = true;
    return FDTD_OK;
}

int setup_resident(fdtd_engine_s* e) {
    if (int rc = plan_resident(e)) return rc;
    if (e->res_ready || !e->res_fits) return FDTD_OK;
    ResArgs& a = e->ra;
    const size_t samples = e->interval ? e->res_samples : 0, esamples = e->energy_on_probe ? samples : 0;
    uint64_t& tot = e->device_bytes;
    const uint64_t before = tot;
    if (e->res_ll.alloc(std::max<long long>(1, 4 * a.ll_pairs), tot, e->stream) ||
        e->res_pval.alloc(a.nentry * samples, tot, e->stream) ||
        e->res_fdval.alloc(a.fd_interval ? (size_t)a.nentry * kMaxRunFd : 0, tot, e->stream) ||
        e->res_seg.alloc(a.seg_stride * esamples, tot, e->stream) ||
        e->res_plane.alloc((e->N[0] - 1) * esamples, tot, e->stream)) {
        // no memory left for it: the half-step kernels need none
        e->res_ll.release();
        e->res_pval.release();
        e->res_fdval.release();
        e->res_seg.release();
        e->res_plane.release();
        tot = before;
        return FDTD_OK;
    }
    a.ll = e->res_ll.p;
    a.pval = e->res_pval.p;
    a.fdval = e->res_fdval.p;
    a.eseg = e->res_seg.p;
    CK(cudaMemsetAsync(e->res_ll.p, 0, e->res_ll.n * sizeof(ulonglong2), e->stream));
    e->res_ready = true;
    return FDTD_OK;
}

uint32_t resident_run(const fdtd_engine_s* e, uint32_t n) {
    n = std::min(n, kMaxRun);
    if (e->interval) n = (uint32_t)std::min<uint64_t>(n, ((uint64_t)e->ts / e->interval + e->res_samples) * e->interval - e->ts);
    const uint32_t f = (uint32_t)e->ra.fd_interval;
    if (f) n = (uint32_t)std::min<uint64_t>(n, ((uint64_t)e->ts / f + kMaxRunFd) * f - e->ts);
    return n;
}

int launch_resident(fdtd_engine_s* e, uint32_t n, cudaStream_t st) {
    ResArgs a = e->ra;
    a.ts0 = (int)e->ts;
    a.nsteps = (int)n;
    if (e->res_tag > kMaxTag) {
        CK(cudaMemsetAsync(e->res_ll.p, 0, e->res_ll.n * sizeof(ulonglong2), st));
        e->res_tag = 0;
    }
    a.tag0 = e->res_tag;
    e->res_tag += n;
    void* args[] = {&e->g, &a, &e->ps};
    CK(cudaLaunchCooperativeKernel(e->res_kernel, dim3((unsigned)(a.p[0] * a.p[1] * a.p[2])),
                                   dim3((unsigned)e->res_threads), args, (size_t)e->res_smem, st));
    const int count = e->interval ? (int)((e->ts + n) / e->interval - e->ts / e->interval) : 0;
    const int first = e->interval ? (int)((e->ts / e->interval + 1) * e->interval) : 0;
    if (count && a.eseg) {
        k_resident_planes<<<dim3(e->N[0] - 1, (unsigned)count), 256, 0, st>>>(e->g, a.eseg, a.seg_stride,
                                                                                   e->res_plane.p);
        e->last_launches += 1;
    }
    k_resident_samples<<<std::max(1, count), 256, 0, st>>>(e->p_ts(), (int)n, count, first, (int)e->interval,
                                                                e->ps, e->g, a.pval, a.nentry, e->res_plane.p,
                                                                a.eseg ? 1 : 0, e->ticket.p, kEps0, kMue0);
    e->last_launches += 2;
    const int f = a.fd_interval, fds = f ? ((int)(e->ts + n) / f - (int)e->ts / f) : 0;
    if (fds) {
        ProbeSet ps = e->ps;
        ps.vals = a.fdval;
        k_fd_accumulate<<<1, 256, std::max<size_t>(8, ps.nprobe * sizeof(double)), st>>>(
            e->p_ts(), (int)(e->ts + n), ps, e->g, e->fd, ((int)e->ts / f + 1) * f, f, fds, a.nentry);
        e->last_launches += 1;
    }
    CK(cudaGetLastError());
    return FDTD_OK;
}

}  // namespace wipems

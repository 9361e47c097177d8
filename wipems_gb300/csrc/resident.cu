// Launch side of the resident timesteps (kernels_resident.cuh): how a grid is
// cut into boxes, the buffers a run needs, and the launches of a run.
#include <cuda_runtime.h>

#include <algorithm>

#include "engine_state.h"
#include "kernels_resident.cuh"

namespace wipems {
namespace {

// box capacities compiled; with UPML the fluxes take their share
constexpr int kNodes[4] = {1536, 3072, 4096, 7680};
template <int NS, bool UPML>
const void* kernel_g(bool geo) {
    return geo ? (const void*)k_resident<NS, UPML, true> : (const void*)k_resident<NS, UPML, false>;
}
const void* kernel_of(int ns, bool upml, bool geo) {
    switch (ns) {
        case kNodes[0]: return upml ? kernel_g<kNodes[0], true>(geo) : kernel_g<kNodes[0], false>(geo);
        case kNodes[1]: return upml ? kernel_g<kNodes[1], true>(geo) : kernel_g<kNodes[1], false>(geo);
        case kNodes[2]: return upml ? kernel_g<kNodes[2], true>(geo) : kernel_g<kNodes[2], false>(geo);
        default: return kernel_g<kNodes[3], false>(geo);
    }
}

constexpr size_t kSampleBytes = (size_t)64 << 20;  // of a run's energy segments
constexpr int kMaxRunSamples = 64;
constexpr int kMaxRunFd = 256;
constexpr uint32_t kMaxRun = 1024;  // timesteps of one launch

}  // namespace

// The cut with the cheapest largest box: its 32-node tasks (eight or fewer
// take the same time), its rows at a cut (which wait for a neighbour), and a
// z cut's lone lanes.
bool resident_plan(const int cov[3], int blocks, int nodes, int p[3]) {
    const int segs = (cov[2] + 31) / 32;
    double best = 1e30;
    for (int pz = 1; pz <= std::min(segs, blocks); ++pz) {
        const int nzc = (segs + pz - 1) / pz;
        for (int py = 1; py <= std::min(cov[1], blocks / pz); ++py) {
            for (int px = 1; px <= std::min(cov[0], blocks / (pz * py)); ++px) {
                const int bx = (cov[0] + px - 1) / px, by = (cov[1] + py - 1) / py, bz = std::min(32 * nzc, cov[2]);
                const long long tasks = (long long)bx * by * nzc;
                if ((long long)bx * by * bz > nodes || tasks > RES_TASKS) continue;
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

int setup_resident(fdtd_engine_s* e) {
    int sms = 0, coop = 0, smem = 0;
    CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, e->device));
    CK(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, e->device));
    CK(cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, e->device));
    ResArgs& a = e->ra;
    const size_t entries = e->h_entries.size();
    for (int k = 0; k < 3; ++k) a.cov[k] = a.ne[k] = e->ti.ne[k];
    const bool up = (e->feat & FEAT_UPML) != 0;
    if (!coop || entries > RES_ENTRIES || !resident_plan(a.cov, sms, kNodes[up ? 2 : 3], a.p)) return FDTD_OK;
    const int segs = (a.cov[2] + 31) / 32, nzc = (segs + a.p[2] - 1) / a.p[2];
    const int bx = (a.cov[0] + a.p[0] - 1) / a.p[0], by = (a.cov[1] + a.p[1] - 1) / a.p[1],
              bz = std::min(32 * nzc, a.cov[2]);
    int ns = kNodes[0];
    for (int k = 1; k < 4 && bx * by * bz > ns; ++k) ns = kNodes[k];
    const int need = res_smem(ns, up);
    if (smem < need + 64) return FDTD_OK;
    e->res_smem = need;
    e->res_threads = 32 * std::min(RES_THREADS / 32, bx * by * nzc);
    e->res_kernel = kernel_of(ns, up, e->geo_on);
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
    int rc;
    uint64_t& tot = e->device_bytes;
    if ((rc = e->res_ll.alloc(std::max<long long>(1, 4 * a.ll_pairs), tot, e->stream)) ||
        (rc = e->res_pval.alloc(std::max<size_t>(1, entries * e->res_samples), tot, e->stream)) ||
        (fd && (rc = e->res_fdval.alloc(std::max<size_t>(1, entries * kMaxRunFd), tot, e->stream))) ||
        (rc = e->res_seg.alloc(a.seg_stride * e->res_samples, tot, e->stream)) ||
        (rc = e->res_plane.alloc((size_t)(e->N[0] - 1) * e->res_samples, tot, e->stream)))
        return rc;
    a.ll = e->res_ll.p;
    a.pval = e->res_pval.p;
    a.fdval = e->res_fdval.p;
    a.eseg = e->energy_on_probe ? e->res_seg.p : nullptr;
    CK(cudaMemsetAsync(e->res_ll.p, 0, e->res_ll.n * sizeof(ulonglong2), e->stream));
    e->resident = true;
    return FDTD_OK;
}

uint32_t resident_run(const fdtd_engine_s* e, uint32_t n) {
    n = std::min(n, kMaxRun);
    if (e->interval) n = (uint32_t)std::min<uint64_t>(n, ((uint64_t)e->ts / e->interval + e->res_samples) * e->interval - e->ts);
    const uint32_t f = (uint32_t)e->ra.fd_interval;
    if (f) n = (uint32_t)std::min<uint64_t>(n, ((uint64_t)e->ts / f + kMaxRunFd) * f - e->ts);
    return n;
}

int launch_resident(fdtd_engine_s* e, uint32_t n) {
    ResArgs a = e->ra;
    a.ts0 = (int)e->ts;
    a.nsteps = (int)n;
    void* args[] = {&e->g, &a, &e->ps};
    CK(cudaLaunchCooperativeKernel(e->res_kernel, dim3((unsigned)(a.p[0] * a.p[1] * a.p[2])),
                                   dim3((unsigned)e->res_threads), args, (size_t)e->res_smem, e->stream));
    const int count = e->interval ? (int)((e->ts + n) / e->interval - e->ts / e->interval) : 0;
    const int first = e->interval ? (int)((e->ts / e->interval + 1) * e->interval) : 0;
    if (count && a.eseg) {
        k_resident_planes<<<dim3(e->N[0] - 1, (unsigned)count), 256, 0, e->stream>>>(e->g, a.eseg, a.seg_stride,
                                                                                   e->res_plane.p);
        e->last_launches += 1;
    }
    k_resident_samples<<<std::max(1, count), 256, 0, e->stream>>>(e->p_ts(), (int)n, count, first, (int)e->interval,
                                                                e->ps, e->g, a.pval, a.nentry, e->res_plane.p,
                                                                a.eseg ? 1 : 0, e->ticket.p, kEps0, kMue0);
    e->last_launches += 2;
    const int f = a.fd_interval, fds = f ? ((int)(e->ts + n) / f - (int)e->ts / f) : 0;
    if (fds) {
        ProbeSet ps = e->ps;
        ps.vals = a.fdval;
        k_fd_accumulate<<<1, 256, std::max<size_t>(8, ps.nprobe * sizeof(double)), e->stream>>>(
            e->p_ts(), (int)(e->ts + n), ps, e->g, e->fd, ((int)e->ts / f + 1) * f, f, fds, a.nentry);
        e->last_launches += 1;
    }
    CK(cudaGetLastError());
    return FDTD_OK;
}

}  // namespace wipems

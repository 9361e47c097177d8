// Resident timesteps: a grid that fits in the shared memory of the whole GPU
// stays there for a run of timesteps.
//
// One block per SM (a cooperative launch, so that all of them run at once)
// owns a box of nodes and keeps its voltages, currents and tuple indices in
// shared memory from the first to the last timestep of the run.  A warp
// takes 32 z-nodes of a row at a time.  What a box needs of its neighbours
// goes through global memory (L2) as 64-bit words {value, tag}, the tag
// counting the timesteps of all runs of the engine (numTS may go back): the
// reader polls the very word it needs, so an exchange costs one store and
// one load, no fence, flag or barrier.  Words of even and odd timesteps lie
// in two buffers: a node's word of timestep n + 2 is stored only after that
// node has read its neighbour's word of n + 1, which the neighbour stored
// after reading the word of n that is being replaced.
//
// A half-step on its own costs a launch (about 3 us, whatever the size) and
// the trip of all fields through L2; here it costs a block barrier and an
// exchange.  Small boxes are bound by the latency of the exchange (1.2 us per
// half-step), large ones by instruction issue (about 115 per 32 nodes).
// Device time per timestep, half-step kernels -> resident:
//   25 x 10 x 31 PEC 6.6 -> 2.5 us      47 x 33 x 61 UPML 8.6 -> 4.5
//   41^3 PEC 7.3 -> 2.8                 61^3 UPML 12.1 -> 5.0
//   65^3 PEC 8.6 -> 4.3                 81^3 UPML 17.8 -> 11.0
//   91^3 PEC 13.7 -> 9.9                98 x 76 x 132 PEC 16.1 -> 13.3
//   102^3 PEC 18.9 -> 15.1              61 x 51 x 71 UPML + RLC 13.8 -> 6.3
//   51 x 42 x 61 Mur 17.3 -> 4.2        91 x 92 x 90 Mur 25.0 -> 10.1
//   21 x 4 x 1001 Mur, Drude 16.0 -> 3.9 (five launches per timestep before)
// so an engine that has the GPU to itself runs every grid that fits resident.
// The same run takes up to 4 % more or less by where its exchange words lie in
// memory (engines of one grid differ by that).
//
// Arithmetic: as update_node (node.cuh).
#pragma once

#include <type_traits>

#include "kernels.cuh"
#include "node.cuh"

namespace wipems {

constexpr int RES_THREADS = 640;   // 96 registers a thread: 768 threads spill
constexpr int RES_TASKS = 320;     // 32-node tasks of a box
constexpr int RES_ENTRIES = 512;   // probe entries whose samples are taken inside the run
// Field components a box keeps: V and I, the UPML fluxes, the Drude states
// and, with RES_LOR, the Lorentz states.
constexpr int RES_LOR = 256;  // beside the FEAT_ bits
__host__ __device__ constexpr int res_comps(int feat) {
    return 6 + ((feat & FEAT_UPML) ? 6 : 0) + ((feat & FEAT_ADE) ? 6 : 0) + ((feat & RES_LOR) ? 6 : 0);
}
// Shared memory of a box of up to NS nodes: the components at a constant
// stride, so that a node's 13 reads share four address registers, the two
// tuple indices, the task tables, the probe entries and, for runs with passes
// after the voltage update, the Mur face nodes of the box (four values and
// two words each) and its lumped RLC edges.
constexpr int RES_MUR = 2048;
constexpr int RES_RLC = 128;
__host__ __device__ constexpr int res_smem(int ns, int feat, bool late) {
    return ns * (res_comps(feat) * 4 + 2 * 2) + 2 * RES_TASKS * 16 + RES_ENTRIES * 8 + (late ? RES_MUR * 24 + RES_RLC * 8 : 0);
}
constexpr unsigned long long RES_WAIT_CYCLES = 4000000000ull;  // ~2 s

// task: {slot of its first node | flags << 16, global offset of it from the
// box's first node, x | y << 16, z}
constexpr uint32_t RT_X = 1u << 16;     // the x neighbour (E: x-1, H: x+1) is in the box
constexpr uint32_t RT_Y = 2u << 16;
constexpr uint32_t RT_ROW = 16u << 16;  // this half-step updates the row
constexpr uint32_t RT_Z = 32u << 16;    // E: node z-1 of lane 0 is in the box

struct ResArgs {
    int cov[3];              // nodes the boxes cover (lines that no timestep changes are left out)
    int p[3];                // boxes per axis
    int ne[3];               // extent of the voltage update
    int ts0, nsteps;         // numTS at the start, timesteps of this run
    uint32_t tag0;           // tags below and up to this one are of earlier runs
    int interval;            // samples after every interval-th timestep (0 = none)
    ulonglong2* ll;          // exchange pairs: [V, I][even, odd][x cuts, y cuts, z cuts]
    long long ll_pairs;      // pairs per field and parity
    float2* eseg;            // energy segments per sample of the run (null = no energies)
    long long seg_stride;
    float* pval;             // probe entry values per sample of the run
    int fd_interval;         // frequency-domain steps: every fd_interval-th timestep (0 = none)
    float* fdval;            // probe entry values per frequency-domain step of the run
    int nentry;
    MurSet mur;              // Mur faces (nface 0 = none)
    RlcSet rlc;              // lumped RLC edges (count 0 = none)
    int* d_err;
};

// first node of box i of p over n nodes
__host__ __device__ __forceinline__ int res_cut(int n, int p, int i) { return (int)((long long)n * i / p); }
// z boxes are whole 32-node segments
__host__ __device__ __forceinline__ int res_cut_z(int n, int p, int i) {
    const int c = 32 * res_cut((n + 31) / 32, p, i);
    return c < n ? c : n;
}

// the two components a neighbour needs of a node, as two tagged words
__device__ __forceinline__ void ll_send(ulonglong2* w, float v0, float v1, uint32_t tag) {
    const unsigned long long t = (unsigned long long)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(w), "l"(t | __float_as_uint(v0)),
                 "l"(t | __float_as_uint(v1))
                 : "memory");
}
// Polls a pair until both words carry the tag (or a later one: a node whose
// current never changes is sent without waiting for its reader, and every
// value it sends is the same); ok turns false when the clock budget runs out.
__device__ __forceinline__ bool ll_load(const ulonglong2* w, uint32_t tag, float& v0, float& v1) {
    unsigned long long a, b;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(w) : "memory");
    v0 = __uint_as_float((uint32_t)a);
    v1 = __uint_as_float((uint32_t)b);
    return (int)((uint32_t)(a >> 32) - tag) >= 0 && (int)((uint32_t)(b >> 32) - tag) >= 0;
}
__device__ __forceinline__ void ll_wait(const ulonglong2* w, uint32_t tag, float& v0, float& v1, bool& ok) {
    if (ll_load(w, tag, v0, v1) || !ok) return;
    const unsigned long long t0 = clock64();
    while (!ll_load(w, tag, v0, v1))
        if (clock64() - t0 > RES_WAIT_CYCLES) {
            ok = false;
            return;
        }
}

// update_node's arithmetic and order on shared-memory states (component
// stride NS): F the node's UPML flux, A and L its Lorentz/Drude states.
template <bool H, int FEAT, bool GEO, int NS>
__device__ __forceinline__ void res_update(const DevGrid& g, float fld[3], const float curl[3], uint32_t t, float* F,
                                           float* A, float* L, int numTS, const GeoF& gf) {
    const DevHalf& T = H ? g.h : g.e;
    const float4 ta = __ldg(&T.main[TAB_MAIN * t]);
    const float4 tb = __ldg(&T.main[TAB_MAIN * t + 1]);
    const float c1[3] = {ta.x, ta.y, ta.z};
    float c2[3] = {ta.w, tb.x, tb.y};
    const uint32_t flags = __float_as_uint(tb.z);
    float ade[3];
    if ((FEAT & FEAT_ADE) && (flags & TF_ADE)) {
        const float4 a0 = __ldg(&T.ade[TAB_ADE * t]);
        const float4 a1 = __ldg(&T.ade[TAB_ADE * t + 1]);
        const float4 a2 = __ldg(&T.ade[TAB_ADE * t + 2]);
        const float kint[3] = {a0.x, a0.y, a0.z};
        const float kext[3] = {a0.w, a1.x, a1.y};
        const float klor[3] = {a1.z, a1.w, a2.x};
#pragma unroll
        for (int n = 0; n < 3; ++n) {
            float a = A[n * NS], f = fld[n];
            if ((FEAT & RES_LOR) && (flags & TF_LOR)) {
                const float l = __fadd_rn(L[n * NS], __fmul_rn(klor[n], a));
                L[n * NS] = l;
                f = __fsub_rn(f, l);
            }
            a = __fadd_rn(__fmul_rn(a, kint[n]), __fmul_rn(kext[n], f));
            A[n * NS] = a;
            ade[n] = a;
        }
    }
#pragma unroll
    for (int n = 0; n < 3; ++n) {
        if (GEO) c2[n] = __fmul_rn(__fmul_rn(__fmul_rn(c2[n], gf.f[n][0]), gf.f[n][1]), gf.f[n][2]);
        c2[n] = __fmul_rn(c2[n], curl[n]);
    }
    if ((FEAT & FEAT_UPML) && (flags & TF_UPML)) {
        const float4 u0 = __ldg(&T.upml[TAB_UPML * t]);
        const float4 u1 = __ldg(&T.upml[TAB_UPML * t + 1]);
        const float4 u2 = __ldg(&T.upml[TAB_UPML * t + 2]);
        const float kp[3] = {u0.x, u0.y, u0.z};
        const float kfo[3] = {u0.w, u1.x, u1.y};
        const float kfn[3] = {u1.z, u1.w, u2.x};
#pragma unroll
        for (int n = 0; n < 3; ++n) {
            const float f0 = F[n * NS];
            const float f = __fsub_rn(__fmul_rn(kp[n], fld[n]), __fmul_rn(kfo[n], f0));
            const float Fn = __fadd_rn(__fmul_rn(f0, c1[n]), c2[n]);
            F[n * NS] = Fn;
            fld[n] = __fadd_rn(f, __fmul_rn(kfn[n], Fn));
        }
    } else {
#pragma unroll
        for (int n = 0; n < 3; ++n) fld[n] = __fadd_rn(__fmul_rn(fld[n], c1[n]), c2[n]);
    }
    if ((FEAT & FEAT_ADE) && (flags & TF_ADE)) {
#pragma unroll
        for (int n = 0; n < 3; ++n) fld[n] = __fsub_rn(fld[n], ade[n]);
    }
    if (flags & TF_EXC) excite_node<H>(g, fld, t, numTS);
}

// Engine_Ext_Mur_ABC on the faces of one box: the three passes of k_mur on
// the voltages in shared memory.  Both lines of a face lie in the box (the
// plan cuts no axis with a Mur face into boxes of one line).  Everything that
// does not change is put into a list once, so a pass is a few instructions
// per face node; the same thread takes a node in every pass.
//   node: .x = slot on the face | slot of the next line << 13 | normal axis
//              << 26 | face << 28 | counts as zero << 31
//         .y = earlier faces that would write component n+1 (6 bits), n+2 (6
//              bits), excitation << 12, tuple << 16
//   val: {cp, cpp, bp, bpp}
template <int NS>
struct ResMur {
    float* sV;
    uint2* node;
    float4* val;
    int count;  // of this box

    __device__ __forceinline__ void init(const DevGrid& g, const MurSet& ms, float* v, const uint16_t* sE, float4* vals,
                                         uint2* nodes, int lx, int ly, int lz, int bx, int by, int bz) {
        sV = v;
        val = vals;
        node = nodes;
        count = 0;
        const int Nl[3] = {g.Nx - 1, g.Ny - 1, g.Nz - 1};
        for (int fi = 0; fi < ms.nface; ++fi) {
            const MurDev F = ms.f[fi];
            const int ny = F.ny;
            const int l0 = ny == 0 ? lx : ny == 1 ? ly : lz, n0 = ny == 0 ? bx : ny == 1 ? by : bz;  // along the normal
            const int lP = ny == 0 ? ly : ny == 1 ? lz : lx, nP = ny == 0 ? by : ny == 1 ? bz : bx;
            const int lQ = ny == 0 ? lz : ny == 1 ? lx : ly, nQ = ny == 0 ? bz : ny == 1 ? bx : by;
            if (F.line < l0 || F.line >= l0 + n0) continue;
            for (int q = threadIdx.x; q < nP * nQ; q += blockDim.x) {
                const int i = q / nQ, j = q - i * nQ;
                auto slot = [&](int line) {
                    const int x = ny == 0 ? line : ny == 1 ? j : i, y = ny == 0 ? i : ny == 1 ? line : j,
                              z = ny == 0 ? j : ny == 1 ? i : line;
                    return (uint32_t)((x * by + y) * bz + z);
                };
                const uint32_t ol = slot(F.line - l0), os = slot(F.shift - l0);
                const int X = ny == 0 ? F.line : ny == 1 ? j + lx : i + lx, Y = ny == 0 ? i + ly : ny == 1 ? F.line : j + ly,
                          Z = ny == 0 ? j + lz : ny == 1 ? i + lz : F.line;
                uint32_t m1 = 0, m2 = 0;
                for (int e = 0; e < fi; ++e) {
                    const int gn = ms.f[e].ny, p = gn == 0 ? X : gn == 1 ? Y : Z;
                    if (p != ms.f[e].line) continue;
                    if (gn != (ny + 1) % 3) m1 |= 1u << e;
                    if (gn != (ny + 2) % 3) m2 |= 1u << e;
                }
                // a last line that the voltage update leaves out counts as zero
                const int P = ny == 0 ? 1 : ny == 1 ? 2 : 0, Q = ny == 0 ? 2 : ny == 1 ? 0 : 1;
                const bool inert = (ms.trim[P] && i + lP == Nl[P]) || (ms.trim[Q] && j + lQ == Nl[Q]);
                const uint32_t t = sE[ol];
                const bool exc = __float_as_uint(__ldg(&g.e.main[TAB_MAIN * t + 1]).z) & TF_EXC;
                const int loc = (i + lP) * F.n1 + j + lQ;
                node[count + q] = make_uint2(ol | os << 13 | (uint32_t)ny << 26 | (uint32_t)fi << 28 | (inert ? 1u << 31 : 0u),
                                             m1 | m2 << 6 | (exc ? 1u << 12 : 0u) | t << 16);
                val[count + q] = make_float4(F.cp[loc], F.cpp[loc], 0.f, 0.f);
            }
            count += nP * nQ;
        }
    }
    // faces that act at numTS ts
    static __device__ __forceinline__ uint32_t active(const MurSet& ms, int ts) {
        uint32_t m = 0;
        for (int fi = 0; fi < ms.nface; ++fi) m |= ts >= ms.f[fi].start_ts ? 1u << fi : 0u;
        return m;
    }
    static __device__ __forceinline__ int comp(int n) { return n >= 3 ? (n - 3) * NS : n * NS; }
    __device__ __forceinline__ void pre(uint32_t act) const {
        for (int q = threadIdx.x; q < count; q += blockDim.x) {
            const uint32_t e = node[q].x;
            if (!(act >> (e >> 28 & 7u) & 1u)) continue;
            const int ol = e & 8191u, os = e >> 13 & 8191u, ny = e >> 26 & 3u;
            const float* vP = sV + comp(ny + 1);
            const float* vQ = sV + comp(ny + 2);
            float4 w = val[q];
            w.z = __fsub_rn(vP[os], __fmul_rn(w.x, vP[ol]));
            w.w = __fsub_rn(vQ[os], __fmul_rn(w.y, vQ[ol]));
            val[q] = w;
        }
    }
    __device__ __forceinline__ void post(uint32_t act) const {
        for (int q = threadIdx.x; q < count; q += blockDim.x) {
            const uint32_t e = node[q].x;
            if (!(act >> (e >> 28 & 7u) & 1u)) continue;
            const int os = e >> 13 & 8191u, ny = e >> 26 & 3u;
            const bool zero = e >> 31;
            float4 w = val[q];
            w.z = __fadd_rn(w.z, __fmul_rn(w.x, zero ? 0.f : sV[comp(ny + 1) + os]));
            w.w = __fadd_rn(w.w, __fmul_rn(w.y, zero ? 0.f : sV[comp(ny + 2) + os]));
            val[q] = w;
        }
    }
    __device__ __forceinline__ void apply(const DevGrid& g, uint32_t act, int ts) const {
        for (int q = threadIdx.x; q < count; q += blockDim.x) {
            const uint2 e = node[q];
            if (!(act >> (e.x >> 28 & 7u) & 1u)) continue;
            const int ol = e.x & 8191u, ny = e.x >> 26 & 3u;
            const float4 w = val[q];
            float v1 = w.z, v2 = w.w;
            if (e.y & 1u << 12) {
                float v[3] = {ny == 0 ? 0.f : ny == 1 ? v2 : v1, ny == 0 ? v1 : ny == 1 ? 0.f : v2,
                              ny == 0 ? v2 : ny == 1 ? v1 : 0.f};
                excite_node<false>(g, v, e.y >> 16, ts);
                v1 = ny == 0 ? v[1] : ny == 1 ? v[2] : v[0];
                v2 = ny == 0 ? v[2] : ny == 1 ? v[0] : v[1];
            }
            if (!(e.y & act & 63u)) sV[comp(ny + 1) + ol] = v1;
            if (!(e.y >> 6 & act & 63u)) sV[comp(ny + 2) + ol] = v2;
        }
    }
};

// LATE: the grid has Mur faces or lumped RLC edges.
template <int NS, int FEAT, bool GEO, bool LATE>
__global__ void __launch_bounds__(RES_THREADS) k_resident(const DevGrid g, const ResArgs a, const ProbeSet ps) {
    extern __shared__ __align__(16) float sm[];
    __shared__ int s_nent, s_nrlc;
    constexpr bool UPML = (FEAT & FEAT_UPML) != 0, ADE = (FEAT & FEAT_ADE) != 0, LOR = (FEAT & RES_LOR) != 0;
    constexpr int NF = res_comps(FEAT), OA = UPML ? 12 : 6;
    float* const sV = sm;
    float* const sI = sm + 3 * NS;
    float* const sFV = sm + 6 * NS;         // UPML only
    float* const sFI = sm + 9 * NS;
    float* const sAV = sm + OA * NS;        // Lorentz/Drude only
    float* const sAI = sm + (OA + 3) * NS;
    float* const sLV = sm + (OA + 6) * NS;  // Lorentz only
    float* const sLI = sm + (OA + 9) * NS;
    uint16_t* const sE = reinterpret_cast<uint16_t*>(sm + NF * NS);
    uint16_t* const sH = sE + NS;
    uint4* const tabE = reinterpret_cast<uint4*>(sm + (NF + 1) * NS);
    uint4* const tabH = tabE + RES_TASKS;
    uint2* const ent = reinterpret_cast<uint2*>(tabH + RES_TASKS);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const int iz = blockIdx.x % a.p[2], iy = (blockIdx.x / a.p[2]) % a.p[1], ix = blockIdx.x / (a.p[2] * a.p[1]);
    const int lx = res_cut(a.cov[0], a.p[0], ix), bx = res_cut(a.cov[0], a.p[0], ix + 1) - lx;
    const int ly = res_cut(a.cov[1], a.p[1], iy), by = res_cut(a.cov[1], a.p[1], iy + 1) - ly;
    const int lz = res_cut_z(a.cov[2], a.p[2], iz), bz = res_cut_z(a.cov[2], a.p[2], iz + 1) - lz;
    const int plane = by * bz;
    const int nzc = (bz + 31) / 32, rows = bx * by, ntask = rows * nzc;
    const long long C = g.comp;
    const long long g0 = (long long)lx * g.sx + (long long)ly * g.Nzp + lz;

    // The tasks that need no neighbour box come first: what the others wait
    // for travels meanwhile.  A thread places each task by counting.
    if (tid == 0) s_nent = s_nrlc = 0;
    auto edgeE = [&](int x, int y, int zc) {
        return (x == 0 && ix > 0) || (y == 0 && iy > 0) || (zc == 0 && iz > 0);
    };
    auto edgeH = [&](int x, int y, int zc) {  // beyond the last box lies at most a line that never changes
        return (x + 1 == bx && lx + bx < g.Nx) || (y + 1 == by && ly + by < g.Ny) ||
               (zc + 1 == nzc && lz + bz < g.Nz);
    };
    // tasks of each kind along z for rows without and with an edge in x or y
    const int freeE = nzc - (iz > 0 ? 1 : 0), freeH = nzc - (lz + bz < g.Nz ? 1 : 0);
    const int rowsE = (bx - (ix > 0 ? 1 : 0)) * (by - (iy > 0 ? 1 : 0));
    const int rowsH = (bx - (lx + bx < g.Nx ? 1 : 0)) * (by - (ly + by < g.Ny ? 1 : 0));
    const int ninE = rowsE * freeE, ninH = rowsH * freeH;
    for (int r = tid; r < rows; r += blockDim.x) {
        const int x = r / by, y = r - x * by;
        // rows without an edge before this one
        const int xe = ix > 0 ? 1 : 0, ye = iy > 0 ? 1 : 0;
        const int fE = max(0, x - xe) * (by - ye) + (x >= xe ? max(0, y - ye) : 0);
        const int xh = bx - (lx + bx < g.Nx ? 1 : 0), yh = by - (ly + by < g.Ny ? 1 : 0);
        const int fH = min(x, xh) * yh + (x < xh ? min(y, yh) : 0);
        int inE = fE * freeE, outE = ninE + r * nzc - inE;
        int inH = fH * freeH, outH = ninH + r * nzc - inH;
        for (int zc = 0; zc < nzc; ++zc) {
            const int z = zc * 32;
            const uint32_t o = (uint32_t)(r * bz + z), go = (uint32_t)(x * g.sx + (long long)y * g.Nzp + z);
            tabE[edgeE(x, y, zc) ? outE++ : inE++] =
                make_uint4(o | (x > 0 ? RT_X : 0u) | (y > 0 ? RT_Y : 0u) | (z > 0 ? RT_Z : 0u) |
                               (lx + x < a.ne[0] && ly + y < a.ne[1] ? RT_ROW : 0u), go,
                           (uint32_t)(x | y << 16), (uint32_t)z);
            tabH[edgeH(x, y, zc) ? outH++ : inH++] =
                make_uint4(o | (x + 1 < bx ? RT_X : 0u) | (y + 1 < by ? RT_Y : 0u) |
                               (lx + x < g.Nx - 1 && ly + y < g.Ny - 1 ? RT_ROW : 0u),
                           go, (uint32_t)(x | y << 16), (uint32_t)z);
        }
    }
    for (int r = warp; r < rows; r += nwarps) {
        const int x = r / by, y = r - x * by;
        const long long go = g0 + (long long)x * g.sx + (long long)y * g.Nzp;
        for (int z = lane; z < bz; z += 32) {
            const int o = r * bz + z;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                sV[c * NS + o] = g.V[c * C + go + z];
                sI[c * NS + o] = g.I[c * C + go + z];
                if (UPML) {
                    sFV[c * NS + o] = g.FV[c * C + go + z];
                    sFI[c * NS + o] = g.FI[c * C + go + z];
                }
                if (ADE) {
                    if (g.AV) sAV[c * NS + o] = g.AV[c * C + go + z];
                    if (LOR && g.LV) sLV[c * NS + o] = g.LV[c * C + go + z];
                    if (g.AI) sAI[c * NS + o] = g.AI[c * C + go + z];
                    if (LOR && g.LI) sLI[c * NS + o] = g.LI[c * C + go + z];
                }
            }
            sE[o] = (uint16_t)load_idx<uint16_t>(g.e.idx, go + z);
            sH[o] = (uint16_t)load_idx<uint16_t>(g.h.idx, go + z);
        }
    }
    __syncthreads();
    for (int k = tid; k < a.nentry; k += blockDim.x) {  // the probe entries in this box
        const ProbeEntry pe = ps.entries[k];
        const int X = (int)(pe.off / g.sx);
        const int rem = (int)(pe.off - (long long)X * g.sx);
        const int Y = rem / g.Nzp, Z = rem - Y * g.Nzp;
        if (X >= a.cov[0] || Y >= a.cov[1] || Z >= a.cov[2]) {
            // on a line that no box covers: no timestep changes it, so the
            // first block writes its value for every sample of the run
            if (blockIdx.x == 0) {
                const float v = (pe.field ? g.I : g.V)[pe.comp * C + pe.off];
                const int ns = a.interval > 0 ? (a.ts0 + a.nsteps) / a.interval - a.ts0 / a.interval : 0;
                const int nf = a.fd_interval > 0 ? (a.ts0 + a.nsteps) / a.fd_interval - a.ts0 / a.fd_interval : 0;
                for (int m = 0; m < ns; ++m) a.pval[(long long)m * a.nentry + k] = v;
                for (int m = 0; m < nf; ++m) a.fdval[(long long)m * a.nentry + k] = v;
            }
            continue;
        }
        const int x = X - lx, y = Y - ly, z = Z - lz;
        if (x < 0 || x >= bx || y < 0 || y >= by || z < 0 || z >= bz) continue;
        ent[atomicAdd(&s_nent, 1)] =
            make_uint2((uint32_t)k, (uint32_t)(((pe.field ? 3 : 0) + pe.comp) * NS + (x * by + y) * bz + z));
    }
    __syncthreads();
    // Exchange pairs of one field and parity: x cuts [cut][y][z], then y cuts
    // [cut][x][z], then z cuts [cut][x][y].  Bases of this box at its low
    // and high cuts (unused where there is none).
    const int oY = (a.p[0] - 1) * a.cov[1] * a.cov[2], oZ = oY + (a.p[1] - 1) * a.cov[0] * a.cov[2];
    const int xl = ((ix - 1) * a.cov[1] + ly) * a.cov[2] + lz, xh = xl + a.cov[1] * a.cov[2];
    const int yl = oY + ((iy - 1) * a.cov[0] + lx) * a.cov[2] + lz, yh = yl + a.cov[0] * a.cov[2];
    const int zl = oZ + ((iz - 1) * a.cov[0] + lx) * a.cov[1] + ly, zh = zl + a.cov[0] * a.cov[1];
    const bool hasx = ix + 1 < a.p[0], hasy = iy + 1 < a.p[1], hasz = iz + 1 < a.p[2];
    const int zE = min(bz, a.ne[2] - lz), zH = min(bz, g.Nz - 1 - lz);  // nodes of a row each half-step updates

    auto send_volt = [&](const uint4 e, int z, float v0, float v1, float v2, ulonglong2* llV, uint32_t tag) {
        const int x = (int)(e.z & 0xffffu), y = (int)(e.z >> 16);
        if (x == 0 && ix > 0) ll_send(llV + (xl + y * a.cov[2] + z), v1, v2, tag);
        if (y == 0 && iy > 0) ll_send(llV + (yl + x * a.cov[2] + z), v0, v2, tag);
        if (z == 0 && iz > 0) ll_send(llV + (zl + x * a.cov[1] + y), v0, v1, tag);
    };
    // passes after the voltage update, in boxes that have any
    ResMur<NS> mur;
    uint2* const rlc = reinterpret_cast<uint2*>(ent + RES_ENTRIES);  // {edge, slot of its voltage}
    bool late = false;
    if (LATE) {
        uint2* const nodes = rlc + RES_RLC;
        mur.init(g, a.mur, sV, sE, reinterpret_cast<float4*>(nodes + RES_MUR), nodes, lx, ly, lz, bx, by, bz);
        for (uint32_t q = tid; q < a.rlc.count; q += blockDim.x) {
            const long long off = a.rlc.off[q];
            const int c = (int)(off / C), r = (int)((off - c * C) % g.sx);
            const int x = (int)((off - c * C) / g.sx) - lx, y = r / g.Nzp - ly, z = r % g.Nzp - lz;
            if (x < 0 || x >= bx || y < 0 || y >= by || z < 0 || z >= bz) continue;
            rlc[atomicAdd(&s_nrlc, 1)] = make_uint2(q, (uint32_t)(c * NS + (x * by + y) * bz + z));
        }
        __syncthreads();
        late = mur.count || s_nrlc;
        mur.pre(mur.active(a.mur, a.ts0));
        __syncthreads();
    }

    bool ok = true;
    int samples = 0, fds = 0;
    for (int k = 0; k < a.nsteps; ++k) {
        const int ts = a.ts0 + k;
        const uint32_t tag = a.tag0 + (uint32_t)k + 1u;  // of this timestep's new values
        ulonglong2* llV = a.ll + (long long)(tag & 1u) * a.ll_pairs;
        ulonglong2* llI = a.ll + (long long)(2u + (tag & 1u)) * a.ll_pairs;
        const ulonglong2* llJ = a.ll + (long long)(2u + ((tag & 1u) ^ 1u)) * a.ll_pairs;  // old currents
        // ------------------------------------------------------- voltages
        auto volt = [&](auto edge, const uint4 e) {
            constexpr bool EDGE = decltype(edge)::value;
            const int z = (int)e.w + lane;
            if (z >= bz) return;
            const int o = (int)(e.x & 0xffffu) + lane;
            const int ox = o - ((e.x & RT_X) ? plane : 0), oy = o - ((e.x & RT_Y) ? bz : 0),
                      oz = o - ((lane > 0 || (e.x & RT_Z)) ? 1 : 0);
            const uint32_t tu = sE[o];
            const float c0 = sI[o], c1 = sI[NS + o], c2 = sI[2 * NS + o];
            // at the domain's wall the neighbour is the node itself
            float i1xm = sI[NS + ox], i2xm = sI[2 * NS + ox];
            float i0ym = sI[oy], i2ym = sI[2 * NS + oy];
            float i0zm = sI[oz], i1zm = sI[NS + oz];
            float v[3] = {sV[o], sV[NS + o], sV[2 * NS + o]};
            const long long go = g0 + e.y + lane;
            if (EDGE) {
                const int x = (int)(e.z & 0xffffu), y = (int)(e.z >> 16);
                const bool nx = x == 0 && ix > 0, ny = y == 0 && iy > 0, nz = z == 0 && iz > 0;
                if (k == 0) {  // the currents of the run's start
                    if (nx) {
                        i1xm = g.I[C + go - g.sx];
                        i2xm = g.I[2 * C + go - g.sx];
                    }
                    if (ny) {
                        i0ym = g.I[go - g.Nzp];
                        i2ym = g.I[2 * C + go - g.Nzp];
                    }
                    if (nz) {
                        i0zm = g.I[go - 1];
                        i1zm = g.I[C + go - 1];
                    }
                } else {
                    if (nx) ll_wait(llJ + (xl + y * a.cov[2] + z), tag - 1u, i1xm, i2xm, ok);
                    if (ny) ll_wait(llJ + (yl + x * a.cov[2] + z), tag - 1u, i0ym, i2ym, ok);
                    if (nz) ll_wait(llJ + (zl + x * a.cov[1] + y), tag - 1u, i0zm, i1zm, ok);
                }
            }
            if (z < zE && (e.x & RT_ROW)) {
            float curl[3];
            curl[0] = __fadd_rn(__fsub_rn(__fsub_rn(c2, i2ym), c1), i1zm);
            curl[1] = __fadd_rn(__fsub_rn(__fsub_rn(c0, i0zm), c2), i2xm);
            curl[2] = __fadd_rn(__fsub_rn(__fsub_rn(c1, i1xm), c0), i0ym);
            GeoF gf;
            if (GEO) gf = geo_factors(g, false, lx + (int)(e.z & 0xffffu), ly + (int)(e.z >> 16), lz + z);
            res_update<false, FEAT, GEO, NS>(g, v, curl, tu, sFV + o, sAV + o, sLV + o, ts, gf);
            sV[o] = v[0];
            sV[NS + o] = v[1];
            sV[2 * NS + o] = v[2];
            }
            if (EDGE && !(LATE && late)) send_volt(e, z, v[0], v[1], v[2], llV, tag);
        };
        int t = warp;
        for (; t < ninE; t += nwarps) volt(std::false_type{}, tabE[t]);
        for (; t < ntask; t += nwarps) volt(std::true_type{}, tabE[t]);
        if (__syncthreads_or(!ok)) break;
        if (LATE && late) {
            // the hooks around the voltage update in the reference's order:
            // Mur post-update, lumped RLC, Mur apply; then the new voltages go out
            const uint32_t act = mur.active(a.mur, ts);
            mur.post(act);
            __syncthreads();
            if (s_nrlc) {
                for (int q = tid; q < s_nrlc; q += blockDim.x) sm[rlc[q].y] = rlc_edge(a.rlc, rlc[q].x, ts, sm[rlc[q].y]);
                __syncthreads();
            }
            mur.apply(g, act, ts);
            __syncthreads();
            for (int q = ninE + warp; q < ntask; q += nwarps) {
                const uint4 e = tabE[q];
                const int z = (int)e.w + lane, o = (int)(e.x & 0xffffu) + lane;
                if (z < bz) send_volt(e, z, sV[o], sV[NS + o], sV[2 * NS + o], llV, tag);
            }
        }
        // ------------------------------------------------------- currents
        const bool sample = a.interval > 0 && (ts + 1) % a.interval == 0;
        auto curr = [&](auto edge, const uint4 e) {
            constexpr bool EDGE = decltype(edge)::value;
            const int z = (int)e.w + lane;
            const int o = min((int)(e.x & 0xffffu) + lane, NS - 1);
            const bool act = z < zH && (e.x & RT_ROW);
            float c0 = 0.f, c1 = 0.f, c2 = 0.f, cu[3] = {0.f, 0.f, 0.f};
            if (act) {
                const int ox = o + ((e.x & RT_X) ? plane : 0), oy = o + ((e.x & RT_Y) ? bz : 0),
                          oz = o + (z + 1 < bz ? 1 : 0);
                const uint32_t tu = sH[o];
                c0 = sV[o];
                c1 = sV[NS + o];
                c2 = sV[2 * NS + o];
                float v1xp = sV[NS + ox], v2xp = sV[2 * NS + ox];
                float v0yp = sV[oy], v2yp = sV[2 * NS + oy];
                float v0zp = sV[oz], v1zp = sV[NS + oz];
                cu[0] = sI[o];
                cu[1] = sI[NS + o];
                cu[2] = sI[2 * NS + o];
                const long long go = g0 + e.y + lane;
                if (EDGE) {
                    const int x = (int)(e.z & 0xffffu), y = (int)(e.z >> 16);
                    // beyond the boxes: the last line, which no timestep changes
                    if (x + 1 == bx) {
                        if (hasx) {
                            ll_wait(llV + (xh + y * a.cov[2] + z), tag, v1xp, v2xp, ok);
                        } else {
                            v1xp = g.V[C + go + g.sx];
                            v2xp = g.V[2 * C + go + g.sx];
                        }
                    }
                    if (y + 1 == by) {
                        if (hasy) {
                            ll_wait(llV + (yh + x * a.cov[2] + z), tag, v0yp, v2yp, ok);
                        } else {
                            v0yp = g.V[go + g.Nzp];
                            v2yp = g.V[2 * C + go + g.Nzp];
                        }
                    }
                    if (z + 1 == bz) {
                        if (hasz) {
                            ll_wait(llV + (zh + x * a.cov[1] + y), tag, v0zp, v1zp, ok);
                        } else {
                            v0zp = g.V[go + 1];
                            v1zp = g.V[C + go + 1];
                        }
                    }
                }
                float curl[3];
                curl[0] = __fadd_rn(__fsub_rn(__fsub_rn(c2, v2yp), c1), v1zp);
                curl[1] = __fadd_rn(__fsub_rn(__fsub_rn(c0, v0zp), c2), v2xp);
                curl[2] = __fadd_rn(__fsub_rn(__fsub_rn(c1, v1xp), c0), v0yp);
                GeoF gf;
                if (GEO) gf = geo_factors(g, true, lx + (int)(e.z & 0xffffu), ly + (int)(e.z >> 16), lz + z);
                res_update<true, FEAT, GEO, NS>(g, cu, curl, tu, sFI + o, sAI + o, sLI + o, ts, gf);
                sI[o] = cu[0];
                sI[NS + o] = cu[1];
                sI[2 * NS + o] = cu[2];
            }
            if (EDGE && z < bz) {
                const int x = (int)(e.z & 0xffffu), y = (int)(e.z >> 16);
                const float s0 = sI[o], s1 = sI[NS + o], s2 = sI[2 * NS + o];  // the old value where nothing changes
                if (x + 1 == bx && hasx) ll_send(llI + (xh + y * a.cov[2] + z), s1, s2, tag);
                if (y + 1 == by && hasy) ll_send(llI + (yh + x * a.cov[2] + z), s0, s2, tag);
                if (z + 1 == bz && hasz) ll_send(llI + (zh + x * a.cov[1] + y), s0, s1, tag);
            }
            if (sample && a.eseg) {
                const int X = lx + (int)(e.z & 0xffffu), Y = ly + (int)(e.z >> 16), Z = lz + (int)e.w;
                energy_segment_to(a.eseg + samples * a.seg_stride, g, X, Y, Z >> 5, act,
                                  (e.x & RT_ROW) && Z < g.Nz - 1, c0, c1, c2, cu[0], cu[1], cu[2]);
            }
        };
        t = warp;
        for (; t < ninH; t += nwarps) curr(std::false_type{}, tabH[t]);
        for (; t < ntask; t += nwarps) curr(std::true_type{}, tabH[t]);
        // the next timestep's Mur pre-update: the voltages stay as they are until then
        if (LATE && late && k + 1 < a.nsteps) mur.pre(mur.active(a.mur, ts + 1));
        if (__syncthreads_or(!ok)) break;
        const bool fd = a.fd_interval > 0 && (ts + 1) % a.fd_interval == 0;
        if (sample || fd) {
            for (int j = tid; j < s_nent; j += blockDim.x) {
                const uint2 en = ent[j];
                if (sample) a.pval[(long long)samples * a.nentry + en.x] = sm[en.y];
                if (fd) a.fdval[(long long)fds * a.nentry + en.x] = sm[en.y];
            }
            samples += sample ? 1 : 0;
            fds += fd ? 1 : 0;
            __syncthreads();
        }
    }
    if (!ok) atomicOr(a.d_err, 8);
    for (int r = warp; r < rows; r += nwarps) {
        const int x = r / by, y = r - x * by;
        const long long go = g0 + (long long)x * g.sx + (long long)y * g.Nzp;
        for (int z = lane; z < bz; z += 32) {
            const int o = r * bz + z;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                g.V[c * C + go + z] = sV[c * NS + o];
                g.I[c * C + go + z] = sI[c * NS + o];
                if (UPML) {
                    g.FV[c * C + go + z] = sFV[c * NS + o];
                    g.FI[c * C + go + z] = sFI[c * NS + o];
                }
                if (ADE) {
                    if (g.AV) g.AV[c * C + go + z] = sAV[c * NS + o];
                    if (LOR && g.LV) g.LV[c * C + go + z] = sLV[c * NS + o];
                    if (g.AI) g.AI[c * C + go + z] = sAI[c * NS + o];
                    if (LOR && g.LI) g.LI[c * C + go + z] = sLI[c * NS + o];
                }
            }
        }
    }
}

// ------------------------------------------------- samples of a resident run
// Plane sums of the energy segments: block (x, m) sums plane x of sample m.
static __global__ void __launch_bounds__(256) k_resident_planes(const DevGrid g, const float2* eseg,
                                                                long long seg_stride, double2* eplane) {
    DevGrid s = g;
    s.eseg = const_cast<float2*>(eseg) + blockIdx.y * seg_stride;
    const double2 r = plane_energy(s, blockIdx.x);
    if (threadIdx.x == 0) eplane[(long long)blockIdx.y * (g.Nx - 1) + blockIdx.x] = r;
}

// Block m records sample m of the run (as advance_sample records one); the
// last block to finish moves the counters.  `count` samples, one block at
// least (a run without samples only moves numTS).
static __global__ void __launch_bounds__(256) k_resident_samples(int* d_ts, int steps, int count, int first_ts,
                                                                 int interval, ProbeSet ps, const DevGrid g,
                                                                 const float* pval, int nentry, const double2* eplane,
                                                                 int energy_valid, unsigned* ticket, double eps0,
                                                                 double mue0) {
    const int m = blockIdx.x, tid = threadIdx.x;
    if (m < count) {
        const int row = *ps.d_nsamp + m;
        if (row < ps.cap) {
            double* rec = ps.ring + (long long)row * ps.row_doubles;
            ProbeSet q = ps;
            q.vals = pval + (long long)m * nentry;
            for (int p = tid >> 5; p < ps.nprobe; p += 8) {
                const double acc = probe_value(q, g, p, 0, tid & 31);
                if ((tid & 31) == 0) rec[2 + p] = acc * ps.weight[p];
            }
            DevGrid s = g;
            s.eplane = const_cast<double2*>(eplane) + (long long)m * (g.Nx - 1);
            const double2 sum = energy_valid ? total_energy(s) : make_double2(0.0, 0.0);
            if (tid == 0) {
                rec[0] = (double)(first_ts + m * interval);
                rec[1] = -1.0;
                if (energy_valid) {
                    const double e = eps0 * sum.x + mue0 * sum.y;
                    if (!isfinite(e)) atomicOr(ps.d_err, 2);
                    rec[1] = e;
                }
            }
        } else if (tid == 0) {
            atomicOr(ps.d_err, 1);
        }
    }
    if (!last_block(ticket, gridDim.x)) return;
    if (tid == 0) {
        *d_ts += steps;
        *ps.d_nsamp = min(*ps.d_nsamp + count, ps.cap);
    }
}

}  // namespace wipems

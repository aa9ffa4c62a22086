// Fused 2D time steps of one shot: the GUI programs' VTI forward modelling
// (CPU_vti2dfd_kernels.c:79-177, GPU_vti2dfd_kernels.cu:209-299), the TTI
// program's (2D-tti-fd+rtm-cuda/Toa_gpu_2dtti_fd_1orderfunction.cu:81-183) and
// the passes of the 2D GPU RTM programs, VTI
// (Toa_gpu2DvtiFdRtmAdcigsLaplace.cu:256-404) and TTI
// (Toa_gpu_2dtti_rtm_adcigs_iorderfunciton.cu:126-228).
//
// A run of steps is one cooperative launch.  A block owns the same tiles, 64
// depths x TX columns, in every step; per tile P with seven columns, Q with
// eight depths, u and w with four either side, the split stresses and the
// model arrive as TMA boxes in shared memory, the next tile's while this one
// is worked on.  The velocities are rebuilt on the tile and on the four-cell
// halos the stresses read, in place in shared memory, then the stresses
// follow and the new level is stored.  One grid barrier a step: half of what
// two half-steps need, and a point costs about 110 B of L2 traffic against
// 250 when each half-step reads its taps there.  A thread owns two
// consecutive depths (one 8-byte vector), whose x taps share a sliding window
// of shared-memory loads.  Every wait is bounded.
//
// The blocks stay for the run because of the two L2 halves: launched anew
// each step, a tile lands on any SM, so on either half, and 93 MB of the
// 1700x601 + 50 shot's 80 MB of state and model moved through DRAM every step;
// with the same SM, 12 MB do (forward: 22.7 to 26 us a step launched per step,
// 17.1 here).  Odd steps walk the tiles backwards, so that what the step before
// left in L2 is read first: nothing forward, where all of it fits, and 41.7
// -> 39.1 us backward, where two sides (140 MB and the gathers) do not.
//
// Between two steps only one thread waits: it brings the first tile's own boxes
// (split stresses, model) before the barrier completes and the shared ones
// after, while the others load the profiles their tile needs and wait for the
// boxes (a barrier of the whole block, and profiles loaded where they are used
// -- an L2 round trip, since the acquire empties L1 -- cost a 101x121 shot 0.7 us
// a step and a 401x401 one 0.9).
//
// Measured against the kernels this replaces (half-steps of one persistent
// launch; tiles kept in shared memory with exchange copies where the grid
// fits that way), us a step: 2401x601 + 50 39.5 -> 18.0; 1200x601 25.0 -> 10.1;
// 600x601 10.9 -> 7.4; 401x401 7.4 -> 5.1; 101x121 + 20 5.4 -> 3.3; RTM program
// 1700x601 forward 26.1 -> 17.1, backward with 70 angles 56.3 -> 36.4.  TTI,
// whose rotated derivatives need both halos of every field (twice the velocity
// work of a tile of 8 columns, 1.6 times of 16): 600x300 11.5 -> 7.5; RTM
// program 1700x601, 65 angles, forward 37.3 -> 24.4, backward 74.0 -> 52.9.
// Large grids are bound by instruction issue (60 % of the slots at 24 warps per
// SM; 325 instructions a point with 8 columns, 200 with 16), small ones by the
// barrier and the TMA round trip.  Tried: four warps with two columns each
// (1.04 times forward, 1.3 backward), split stresses and model from L2 into
// registers instead of TMA (1.05 and 1.15), flags of the neighbours' blocks
// instead of the barrier (0.95 where a block has one tile, 1.3 where several).
//
// The backward pass of the RTM program takes the source side and the
// receiver side of a tile one after the other, the source side's new values
// waiting in registers for the image; the ring and the record of the next
// step of the run go into the new level as it is stored.
#include "step2d.cuh"
#include "adcig.cuh"
#include "gridsync.cuh"
#include "tc_util.cuh"
#include <algorithm>
#include <cmath>
#include <cstring>
#include <cudaTypedefs.h>

namespace geo {

__constant__ float cs_fd[4] = {1.196289f, -0.0797526f, 0.009570313f, -0.0006975447f};
__constant__ double cs_gauss[49];   // exp(-x^2-z^2) on the 7x7 source window
__constant__ float cs_thr[128];     // angle-bin thresholds (largest cosine of bins >= k)
__constant__ float cs_cos[128];     // cosf(ia*pi/180) per bin

namespace {

constexpr int kTz = 64, kThreads = 256;
constexpr int kQz = kTz + 16, kWz = kTz + 8;   // depths of a Q and a w box

// Boxes of a tile in a stage (floats): P, Q, u, w, the four split stresses,
// the three model arrays and, TTI, cos and sin of the tilt.  The rotated
// derivatives read every field along both axes, so TTI boxes have both halos.
template <bool TTI, int TX>
struct Box {
    static constexpr int zp = TTI ? kQz : kTz, zu = TTI ? kWz : kTz;      // depths of a P and a u box
    static constexpr int xq = TTI ? TX + 14 : TX, xw = TTI ? TX + 8 : TX; // columns of a Q and a w box
    static constexpr int hz = TTI ? 8 : 0, hu = TTI ? 4 : 0;              // depths above the tile in P and u
    static constexpr int hq = TTI ? 7 : 0, hw = TTI ? 4 : 0;              // columns left of it in Q and w
    static constexpr int q = (TX + 14) * zp, u = q + xq * kQz, w = u + (TX + 8) * zu, s = w + xw * kWz,
                         m = s + 4 * TX * kTz, t = m + 3 * TX * kTz, all = t + (TTI ? 2 * (TX + 8) * kWz : 0);
    static_assert(q % 32 == 0 && u % 32 == 0 && w % 32 == 0 && s % 32 == 0 && t % 32 == 0 && all % 32 == 0, "128-byte boxes");
};
constexpr size_t step_smem(int tx, int stages, bool tti) {
    return (size_t)stages * 4 *
           (tti ? (tx == 8 ? Box<true, 8>::all : Box<true, 16>::all) : tx == 8 ? Box<false, 8>::all : Box<false, 16>::all);
}

__device__ __forceinline__ float2 lds2(const float *p) { return *reinterpret_cast<const float2 *>(p); }
__device__ __forceinline__ void sts2(float *p, float2 v) { *reinterpret_cast<float2 *>(p) = v; }
__device__ __forceinline__ float2 ldg2(const float *p) { return __ldg(reinterpret_cast<const float2 *>(p)); }
__device__ __forceinline__ float &at2(float2 &v, int j) { return j ? v.y : v.x; }

// sum_m c_m (a_m - b_m), accumulated from 0 in the programs' order
__device__ __forceinline__ float d8(float a0, float b0, float a1, float b1, float a2, float b2, float a3, float b3) {
    float d = 0.0f;
    d += cs_fd[0] * (a0 - b0);
    d += cs_fd[1] * (a1 - b1);
    d += cs_fd[2] * (a2 - b2);
    d += cs_fd[3] * (a3 - b3);
    return d;
}
// over eight vectors a(-3) .. a(+4) (or a(-4) .. a(+3))
__device__ __forceinline__ float2 dx8(const float2 *q) {
    return make_float2(d8(q[4].x, q[3].x, q[5].x, q[2].x, q[6].x, q[1].x, q[7].x, q[0].x),
                       d8(q[4].y, q[3].y, q[5].y, q[2].y, q[6].y, q[1].y, q[7].y, q[0].y));
}
// along z at the pair p points to; SHIFT 1 forward, 0 backward stagger
template <int SHIFT>
__device__ __forceinline__ float2 dz8(const float *p) {
    float e[10];
#pragma unroll
    for (int k = 0; k < 5; k++) {
        const float2 t = lds2(p - 4 + 2 * k);
        e[2 * k] = t.x;
        e[2 * k + 1] = t.y;
    }
    const float *a = e + 4 + SHIFT, *b = a + 1;
    return make_float2(d8(a[0], a[-1], a[1], a[-2], a[2], a[-3], a[3], a[-4]),
                       d8(b[0], b[-1], b[1], b[-2], b[2], b[-3], b[3], b[-4]));
}

__device__ __forceinline__ void tma3(float *dst, const CUtensorMap *map, int z, int x, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::
            "r"(tc::su32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(z), "r"(x), "r"(0), "r"(tc::su32(bar))
        : "memory");
}

// Wait for the boxes: 2 s at most, 1 ms once a step has given up.
__device__ __forceinline__ bool boxes_here(uint64_t *bar, uint32_t parity, const int *err) {
    if (tc::mbar_wait(bar, parity, 1000000ull)) return true;
    return !*(const volatile int *)err && tc::mbar_wait(bar, parity);
}

// The TTI programs' velocity update (Toa_gpu_2dtti_fd_1orderfunction.cu:81-112)
// of a pair of points, in place; on: which of them are on the updated grid.
__device__ __forceinline__ void tti_vel(const SGrid &g, float c1, float c2, float2 cz1, float2 cz2, float2 ct, float2 sn, float2 Px, float2 Pz,
                                        float2 Qx, float2 Qz, bool on0, bool on1, float *pu, float *pw) {
    float2 u = lds2(pu), w = lds2(pw);
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const float C = at2(ct, j), S = at2(sn, j), k2 = c2 * at2(cz2, j), k1 = c1 * at2(cz1, j);
        const float un = k2 * at2(u, j) - k1 * (C * g.dtx * at2(Px, j) - S * g.dtz * at2(Pz, j));
        const float wn = k2 * at2(w, j) - k1 * (S * g.dtx * at2(Qx, j) + C * g.dtz * at2(Qz, j));
        if (j ? on1 : on0) {
            at2(u, j) = un;
            at2(w, j) = wn;
        }
    }
    sts2(pu, u);
    sts2(pw, w);
}

// Position in the ring of wavefield_bndr (:532), -1 off it.
__device__ __forceinline__ int ring_at(const SGrid &g, int ix, int iz) {
    const int n = g.npd;
    if (ix >= n && ix < n + g.nx) {
        if (iz == n - 1) return ix - n;
        if (iz == n + g.nz + 1) return g.nx + ix - n;
    }
    if (iz >= n && iz < n + g.nz) {
        if (ix == n - 1) return 2 * g.nx + iz - n;
        if (ix == n + g.nx + 1) return 2 * g.nx + g.nz + iz - n;
    }
    return -1;
}

struct Maps {
    SMaps m[2][2];   // side, level
    CUtensorMap model, trig;
};

template <int KIND, bool TTI, int NC>
__global__ void __launch_bounds__(kThreads, NC == 1 ? 3 : 2)
    k_step2d(const __grid_constant__ Maps tm, const __grid_constant__ SStep a, int ntiles, int stages) {
    constexpr int W = kThreads / 32, TX = W * NC;
    using B = Box<TTI, TX>;
    constexpr int SF = B::all;
    constexpr bool BWD = KIND == SK_GBWD;
    extern __shared__ __align__(128) float sm[];
    __shared__ __align__(8) uint64_t bar[2];
    __shared__ int s_abort;
    const SGrid &g = a.g;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ntz = (g.nnz + kTz - 1) / kTz, zl = 2 * lane, c0 = warp * NC, ldz = g.ldz;
    // this block's items of a step: its tiles, backward both sides of each,
    // one after the other
    const int nb = ((ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1) * (BWD ? 2 : 1);
    unsigned base = 0;   // items of the steps before
    const int step_z = (int)gridDim.x % ntz * kTz, step_x = (int)gridDim.x / ntz * TX;
    // boxes of item k: what other blocks do not write, and what they do
    auto fetch_own = [&](int k, int f, int z, int x) {
        const int st = (base + k) & (stages - 1);
        uint64_t *b = &bar[st];
        float *s = sm + st * SF;
        tc::mbar_expect_tx(b, SF * 4);
        tma3(s + B::s, &tm.m[f][0].S, z, x, b);
        tma3(s + B::m, &tm.model, z, x, b);
        if (TTI) tma3(s + B::t, &tm.trig, z - 4, x - 4, b);
    };
    auto fetch_shared = [&](int k, int f, int z, int x, int lev) {
        const int st = (base + k) & (stages - 1);
        uint64_t *b = &bar[st];
        float *s = sm + st * SF;
        const SMaps &m = tm.m[f][lev];
        tc::tma2(s, &m.P, z - B::hz, x - 7, b);
        tc::tma2(s + B::q, &m.Q, z - 8, x - B::hq, b);
        tc::tma2(s + B::u, &m.u, z - B::hu, x - 4, b);
        tc::tma2(s + B::w, &m.w, z - 4, x - B::hw, b);
    };
    auto fetch = [&](int k, int f, int z, int x, int lev) {
        fetch_own(k, f, z, x);
        fetch_shared(k, f, z, x, lev);
    };
    if (tid == 0) {
        for (int k = 0; k < stages; k++) tc::mbar_init(&bar[k], 1);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (ld_acquire_u32(reinterpret_cast<const unsigned *>(a.err))) return;   // an earlier run gave up
    __syncthreads();
    float2 sv[NC][4];   // source side's new P, Q, u, w, for the image
    const int steps = BWD ? a.it0 - a.it1 + 1 : a.it1 - a.it0;
    for (int s = 0; s < steps; s++, base += nb) {
        const int it = BWD ? a.it0 - s : a.it0 + s, lev = (a.lev + s) & 1, next = BWD && it > a.it1 ? it - 1 : -1;
        const bool src_on = BWD ? false : a.on[it] != 0;
        const float amp = BWD ? 0.0f : a.amp[it];
        const bool rev = s & 1;
        const int t_first = blockIdx.x + (rev ? (BWD ? nb / 2 - 1 : nb - 1) * gridDim.x : 0);
        const int z_first = t_first % ntz * kTz, x_first = t_first / ntz * TX;
        if (tid == 0) {   // the others wait for the boxes
            fetch_own(0, 0, z_first, x_first);
            if (s && !grid_wait(a.bar, (unsigned)s * gridDim.x, a.err)) {
                s_abort = 1;
            } else {
                // other blocks' stores of the step before, then TMA reads of them
                asm volatile("fence.proxy.async;" ::: "memory");
                fetch_shared(0, 0, z_first, x_first, lev);
            }
        }
        int z0 = z_first, x0 = x_first, zn = z0, xn = x0;   // this item's tile, the next item's
        for (int k = 0; k < nb; k++, z0 = zn, x0 = xn) {
            const int side = BWD ? k & 1 : 0, zo = z0 + zl;
            if (!BWD || side) {
                zn += rev ? -step_z : step_z;
                xn += rev ? -step_x : step_x;
                if (zn >= ntz * kTz) {
                    zn -= ntz * kTz;
                    xn += TX;
                }
                if (zn < 0) {
                    zn += ntz * kTz;
                    xn -= TX;
                }
            }
            if (k == 0 && stages > 1 && nb > 1 && tid == 0) fetch(1, BWD ? 1 : 0, zn, xn, lev);
            const bool ring = !(KIND == SK_GFWD || KIND == SK_GBWD) ? false :
                (z0 < g.npd && z0 + kTz >= g.npd) || (z0 <= g.npd + g.nz + 1 && z0 + kTz > g.npd + g.nz + 1) ||
                (x0 < g.npd && x0 + TX >= g.npd) || (x0 <= g.npd + g.nx + 1 && x0 + TX > g.npd + g.nx + 1);
            const int st = (base + k) & (stages - 1);
            float *sP = sm + st * SF, *sQ = sP + B::q, *sU = sP + B::u, *sW = sP + B::w;
            const float *sS = sP + B::s, *sM = sP + B::m, *sT = sP + B::t;
            const bool z0u = zo >= 4 && zo < g.nnz - 4, z1u = zo + 1 >= 4 && zo + 1 < g.nnz - 4;
            const int zc = min(zo, ldz - 2);   // profiles of the pair
            const float2 cz1 = ldg2(g.zp + zc), cz2 = ldg2(g.zp + ldz + zc), az1 = ldg2(g.zp + 2 * ldz + zc),
                         az2 = ldg2(g.zp + 3 * ldz + zc);
            constexpr int NU = (TX + 7 + W - 1) / W;   // columns of u a warp
            float cu1[NU], cu2[NU], ca1[NC], ca2[NC];
#pragma unroll
            for (int j = 0; j < NU; j++) {
                const int ix = min(max(x0 - 4 + warp * NU + j, 0), g.nnx - 1);
                cu1[j] = __ldg(g.cx1 + ix);
                cu2[j] = __ldg(g.cx2 + ix);
            }
#pragma unroll
            for (int c = 0; c < NC; c++) {
                const int ix = min(x0 + c0 + c, g.nnx - 1);
                ca1[c] = __ldg(g.ax1 + ix);
                ca2[c] = __ldg(g.ax2 + ix);
            }
            if (!boxes_here(&bar[st], ((base + k) >> (stages - 1)) & 1, a.err)) *(volatile int *)&s_abort = 1;
            if ((KIND == SK_GPU || KIND == SK_GFWD) && src_on) {
                // point source: P,Q += amp before the velocity update, on this
                // block's copies of the source cell
                const int px = a.ixs - (x0 - 7), pz = a.izs - (z0 - B::hz), qx = a.ixs - (x0 - B::hq), qz = a.izs - (z0 - 8);
                const bool inP = px >= 0 && px < TX + 14 && pz >= 0 && pz < B::zp, inQ = qx >= 0 && qx < B::xq && qz >= 0 && qz < kQz;
                if (inP || inQ) {
                    __syncthreads();
                    if (tid == 0 && inP) sP[px * B::zp + pz] += amp;
                    if (tid == 0 && inQ) sQ[qx * kQz + qz] += amp;
                    __syncthreads();
                }
            }
            float2 wn[NC];
            if constexpr (TTI) {
                // u and w at once, on the columns of the tile and its halos
                const int u0 = warp * NU;
                const float *pP = sP + B::hz + zl, *pQ = sQ + 8 + zl;
                float2 p[8], q[8];
#pragma unroll
                for (int j = 0; j < 7; j++) {
                    p[j + 1] = lds2(pP + min(u0 + j, TX + 13) * kQz);
                    q[j + 1] = lds2(pQ + min(u0 + j, TX + 13) * kQz);
                }
#pragma unroll
                for (int j = 0; j < NU; j++) {
                    const int uc = u0 + j, ix = x0 - 4 + uc, n = min(uc + 7, TX + 13) * kQz;
#pragma unroll
                    for (int m = 0; m < 7; m++) {
                        p[m] = p[m + 1];
                        q[m] = q[m + 1];
                    }
                    p[7] = lds2(pP + n);
                    q[7] = lds2(pQ + n);
                    if (uc < TX + 7 && ix >= 4 && ix < g.nnx - 4) {
                        const float2 Pz = dz8<1>(pP + (uc + 3) * kQz), Qz = dz8<1>(pQ + (uc + 3) * kQz);
                        tti_vel(g, cu1[j], cu2[j], cz1, cz2, lds2(sT + uc * kWz + zl + 4), lds2(sT + (TX + 8 + uc) * kWz + zl + 4), dx8(p),
                                Pz, dx8(q), Qz, z0u, z1u, sU + uc * kWz + zl + 4, sW + uc * kWz + zl + 4);
                    }
                }
                // and on the four depths above and below the tile's columns
                if (tid >= 32 * W - 4 * TX) {
                    const int col = (tid - 32 * W + 4 * TX) >> 2, k4 = tid & 3, zr = k4 < 2 ? 2 * k4 - 4 : kTz + 2 * (k4 - 2);
                    const int iz = z0 + zr, ix = x0 + col, i0 = min(max(iz, 0), ldz - 2);
                    const bool h0 = iz >= 4 && iz < g.nnz - 4, h1 = iz + 1 >= 4 && iz + 1 < g.nnz - 4;
                    if (ix >= 4 && ix < g.nnx - 4 && (h0 || h1)) {
                        const float *hP = sP + (col + 7) * kQz + zr + 8, *hQ = sQ + (col + 7) * kQz + zr + 8;
#pragma unroll
                        for (int m = 0; m < 8; m++) {
                            p[m] = lds2(hP + (m - 3) * kQz);
                            q[m] = lds2(hQ + (m - 3) * kQz);
                        }
                        const int uc = col + 4, z4 = zr + 4;
                        tti_vel(g, __ldg(g.cx1 + ix), __ldg(g.cx2 + ix), ldg2(g.zp + i0), ldg2(g.zp + ldz + i0), lds2(sT + uc * kWz + z4),
                                lds2(sT + (TX + 8 + uc) * kWz + z4), dx8(p), dz8<1>(hP), dx8(q), dz8<1>(hQ), h0, h1,
                                sU + uc * kWz + z4, sW + uc * kWz + z4);
                    }
                }
            } else {
                // u on the tile's columns and its halos: NU consecutive columns a
                // warp, column uc at x = x0 - 4 + uc, taps P box columns uc .. uc+7
                const int u0 = warp * NU;
                float2 pq[8];
#pragma unroll
                for (int j = 0; j < 7; j++) pq[j + 1] = lds2(sP + min(u0 + j, TX + 13) * kTz + zl);
#pragma unroll
                for (int j = 0; j < NU; j++) {
                    const int uc = u0 + j, ix = x0 - 4 + uc;
#pragma unroll
                    for (int m = 0; m < 7; m++) pq[m] = pq[m + 1];
                    pq[7] = lds2(sP + min(uc + 7, TX + 13) * kTz + zl);
                    if (uc < TX + 7 && ix >= 4 && ix < g.nnx - 4) {
                        const float c1 = cu1[j] * g.dtx, c2 = cu2[j];
                        const float2 xx = dx8(pq), uo = lds2(sU + uc * kTz + zl);
                        sts2(sU + uc * kTz + zl,
                             make_float2(z0u ? c2 * uo.x - c1 * xx.x : uo.x, z1u ? c2 * uo.y - c1 * xx.y : uo.y));
                    }
                }
                // w of the own points, and of the four depths above and below
#pragma unroll
                for (int c = 0; c < NC; c++) {
                    float *pw = sW + (c0 + c) * kWz + zl + 4;
                    const int ix = x0 + c0 + c;
                    const bool xu = ix >= 4 && ix < g.nnx - 4;
                    const float2 zz = dz8<1>(sQ + (c0 + c) * kQz + zl + 8), wo = lds2(pw);
                    wn[c] = make_float2(xu && z0u ? cz2.x * wo.x - cz1.x * g.dtz * zz.x : wo.x,
                                        xu && z1u ? cz2.y * wo.y - cz1.y * g.dtz * zz.y : wo.y);
                    sts2(pw, wn[c]);
                }
                // (by the last warps, which have fewer columns of u)
                if (tid >= 32 * W - 4 * TX) {
                    const int col = (tid - 32 * W + 4 * TX) >> 2, q = tid & 3, zr = q < 2 ? 2 * q - 4 : kTz + 2 * (q - 2), iz = z0 + zr, ix = x0 + col;
                    if (ix >= 4 && ix < g.nnx - 4) {
                        float *pw = sW + col * kWz + zr + 4;
                        const float2 zz = dz8<1>(sQ + col * kQz + zr + 8), wo = lds2(pw);
                        const int i0 = min(max(iz, 0), ldz - 1), i1 = min(max(iz + 1, 0), ldz - 1);
                        float2 r = wo;
                        if (iz >= 4 && iz < g.nnz - 4) r.x = g.zp[ldz + i0] * wo.x - g.zp[i0] * g.dtz * zz.x;
                        if (iz + 1 >= 4 && iz + 1 < g.nnz - 4) r.y = g.zp[ldz + i1] * wo.y - g.zp[i1] * g.dtz * zz.y;
                        sts2(pw, r);
                    }
                }
            }
            const int gz = zo - g.npd;
            bool in[NC][2];
            float im[NC][2];   // illumination or image of the interior points
            if (KIND == SK_GFWD || KIND == SK_GBWD) {
#pragma unroll
                for (int c = 0; c < NC; c++)
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        const int gx = x0 + c0 + c - g.npd;
                        in[c][j] = gx >= 0 && gx < g.nx && gz + j >= 0 && gz + j < g.nz;
                        im[c][j] = in[c][j] && (!BWD || side) ? (BWD ? a.mig : a.ill)[(long)gx * g.nz + gz + j] : 0.0f;
                    }
            }
            tc::fence_async_smem();
            __syncthreads();
            if (*(volatile int *)&s_abort) {   // boxes never came: report, let the copies end and leave
                if (tid == 0) {
                    atomicExch(a.err, 1);
                    for (int j = 0; j < stages; j++) tc::mbar_wait(&bar[(base + k + j) & (stages - 1)], ((base + k + j) >> (stages - 1)) & 1, 1000000ull);
                }
                return;
            }
            // every thread is past the item before: its stage takes the next one
            if (tid == 0 && stages > 1 && k >= 1 && k + 1 < nb) fetch(k + 1, BWD ? (k + 1) & 1 : 0, zn, xn, lev);
            const int n = lev ^ 1;
            const SField &F = a.f[side];
            float2 q[8], r8[8];   // u, and TTI w, of eight columns
            const float *pU = sU + B::hu + zl, *pW = sW + 4 + zl;
#pragma unroll
            for (int j = 0; j < 7; j++) {
                q[j + 1] = lds2(pU + (c0 + j) * B::zu);
                if (TTI) r8[j + 1] = lds2(pW + (c0 + j) * kWz);
            }
#pragma unroll
            for (int c = 0; c < NC; c++) {
#pragma unroll
                for (int j = 0; j < 7; j++) {
                    q[j] = q[j + 1];
                    if (TTI) r8[j] = r8[j + 1];
                }
                q[7] = lds2(pU + (c0 + c + 7) * B::zu);
                if (TTI) {
                    r8[7] = lds2(pW + (c0 + c + 7) * kWz);
                    wn[c] = r8[4];
                }
                const int ix = x0 + c0 + c, gx = ix - g.npd;
                const long o = (long)ix * ldz + zo;
                const bool xu = ix >= 4 && ix < g.nnx - 4, up[2] = {xu && z0u, xu && z1u};
                if (KIND != SK_GFWD && KIND != SK_GBWD && !(up[0] || up[1])) continue;
                // points off the updated band hold zeros in every array but P
                // and Q on the ring, which is written below
                float2 Pn = make_float2(0.0f, 0.0f), Qn = Pn;
                if (up[0] || up[1]) {
                    const float2 xx = dx8(q), zz = dz8<0>(pW + (c0 + c + B::hw) * kWz);
                    float2 uz, wx, ct, sn;
                    if (TTI) {
                        uz = dz8<0>(pU + (c0 + c + 4) * B::zu);
                        wx = dx8(r8);
                        ct = lds2(sT + (c0 + c + 4) * kWz + zl + 4);
                        sn = lds2(sT + (TX + 12 + c0 + c) * kWz + zl + 4);
                    }
                    const float ax1 = ca1[c], ax2 = ca2[c];
                    const int so = (c0 + c) * kTz + zl;
                    float2 T[4], M[3];
#pragma unroll
                    for (int j = 0; j < 4; j++) T[j] = lds2(sS + j * TX * kTz + so);
#pragma unroll
                    for (int j = 0; j < 3; j++) M[j] = lds2(sM + j * TX * kTz + so);
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        const float v = at2(M[0], j), e = at2(M[1], j), d = at2(M[2], j);
                        const float X = j ? xx.y : xx.x, Z = j ? zz.y : zz.x, z1 = j ? az1.y : az1.x, z2 = j ? az2.y : az2.x;
                        float px, pz, qx, qz;
                        if constexpr (TTI) {
                            const float C = at2(ct, j), S = at2(sn, j), k2 = ax2 * z2, k1 = ax1 * z1;
                            const float A = C * g.dtx * X - S * g.dtz * at2(uz, j), Bz = S * g.dtx * at2(wx, j) + C * g.dtz * Z;
                            px = k2 * at2(T[0], j) - k1 * v * v * e * A;
                            pz = k2 * at2(T[1], j) - k1 * v * v * d * Bz;
                            qx = k2 * at2(T[2], j) - k1 * v * v * d * A;
                            qz = k2 * at2(T[3], j) - k1 * v * v * Bz;
                        } else {
                            px = ax2 * at2(T[0], j) - ax1 * v * v * e * g.dtx * X;
                            pz = z2 * at2(T[1], j) - z1 * v * v * d * g.dtz * Z;
                            qx = ax2 * at2(T[2], j) - ax1 * v * v * d * g.dtx * X;
                            qz = z2 * at2(T[3], j) - z1 * v * v * g.dtz * Z;
                        }
                        float P = px + pz, Q = qx + qz;
                        if (KIND == SK_CPU) {
                            // 7x7 Gaussian source window, added after the split sum
                            float s = 0.0f;
                            const int rx = ix - a.ixs, rz = zo + j - a.izs;
                            if (src_on && rx >= -3 && rx <= 3 && rz >= -3 && rz <= 3)
                                s = (float)((double)amp * cs_gauss[(rx + 3) * 7 + (rz + 3)]);
                            P = P + s;
                            Q = Q + s;
                        }
                        if (!up[j]) continue;
                        at2(T[0], j) = px;
                        at2(T[1], j) = pz;
                        at2(T[2], j) = qx;
                        at2(T[3], j) = qz;
                        at2(Pn, j) = P;
                        at2(Qn, j) = Q;
                    }
                    sts2(F.px + o, T[0]);
                    sts2(F.pz + o, T[1]);
                    sts2(F.qx + o, T[2]);
                    sts2(F.qz + o, T[3]);
                    sts2(F.u[n] + o, q[4]);
                    sts2(F.w[n] + o, wn[c]);
                }
                if (KIND == SK_CPU || KIND == SK_GPU) {
                    sts2(F.P[n] + o, Pn);
                    sts2(F.Q[n] + o, Qn);
                    const int j = a.rec_iz - zo;
                    if ((j == 0 || j == 1) && gx >= 0 && gx < g.nx && (!TTI || up[j])) {
                        const float P = j ? Pn.y : Pn.x;
                        if (TTI) a.rec[it + (long)a.nt * gx] = P;   // the TTI program's record is trace-major
                        else a.rec[(long)it * g.nx + gx] = a.rec_scale == 2.0f ? P + P : P * a.rec_scale;
                    }
                    continue;
                }
                if (ix >= g.nnx) continue;
                const int r[2] = {ring && zo < g.nnz ? ring_at(g, ix, zo) : -1, ring && zo + 1 < g.nnz ? ring_at(g, ix, zo + 1) : -1};
                const long m = (long)gx * g.nz + gz;
                if (KIND == SK_GFWD) {
                    // record (shot_record :498), ring save (wavefield_bndr :532,
                    // cells off the band with their unchanged zeros), illumination
                    // (cal_illumination :654)
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        const float P = j ? Pn.y : Pn.x, Q = j ? Qn.y : Qn.x;
                        if (r[j] >= 0) {
                            a.bp[(long)it * a.L + r[j]] = P;
                            a.bq[(long)it * a.L + r[j]] = Q;
                        }
                        if (in[c][j]) {
                            if (gz + j == 0) a.rec[(long)it * g.nx + gx] = P;
                            float v = im[c][j] + (P * P + Q * Q);
                            if (v <= 0.0f) v = 1.0f;
                            a.ill[m + j] = v;
                        }
                    }
                    if (up[0] || up[1]) {
                        sts2(F.P[n] + o, Pn);
                        sts2(F.Q[n] + o, Qn);
                    }
                } else if (side == 0) {
                    sv[c][0] = Pn;
                    sv[c][1] = Qn;
                    sv[c][2] = q[4];
                    sv[c][3] = wn[c];
                    // the next step's ring in place in the new level
                    if (next >= 0) {
#pragma unroll
                        for (int j = 0; j < 2; j++)
                            if (r[j] >= 0) {
                                at2(Pn, j) = a.bp[(long)next * a.L + r[j]];
                                at2(Qn, j) = a.bq[(long)next * a.L + r[j]];
                            }
                    }
                    if (up[0] || up[1] || r[0] >= 0 || r[1] >= 0) {
                        sts2(F.P[n] + o, Pn);
                        sts2(F.Q[n] + o, Qn);
                    }
                } else if (up[0] || up[1]) {
                    // image (cal_migration :679) and Poynting gathers (:718-766)
                    // (gathers at gx = 0, dcdp, ... below nx / dcdp * dcdp)
                    const int ga = !a.adcig || gx < 0 ? -1 : a.dcdp == 1 ? gx : gx % a.dcdp || gx / a.dcdp >= g.nx / a.dcdp ? -1 : gx / a.dcdp;
                    float *ag[2] = {nullptr, nullptr}, av[2], old[2];
#pragma unroll
                    for (int j = 0; j < 2; j++) {
                        if (!in[c][j]) continue;
                        const float sP_ = at2(sv[c][0], j), gP = at2(Pn, j);
                        // a zero product adds nothing to any bin (the sums start at +0
                        // and never become -0): most points ahead of the wavefronts
                        // (1700x601 backward 38.9 -> 36.4 us a step)
                        const float sg = sP_ * gP;
                        if (ga < 0 || sg == 0.0f) continue;
                        const float Ssx = -sP_ * at2(sv[c][2], j), Ssz = -at2(sv[c][1], j) * at2(sv[c][3], j);
                        const float Sgx = gP * at2(q[4], j), Sgz = at2(Qn, j) * at2(wn[c], j);
                        const float b1 = Ssx * Ssx + Ssz * Ssz, b2 = Sgx * Sgx + Sgz * Sgz;
                        const int ia = poynting_bin(Ssx * Sgx + Ssz * Sgz, b1, b2, cs_thr, a.nangle);
                        if (ia < 0) continue;
                        const float co = cs_cos[ia];
                        av[j] = sg * co * co * co;
                        ag[j] = a.adcig + gz + j + (long)g.nz * ia + (long)g.nz * a.nangle * ga;
                        old[j] = __ldcs(ag[j]);
                    }
#pragma unroll
                    for (int j = 0; j < 2; j++)
                        if (in[c][j]) a.mig[m + j] = im[c][j] + at2(sv[c][0], j) * at2(Pn, j);
                    // the next step's record in place in the new level
                    if (next >= 0 && gx >= 0 && gx < g.nx && (gz == 0 || gz == -1)) {
                        const float v = a.rec[(long)next * g.nx + gx];
                        at2(Pn, -gz) = v;
                        at2(Qn, -gz) = v;
                    }
                    sts2(F.P[n] + o, Pn);
                    sts2(F.Q[n] + o, Qn);
#pragma unroll
                    for (int j = 0; j < 2; j++)
                        if (ag[j]) __stcs(ag[j], old[j] + av[j]);
                }
            }
            if (stages == 1 && k + 1 < nb) {   // one stage: the next item's boxes once all are done with this one's
                __syncthreads();
                if (tid == 0) fetch(k + 1, BWD ? (k + 1) & 1 : 0, zn, xn, lev);
            }
        }
        // this step's stores before the next step's TMA reads of them
        asm volatile("fence.proxy.async;" ::: "memory");
        __syncthreads();
        if (tid == 0) grid_arrive(a.bar);
    }
}

// Ring (entry k at ring_at's position) and record of step it.  Over their
// cells only: it runs before every backward run of steps (a 600-step shot of
// 1700x601 + 50 took 33.75 ms with a pass over the whole grid, 33.52 so).
__global__ void k_step2d_restore(const __grid_constant__ SStep a, int it, int lev) {
    const SGrid &g = a.g;
    const int n = g.npd;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < a.L + g.nx; k += gridDim.x * blockDim.x) {
        if (k >= a.L) {
            const int gx = k - a.L;
            const long o = (long)(n + gx) * g.ldz + n;
            a.f[1].P[lev][o] = a.f[1].Q[lev][o] = a.rec[(long)it * g.nx + gx];
            continue;
        }
        int ix, iz;
        if (k < 2 * g.nx) {
            ix = n + (k < g.nx ? k : k - g.nx);
            iz = k < g.nx ? n - 1 : n + g.nz + 1;
        } else {
            const int q = k - 2 * g.nx;
            ix = q < g.nz ? n - 1 : n + g.nx + 1;
            iz = n + (q < g.nz ? q : q - g.nz);
        }
        const long o = (long)ix * g.ldz + iz;
        a.f[0].P[lev][o] = a.bp[(long)it * a.L + k];
        a.f[0].Q[lev][o] = a.bq[(long)it * a.L + k];
    }
}

template <int NC>
const void *step_fn(StepKind k) {
    switch (k) {
        case SK_CPU: return (const void *)k_step2d<SK_CPU, false, NC>;
        case SK_GPU: return (const void *)k_step2d<SK_GPU, false, NC>;
        case SK_GFWD: return (const void *)k_step2d<SK_GFWD, false, NC>;
        default: return (const void *)k_step2d<SK_GBWD, false, NC>;
    }
}
const void *step_fn(StepKind k, bool tti, int tx) {
    if (!tti) return tx == 8 ? step_fn<1>(k) : step_fn<2>(k);
    switch (k) {
        case SK_GFWD: return (const void *)k_step2d<SK_GFWD, true, 1>;
        case SK_GBWD: return (const void *)k_step2d<SK_GBWD, true, 1>;
        default: return tx == 8 ? (const void *)k_step2d<SK_GPU, true, 1> : (const void *)k_step2d<SK_GPU, true, 2>;
    }
}

PFN_cuTensorMapEncodeTiled_v12000 g_enc = nullptr;

// Boxes of boxz x boxx of `arrays` arrays that lie one behind the other.
int box_map(CUtensorMap *map, const float *base, const SGrid &g, int boxz, int boxx, int arrays) {
    if (!g_enc) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        GEO_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q));
        if (!fn || q != cudaDriverEntryPointSuccess) return fail(GEO_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
        g_enc = (PFN_cuTensorMapEncodeTiled_v12000)fn;
    }
    cuuint64_t dims[3] = {(cuuint64_t)g.nnz, (cuuint64_t)g.nnx, (cuuint64_t)arrays};
    cuuint64_t strides[2] = {(cuuint64_t)g.ldz * 4, (cuuint64_t)g.ldz * g.nnx * 4};
    cuuint32_t box[3] = {(cuuint32_t)boxz, (cuuint32_t)boxx, (cuuint32_t)arrays}, es[3] = {1, 1, 1};
    const CUresult r = g_enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, arrays > 1 ? 3 : 2, const_cast<float *>(base), dims,
                             strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(GEO_ERR_CUDA, "cuTensorMapEncodeTiled (2D step) failed (%d)", (int)r);
    return GEO_OK;
}

}  // namespace

int Fused2D::maps(const SGrid &g, const SField &f, int side) {
    SMaps *out = m[side];
    for (int l = 0; l < 2; l++) {
        GEO_TRY(box_map(&out[l].P, f.P[l], g, tti ? kQz : kTz, tx + 14, 1));
        GEO_TRY(box_map(&out[l].Q, f.Q[l], g, kQz, tti ? tx + 14 : tx, 1));
        GEO_TRY(box_map(&out[l].u, f.u[l], g, tti ? kWz : kTz, tx + 8, 1));
        GEO_TRY(box_map(&out[l].w, f.w[l], g, kWz, tti ? tx + 8 : tx, 1));
        GEO_TRY(box_map(&out[l].S, f.px, g, kTz, tx, 4));
    }
    return GEO_OK;
}

int Fused2D::model(const SGrid &g, const float *p, const float *trig) {
    if (tti) GEO_TRY(box_map(&mt, trig, g, kWz, tx + 8, 2));
    else memset(&mt, 0, sizeof mt);
    return box_map(&mm, p, g, kTz, tx, 3);
}

// Tiles of 8 columns (three or four blocks per SM) or 16 (two; a quarter less
// halo work): the fewer columns on the busiest SM, each tile's halo counted as
// one (VTI) or six (TTI, whose halos cost both velocities).  us a step with 8
// and with 16: VTI 601 deep 2401 wide 19.7 and 18.0, 600 8.5 and 7.4, 300 6.3
// and 4.9, the RTM program's 1700 forward 17.1 and 17.6, 401x401 6.5 and 5.0,
// 250x250 4.1 and 4.1, 101x121 3.3 and 3.9; TTI 600x300 8.1 and 7.5, 1500x600
// 21 and 19.2, 200x150 3.8 and 4.8.  The TTI RTM passes take 8: 1100x450 15.2
// and 16.4 forward, 31.3 and 37.8 backward.  VTI takes one stage where every
// tile has its own block, two where blocks walk several; TTI tiles are heavier
// and always take one (three blocks per SM instead of two beat the prefetch).
int Fused2D::plan(StepKind k, bool tti_, const SGrid &g, int fixed) {
    kind = k;
    tti = tti_;
    if (k == SK_CPU) GEO_TRY(load_step2d_gauss());
    int dev = 0, sms = 0, coop = 0;
    GEO_CUDA(cudaGetDevice(&dev));
    GEO_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    GEO_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    long best = 0;
    for (int nc = 1; nc <= 2 && coop; nc++) {
        const int t = nc * kThreads / 32;
        const void *fn = step_fn(k, tti, t);
        if (fixed && t != fixed) continue;
        if (tti && k != SK_GPU && t != 8) continue;   // no such kernel (step_fn)
        const int n = ((g.nnz + kTz - 1) / kTz) * ((g.nnx + t - 1) / t);
        GEO_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)step_smem(t, 2, tti)));
        for (int st = k == SK_GBWD && !tti ? 2 : 1; st <= 2; st++) {
            int occ = 0;
            GEO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kThreads, step_smem(t, st, tti)));
            if (occ < 1 || (st == 1 && !tti && n > occ * sms)) continue;
            const long cost = (n + sms - 1L) / sms * (t + (tti ? 6 : 1));
            if (!best || cost < best) {
                best = cost;
                tx = t;
                tiles = n;
                stages = st;
                grid = std::min(n, occ * sms);
            }
            break;
        }
    }
    if (!best && coop && fixed) return fail(GEO_ERR_ARG, "2D step: no tiles of %d columns", fixed);
    if (!best) return fail(GEO_ERR_CUDA, "2D step: cooperative launch unavailable");
    return GEO_OK;
}

void step2d_fields(float *p, size_t n, SField &f) {
    float **q[12] = {&f.u[0], &f.u[1], &f.w[0], &f.w[1], &f.P[0], &f.P[1], &f.Q[0], &f.Q[1], &f.px, &f.pz, &f.qx, &f.qz};
    for (int k = 0; k < 12; k++) *q[k] = p + k * n;
}

int load_step2d_angles(const float *thr, const float *cs, cudaStream_t s) {
    GEO_CUDA(cudaMemcpyToSymbolAsync(cs_thr, thr, sizeof cs_thr, 0, cudaMemcpyDeviceToDevice, s));
    GEO_CUDA(cudaMemcpyToSymbolAsync(cs_cos, cs, sizeof cs_cos, 0, cudaMemcpyDeviceToDevice, s));
    return GEO_OK;
}

int load_step2d_gauss() {
    static OncePerDevice once;
    return once.run([]() -> int {
        double g[49];
        for (int x = -3; x <= 3; x++)
            for (int z = -3; z <= 3; z++) g[(x + 3) * 7 + (z + 3)] = std::exp((double)(-z * z - x * x));
        GEO_CUDA(cudaMemcpyToSymbol(cs_gauss, g, sizeof g));
        return GEO_OK;
    });
}

int Fused2D::run(const SStep &a, cudaStream_t s) const {
    const long long steps = std::abs((long long)a.it1 - a.it0) + 1;
    if (steps * grid >= 4000000000LL) return fail(GEO_ERR_ARG, "too many steps for one launch");
    Maps tm;
    for (int f = 0; f < 2; f++)
        for (int l = 0; l < 2; l++) tm.m[f][l] = m[kind == SK_GBWD ? f : 0][l];
    tm.model = mm;
    tm.trig = mt;
    GEO_CUDA(cudaMemsetAsync(a.bar, 0, 4, s));
    int n = tiles, st = stages;
    void *args[] = {(void *)&tm, (void *)&a, (void *)&n, (void *)&st};
    GEO_CUDA(cudaLaunchCooperativeKernel(step_fn(kind, tti, tx), dim3(grid), dim3(kThreads), args,
                                         step_smem(tx, stages, tti), s));
    return check_launch("step2d");
}

int launch_step2d_restore(const SStep &a, int it, int lev, cudaStream_t s) {
    k_step2d_restore<<<std::min((a.L + a.g.nx + 255) / 256, 152 * 8), 256, 0, s>>>(a, it, lev);
    return check_launch("step2d_restore");
}

}  // namespace geo

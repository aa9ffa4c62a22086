// 2D VTI staggered-grid half-steps of single-shot forward modelling: the MPI
// form, and every form's runs in a caller's scratch (noalloc.cu).  The CPU
// and GPU forms otherwise take the fused steps of step2d.cu.
//
// The half-step kernels walk a shot's tiles with a persistent grid; a tile
// is 32 z-points (one warp, z contiguous in memory) by `blockDim.y`
// x-columns.
//
// Arithmetic keeps the reference's operation order exactly (the library is
// compiled with contraction off), so results are bit-identical to the
// reference CPU code and to the oracle:
//   velocity  CPU_vti2dfd_kernels.c:79-106 / GPU_vti2dfd_kernels.cu:209-238
//   stress    CPU_vti2dfd_kernels.c:108-177 / GPU_vti2dfd_kernels.cu:240-299
//             MPI program Toa_rtm_vti_adcig_cdp.c:1227-1327 (rho*vp^2 form,
//             pz/qx chains in double after pow(1+2del, 0.5))
#include "geo_internal.h"
#include "tc_util.cuh"
#include "gridsync.cuh"
#include "softcvt.cuh"
#include <algorithm>
#include <cmath>

namespace geo {

__constant__ float c_fd[4] = {1.196289f, -0.0797526f, 0.009570313f, -0.0006975447f};
// exp(-x^2-z^2) on the 7x7 source window, x,z in [-3,3] (ptsource,
// CPU_vti2dfd_kernels.c:72); filled from the host's exp() at load.
__constant__ double c_gauss[49];

static int ensure_gauss() {
    static OncePerDevice once;
    return once.run([]() -> int {
        double g[49];
        for (int x = -3; x <= 3; x++)
            for (int z = -3; z <= 3; z++) g[(x + 3) * 7 + (z + 3)] = std::exp((double)(-z * z - x * x));
        GEO_CUDA(cudaMemcpyToSymbol(c_gauss, g, sizeof g));
        return GEO_OK;
    });
}

struct Tile2D {
    const Shot2D *sh;
    int ix, iz;
};

__device__ __forceinline__ bool locate(const Shot2D *shots, const int *item_shot, int item, Tile2D &t) {
    const int s = item_shot[item];
    const Shot2D *sh = shots + s;
    const int tile = item - sh->tile_base;
    const int tz = tile % sh->ntz, tx = tile / sh->ntz;
    t.sh = sh;
    t.iz = tz * 32 + threadIdx.x;
    t.ix = tx * blockDim.y + threadIdx.y;
    return t.ix >= 4 && t.ix < sh->nnx - 4 && t.iz >= 4 && t.iz < sh->nnz - 4;
}

// Reads of neighbours' values.  Kernels of one half-step read fields that
// no thread of the launch writes, through the read-only path (NC); the
// persistent shot kernel reads values other blocks wrote before a grid
// barrier, through L2 (the read-only path is not coherent with them).
template <bool NC>
__device__ __forceinline__ float ldf(const float *p) {
    return NC ? __ldg(p) : __ldcg(p);
}

// P/Q read for the velocity update.  The GPU-form source (P,Q += amp at one
// cell before the velocity update, GPU_vti2dfd_kernels.cu:423) is applied on
// the fly to the taps that touch the source cell.
template <bool PT_SRC, bool NC>
__device__ __forceinline__ float tap(const float *a, long idx, long src, float amp) {
    float v = NC ? a[idx] : __ldcg(a + idx);
    if (PT_SRC && idx == src) v = v + amp;
    return v;
}

// Velocity update of one updated point (ix, iz) of a shot.
template <int VARIANT, bool NC>
__device__ __forceinline__ void vel_point(const Shot2D &sh, int ix, int iz, const Step2D &st) {
    const int nnz = sh.nnz;
    const long id = (long)ix * nnz + iz;
    const bool pt_src = VARIANT == V_GPU && st.src_on;
    const long src = (long)sh.ixs * nnz + sh.izs;
    const bool near = pt_src && ((iz == sh.izs && abs(ix - sh.ixs) <= 4) || (ix == sh.ixs && abs(iz - sh.izs) <= 4));
    const float *P = sh.P, *Q = sh.Q;
    float xx = 0.0f, zz = 0.0f;
    if (near) {
#pragma unroll
        for (int im = 0; im < 4; im++) {
            xx += c_fd[im] * (tap<true, NC>(P, id + (im + 1) * nnz, src, st.amp) - tap<true, NC>(P, id - im * nnz, src, st.amp));
            zz += c_fd[im] * (tap<true, NC>(Q, id + im + 1, src, st.amp) - tap<true, NC>(Q, id - im, src, st.amp));
        }
    } else {
#pragma unroll
        for (int im = 0; im < 4; im++) {
            xx += c_fd[im] * (ldf<NC>(P + id + (im + 1) * nnz) - ldf<NC>(P + id - im * nnz));
            zz += c_fd[im] * (ldf<NC>(Q + id + im + 1) - ldf<NC>(Q + id - im));
        }
    }
    // u1 = coffx2*u0 - coffx1*dtx*xx (the MPI copy's extra *rho is *1.0f)
    sh.u[id] = sh.cx2[ix] * sh.u[id] - sh.cx1[ix] * sh.dtx * xx;
    sh.w[id] = sh.cz2[iz] * sh.w[id] - sh.cz1[iz] * sh.dtz * zz;
}

template <int VARIANT>
__global__ void __launch_bounds__(256) k_vel2d(const Shot2D *__restrict__ shots, const int *__restrict__ item_shot,
                                               int nitems, Step2D st) {
    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
        Tile2D t;
        if (!locate(shots, item_shot, item, t)) continue;
        vel_point<VARIANT, true>(*t.sh, t.ix, t.iz, st);
    }
}

// Stress update of one updated point (ix, iz) of a shot, with the record.
template <int VARIANT, bool NC>
__device__ __forceinline__ void stress_point(const Shot2D &sh, int ix, int iz, const Step2D &st) {
    const int nnz = sh.nnz;
    const long id = (long)ix * nnz + iz;
    const float vp = __ldg(sh.vp + id);
    // the MPI form's arithmetic carries its pz and qx chains in double
    // (their fixed factors kz, kx formed once per shot in the program's
    // order)
    constexpr bool dpw = VARIANT == V_MPI;
    float e2 = __ldg(sh.e2 + id), d2 = 0.0f;
    double kz = 0.0, kx = 0.0;
    if (dpw) {
        kz = __ldg(sh.kz + id);
        kx = __ldg(sh.kx + id);
    } else {
        d2 = __ldg(sh.d2 + id);
    }
    if (st.taper) {
        const int bx = ix - sh.tx0, bz = iz - sh.tz0;
        if (bx >= 0 && bx < kTB && bz >= 0 && bz < kTB) {
            e2 = sh.te2[bx * kTB + bz];
            if (dpw) {
                kz = sh.tkz[bx * kTB + bz];
                kx = sh.tkx[bx * kTB + bz];
            } else {
                d2 = sh.td2[bx * kTB + bz];
            }
        }
    }
    const float ax1 = sh.ax1[ix], ax2 = sh.ax2[ix], az1 = sh.az1[iz], az2 = sh.az2[iz];
    float xx = 0.0f, zz = 0.0f;
#pragma unroll
    for (int im = 0; im < 4; im++) {
        xx += c_fd[im] * (ldf<NC>(sh.u + id + im * nnz) - ldf<NC>(sh.u + id - (im + 1) * nnz));
        zz += c_fd[im] * (ldf<NC>(sh.w + id + im) - ldf<NC>(sh.w + id - im - 1));
    }
    float px = sh.px[id], pz = sh.pz[id], qx = sh.qx[id], qz = sh.qz[id];
    if (VARIANT == V_MPI) {
        px = ax2 * px - ax1 * vp * e2 * sh.dtx * xx;
        // the conversions on the integer pipe (softcvt.cuh): same bits
        pz = d2f_rn(f2d_exact(az2 * pz) - kz * f2d_exact(zz));
        qx = d2f_rn(f2d_exact(ax2 * qx) - kx * f2d_exact(xx));
        qz = az2 * qz - az1 * vp * sh.dtz * zz;
    } else {
        px = ax2 * px - ax1 * vp * vp * e2 * sh.dtx * xx;
        pz = az2 * pz - az1 * vp * vp * d2 * sh.dtz * zz;
        qx = ax2 * qx - ax1 * vp * vp * d2 * sh.dtx * xx;
        qz = az2 * qz - az1 * vp * vp * sh.dtz * zz;
    }
    sh.px[id] = px; sh.pz[id] = pz; sh.qx[id] = qx; sh.qz[id] = qz;
    float P = px + pz, Q = qx + qz;
    if (VARIANT == V_CPU || VARIANT == V_MPI) {
        // Gaussian source window, added after the split sum
        float s = 0.0f;
        if (st.src_on) {
            const int rx = ix - sh.ixs, rz = iz - sh.izs;
            if (rx >= -3 && rx <= 3 && rz >= -3 && rz <= 3)
                s = (float)((double)st.amp * c_gauss[(rx + 3) * 7 + (rz + 3)]);
        }
        P = P + s;
        Q = Q + s;
    }
    sh.P[id] = P;
    sh.Q[id] = Q;
    // receiver gather at rec_iz, time-major
    const int gx = ix - sh.npd;
    if (iz == sh.rec_iz && gx >= 0 && gx < sh.nx)
        sh.rec_p[(long)st.it * sh.nx + gx] = sh.rec_scale == 2.0f ? P + P : P * sh.rec_scale;
}

template <int VARIANT>
__global__ void __launch_bounds__(256) k_stress2d(const Shot2D *__restrict__ shots, const int *__restrict__ item_shot,
                                                  int nitems, Step2D st) {
    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
        Tile2D t;
        if (!locate(shots, item_shot, item, t)) continue;
        stress_point<VARIANT, true>(*t.sh, t.ix, t.iz, st);
    }
}

// ------------------------------------------------------ persistent shot
// A whole forward run of a single shot of the MPI form in one cooperative
// launch: per step the velocity half-step over every tile, a grid barrier, the stress half-step
// with the record, a grid barrier.  Same per-point arithmetic as the
// per-half-step kernels; neighbours' values are read through L2.
__global__ void __launch_bounds__(512) k_fd2d_shot(const Shot2D *__restrict__ shots,
                                                   const int *__restrict__ item_shot, int nitems, Persist2D a) {
    unsigned k = 0;
    for (int it = 0; it < a.nt; it++) {
        Step2D st;
        st.it = it;
        st.amp = a.amp[it];
        st.src_on = a.on[it];
        st.taper = a.taper;
        for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
            Tile2D t;
            if (locate(shots, item_shot, item, t)) vel_point<V_MPI, false>(*t.sh, t.ix, t.iz, st);
        }
        if (!grid_barrier(a.bar, ++k * gridDim.x, a.err)) return;
        for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
            Tile2D t;
            if (locate(shots, item_shot, item, t)) stress_point<V_MPI, false>(*t.sh, t.ix, t.iz, st);
        }
        if (!grid_barrier(a.bar, ++k * gridDim.x, a.err)) return;
    }
}

int launch_fd2d_shot(const Shot2D *d_shots, const int *d_item_shot, int nitems, int by, Persist2D a, cudaStream_t s) {
    const void *fn = (const void *)k_fd2d_shot;
    GEO_TRY(ensure_gauss());
    int dev = 0, sms = 0, occ = 0, coop = 0;
    GEO_CUDA(cudaGetDevice(&dev));
    GEO_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    GEO_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    GEO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, 32 * by, 0));
    if (!coop || occ < 1) return fail(GEO_ERR_CUDA, "cooperative launch unavailable");
    // every block resident at once (the barrier needs it; the cooperative
    // launch checks it), blocks walking the tiles when there are more
    const int grid = std::min(nitems, occ * sms);
    if ((long long)grid * 2 * a.nt >= 4000000000LL) return fail(GEO_ERR_ARG, "too many steps for one launch");
    dim3 block(32, by);
    void *args[] = {(void *)&d_shots, (void *)&d_item_shot, (void *)&nitems, (void *)&a};
    GEO_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), block, args, 0, s));
    return check_launch("fd2d_shot");
}

template <int V>
static void vel_dispatch(const Shot2D *d_shots, const int *d_item_shot, int nitems, dim3 grid, dim3 block,
                         Step2D st, cudaStream_t s) {
    k_vel2d<V><<<grid, block, 0, s>>>(d_shots, d_item_shot, nitems, st);
}

int launch_vel2d(int variant, const Shot2D *d_shots, const int *d_item_shot, int nitems, int by, int grid,
                 Step2D st, cudaStream_t s) {
    dim3 block(32, by), g(grid);
    switch (variant) {
        case V_CPU: vel_dispatch<V_CPU>(d_shots, d_item_shot, nitems, g, block, st, s); break;
        case V_GPU: vel_dispatch<V_GPU>(d_shots, d_item_shot, nitems, g, block, st, s); break;
        default: vel_dispatch<V_MPI>(d_shots, d_item_shot, nitems, g, block, st, s); break;
    }
    return check_launch("vel2d");
}

int launch_stress2d(int variant, const Shot2D *d_shots, const int *d_item_shot, int nitems, int by, int grid,
                    Step2D st, cudaStream_t s) {
    GEO_TRY(ensure_gauss());
    dim3 block(32, by), g(grid);
    switch (variant) {
        case V_CPU: k_stress2d<V_CPU><<<g, block, 0, s>>>(d_shots, d_item_shot, nitems, st); break;
        case V_GPU: k_stress2d<V_GPU><<<g, block, 0, s>>>(d_shots, d_item_shot, nitems, st); break;
        default: k_stress2d<V_MPI><<<g, block, 0, s>>>(d_shots, d_item_shot, nitems, st); break;
    }
    return check_launch("stress2d");
}

}  // namespace geo

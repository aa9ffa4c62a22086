// 2D TTI (tilted VTI) staggered-grid FD with the semantics of the GPU TTI
// program (2D-tti-fd+rtm-cuda/Toa_gpu_2dtti_fd_1orderfunction.cu):
//   update_vel (:81-112)     u <- cx2 cz2 u - cx1 cz1 (cos t dtx dP/dx - sin t dtz dP/dz)
//                            w <- cx2 cz2 w - cx1 cz1 (sin t dtx dQ/dx + cos t dtz dQ/dz)
//   update_stress (:114-183) px,pz,qx,qz with the same rotated derivatives of
//                            u and w, P = px + pz, Q = qx + qz
// with the sponge applied as products of the x and z profiles, the point
// source added to P and Q before the velocity update (add_source :47-79),
// the record taken from P at the surface row after each step
// (shot_record :273-283) and padded-P snapshots every snap_every steps from
// snap_every on (:451-456).  The program swaps its old/new pointers without
// keeping two buffers (u0 = u1 after the first step), so every field is in
// effect updated in place.
// cos and sin of the tilt are formed once on the device (cosf/sinf of the
// angle in radians, theta * pi/180 as the program converts it).
// The program launches four kernels per step; here the steps between two
// host events (a snapshot, a watchdog scan) are one launch of the fused steps
// of step2d.cu.
#include "geo_internal.h"
#include <algorithm>
#include "model2d.cuh"
#include "step2d.cuh"
#include <cmath>
#include <vector>

namespace geo {

// cos and sin of the tilt (radians, in place: th -> cos, sin into sn).  The
// 2D TTI programs evaluate cos(theta[id]) and sin(theta[id]) of their float
// tilt inside their kernels (Toa_gpu_2dtti_fd_1orderfunction.cu:106-107,
// :168-175; Toa_gpu_2dtti_rtm_adcigs_iorderfunciton.cu:155-156, :216-222),
// i.e. the device's single-precision cosf and sinf; the tables are formed
// here with the same device functions, so they hold the programs' values.
__global__ void k_tilt_trig(float *th_cos, float *sn, size_t n) {
    for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
        const float t = th_cos[k];
        th_cos[k] = cosf(t);
        sn[k] = sinf(t);
    }
}

int launch_tilt_trig(float *th_cos, float *sn, size_t n, cudaStream_t s) {
    const int grid = (int)std::min<size_t>((n + 255) / 256, 152 * 8);
    k_tilt_trig<<<grid, 256, 0, s>>>(th_cos, sn, n);
    return check_launch("tilt_trig");
}

}  // namespace geo

using namespace geo;

extern "C" int geo_tti2d_shot(const geo_fd2d_desc *desc, const float *v, const float *e, const float *d,
                              const float *theta, float *shot, float *snap, int snap_every, int mem, void *stream) {
    if (!desc || !v || !e || !d || !theta || !shot) return fail(GEO_ERR_ARG, "null argument");
    const geo_fd2d_desc &D = *desc;
    if (D.nx < 2 || D.nz < 2 || D.npd < 5 || D.nt < 1) return fail(GEO_ERR_ARG, "grid too small (npd must be >= 5)");
    if (!(D.dt > 0) || !(D.dx > 0) || !(D.dz > 0) || !(D.favg > 0)) return fail(GEO_ERR_ARG, "bad spacing");
    if (mem != GEO_MEM_HOST && mem != GEO_MEM_DEVICE) return fail(GEO_ERR_ARG, "bad mem kind");
    if (snap && snap_every < 1) return fail(GEO_ERR_ARG, "snap_every must be >= 1");
    const int nx = D.nx, nz = D.nz, npd = D.npd, nt = D.nt;
    const int nnx = nx + 2 * npd, nnz = nz + 2 * npd;
    const int ldz = (nnz + 3) / 4 * 4;   // columns of a pitch that TMA takes
    const size_t n = (size_t)nnx * ldz, mid = (size_t)nnx * nnz / 2;
    if (D.rec_iz < 0 || D.rec_iz >= nnz) return fail(GEO_ERR_ARG, "receiver row outside the grid");
    cudaStream_t s = (cudaStream_t)stream;
    Raw2D raw;
    GEO_TRY(raw.open(nx, nz, v, e, d, theta, mem, s));
    // source cell (add_source :71-72), shot is 1-based
    const float fsx = D.fs + (D.is - 1) * D.ds;
    const int ixs = (int)(fsx + 0.5f) + npd - 1, izs = (int)(D.zs + 0.5f) + npd - 1;
    // SV taper centre (fs+(is-1)ds+npml, zs+npml) (:131-132): one cell right/down of the source cell
    const int cx = ixs + 1, cz = izs + 1;
    std::vector<unsigned long long> pick;
    auto at = [&](int a, int ix, int iz) {   // padded position
        return raw_at(a, raw, std::min(std::max(ix - npd, 0), nx - 1), std::min(std::max(iz - npd, 0), nz - 1));
    };
    pick.push_back(at(0, (int)(mid / nnz), (int)(mid % nnz)));
    if (D.sv)
        for (int a = 1; a <= 2; a++)
            for (int b = 0; b < kTB * kTB; b++) pick.push_back(at(a, cx - kTB / 2 + b / kTB, cz - kTB / 2 + b % kTB));
    RawStats rs;
    GEO_TRY(raw_stats(raw, pick, rs, s));
    if (ixs < 4 || ixs >= nnx - 4 || izs < 4 || izs >= nnz - 4) return fail(GEO_ERR_ARG, "source outside the grid");
    GEO_TRY(check_stability(V_GPU, 2, rs.vmin, rs.vmax, D.dt, D.dx, D.dx, D.dz, D.favg));
    // sponge (get_d0 :186-189 from the padded centre velocity; initial_coffe :227-271)
    const float d0 = sponge_d0(V_GPU, 2, 0.0f, rs.val[0], npd, D.dx, D.dx, D.dz);
    std::vector<float> prof(4 * (size_t)(nnx + ldz), 1.0f);
    float *q = prof.data();
    sponge_profiles(V_GPU, nx, npd, D.dt, d0, q, q + nnx, q + 2 * nnx, q + 3 * nnx);
    q += 4 * nnx;
    sponge_profiles(V_GPU, nz, npd, D.dt, d0, q, q + ldz, q + 2 * ldz, q + 3 * ldz);
    std::vector<float> amp;
    std::vector<uint8_t> on;
    source_amplitudes(V_GPU, nt, D.dt, D.favg, D.pfac, D.wtype, amp, on);
    Blob small;
    const size_t o_prof = small.put(prof), o_amp = small.put(amp), o_on = small.put(on);
    size_t o_te2 = 0, o_td2 = 0;
    Taper2D tp;
    if (D.sv) {
        sv_taper_2d(V_GPU, nnx, nnz, cx, cz, rs.val.data() + 1, rs.val.data() + 1 + kTB * kTB, tp);
        std::vector<float> te2(kTB * kTB), td2(kTB * kTB);
        for (int b = 0; b < kTB * kTB; b++) {
            te2[b] = 1 + 2 * tp.e[b];
            td2[b] = sqrtf(1 + 2 * tp.d[b]);
        }
        o_te2 = small.put(te2);
        o_td2 = small.put(td2);
    }
    GEO_TRY(small.upload(s));
    // one allocation: the cleared state (fields, record, barrier and error
    // words), then vp, 1+2eps, sqrtf(1+2del) and the tilt in radians as
    // read_file converts it (:235), whose cos and sin are formed on the
    // device (launch_tilt_trig) as the program's kernels form them
    Arena ar;
    float *fb = nullptr, *drec = nullptr, *model = nullptr;
    unsigned *sync = nullptr;
    size_t clear = 0;
    for (int pass = 0; pass < 2; pass++) {
        fb = ar.take<float>(12 * n);
        drec = ar.take<float>((size_t)nx * nt);
        sync = ar.take<unsigned>(2);
        clear = ar.off;
        model = ar.take<float>(5 * n);
        if (pass == 0) GEO_TRY(ar.alloc());
    }
    GEO_CUDA(cudaMemsetAsync(ar.buf.p, 0, clear, s));
    ModelJob job{};
    job.nx = nx; job.nz = nz; job.npd = npd; job.ldz = ldz;
    job.vp = model; job.e2 = model + n; job.d2 = model + 2 * n; job.rad = model + 3 * n;
    GEO_TRY(launch_model2d(raw, {job}, s));
    if (D.sv)
        GEO_TRY(launch_box2d(job.e2, job.d2, nnx, ldz, tp.x0, tp.z0, kTB, small.at<float>(o_te2), small.at<float>(o_td2),
                             s));
    GEO_TRY(launch_tilt_trig(model + 3 * n, model + 4 * n, n, s));
    SStep a{};
    SGrid &g = a.g;
    g.nnx = nnx; g.nnz = nnz; g.ldz = ldz; g.npd = npd; g.nx = nx; g.nz = nz;
    g.dtx = D.dt / D.dx;
    g.dtz = D.dt / D.dz;
    const float *pp = small.at<float>(o_prof);
    g.cx1 = pp; g.cx2 = pp + nnx; g.ax1 = pp + 2 * nnx; g.ax2 = pp + 3 * nnx;
    g.zp = pp + 4 * nnx;
    step2d_fields(fb, n, a.f[0]);
    a.amp = small.at<float>(o_amp);
    a.on = small.at<unsigned char>(o_on);
    a.ixs = ixs;
    a.izs = izs;
    a.rec = drec;
    a.rec_iz = D.rec_iz;
    a.nt = nt;
    a.bar = sync;
    a.err = reinterpret_cast<int *>(sync) + 1;
    const cudaMemcpyKind kout = mem == GEO_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
    Fused2D plan;
    GEO_TRY(plan.plan(SK_GPU, true, g));
    GEO_TRY(plan.maps(g, a.f[0], 0));
    GEO_TRY(plan.model(g, model, model + 3 * n));
    Watchdog wd;
    GEO_TRY(wd.open());
    // runs of steps between the host's work: a snapshot after step it
    // (it % snap_every == 0, it > 0) and the watchdog's scan end a run
    for (int it0 = 0; it0 < nt;) {
        int it1 = it0;
        while (true) {
            const int it = it1++;
            const bool snap_due = snap && it % snap_every == 0 && it != 0;
            const bool watch_due = wd.every > 0 && (it + 1) % wd.every == 0;
            if (snap_due || watch_due || it1 == nt) break;
        }
        if ((long long)plan.grid * (it1 - it0 + 1) >= 4000000000LL) it1 = it0 + (int)(1900000000LL / plan.grid);
        a.it0 = it0;
        a.it1 = it1;
        GEO_TRY(plan.run(a, s));
        a.lev = (a.lev + it1 - it0) & 1;
        const float *P = a.f[0].P[a.lev];
        const int it = it1 - 1;
        if (snap && it % snap_every == 0 && it != 0)
            GEO_CUDA(cudaMemcpy2DAsync(snap + (size_t)(it / snap_every - 1) * nnx * nnz, (size_t)nnz * 4, P, (size_t)ldz * 4,
                                       (size_t)nnz * 4, nnx, kout, s));
        const int w = wd.check(P, n, it, it == nt - 1, s);
        if (w == GEO_ERR_NAN) break;
        GEO_TRY(w);
        it0 = it1;
    }
    int err = 0;
    GEO_CUDA(cudaMemcpyAsync(&err, a.err, 4, cudaMemcpyDeviceToHost, s));
    GEO_CUDA(cudaStreamSynchronize(s));
    if (err) return fail(GEO_ERR_CUDA, "2D TTI shot: a device-side wait timed out");
    GEO_TRY(wd.verdict(s, "2D TTI shot"));
    GEO_CUDA(cudaMemcpyAsync(shot, drec, (size_t)nx * nt * 4, kout, s));
    GEO_CUDA(cudaStreamSynchronize(s));
    return GEO_OK;
}

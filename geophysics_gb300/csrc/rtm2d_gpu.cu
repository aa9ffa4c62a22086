// 2D RTM with the semantics of the 2D GPU RTM program
// (2D-vti-fd+rtm-cuda/Toa_gpu2DvtiFdRtmAdcigsLaplace.cu, RTM() :1184-1566).
// Per shot:
//   forward, SV taper on (R=18, r=7, update_stress :303-404): point source
//     before the velocity update (add_source :204), record P at row npml
//     (shot_record :498), save the ring of P,Q (wavefield_bndr :532: rows
//     npml-1 and npml+nz+1, columns npml-1 and npml+nx+1), source
//     illumination ill += P*P + Q*Q, then <= 0 -> 1 (cal_illumination :654);
//   direct-wave mute of the record (mute_directwave :614, tt = 20 in the
//     program) -- the program launches one thread per sample rounded up to
//     512 without a bound on the sample index, so the surplus threads zero
//     samples of later traces; those samples are zeroed too;
//   backward, SV taper off: restore the ring into the source field and step
//     it forward, write the record into P and Q of the receiver field at row
//     npml (shot_record with record = false) and step it, image mig += sP*gP
//     (cal_migration :679) and the Poynting angle gathers (Poynting_Adcigs
//     :718-766).
// After the shots: mig /= ill, gathers /= ill (migration_illum :700,
// adcigs_illum :768), the adjoint Laplacian of the image and of the angle
// stack (stk_adcigs :799).  The image kernels of the program run over
// nnx*nnz threads on nx*nz arrays (an overrun); here they cover nx*nz.
// The steps are those of step2d.cu.
//
// The 2D TTI GPU RTM program (2D-tti-fd+rtm-cuda/
// Toa_gpu_2dtti_rtm_adcigs_iorderfunciton.cu, main :500-800) has the same
// shot structure and runs through the same driver with its own choices:
// the TTI update_vel / update_stress (:126-228) over the tilt field, SV taper
// R=15, r=4, a mute with a sample bound whose direct-wave velocity is
// vp[1]*(1+(sqrtf(1+2 eps[1])-1)*cos(theta[1])) (:336-358, tt = 30 in the
// program), its own sponge (d0 with 3.0 in place of 10.0, whole-cell
// distances for both profile pairs; :230-233, :289-320), gathers at every
// dcdp-th CDP (Poynting_Adcigs :454-486,
// adcigs_illum :488-498), no angle stack and no readFile checks.  Where the
// program's adcigs_illum bound ((nx*nz)/dcdp*na) runs past its gathers
// array (nx not a multiple of dcdp) it divides floats beyond the array;
// here only the nx/dcdp gathers are divided.
#include "geo_internal.h"
#include "adcig.cuh"
#include "model2d.cuh"
#include "step2d.cuh"
#include <cmath>
#include <cstring>
#include <vector>

namespace geo {

// Zero samples lo <= it < hi of every trace, as flat positions ix*nt + it of
// the trace-major record inside it (the record itself is time-major).
__global__ void k_g_mute(float *rec, const int *lo, const int *hi, int nx, int nt) {
    const int it = blockIdx.x * blockDim.x + threadIdx.x;
    for (int ix = blockIdx.y; ix < nx; ix += gridDim.y) {
        if (it < lo[ix] || it >= hi[ix]) continue;
        const long j = (long)ix * nt + it;
        if (j < (long)nx * nt) rec[(j % nt) * nx + j / nt] = 0.0f;
    }
}

// gathers [ixa][ia][iz] /= ill[ixa*dcdp][iz]
__global__ void k_g_adcig_norm(float *adcig, const float *ill, int nxa, int nz, int nangle, int dcdp) {
    const long n = (long)nxa * nz * nangle;
    for (long k = blockIdx.x * (long)blockDim.x + threadIdx.x; k < n; k += (long)gridDim.x * blockDim.x) {
        const int ix = (int)(k / ((long)nz * nangle)) * dcdp, iz = (int)(k % nz);
        adcig[k] = adcig[k] / ill[iz + (long)nz * ix];
    }
}

// angle stack (stk_adcigs :799-818): stk = 0, += over the angles in order
__global__ void k_g_stack_angles(const float *adcig, float *stk, int nx, int nz, int nangle) {
    const long n = (long)nx * nz;
    for (long o = blockIdx.x * (long)blockDim.x + threadIdx.x; o < n; o += (long)gridDim.x * blockDim.x) {
        const int ix = (int)(o / nz), iz = (int)(o % nz);
        float s = 0.0f;
        for (int ia = 0; ia < nangle; ia++) s += adcig[(long)ix * nangle * nz + (long)ia * nz + iz];
        stk[o] = s;
    }
}

// The programs' bin of a cosine a: (int)((float)(0.5*acosf(a)*180.0/pi) / (dangle*1.0)),
// with the device's acosf, as their Poynting_Adcigs kernels evaluate it.
__device__ int ref_gpu_bin(float a, int dangle) {
    const float deg = (float)(0.5 * acosf(a) * 180.0 / kPiGui);
    return (int)(deg / (dangle * 1.0));
}

// Float keys ordered like the floats they encode.
__device__ uint32_t okey(float f) {
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__device__ float kfloat(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// One thread per bin k < kMaxAngles: thr[k] = largest float a in [-1,1]
// with bin(a) >= k+1 (binary search over the ordered float keys; bin is
// non-increasing in a), -2 where none is; cs[k] = cosf(k*pi/180).  Both
// come from the device's acosf and cosf, the functions the programs'
// kernels call, so the tables give their bins and weights bit for bit.
__global__ void k_angle_tables(float *thr, float *cs, int nangle, int dangle) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= kMaxAngles) return;
    cs[k] = k < nangle ? cosf((float)(k * kPiGui / 180.0)) : 0.0f;
    float t = -2.0f;
    if (k < nangle && ref_gpu_bin(-1.0f, dangle) >= k + 1) {
        uint32_t a = okey(-1.0f), b = okey(1.0f);
        while (a < b) {
            const uint32_t m = a + (b - a + 1) / 2;
            if (ref_gpu_bin(kfloat(m), dangle) >= k + 1) a = m;
            else b = m - 1;
        }
        t = kfloat(a);
    }
    thr[k] = t;
}

int adcig_angle_tables(int nangle, int dangle, float *thr, float *cs, cudaStream_t s) {
    k_angle_tables<<<1, kMaxAngles, 0, s>>>(thr, cs, nangle, dangle);
    return check_launch("angle_tables");
}

__device__ float g_angle_stage[2 * kMaxAngles];

static int gpu_adcig_tables(int nangle, int dangle, cudaStream_t s) {
    void *stage = nullptr;
    GEO_CUDA(cudaGetSymbolAddress(&stage, g_angle_stage));
    float *st = static_cast<float *>(stage);
    GEO_TRY(adcig_angle_tables(nangle, dangle, st, st + kMaxAngles, s));
    return load_step2d_angles(st, st + kMaxAngles, s);
}

// readFile's checks (:930-965): grid spacing for the frequency, dt, dispersion, stability.
static int gpu_rtm_checks(const geo_rtm2d_gpu_desc &D, float vmin, float vmax) {
    const float H_min = D.dx < D.dz ? D.dx : D.dz;
    const float dt_max = (float)(0.5 * H_min / vmin), dxz_max = (float)(vmax / D.favg * 0.2);
    if (dxz_max < D.dz || dxz_max < D.dx) return fail(GEO_ERR_CFL, "grid spacing too coarse for favg (redefine dx, dz)");
    if (dt_max < D.dt) return fail(GEO_ERR_CFL, "dt too large (redefine dt)");
    if (D.favg >= vmin / (5.0 * (D.dx > D.dz ? D.dx : D.dz))) return fail(GEO_ERR_CFL, "non-dispersion relation not satisfied");
    const float tmp = (float)(D.dt * vmax * sqrtf((float)(1.0 / (D.dx * D.dx) + 1.0 / (D.dz * D.dz))));
    if (tmp >= 0.777f) return fail(GEO_ERR_CFL, "stability condition not satisfied (%g >= 0.777)", tmp);
    return GEO_OK;
}

static int grid_of_n(long n) { return (int)std::min<long>((n + 255) / 256, 152L * 16); }

}  // namespace geo

namespace geo {

// What differs between the two GPU RTM programs that share this driver.
struct GpuRtmProgram {
    bool tti;            // TTI stencil over a tilt field (theta, degrees)
    int taper_R, taper_r;  // SV taper radii of the forward stress update
    bool mute_overrun;   // the mute launch has no sample bound (VTI program)
    bool checks;         // readFile's dispersion / stability checks (VTI program)
};

static int gpu_rtm_run(const GpuRtmProgram &prog, const geo_rtm2d_gpu_desc &D, const float *v, const float *e,
                       const float *d, const float *theta, const float *obs, float *mig_lap, float *illum,
                       float *adcigs, float *stk_lap, float *shots, int mem, void *stream) {
    if (D.nx < 2 || D.nz < 2 || D.npml < 5 || D.nt < 1 || D.ns < 1) return fail(GEO_ERR_ARG, "bad sizes");
    if (!(D.dt > 0) || !(D.dx > 0) || !(D.dz > 0) || !(D.favg > 0)) return fail(GEO_ERR_ARG, "bad spacing");
    if (D.nangle < 1 || D.nangle > 128 || D.dangle < 1) return fail(GEO_ERR_ARG, "nangle must be 1..128, dangle >= 1");
    const int dcdp = D.dcdp > 0 ? D.dcdp : 1;
    if (dcdp > D.nx) return fail(GEO_ERR_ARG, "dcdp exceeds nx");
    if (dcdp != 1 && !prog.tti) return fail(GEO_ERR_ARG, "the VTI program forms gathers at every CDP (dcdp 0 or 1)");
    if (mem != GEO_MEM_HOST && mem != GEO_MEM_DEVICE) return fail(GEO_ERR_ARG, "bad mem kind");
    const int nx = D.nx, nz = D.nz, npml = D.npml, nt = D.nt, nnx = nx + 2 * npml, nnz = nz + 2 * npml;
    // columns of the fused step's arrays are of a pitch that TMA takes
    const int ldz = (nnz + 3) / 4 * 4, mid = (int)((size_t)nnx * nnz / 2 / nnz);
    const size_t n0 = (size_t)nx * nz, n = (size_t)nnx * ldz;
    cudaStream_t s = (cudaStream_t)stream;
    Raw2D raw;
    GEO_TRY(raw.open(nx, nz, v, e, d, prog.tti ? theta : nullptr, mem, s));
    // the values the host formulas read: vp at the padded centre (d0), vp and
    // eps at padded index 1 (the mute: the model's first cell, the sponge
    // being at least five wide), eps and del on every shot's SV taper box
    // (centre fs+(is-1)ds+npml, zs+npml)
    const int TR = prog.taper_R, tr = prog.taper_r, nb = 2 * TR + 1;
    auto at = [&](int a, int ix, int iz) {   // padded position
        return raw_at(a, raw, std::min(std::max(ix - npml, 0), nx - 1), std::min(std::max(iz - npml, 0), nz - 1));
    };
    std::vector<unsigned long long> pick;
    pick.push_back(at(0, mid, (int)((size_t)nnx * nnz / 2 % nnz)));
    pick.push_back(at(0, 0, 1));
    pick.push_back(at(1, 0, 1));
    for (int is = 1; is <= D.ns; is++) {
        const int cx = D.fs + (is - 1) * D.ds + npml, cz = D.zs + npml;
        for (int b = 0; b < nb * nb; b++) {
            pick.push_back(at(1, cx - TR + b / nb, cz - TR + b % nb));
            pick.push_back(at(2, cx - TR + b / nb, cz - TR + b % nb));
        }
    }
    RawStats rs;
    GEO_TRY(raw_stats(raw, pick, rs, s));
    if (prog.checks) GEO_TRY(gpu_rtm_checks(D, rs.vmin, rs.vmax));
    for (int is = 1; is <= D.ns; is++) {
        const int ixs = D.fs + (is - 1) * D.ds + npml - 1, izs = D.zs + npml - 1;
        if (ixs < 4 || ixs >= nnx - 4 || izs < 4 || izs >= nnz - 4) return fail(GEO_ERR_ARG, "shot %d outside the grid", is);
    }
    // get_d0 and initial_coffe of the program (VTI :110-118; TTI :230-233, :289-320)
    const Variant sp = prog.tti ? V_TTIRTM : V_GPU;
    const float d0 = sponge_d0(sp, 2, 0.0f, rs.val[0], npml, D.dx, D.dx, D.dz);
    std::vector<float> prof(4 * (size_t)(nnx + ldz), 1.0f);
    float *q = prof.data();
    sponge_profiles(sp, nx, npml, D.dt, d0, q, q + nnx, q + 2 * nnx, q + 3 * nnx);
    q += 4 * nnx;
    sponge_profiles(sp, nz, npml, D.dt, d0, q, q + ldz, q + 2 * ldz, q + 3 * ldz);
    std::vector<float> amp;
    std::vector<uint8_t> on;
    source_amplitudes(V_GPU, nt, D.dt, D.favg, D.pfac, D.wtype, amp, on);
    Blob small;
    const size_t o_prof = small.put(prof), o_amp = small.put(amp), o_on = small.put(on);
    // tapered 1+2eps, sqrtf(1+2del) of every shot's box
    std::vector<size_t> o_te2(D.ns), o_td2(D.ns);
    for (int is = 1; is <= D.ns; is++) {
        std::vector<float> te2(nb * nb), td2(nb * nb);
        const float *box = rs.val.data() + 3 + (size_t)(is - 1) * 2 * nb * nb;
        for (int b = 0; b < nb * nb; b++) {
            const int rx = b / nb - TR, rz = b % nb - TR, q2 = rx * rx + rz * rz;
            float ee = box[2 * b], dd = box[2 * b + 1];
            if (q2 <= tr * tr) {
                ee = dd = 0.0f;
            } else if (q2 <= TR * TR) {
                const double gq = 0.5 * (1 - std::cos(kPiGui * ((sqrtf((float)q2) - tr) * 4.0 / (TR * 3.0 - 1))));
                ee = (float)(gq * ee);
                dd = (float)(gq * dd);
            }
            te2[b] = 1 + 2 * ee;
            td2[b] = sqrtf(1 + 2 * dd);
        }
        o_te2[is - 1] = small.put(te2);
        o_td2[is - 1] = small.put(td2);
    }
    GEO_TRY(small.upload(s));
    float mu_v = rs.val[1] * sqrtf(1 + 2 * rs.val[2]);   // direct-wave velocity of the VTI program's mute
    const int L = 2 * nx + 2 * nz;
    const int nxa = nx / dcdp;
    const size_t nag = (size_t)D.nangle * nz * nxa;
    const bool gathers = adcigs || stk_lap;
    // one allocation; the state a shot starts from is cleared together
    Arena ar;
    float *fS = nullptr, *fR = nullptr, *rec = nullptr, *ring = nullptr, *mig = nullptr, *ill = nullptr, *ag = nullptr;
    float *dvp = nullptr, *dtvp = nullptr, *dct = nullptr, *dsn = nullptr;
    float *lap = nullptr, *stk = nullptr, *trs = nullptr;
    int *mlo = nullptr;
    unsigned *sync = nullptr;
    size_t shot_end = 0, clear_end = 0;
    for (int pass = 0; pass < 2; pass++) {
        fS = ar.take<float>(12 * n);
        fR = ar.take<float>(12 * n);
        rec = ar.take<float>((size_t)nt * nx);
        ring = ar.take<float>((size_t)2 * nt * L);
        shot_end = ar.off;
        mig = ar.take<float>(n0);
        ill = ar.take<float>(n0);
        if (gathers) ag = ar.take<float>(nag);
        sync = ar.take<unsigned>(2);
        clear_end = ar.off;
        dvp = ar.take<float>(3 * n);    // vp, 1+2eps, sqrtf(1+2del)
        dtvp = ar.take<float>(3 * n);   // the shot's, with the SV taper
        if (prog.tti) {
            dct = ar.take<float>(2 * n);   // cos and sin of the tilt
            dsn = dct + n;
        }
        lap = ar.take<float>(n0);
        if (stk_lap) stk = ar.take<float>(n0);
        if (shots || obs) trs = ar.take<float>((size_t)nt * nx);
        mlo = ar.take<int>(2 * (size_t)nx);
        if (pass == 0) GEO_TRY(ar.alloc());
    }
    float *de2 = dvp + n, *dd2 = de2 + n, *dte2 = dtvp + n, *dtd2 = dte2 + n;
    GEO_CUDA(cudaMemsetAsync(ar.buf.p, 0, clear_end, s));
    ModelJob job{};
    job.nx = nx; job.nz = nz; job.npd = npml; job.ldz = ldz;
    job.vp = dvp; job.e2 = de2; job.d2 = dd2; job.rad = dct;
    GEO_TRY(launch_model2d(raw, {job}, s));
    if (prog.tti) {
        // tilt in radians as read_file converts it (theta *= pi/180); its cos
        // and sin as the program's kernels form them
        GEO_TRY(launch_tilt_trig(dct, dsn, n, s));
        // mute_directwave of the TTI program: vp[1]*(1+(sqrtf(1+2 eps[1])-1)*cos(theta[1]))
        float c1 = 0.0f;
        GEO_CUDA(cudaMemcpyAsync(&c1, dct + 1, 4, cudaMemcpyDeviceToHost, s));
        GEO_CUDA(cudaStreamSynchronize(s));
        mu_v = rs.val[1] * (1 + (sqrtf(1 + 2 * rs.val[2]) - 1) * c1);
    }
    if (gathers) GEO_TRY(gpu_adcig_tables(D.nangle, D.dangle, s));
    SStep st{};
    SGrid &g = st.g;
    g.nnx = nnx; g.nnz = nnz; g.ldz = ldz; g.npd = npml; g.nx = nx; g.nz = nz;
    g.dtx = D.dt / D.dx;
    g.dtz = D.dt / D.dz;
    const float *pp = small.at<float>(o_prof);
    g.cx1 = pp; g.cx2 = pp + nnx; g.ax1 = pp + 2 * nnx; g.ax2 = pp + 3 * nnx;
    g.zp = pp + 4 * nnx;
    step2d_fields(fS, n, st.f[0]);
    step2d_fields(fR, n, st.f[1]);
    float *bp = ring, *bq = bp + (size_t)nt * L;
    const int gi = grid_of_n((long)n0);
    const cudaMemcpyKind kout = mem == GEO_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
    const cudaMemcpyKind kin = mem == GEO_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
    st.amp = small.at<float>(o_amp);
    st.on = small.at<unsigned char>(o_on);
    st.izs = D.zs + npml - 1;
    st.rec = rec;
    st.bp = bp; st.bq = bq; st.ill = ill; st.mig = mig; st.adcig = ag;
    st.L = L; st.nangle = D.nangle; st.dcdp = dcdp;
    st.bar = sync;
    st.err = reinterpret_cast<int *>(sync) + 1;
    Fused2D fwd, bwd;
    GEO_TRY(fwd.plan(SK_GFWD, prog.tti, g));
    GEO_TRY(fwd.maps(g, st.f[0], 0));
    GEO_TRY(fwd.model(g, dtvp, dct));
    GEO_TRY(bwd.plan(SK_GBWD, prog.tti, g));
    for (int f = 0; f < 2; f++) GEO_TRY(bwd.maps(g, st.f[f], f));
    GEO_TRY(bwd.model(g, dvp, dct));
    Watchdog wd;
    GEO_TRY(wd.open());
    for (int is = 1; is <= D.ns; is++) {
        // the shot's tapered model: the untapered one with its box replaced
        GEO_CUDA(cudaMemcpyAsync(dtvp, dvp, 3 * n * 4, cudaMemcpyDeviceToDevice, s));
        GEO_TRY(launch_box2d(dte2, dtd2, nnx, ldz, D.fs + (is - 1) * D.ds + npml - TR, D.zs + npml - TR, nb,
                             small.at<float>(o_te2[is - 1]), small.at<float>(o_td2[is - 1]), s));
        if (is > 1) GEO_CUDA(cudaMemsetAsync(ar.buf.p, 0, shot_end, s));
        st.ixs = D.fs + (is - 1) * D.ds + npml - 1;
        st.lev = 0;
        // runs of steps between the watchdog's scans, one launch each
        for (st.it0 = 0; st.it0 < nt; st.it0 = st.it1) {
            st.it1 = st.it0 + 1;
            while (st.it1 < nt && !(wd.every > 0 && st.it1 % wd.every == 0)) st.it1++;
            GEO_TRY(fwd.run(st, s));
            st.lev = (st.lev + st.it1 - st.it0) & 1;
            const int w = wd.check(st.f[0].P[st.lev], n, st.it1 - 1, st.it1 == nt, s);
            if (w == GEO_ERR_NAN) break;
            GEO_TRY(w);
        }
        GEO_TRY(wd.verdict(s, "2D RTM forward pass"));
        // direct-wave mute (GPU form, tt), exactly as the program's kernel
        // writes it.  VTI program: thread it < nt rounded up to 512 zeroes
        // flat sample ix*nt + it of the trace-major record for every trace
        // ix whose window holds it -- past nt that lands on later traces.
        // TTI program: one thread per sample, bounded.
        {
            std::vector<int> lohi(2 * (size_t)nx);
            const int nt512 = prog.mute_overrun ? (nt + 511) / 512 * 512 : nt;
            for (int ix = 0; ix < nx; ix++) {
                const float mu_x = D.dx * std::abs(ix - D.fs - (is - 1) * D.ds), mu_z = D.dz * D.zs;
                const float mu_t0 = sqrtf((float)(std::pow(mu_x, 2) + std::pow(mu_z, 2))) / mu_v;
                const int mu_t = (int)(2.0 / (D.dt * D.favg));
                const int mu_nt = (int)(mu_t0 / D.dt) + mu_t + D.mute_tt;
                lohi[ix] = std::max(0, (int)(mu_t0 / D.dt) - D.mute_tt + 1);
                lohi[nx + ix] = std::min(mu_nt, nt512);
            }
            GEO_CUDA(cudaMemcpyAsync(mlo, lohi.data(), lohi.size() * 4, cudaMemcpyHostToDevice, s));
            k_g_mute<<<dim3((nt512 + 255) / 256, std::min(nx, 65535)), 256, 0, s>>>(rec, mlo, mlo + nx, nx, nt);
            GEO_TRY(check_launch("grtm_mute"));
            GEO_CUDA(cudaStreamSynchronize(s));
        }
        if (shots) {
            GEO_TRY(launch_transpose_records(rec, trs, nx, nt, s));
            GEO_CUDA(cudaMemcpyAsync(shots + (size_t)(is - 1) * nx * nt, trs, (size_t)nx * nt * 4, kout, s));
        }
        if (obs) {
            // observed shot (trace-major nx*nt) replaces the modelled record
            GEO_CUDA(cudaMemcpyAsync(trs, obs + (size_t)(is - 1) * nx * nt, (size_t)nx * nt * 4, kin, s));
            GEO_TRY(launch_transpose_records(trs, rec, nt, nx, s));
        }
        // runs of steps between the watchdog's scans (after backward step it
        // when (nt - it) is a multiple of the interval), one launch each
        for (st.it0 = nt - 1; st.it0 >= 0; st.it0 = st.it1 - 1) {
            st.it1 = st.it0;
            while (st.it1 > 0 && !(wd.every > 0 && (nt - st.it1) % wd.every == 0)) st.it1--;
            GEO_TRY(launch_step2d_restore(st, st.it0, st.lev, s));   // after the scan, which sees a step's own values
            GEO_TRY(bwd.run(st, s));
            st.lev = (st.lev + st.it0 - st.it1 + 1) & 1;
            const int w = wd.check(st.f[1].P[st.lev], n, nt - 1 - st.it1, st.it1 == 0, s);
            if (w == GEO_ERR_NAN) break;
            GEO_TRY(w);
        }
        GEO_TRY(wd.verdict(s, "2D RTM backward pass"));
    }
    {
        int err = 0;
        GEO_CUDA(cudaMemcpyAsync(&err, st.err, 4, cudaMemcpyDeviceToHost, s));
        GEO_CUDA(cudaStreamSynchronize(s));
        if (err) return fail(GEO_ERR_CUDA, "2D RTM: a device-side wait timed out");
    }
    GEO_TRY(launch_normalize_image(mig, ill, n0, s));
    GEO_TRY(launch_laplace2d(nx, nz, mig, lap, s));
    GEO_CUDA(cudaMemcpyAsync(mig_lap, lap, n0 * 4, kout, s));
    if (illum) GEO_CUDA(cudaMemcpyAsync(illum, ill, n0 * 4, kout, s));
    if (gathers) {
        k_g_adcig_norm<<<grid_of_n((long)nag), 256, 0, s>>>(ag, ill, nxa, nz, D.nangle, dcdp);
        GEO_TRY(check_launch("grtm_adcig_norm"));
        if (adcigs) GEO_CUDA(cudaMemcpyAsync(adcigs, ag, nag * 4, kout, s));
        if (stk_lap) {
            k_g_stack_angles<<<gi, 256, 0, s>>>(ag, stk, nx, nz, D.nangle);
            GEO_TRY(check_launch("grtm_stack_angles"));
            GEO_TRY(launch_laplace2d(nx, nz, stk, lap, s));
            GEO_CUDA(cudaMemcpyAsync(stk_lap, lap, n0 * 4, kout, s));
        }
    }
    GEO_CUDA(cudaStreamSynchronize(s));
    return GEO_OK;
}

}  // namespace geo

using namespace geo;

extern "C" int geo_rtm2d_gpu(const geo_rtm2d_gpu_desc *desc, const float *v, const float *e, const float *d,
                             const float *obs, float *mig_lap, float *illum, float *adcigs, float *stk_lap,
                             float *shots, int mem, void *stream) {
    if (!desc || !v || !e || !d || !mig_lap) return fail(GEO_ERR_ARG, "null argument");
    const GpuRtmProgram vti{false, 18, 7, true, true};
    return gpu_rtm_run(vti, *desc, v, e, d, nullptr, obs, mig_lap, illum, adcigs, stk_lap, shots, mem, stream);
}

extern "C" int geo_rtm2d_tti(const geo_rtm2d_gpu_desc *desc, const float *v, const float *e, const float *d,
                             const float *theta, const float *obs, float *mig_lap, float *illum, float *adcigs,
                             float *shots, int mem, void *stream) {
    if (!desc || !v || !e || !d || !theta || !mig_lap) return fail(GEO_ERR_ARG, "null argument");
    const GpuRtmProgram tti{true, 15, 4, false, false};
    return gpu_rtm_run(tti, *desc, v, e, d, theta, obs, mig_lap, illum, adcigs, nullptr, shots, mem, stream);
}

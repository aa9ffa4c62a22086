// 2D drivers: single-shot forward modelling (fused steps of step2d.cu; the
// MPI form the half-steps of fd2d.cu) and batched RTM (fused steps of
// march2d.cu over every shot, the time loops captured once into CUDA graphs
// and replayed).
#include "geo_internal.h"
#include "model2d.cuh"
#include "march2d.cuh"
#include "step2d.cuh"
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>

namespace geo {

// One shot's window of the model and its source.
struct ShotGeom {
    int nx, col0;        // window width, model column of window column 0
    float srcx, srcz;    // source position inside the window, 1-based
};

// The shots of one run on the device: model and state in one allocation,
// the profiles and taper boxes in another.
struct ShotSet {
    Variant var;
    int nz, npd, nnz;
    bool taper;
    std::vector<ShotGeom> G;
    RawStats st;
    float v00, e00;               // model values at unpadded (0, 0)
    std::vector<float> mu_v;      // MPI mute velocity of each shot
    Arena mem;
    Blob small;
    static constexpr int kPick = 3 + 3 * kTB * kTB;   // centre v, v(1,1), e(1,1); v, e, d on the taper box
    void source(int k, int &ixs, int &izs) const {
        // source cell: (int)(fs+0.5)+npd-1 (CPU_vti2dfd_kernels.c:65-66)
        ixs = (int)(G[k].srcx + 0.5) + npd - 1;
        izs = (int)(G[k].srcz + 0.5) + npd - 1;
    }
    // CPU/MPI circle centre = the source cell; GPU form centre is
    // (fs+(is-1)ds+npd, zs+npd), one cell right/down of it
    void centre(int k, int &cx, int &cz) const {
        source(k, cx, cz);
        if (var == V_GPU) {
            cx++;
            cz++;
        }
    }
    int read(const Raw2D &raw, cudaStream_t s);
    // profiles and taper box of shot k: offsets in `small`
    struct Off {
        size_t xprof, zprof, te2, td2;        // xprof cx1 cx2 ax1 ax2; zprof cz1 cz2 az1 az2, ldz each
        Taper2D box;
        std::vector<float> vbox;              // v on the taper box
        std::vector<float> p[8];
    };
    void tables(int k, float dx, float dz, float dt, int ldz, Off &o);
};

// The model values the set-up formulas read, with the model check.
int ShotSet::read(const Raw2D &raw, cudaStream_t s) {
    std::vector<unsigned long long> pick;
    pick.reserve(2 + G.size() * kPick);
    pick.push_back(raw_at(0, raw, 0, 0));
    pick.push_back(raw_at(1, raw, 0, 0));
    for (size_t k = 0; k < G.size(); k++) {
        const int nx = G[k].nx, nnx = nx + 2 * npd;
        auto at = [&](int a, int ix, int iz) {   // padded position
            const int sx = std::min(std::max(ix - npd, 0), nx - 1) + G[k].col0;
            const int sz = std::min(std::max(iz - npd, 0), nz - 1);
            return raw_at(a, raw, std::min(sx, raw.nx - 1), sz);
        };
        const size_t c = (size_t)nnx * nnz / 2;
        pick.push_back(at(0, (int)(c / nnz), (int)(c % nnz)));
        pick.push_back(at(0, 1 + npd, 1 + npd));
        pick.push_back(at(1, 1 + npd, 1 + npd));
        int cx, cz;
        centre(k, cx, cz);
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < kTB * kTB; b++)
                pick.push_back(taper ? at(a, cx - kTB / 2 + b / kTB, cz - kTB / 2 + b % kTB) : 0);
    }
    GEO_TRY(raw_stats(raw, pick, st, s));
    v00 = st.val[0];
    e00 = st.val[1];
    return GEO_OK;
}

// The sponge profiles (of pitch ldz along z, ones beyond nnz), taper box and
// mute velocity of shot k; var picks the reference program's formulas.
void ShotSet::tables(int k, float dx, float dz, float dt, int ldz, Off &o) {
    const ShotGeom &g = G[k];
    const int nnx = g.nx + 2 * npd;
    const float *val = st.val.data() + 2 + (size_t)k * kPick;
    float vpmax = 0.0f;
    for (int c = 0; c < g.nx; c++) vpmax = std::max(vpmax, st.colmax[std::min(c + g.col0, (int)st.colmax.size() - 1)]);
    const float d0 = sponge_d0(var, 2, vpmax, val[0], npd, dx, dx, dz);
    mu_v.resize(G.size());
    mu_v[k] = val[1] * sqrtf(1 + 2 * val[2]);
    for (int q = 0; q < 8; q++) o.p[q].assign(q < 4 ? nnx : ldz, 1.0f);
    sponge_profiles(var, g.nx, npd, dt, d0, o.p[0].data(), o.p[1].data(), o.p[2].data(), o.p[3].data());
    sponge_profiles(var, nz, npd, dt, d0, o.p[4].data(), o.p[5].data(), o.p[6].data(), o.p[7].data());
    std::vector<float> px, pz;
    for (int q = 0; q < 4; q++) {
        px.insert(px.end(), o.p[q].begin(), o.p[q].end());
        pz.insert(pz.end(), o.p[4 + q].begin(), o.p[4 + q].end());
    }
    o.xprof = small.put(px);
    o.zprof = small.put(pz);
    if (!taper) return;
    int cx, cz;
    centre(k, cx, cz);
    const float *vbox = val + 3;
    o.vbox.assign(vbox, vbox + kTB * kTB);
    sv_taper_2d(var, nnx, nnz, cx, cz, vbox + kTB * kTB, vbox + 2 * kTB * kTB, o.box);
    std::vector<float> te2(kTB * kTB), td2(kTB * kTB);
    for (int b = 0; b < kTB * kTB; b++) {
        te2[b] = 1 + 2 * o.box.e[b];
        td2[b] = sqrtf(1 + 2 * o.box.d[b]);
    }
    o.te2 = small.put(te2);
    o.td2 = small.put(td2);
}

// One shot of the MPI form on the device for the half-steps of fd2d.cu.
struct SingleShot {
    ShotSet X;
    Shot2D S{};
    size_t o_amp = 0, o_on = 0;
    int build(const Raw2D &raw, float dx, float dz, float dt, const std::vector<float> &amp,
              const std::vector<uint8_t> &on, int nt, cudaStream_t s);
};

int SingleShot::build(const Raw2D &raw, float dx, float dz, float dt, const std::vector<float> &amp,
                      const std::vector<uint8_t> &on, int nt, cudaStream_t s) {
    const int nx = X.G[0].nx, nz = X.nz, npd = X.npd, nnx = nx + 2 * npd, nnz = X.nnz;
    // the MPI program's pz and qx chains are
    //   (double)(az2*pz) - (double)(az1*vp) * pow(1+2del,0.5) * (double)dtz * (double)zz
    // (and with ax, dtx, xx for qx), evaluated left to right; every factor but
    // zz is fixed for the shot, so the product of the first three is formed
    // once, in the same order and precision (ModelJob::kz), and the kernel
    // issues one double multiply and one double subtraction per chain.  The
    // program's pow runs on the host, once per model point.
    const double ddtx = (double)(dt / dx), ddtz = (double)(dt / dz);
    DevBuf d_pw;
    GEO_TRY(upload_pow_half(raw, d_pw, s));
    ShotSet::Off o;
    X.tables(0, dx, dz, dt, nnz, o);
    std::vector<double> tkz(kTB * kTB, 0.0), tkx(kTB * kTB, 0.0);
    for (int b = 0; b < kTB * kTB; b++) {
        const int ix = o.box.x0 + b / kTB, iz = o.box.z0 + b % kTB;
        if (ix < 0 || ix >= nnx || iz < 0 || iz >= nnz) continue;
        const double pw = std::pow((double)(1 + 2 * o.box.d[b]), 0.5);
        const float vpk = 1.0f * (o.vbox[b] * o.vbox[b]);
        tkz[b] = (double)(o.p[6][iz] * vpk) * pw * ddtz;
        tkx[b] = (double)(o.p[2][ix] * vpk) * pw * ddtx;
    }
    const size_t o_tkz = X.small.put(tkz), o_tkx = X.small.put(tkx);
    o_amp = X.small.put(amp);
    o_on = X.small.put(on);
    GEO_TRY(X.small.upload(s));
    const size_t n = (size_t)nnx * nnz;
    ModelJob j{};
    size_t clear = 0;
    for (int pass = 0; pass < 2; pass++) {   // sizes, then addresses
        float **dst[8] = {&S.u, &S.w, &S.P, &S.Q, &S.px, &S.pz, &S.qx, &S.qz};
        for (auto d : dst) *d = X.mem.take<float>(n);
        S.rec_p = X.mem.take<float>((size_t)nt * nx);
        clear = X.mem.off;
        j.vp = X.mem.take<float>(n);
        j.e2 = X.mem.take<float>(n);
        j.kz = X.mem.take<double>(n);
        j.kx = X.mem.take<double>(n);
        if (pass == 0) GEO_TRY(X.mem.alloc());
    }
    S.nnx = nnx; S.nnz = nnz; S.npd = npd; S.nx = nx; S.nz = nz;
    S.dtx = dt / dx; S.dtz = dt / dz;
    const float *xp = X.small.at<float>(o.xprof), *zp = X.small.at<float>(o.zprof);
    S.cx1 = xp; S.cx2 = xp + nnx; S.ax1 = xp + 2 * nnx; S.ax2 = xp + 3 * nnx;
    S.cz1 = zp; S.cz2 = zp + nnz; S.az1 = zp + 2 * nnz; S.az2 = zp + 3 * nnz;
    X.source(0, S.ixs, S.izs);
    S.tx0 = o.box.x0;
    S.tz0 = o.box.z0;
    S.te2 = X.small.at<float>(o.te2);
    S.tkz = X.small.at<double>(o_tkz);
    S.tkx = X.small.at<double>(o_tkx);
    j.nx = nx; j.nz = nz; j.npd = npd; j.ldz = nnz;
    j.vp2 = 1;   // vp <- rho*vp^2 with rho == 1 (Toa_rtm_vti_adcig_cdp.c:641)
    j.pw = d_pw.as<double>();
    j.ax1 = S.ax1; j.az1 = S.az1;
    j.ddtx = ddtx; j.ddtz = ddtz;
    S.vp = j.vp; S.e2 = j.e2; S.kz = j.kz; S.kx = j.kx;
    GEO_TRY(launch_model2d(raw, {j}, s));
    GEO_CUDA(cudaMemsetAsync(X.mem.buf.p, 0, clear, s));
    return GEO_OK;
}

// One shot of the CPU or GPU form on the device for the fused steps of
// step2d.cu.
struct FusedShot {
    ShotSet X;
    SStep st{};
    Fused2D plan;
    size_t n = 0;                 // floats of an array
    int build(const Raw2D &raw, float dx, float dz, float dt, const std::vector<float> &amp,
              const std::vector<uint8_t> &on, int nt, cudaStream_t s);
    const float *P() const { return st.f[0].P[st.lev]; }
};

int FusedShot::build(const Raw2D &raw, float dx, float dz, float dt, const std::vector<float> &amp,
                     const std::vector<uint8_t> &on, int nt, cudaStream_t s) {
    const int nx = X.G[0].nx, nz = X.nz, npd = X.npd, nnx = nx + 2 * npd, nnz = X.nnz, ldz = (nnz + 3) / 4 * 4;
    ShotSet::Off o;
    X.tables(0, dx, dz, dt, ldz, o);
    const size_t o_amp = X.small.put(amp), o_on = X.small.put(on);
    GEO_TRY(X.small.upload(s));
    n = (size_t)nnx * ldz;
    float *f = nullptr, *model = nullptr;
    unsigned *sync = nullptr;
    size_t clear = 0;
    for (int pass = 0; pass < 2; pass++) {   // sizes, then addresses
        f = X.mem.take<float>(12 * n);
        st.rec = X.mem.take<float>((size_t)nt * nx);
        sync = X.mem.take<unsigned>(2);
        clear = X.mem.off;
        model = X.mem.take<float>(3 * n);
        if (pass == 0) GEO_TRY(X.mem.alloc());
    }
    SGrid &g = st.g;
    g.nnx = nnx; g.nnz = nnz; g.ldz = ldz; g.npd = npd; g.nx = nx; g.nz = nz;
    g.dtx = dt / dx; g.dtz = dt / dz;
    const float *xp = X.small.at<float>(o.xprof);
    g.cx1 = xp; g.cx2 = xp + nnx; g.ax1 = xp + 2 * nnx; g.ax2 = xp + 3 * nnx;
    g.zp = X.small.at<float>(o.zprof);
    step2d_fields(f, n, st.f[0]);
    X.source(0, st.ixs, st.izs);
    st.amp = X.small.at<float>(o_amp);
    st.on = X.small.at<unsigned char>(o_on);
    st.bar = sync;
    st.err = reinterpret_cast<int *>(sync) + 1;
    ModelJob j{};
    j.nx = nx; j.nz = nz; j.npd = npd; j.ldz = ldz;
    j.vp = model; j.e2 = model + n; j.d2 = model + 2 * n;
    GEO_TRY(launch_model2d(raw, {j}, s));
    if (X.taper)
        GEO_TRY(launch_box2d(j.e2, j.d2, nnx, ldz, o.box.x0, o.box.z0, kTB, X.small.at<float>(o.te2),
                             X.small.at<float>(o.td2), s));
    GEO_CUDA(cudaMemsetAsync(X.mem.buf.p, 0, clear, s));
    // GEO_FD2D_TILE=TZxTX: tiles of 16 columns from TX 16, of 8 below; a shape
    // no block could hold with its whole state is refused as it always was
    int tz = 0, tx = 0;
    if (const char *e = getenv("GEO_FD2D_TILE"))
        if (sscanf(e, "%dx%d", &tz, &tx) != 2 || tx < 4 || tx > 128) tx = 0;
    GEO_TRY(plan.plan(X.var == V_CPU ? SK_CPU : SK_GPU, false, g, !tx ? 0 : tx < 16 ? 8 : 16));
    if (tx && tz >= 32 && tz <= 256 && !(tz & (tz - 1)) && plan.stages == 1 && 11L * tx * tz + 21L * (tx + tz) > 56320)
        return fail(GEO_ERR_ARG, "GEO_FD2D_TILE %dx%d: tile too large", tz, tx);
    GEO_TRY(plan.maps(g, st.f[0], 0));
    return plan.model(g, model);
}

// A group of consecutive shots of a batched RTM on the device for the fused
// steps: M[k] is shot first + k of the set.
struct MarchBatch {
    ShotSet &X;
    const int first, ns;
    std::vector<March2D> M;
    DevBuf d_M, d_items[2];
    std::vector<int4> items[2];   // forward, backward
    const bool fast, adcig;
    bool wide = false;
    MarchBatch(ShotSet &set, int first_, int ns_, bool fast_, bool adcig_)
        : X(set), first(first_), ns(ns_), fast(fast_), adcig(adcig_) {}
    int build(const Raw2D &raw, float dx, float dz, float dt, int nt, cudaStream_t s);
    int clear_side(int k, int slots, cudaStream_t s) {
        GEO_CUDA(cudaMemsetAsync(M[k].f, 0, (size_t)slots * M[k].n * 4, s));
        return GEO_OK;
    }
    int work(bool backward);
    int step(bool backward, const MarchStep &st, cudaStream_t s) {
        return launch_march2d(backward, fast, adcig, wide, d_M.as<March2D>(), d_items[backward].as<int4>(),
                              (int)items[backward].size(), st, s);
    }
};

// Strips of at most 120 depths and chunks of columns.  A chunk repeats 14
// columns' worth of P and 7 of u, so long chunks save work; short ones
// balance it, since warps on a wavefront's rim take longer (ziv.cuh).
//
// Work for several waves of warps: four waves, within 8 and 48 columns.  16
// shots of 401-1199 columns x 601 take 182 us a forward and 328 us a backward
// step with chunks of about 12, 200 and 376 us with one wave (35 and 70
// columns).
//
// Work that one wave takes in chunks of 8 or fewer: the shortest chunks that
// leave it one wave.  There a step lasts as long as a warp's march, about 8 us
// and 3 a column (2 in the fast form, 9 backward with gathers on full
// wavefields), and half the warps idle.  us a forward and a backward step
// together, chunks of 8 and by the rule: one shot 61x101 + 30 54.9 and 18.4,
// 201x301 64.8 and 22.7, four of 201x301 69.0 and 40.4, eight 78.5 and 62,
// three of 401x401 76.9 and 55.4.
int MarchBatch::work(bool backward) {
    const int nnz = X.nnz, depths = nnz - 8;
    const int strips = (depths + 119) / 120, len = ((depths + strips - 1) / strips + 3) / 4 * 4;
    int res = 0;
    GEO_TRY(march2d_resident(backward, fast, adcig, &res));
    auto chunks = [&](int k, int chunk) { return (M[k].nnx - 8 + chunk - 1) / chunk; };
    int chunk = 0;
    for (int c = 1; c <= 8 && !chunk; c++) {
        long n = 0;
        for (int k = 0; k < ns; k++) n += (long)strips * chunks(k, c);
        if (n <= res) chunk = c;
    }
    const bool one_wave = chunk != 0;
    if (!one_wave) {
        long cols = 0;
        for (int k = 0; k < ns; k++) cols += (long)strips * (M[k].nnx - 8);
        chunk = (int)std::min(48L, std::max(8L, cols / (4L * res)));
    }
    if (const char *e = getenv("GEO_RTM2D_CHUNK"))
        if (const int c = atoi(e); c > 0) chunk = std::min(c, 1 << 20);
    std::vector<int4> &v = items[backward];
    v.clear();
    for (int k = 0; k < ns; k++) {
        const int w = M[k].nnx - 8, nc = one_wave ? chunks(k, chunk) : std::max(1, (w + chunk / 2) / chunk);
        for (int t = 0; t < strips; t++)
            for (int c = 0; c < nc; c++)
                v.push_back(make_int4(k | (len / 4) << 24, t * len, 4 + (int)((long)w * c / nc), 4 + (int)((long)w * (c + 1) / nc)));
    }
    return GEO_OK;
}

int MarchBatch::build(const Raw2D &raw, float dx, float dz, float dt, int nt, cudaStream_t s) {
    const int npd = X.npd, nz = X.nz, nnz = X.nnz, ldz = (nnz + 3) / 4 * 4;
    const ShotGeom *const G = X.G.data() + first;
    X.small.h.clear();
    X.mem.buf.release();   // the last group's
    X.mem.off = 0;
    DevBuf d_pw;
    if (!fast) GEO_TRY(upload_pow_half(raw, d_pw, s));
    std::vector<ShotSet::Off> off(ns);
    std::vector<size_t> o_tpw2(ns), o_tpw(ns);
    for (int k = 0; k < ns; k++) {
        X.tables(first + k, dx, dz, dt, ldz, off[k]);
        if (fast) continue;
        std::vector<double> pw(kTB * kTB);
        std::vector<float> p2(2 * kTB * kTB);
        for (int b = 0; b < kTB * kTB; b++) {
            pw[b] = std::pow((double)(1 + 2 * off[k].box.d[b]), 0.5);
            p2[2 * b] = (float)pw[b];
            p2[2 * b + 1] = (float)(pw[b] - (double)p2[2 * b]);
        }
        o_tpw[k] = X.small.put(pw);
        o_tpw2[k] = X.small.put(p2);
    }
    GEO_TRY(X.small.upload(s));
    M.assign(ns, March2D{});
    std::vector<ModelJob> jobs(ns, ModelJob{});
    for (int pass = 0; pass < 2; pass++) {   // sizes, then addresses
        for (int k = 0; k < ns; k++) {
            const int nx = G[k].nx, nnx = nx + 2 * npd;
            const size_t n = (size_t)nnx * ldz, L = 2 * (size_t)nx + 2 * (size_t)nz;
            March2D &m = M[k];
            m.n = (unsigned)n;
            if ((double)MS_SLOTS * n >= 4294967296.0) wide = true;
            m.f = X.mem.take<float>((fast ? MS_PL : MS_SLOTS) * n);
            if (!fast) m.pw = jobs[k].pwd = X.mem.take<double>(n);
            if (adcig) m.adcig = X.mem.take<float>((size_t)kAdcigAngles * nx * nz);
            m.rec_p = X.mem.take<float>((size_t)nt * nx);
            m.rec_q = X.mem.take<float>((size_t)nt * nx);
            m.edge_p = X.mem.take<float>((size_t)nt * L);
            m.edge_q = X.mem.take<float>((size_t)nt * L);
        }
        X.mem.take<float>(1024);   // the last column's rows run past it
        if (pass == 0) GEO_TRY(X.mem.alloc());
    }
    for (int k = 0; k < ns; k++) {
        March2D &m = M[k];
        const int nx = G[k].nx;
        m.nnx = nx + 2 * npd; m.nnz = nnz; m.ldz = ldz; m.npd = npd; m.nx = nx; m.nz = nz;
        m.dtx = dt / dx; m.dtz = dt / dz;
        const float *xp = X.small.at<float>(off[k].xprof);
        m.cx1 = xp; m.cx2 = xp + m.nnx; m.ax1 = xp + 2 * m.nnx; m.ax2 = xp + 3 * m.nnx;
        m.cz1 = X.small.at<float>(off[k].zprof);
        m.tx0 = off[k].box.x0;
        m.tz0 = off[k].box.z0;
        m.te2 = X.small.at<float>(off[k].te2);
        m.td2 = X.small.at<float>(off[k].td2);
        if (!fast) {
            m.tpw = X.small.at<double>(o_tpw[k]);
            m.tpw2 = X.small.at<float2>(o_tpw2[k]);
        }
        X.source(first + k, m.ixs, m.izs);
        ModelJob &j = jobs[k];
        const size_t n = m.n;
        j.nx = nx; j.nz = nz; j.npd = npd; j.ldz = ldz; j.col0 = G[k].col0;
        j.vp2 = 1;   // vp <- rho*vp^2 with rho == 1 (Toa_rtm_vti_adcig_cdp.c:641)
        j.vp = m.f + MS_VP * n;
        j.e2 = m.f + MS_E2 * n;
        if (fast) {
            j.d2 = m.f + MS_D2 * n;
        } else {
            j.ph = m.f + MS_D2 * n;
            j.pl = m.f + MS_PL * n;
            j.pw = d_pw.as<double>();
        }
        // the model's slots, whose pitch columns beyond nnz are never used, stay as allocated
        GEO_TRY(clear_side(k, MS_STATE, s));
        if (adcig) GEO_CUDA(cudaMemsetAsync(m.adcig, 0, (size_t)kAdcigAngles * nx * nz * 4, s));
        GEO_CUDA(cudaMemsetAsync(m.rec_p, 0, (size_t)nt * nx * 4, s));
        GEO_CUDA(cudaMemsetAsync(m.rec_q, 0, (size_t)nt * nx * 4, s));
    }
    GEO_TRY(launch_model2d(raw, jobs, s));
    GEO_TRY(d_M.alloc(ns * sizeof(March2D)));
    GEO_CUDA(cudaMemcpyAsync(d_M.p, M.data(), ns * sizeof(March2D), cudaMemcpyHostToDevice, s));
    for (int b = 0; b < 2; b++) {
        GEO_TRY(work(b));
        GEO_TRY(d_items[b].alloc(items[b].size() * sizeof(int4)));
        GEO_CUDA(cudaMemcpyAsync(d_items[b].p, items[b].data(), items[b].size() * sizeof(int4), cudaMemcpyHostToDevice, s));
    }
    return GEO_OK;
}

// Work list: item -> shot.  Tiles are 32 (z) x by (x).
static void build_items(std::vector<Shot2D> &S, int by, std::vector<int> &item_shot) {
    item_shot.clear();
    for (size_t k = 0; k < S.size(); k++) {
        S[k].ntz = (S[k].nnz + 31) / 32;
        const int ntx = (S[k].nnx + by - 1) / by;
        S[k].tile_base = (int)item_shot.size();
        item_shot.insert(item_shot.end(), (size_t)S[k].ntz * ntx, (int)k);
    }
}

struct Batch2D {
    std::vector<Shot2D> S;
    std::vector<int> items;
    DevBuf d_S, d_items;
    int by = 8, grid = 1;
    int upload(int by_, int blocks_per_sm, cudaStream_t s) {
        by = by_;
        build_items(S, by, items);
        const int nitems = (int)items.size();
        grid = std::max(1, std::min(nitems, sm_count() * blocks_per_sm));
        GEO_TRY(d_S.alloc(S.size() * sizeof(Shot2D)));
        GEO_TRY(d_items.alloc(items.size() * 4));
        GEO_CUDA(cudaMemcpyAsync(d_S.p, S.data(), S.size() * sizeof(Shot2D), cudaMemcpyHostToDevice, s));
        GEO_CUDA(cudaMemcpyAsync(d_items.p, items.data(), items.size() * 4, cudaMemcpyHostToDevice, s));
        GEO_CUDA(cudaStreamSynchronize(s));
        return GEO_OK;
    }
    int vel(Step2D st, cudaStream_t s) {
        return launch_vel2d(V_MPI, d_S.as<Shot2D>(), d_items.as<int>(), (int)items.size(), by, grid, st, s);
    }
    int stress(Step2D st, cudaStream_t s) {
        return launch_stress2d(V_MPI, d_S.as<Shot2D>(), d_items.as<int>(), (int)items.size(), by, grid, st, s);
    }
};

// GEO_ERR_NOMEM where the device has no room for a graph.
static int no_memory(cudaError_t e, const char *what) {
    if (e == cudaSuccess) return GEO_OK;
    if (e == cudaErrorMemoryAllocation) cudaGetLastError();
    return fail(e == cudaErrorMemoryAllocation ? GEO_ERR_NOMEM : GEO_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

// Graph of a range of steps; capture on a private stream.
struct Graph {
    cudaGraph_t g = nullptr;
    cudaGraphExec_t x = nullptr;
    long long kernels = 0;     // kernel nodes, counted once per replay
    int launch(cudaStream_t s) {
        GEO_TRY(no_memory(cudaGraphLaunch(x, s), "graph launch"));
        count_launch(kernels);
        return GEO_OK;
    }
    ~Graph() {
        if (x) cudaGraphExecDestroy(x);
        if (g) cudaGraphDestroy(g);
    }
};

template <class F>
static int capture(Graph &G, cudaStream_t cs, F &&body) {
    GEO_CUDA(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
    const long long before = launches_so_far();
    int st = body();
    G.kernels = launches_so_far() - before;
    count_launch(-G.kernels);   // captured, not yet run
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamEndCapture(cs, &g);
    if (st != GEO_OK) {
        if (g) cudaGraphDestroy(g);
        return st;
    }
    if (e != cudaSuccess) return fail(GEO_ERR_CUDA, "graph capture: %s", cudaGetErrorString(e));
    G.g = g;
    return no_memory(cudaGraphInstantiate(&G.x, g, 0), "graph instantiation");
}

// Event-ordered hand-off between the caller's stream and a private one.
struct SideStream {
    cudaStream_t cs = nullptr;
    cudaEvent_t ev = nullptr;
    int open(cudaStream_t user) {
        GEO_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
        GEO_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
        GEO_CUDA(cudaEventRecord(ev, user));
        GEO_CUDA(cudaStreamWaitEvent(cs, ev, 0));
        return GEO_OK;
    }
    ~SideStream() {
        if (cs) {
            cudaStreamSynchronize(cs);
            cudaStreamDestroy(cs);
        }
        if (ev) cudaEventDestroy(ev);
    }
};

}  // namespace geo

using namespace geo;

// ---------------------------------------------------------------- FD 2D
extern "C" int geo_fd2d_shot(const geo_fd2d_desc *desc, const float *v, const float *e, const float *d,
                             float *shot, float *snap, int snap_every, int mem, void *stream) {
    if (!desc || !v || !e || !d || !shot) return fail(GEO_ERR_ARG, "null argument");
    const geo_fd2d_desc &D = *desc;
    if (D.nx < 2 || D.nz < 2 || D.npd < 5 || D.nt < 1) return fail(GEO_ERR_ARG, "grid too small (npd >= 5)");
    if (D.variant < GEO_VARIANT_CPU || D.variant > GEO_VARIANT_MPI) return fail(GEO_ERR_ARG, "bad variant");
    if (!(D.dt > 0) || !(D.dx > 0) || !(D.dz > 0) || !(D.favg > 0)) return fail(GEO_ERR_ARG, "bad spacing");
    const int nnx = D.nx + 2 * D.npd, nnz = D.nz + 2 * D.npd;
    if (D.rec_iz < 4 || D.rec_iz >= nnz - 4) return fail(GEO_ERR_ARG, "receiver row outside grid");
    cudaStream_t s = (cudaStream_t)stream;
    const Variant var = (Variant)D.variant;
    SideStream ss;
    GEO_TRY(ss.open(s));
    Raw2D raw;
    GEO_TRY(raw.open(D.nx, D.nz, v, e, d, nullptr, mem, ss.cs));
    const bool taper = var == V_MPI || D.sv;
    SingleShot shot1;
    FusedShot fused;
    ShotSet &X = var == V_MPI ? shot1.X : fused.X;
    X.var = var;
    X.nz = D.nz; X.npd = D.npd; X.nnz = nnz;
    X.taper = taper;
    X.G = {ShotGeom{D.nx, 0, D.fs + (D.is - 1) * D.ds, D.zs}};
    GEO_TRY(X.read(raw, ss.cs));
    GEO_TRY(check_stability(var, 2, X.st.vmin, X.st.vmax, D.dt, D.dx, D.dx, D.dz, D.favg));
    int ixs, izs;
    X.source(0, ixs, izs);
    if (ixs < 4 || ixs >= nnx - 4 || izs < 4 || izs >= nnz - 4)
        return fail(GEO_ERR_ARG, "source outside the updated grid");
    if (var == V_CPU || var == V_MPI)
        if (ixs - 3 < 0 || ixs + 3 >= nnx || izs - 3 < 0 || izs + 3 >= nnz)
            return fail(GEO_ERR_ARG, "source window outside grid");
    std::vector<float> amp;
    std::vector<uint8_t> on;
    source_amplitudes(var, D.nt, D.dt, D.favg, D.pfac, D.wtype, amp, on);
    const size_t nn = (size_t)nnx * nnz;
    const bool snaps = snap && snap_every > 0;
    const cudaMemcpyKind ksnap = mem == GEO_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
    Watchdog wd;
    GEO_TRY(wd.open());
    DevBuf d_sync;
    Batch2D B;
    float *rec = nullptr;
    int *errw = nullptr;
    if (var != V_MPI) {
        GEO_TRY(fused.build(raw, D.dx, D.dz, D.dt, amp, on, D.nt, ss.cs));
        SStep &st = fused.st;
        rec = st.rec;
        errw = st.err;
        st.rec_iz = D.rec_iz;
        st.rec_scale = D.rec_scale;
        // one launch per run of steps between snapshots
        for (st.it0 = 0; st.it0 < D.nt; st.it0 = st.it1) {
            st.it1 = snaps ? st.it0 + 1 : D.nt;
            while (st.it1 < D.nt && (st.it1 - 1) % snap_every != 0) st.it1++;
            GEO_TRY(fused.plan.run(st, ss.cs));
            st.lev = (st.lev + st.it1 - st.it0) & 1;
            const int it = st.it1 - 1;
            if (snaps && it % snap_every == 0)
                GEO_CUDA(cudaMemcpy2DAsync(snap + (size_t)(it / snap_every) * nn, (size_t)nnz * 4, fused.P(),
                                           (size_t)st.g.ldz * 4, (size_t)nnz * 4, nnx, ksnap, ss.cs));
            if (wd.every > 0) {
                GEO_TRY(wd.scan(fused.P(), fused.n, it + 1, ss.cs));
                if (wd.tripped()) break;
            }
        }
    } else {
        GEO_TRY(shot1.build(raw, D.dx, D.dz, D.dt, amp, on, D.nt, ss.cs));
        GEO_TRY(d_sync.alloc(8));
        GEO_TRY(d_sync.zero(ss.cs));
        errw = d_sync.as<int>() + 1;
        B.S = {shot1.S};
        B.S[0].rec_iz = D.rec_iz;
        B.S[0].rec_scale = D.rec_scale;
        rec = B.S[0].rec_p;
        GEO_TRY(B.upload(snaps ? 8 : 16, 8, ss.cs));
        for (int it = 0; snaps && it < D.nt; it++) {
            Step2D st{};
            st.it = it;
            st.amp = amp[it];
            st.src_on = on[it];
            st.taper = 1;
            GEO_TRY(B.vel(st, ss.cs));
            GEO_TRY(B.stress(st, ss.cs));
            if (it % snap_every == 0)
                GEO_CUDA(cudaMemcpyAsync(snap + (size_t)(it / snap_every) * nn, B.S[0].P, nn * 4, ksnap, ss.cs));
            if (wd.every > 0 && ((it + 1) % wd.every == 0 || it == D.nt - 1)) {
                GEO_TRY(wd.scan(B.S[0].P, nn, it + 1, ss.cs));
                if (wd.tripped()) break;
            }
        }
        if (!snaps) {
            // the whole shot in one cooperative launch (grid barriers between
            // the half-steps, bounded waits reported through an error word)
            Persist2D a{};
            a.nt = D.nt;
            a.taper = 1;
            a.amp = X.small.at<float>(shot1.o_amp);
            a.on = X.small.at<unsigned char>(shot1.o_on);
            a.bar = d_sync.as<unsigned>();
            a.err = errw;
            GEO_TRY(launch_fd2d_shot(B.d_S.as<Shot2D>(), B.d_items.as<int>(), (int)B.items.size(), B.by, a, ss.cs));
        }
    }
    int err = 0;
    GEO_CUDA(cudaMemcpyAsync(&err, errw, 4, cudaMemcpyDeviceToHost, ss.cs));
    GEO_CUDA(cudaStreamSynchronize(ss.cs));
    if (err) return fail(GEO_ERR_CUDA, "2D shot: a device-side wait timed out");
    // what a launch left unscanned
    if (wd.every > 0 && (var != V_MPI || !snaps)) {
        if (var == V_MPI) GEO_TRY(wd.scan(B.S[0].P, nn, D.nt, ss.cs));
        GEO_TRY(wd.scan(rec, (size_t)D.nx * D.nt, D.nt, ss.cs));
    }
    GEO_TRY(wd.verdict(ss.cs, "2D shot"));
    DevBuf mlo, mhi, out;
    if (D.mute_tt > 0) {
        std::vector<int> lo, hi;
        // vp[1]*sqrtf(1+2*eps[1]) of the padded model (GPU_vti2dfd_kernels.cu:167):
        // the sponge is at least five cells wide, so the model's first cell
        const float mu_v = X.v00 * sqrtf(1 + 2 * X.e00);
        mute_window_gpu2d(D.nx, D.nt, D.dt, D.favg, D.dx, D.dz, (int)D.fs, (int)D.ds, (int)D.zs, D.is, mu_v, D.mute_tt,
                          lo, hi);
        GEO_TRY(mlo.alloc(lo.size() * 4));
        GEO_TRY(mhi.alloc(hi.size() * 4));
        GEO_CUDA(cudaMemcpyAsync(mlo.p, lo.data(), lo.size() * 4, cudaMemcpyHostToDevice, ss.cs));
        GEO_CUDA(cudaMemcpyAsync(mhi.p, hi.data(), hi.size() * 4, cudaMemcpyHostToDevice, ss.cs));
        GEO_TRY(launch_mute_records(rec, D.nx, D.nt, mlo.as<int>(), mhi.as<int>(), ss.cs));
    }
    const size_t rbytes = (size_t)D.nx * D.nt * 4;
    if (mem == GEO_MEM_DEVICE) {
        GEO_TRY(launch_transpose_records(rec, shot, D.nx, D.nt, ss.cs));
    } else {
        GEO_TRY(out.alloc(rbytes));
        GEO_TRY(launch_transpose_records(rec, out.as<float>(), D.nx, D.nt, ss.cs));
        GEO_CUDA(cudaMemcpyAsync(shot, out.p, rbytes, cudaMemcpyDeviceToHost, ss.cs));
    }
    GEO_CUDA(cudaStreamSynchronize(ss.cs));
    return GEO_OK;
}

// ---------------------------------------------------------------- RTM 2D
extern "C" int geo_rtm2d_batch(const geo_rtm2d_desc *desc, const float *v, const float *e, const float *d,
                               float *image, float *per_shot, int mem, void *stream) {
    return geo_rtm2d_batch_adcig(desc, v, e, d, image, per_shot, nullptr, mem, stream);
}

extern "C" int geo_rtm2d_batch_adcig(const geo_rtm2d_desc *desc, const float *v, const float *e, const float *d,
                                     float *image, float *per_shot, float *adcig, int mem, void *stream) {
    if (!desc || !v || !e || !d || !image || !desc->shot_x || !desc->shot_nxs) return fail(GEO_ERR_ARG, "null argument");
    const geo_rtm2d_desc &D = *desc;
    if (D.nx < 2 || D.nz < 2 || D.npd < 5 || D.nt < 1 || D.ns < 1) return fail(GEO_ERR_ARG, "bad sizes");
    if (!(D.dt_ms > 0) || !(D.dx > 0) || !(D.dz > 0) || !(D.favg > 0)) return fail(GEO_ERR_ARG, "bad spacing");
    for (int k = 0; k < D.ns; k++) {
        const int nxs = D.shot_nxs[k], kk = D.shot_x[k];
        if (nxs < 3 || nxs % 2 == 0) return fail(GEO_ERR_ARG, "shot %d: window width must be odd and >= 3", k);
        // the reference exits when a window leaves the model (Toa_rtm_vti_adcig_cdp.c:283-292)
        if (kk < nxs / 2 + 1 || kk + nxs / 2 > D.nx) return fail(GEO_ERR_WINDOW, "shot %d window leaves model", k);
    }
    if (D.zs < 1 || D.zs + D.npd - 1 + 3 >= D.nz + 2 * D.npd) return fail(GEO_ERR_ARG, "bad source depth");
    if (D.mode != GEO_MODE_EXACT && D.mode != GEO_MODE_FAST) return fail(GEO_ERR_ARG, "bad mode %d", D.mode);
    const int fast = D.mode == GEO_MODE_FAST;
    cudaStream_t s = (cudaStream_t)stream;
    SideStream ss;
    GEO_TRY(ss.open(s));
    Raw2D raw;
    GEO_TRY(raw.open(D.nx, D.nz, v, e, d, nullptr, mem, ss.cs));
    const float dt = D.dt_ms / 1000;
    const int nt = D.nt, nz = D.nz, npd = D.npd;
    ShotSet X;
    X.var = V_MPI;
    X.nz = nz; X.npd = npd; X.nnz = nz + 2 * npd;
    X.taper = true;
    for (int k = 0; k < D.ns; k++) {
        const int nxs = D.shot_nxs[k], kk = D.shot_x[k];
        // window column c <- model column c + k - nxs/2, clamped into the pad;
        // shot position inside its window: fs = nxs/2+1, ds = 0
        X.G.push_back(ShotGeom{nxs, kk - nxs / 2, (float)(nxs / 2 + 1), (float)D.zs});
    }
    GEO_TRY(X.read(raw, ss.cs));
    GEO_TRY(check_stability(V_MPI, 2, X.st.vmin, X.st.vmax, dt, D.dx, D.dx, D.dz, D.favg));
    std::vector<float> amp;
    std::vector<uint8_t> on;
    source_amplitudes(V_MPI, nt, dt, D.favg, D.pfac, 1, amp, on);
    GEO_TRY(load_march_tables(adcig != nullptr, ss.cs));
    Watchdog wd;
    GEO_TRY(wd.open());
    const size_t nimg = (size_t)D.nx * nz;
    const cudaMemcpyKind kout = mem == GEO_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
    DevBuf stack, lap, gathers;
    GEO_TRY(stack.alloc(nimg * 4));
    GEO_TRY(stack.zero(ss.cs));
    if (D.laplace) GEO_TRY(lap.alloc(nimg * 4));
    if (adcig) {
        GEO_TRY(gathers.alloc((size_t)kAdcigAngles * nimg * 4));
        GEO_TRY(gathers.zero(ss.cs));
    }
    std::vector<size_t> shot_off(D.ns + 1, 0);   // of the per-shot images
    for (int k = 0; k < D.ns; k++) shot_off[k + 1] = shot_off[k] + (size_t)D.shot_nxs[k] * nz;
    DevBuf d_err;
    GEO_TRY(d_err.alloc(4));
    GEO_TRY(d_err.zero(ss.cs));
    auto step = [&](int it, int k) {   // k-th step of its pass
        MarchStep st{};
        st.it = it;
        st.lev = k & 1;
        st.inject = -1;
        st.err = d_err.as<int>();
        st.ddtx = (double)(dt / D.dx);
        st.ddtz = (double)(dt / D.dz);
        st.dhx = (float)st.ddtx; st.dlx = (float)(st.ddtx - (double)st.dhx);
        st.dhz = (float)st.ddtz; st.dlz = (float)(st.ddtz - (double)st.dhz);
        return st;
    };
    // Shots first .. first + n - 1, both passes, their images and gathers added
    // to the stacks.  Memory is taken before anything is added.
    auto group = [&](int first, int n) -> int {
        MarchBatch B(X, first, n, fast != 0, adcig != nullptr);
        GEO_TRY(B.build(raw, D.dx, D.dz, dt, nt, ss.cs));
        const int *nxs = D.shot_nxs + first;
        const March2D *d_M = B.d_M.as<March2D>();
        int maxline = 0, traces = 0;
        // after the backward pass the source side's fields are done with: image
        // and illumination of a shot lie there without the sponge
        std::vector<float *> imgs(2 * (size_t)n);   // images, then illuminations
        std::vector<int> offs(n);
        std::vector<const float *> ap(adcig ? (size_t)kAdcigAngles * n : 0);   // gathers, an angle after the other
        for (int k = 0; k < n; k++) {
            maxline = std::max(maxline, 2 * nxs[k] + 2 * nz);
            traces += nxs[k];
            imgs[k] = B.M[k].f + (size_t)MS_P * B.M[k].n;
            imgs[n + k] = B.M[k].f + (size_t)MS_Q * B.M[k].n;
            offs[k] = D.shot_x[first + k] - nxs[k] / 2 - 1;
            for (size_t ia = 0; ia < ap.size() / n; ia++) ap[ia * n + k] = B.M[k].adcig + ia * nxs[k] * nz;
        }
        DevBuf d_mute, d_imgs, d_offs, d_wid, d_aptr;
        GEO_TRY(d_mute.alloc((size_t)traces * 4));
        GEO_TRY(d_imgs.alloc(imgs.size() * sizeof(float *)));
        GEO_TRY(d_offs.alloc(n * 4));
        GEO_TRY(d_wid.alloc(n * 4));
        if (adcig) GEO_TRY(d_aptr.alloc(ap.size() * sizeof(float *)));
        // non-finite detector: after every wd.every steps (and the last) the
        // graphs scan every shot's P; the verdict follows each pass
        auto watched = [&](int k) { return wd.every > 0 && ((k + 1) % wd.every == 0 || k == nt - 1); };
        auto watch = [&](int k, int nf, int lev) {
            return watched(k) ? launch_march_watch(d_M, n, nf, lev, wd.word(), k + 1, ss.cs) : (int)GEO_OK;
        };
        // forward: source side only, with records and edge lines
        {
            Graph G;
            GEO_TRY(capture(G, ss.cs, [&]() -> int {
                for (int it = 0; it < nt; it++) {
                    MarchStep st = step(it, it);
                    st.amp = amp[it];
                    st.src_on = on[it];
                    GEO_TRY(B.step(false, st, ss.cs));
                    GEO_TRY(watch(it, 1, st.lev ^ 1));
                }
                return GEO_OK;
            }));
            GEO_TRY(G.launch(ss.cs));
        }
        GEO_TRY(wd.verdict(ss.cs, "batched 2D RTM forward pass"));
        // mute both records (tt = 285) and restart the source side from zero
        std::vector<int> mute;
        for (int k = 0; k < n; k++) {
            std::vector<int> lo, hi;
            mute_window_mpi(nxs[k], nt, D.dt_ms, D.favg, D.dx, D.dz, nxs[k] / 2 + 1, 0, D.zs, first + k + 1,
                            X.mu_v[first + k], 285, lo, hi);
            mute.insert(mute.end(), hi.begin(), hi.end());
        }
        GEO_CUDA(cudaMemcpyAsync(d_mute.p, mute.data(), mute.size() * 4, cudaMemcpyHostToDevice, ss.cs));
        for (int k = 0, o = 0; k < n; o += nxs[k++]) {
            const int *hi = d_mute.as<int>() + o;
            GEO_TRY(launch_mute_records(B.M[k].rec_p, nxs[k], nt, nullptr, hi, ss.cs));
            GEO_TRY(launch_mute_records(B.M[k].rec_q, nxs[k], nt, nullptr, hi, ss.cs));
            GEO_TRY(B.clear_side(k, MS_SIDE, ss.cs));
        }
        // backward: both propagations with fused imaging; each step's lines and
        // records go into the level it reads, as the step before stores that
        // level, or by a launch of their own before the first step and after a
        // scan, which is to see the step's own values
        {
            Graph G;
            GEO_TRY(capture(G, ss.cs, [&]() -> int {
                GEO_TRY(launch_march_inject(d_M, n, maxline, nt - 1, 0, ss.cs));
                for (int it = nt - 1; it >= 0; it--) {
                    const int k = nt - 1 - it;
                    MarchStep st = step(it, k);
                    st.inject = watched(k) ? -1 : it - 1;
                    GEO_TRY(B.step(true, st, ss.cs));
                    GEO_TRY(watch(k, 2, st.lev ^ 1));
                    if (watched(k) && it > 0) GEO_TRY(launch_march_inject(d_M, n, maxline, it - 1, st.lev ^ 1, ss.cs));
                }
                return GEO_OK;
            }));
            GEO_TRY(G.launch(ss.cs));
        }
        int gave_up = 0;
        GEO_CUDA(cudaMemcpyAsync(&gave_up, d_err.p, 4, cudaMemcpyDeviceToHost, ss.cs));
        GEO_TRY(wd.verdict(ss.cs, "batched 2D RTM backward pass"));
        GEO_CUDA(cudaStreamSynchronize(ss.cs));
        if (gave_up) return fail(GEO_ERR_CUDA, "batched 2D RTM: a pipeline wait timed out");
        // normalise per shot, stack in shot order
        GEO_CUDA(cudaMemcpyAsync(d_imgs.p, imgs.data(), imgs.size() * sizeof(float *), cudaMemcpyHostToDevice, ss.cs));
        GEO_CUDA(cudaMemcpyAsync(d_offs.p, offs.data(), n * 4, cudaMemcpyHostToDevice, ss.cs));
        GEO_CUDA(cudaMemcpyAsync(d_wid.p, nxs, n * 4, cudaMemcpyHostToDevice, ss.cs));
        GEO_TRY(launch_march_image(d_M, n, d_imgs.as<float *>(), d_imgs.as<float *>() + n, ss.cs));
        GEO_TRY(launch_stack_image(stack.as<float>(), nz, d_imgs.as<const float *const>(), d_offs.as<int>(),
                                   d_wid.as<int>(), n, D.nx, ss.cs));
        if (adcig) {
            // per shot: divide by the source illumination (Toa_rtm_vti_adcig_cdp.c:1083-1090), then stack
            // every angle plane in shot order into [90][nx][nz] (adcig_ns0)
            for (int q = 0; q < n; q++)
                GEO_TRY(launch_normalize_planes(B.M[q].adcig, imgs[n + q], (size_t)nxs[q] * nz, kAdcigAngles, ss.cs));
            GEO_CUDA(cudaMemcpyAsync(d_aptr.p, ap.data(), ap.size() * sizeof(float *), cudaMemcpyHostToDevice, ss.cs));
            for (int ia = 0; ia < kAdcigAngles; ia++)
                GEO_TRY(launch_stack_image(gathers.as<float>() + ia * nimg, nz,
                                           d_aptr.as<const float *const>() + (size_t)ia * n, d_offs.as<int>(),
                                           d_wid.as<int>(), n, D.nx, ss.cs));
        }
        for (int k = 0; k < n && per_shot; k++)
            GEO_CUDA(cudaMemcpyAsync(per_shot + shot_off[first + k], imgs[k], (size_t)nxs[k] * nz * 4, kout, ss.cs));
        GEO_CUDA(cudaStreamSynchronize(ss.cs));
        return GEO_OK;
    };
    // All shots together where they fit (a shot takes 128 B a padded point in
    // the exact form, 116 in the fast one, and its records and edge lines), else
    // in the largest of halved groups that do: the stacks add in shot order
    // either way, so the images are the same.
    int n = D.ns;
    if (const char *e = getenv("GEO_RTM2D_GROUP"))
        if (const int k = atoi(e); k > 0) n = std::min(n, k);
    for (int first = 0; first < D.ns;) {
        n = std::min(n, D.ns - first);
        const int rc = group(first, n);
        if (rc == GEO_ERR_NOMEM && n > 1) {
            n = (n + 1) / 2;
            continue;
        }
        GEO_TRY(rc);
        first += n;
    }
    const float *result = stack.as<float>();
    if (D.laplace) {
        GEO_TRY(launch_laplace2d(D.nx, nz, stack.as<float>(), lap.as<float>(), ss.cs));
        result = lap.as<float>();
    }
    GEO_CUDA(cudaMemcpyAsync(image, result, nimg * 4, kout, ss.cs));
    if (adcig) GEO_CUDA(cudaMemcpyAsync(adcig, gathers.p, (size_t)kAdcigAngles * nimg * 4, kout, ss.cs));
    GEO_CUDA(cudaStreamSynchronize(ss.cs));
    return GEO_OK;
}

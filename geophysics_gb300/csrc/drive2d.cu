// 2D drivers: single-shot forward modelling and batched RTM.
//
// Both build per-shot Shot2D descriptors and step them with the batched
// kernels of fd2d.cu.  A batch time step is one persistent launch per phase
// (velocity, stress) covering every shot's tiles; the time loops are
// captured once into CUDA graphs and replayed.
#include "geo_internal.h"
#include "model2d.cuh"
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <memory>
#include <tuple>

namespace geo {

static int sm_count() {
    static int n = 0;
    if (!n) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 1;
    }
    return n;
}

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
    std::vector<Shot2D> S;
    RawStats st;
    float v00, e00;               // model values at unpadded (0, 0)
    std::vector<float> mu_v;      // MPI mute velocity of each shot
    Arena mem;
    Blob small;
    size_t o_amp = 0, o_on = 0;
    // cleared state: fields of side 0 of every shot, then of side 1, images
    // and gathers, records
    size_t z_side0 = 0, z_side1 = 0, z_img = 0, z_rec = 0, z_end = 0;
    int clear(size_t from, size_t to, cudaStream_t s) {
        if (to > from) GEO_CUDA(cudaMemsetAsync(mem.buf.as<char>() + from, 0, to - from, s));
        return GEO_OK;
    }
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
    int build(const Raw2D &raw, float dx, float dz, float dt, const std::vector<float> &amp,
              const std::vector<uint8_t> &on, int nfields, int nt, bool edges, bool image, bool adcig, bool fast,
              cudaStream_t s);
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

// Propagation coefficients and state of every shot; var picks the reference
// program's formulas.
int ShotSet::build(const Raw2D &raw, float dx, float dz, float dt, const std::vector<float> &amp,
                   const std::vector<uint8_t> &on, int nfields, int nt, bool edges, bool image, bool adcig, bool fast,
                   cudaStream_t s) {
    const int ns = (int)G.size();
    // the MPI program's pz and qx chains are
    //   (double)(az2*pz) - (double)(az1*vp) * pow(1+2del,0.5) * (double)dtz * (double)zz
    // (and with ax, dtx, xx for qx), evaluated left to right; every factor but
    // zz is fixed for the shot, so the product of the first three is formed
    // once, in the same order and precision (ModelJob::kz), and the kernel
    // issues one double multiply and one double subtraction per chain.  The
    // program's pow runs on the host, once per model point.
    const bool kchain = var == V_MPI && !fast;
    const double ddtx = (double)(dt / dx), ddtz = (double)(dt / dz);
    S.assign(ns, Shot2D{});
    mu_v.resize(ns);
    DevBuf d_pw;
    if (kchain) {
        const size_t n0 = (size_t)raw.nx * raw.nz;
        std::vector<float> hd(n0);
        std::vector<double> pw(n0);
        GEO_CUDA(cudaMemcpyAsync(hd.data(), raw.a[2], n0 * 4, cudaMemcpyDeviceToHost, s));
        GEO_CUDA(cudaStreamSynchronize(s));
        host_pow_half(hd.data(), n0, pw.data());
        GEO_TRY(d_pw.alloc(n0 * 8));
        GEO_CUDA(cudaMemcpyAsync(d_pw.p, pw.data(), n0 * 8, cudaMemcpyHostToDevice, s));
        GEO_CUDA(cudaStreamSynchronize(s));   // pw is freed below
    }
    struct Off {
        size_t prof[8], te2, td2, tkz, tkx;
    };
    std::vector<Off> off(ns);
    for (int k = 0; k < ns; k++) {
        const ShotGeom &g = G[k];
        const int nnx = g.nx + 2 * npd;
        const float *val = st.val.data() + 2 + (size_t)k * kPick;
        float vpmax = 0.0f;
        for (int c = 0; c < g.nx; c++) vpmax = std::max(vpmax, st.colmax[std::min(c + g.col0, raw.nx - 1)]);
        const float d0 = sponge_d0(var, 2, vpmax, val[0], npd, dx, dx, dz);
        mu_v[k] = val[1] * sqrtf(1 + 2 * val[2]);
        std::vector<float> p[8];
        for (int q = 0; q < 8; q++) p[q].resize(q < 4 ? nnx : nnz);
        sponge_profiles(var, g.nx, npd, dt, d0, p[0].data(), p[1].data(), p[2].data(), p[3].data());
        sponge_profiles(var, nz, npd, dt, d0, p[4].data(), p[5].data(), p[6].data(), p[7].data());
        for (int q = 0; q < 8; q++) off[k].prof[q] = small.put(p[q]);
        Shot2D &h = S[k];
        source(k, h.ixs, h.izs);
        h.tx0 = h.tz0 = -100000;
        if (!taper) continue;
        int cx, cz;
        centre(k, cx, cz);
        Taper2D tp;
        const float *vbox = val + 3;
        sv_taper_2d(var, nnx, nnz, cx, cz, vbox + kTB * kTB, vbox + 2 * kTB * kTB, tp);
        h.tx0 = tp.x0;
        h.tz0 = tp.z0;
        std::vector<float> te2(kTB * kTB, 1.0f), td2(kTB * kTB, 1.0f);
        for (int b = 0; b < kTB * kTB; b++) {
            te2[b] = 1 + 2 * tp.e[b];
            td2[b] = sqrtf(1 + 2 * tp.d[b]);
        }
        off[k].te2 = small.put(te2);
        off[k].td2 = small.put(td2);
        if (!kchain) continue;
        std::vector<double> tkz(kTB * kTB, 0.0), tkx(kTB * kTB, 0.0);
        for (int b = 0; b < kTB * kTB; b++) {
            const int ix = tp.x0 + b / kTB, iz = tp.z0 + b % kTB;
            if (ix < 0 || ix >= nnx || iz < 0 || iz >= nnz) continue;
            const double pw = std::pow((double)(1 + 2 * tp.d[b]), 0.5);
            const float vpk = 1.0f * (vbox[b] * vbox[b]);
            tkz[b] = (double)(p[6][iz] * vpk) * pw * ddtz;
            tkx[b] = (double)(p[2][ix] * vpk) * pw * ddtx;
        }
        off[k].tkz = small.put(tkz);
        off[k].tkx = small.put(tkx);
    }
    o_amp = small.put(amp);
    o_on = small.put(on);
    GEO_TRY(small.upload(s));
    // two passes: sizes, then addresses
    std::vector<ModelJob> jobs(ns);
    for (int pass = 0; pass < 2; pass++) {
        z_side0 = 0;
        for (int f = 0; f < nfields; f++) {
            if (f == 1) z_side1 = mem.off;
            for (int k = 0; k < ns; k++) {
                const size_t n = (size_t)(G[k].nx + 2 * npd) * nnz;
                float **dst[8] = {&S[k].u[f], &S[k].w[f], &S[k].P[f], &S[k].Q[f],
                                  &S[k].px[f], &S[k].pz[f], &S[k].qx[f], &S[k].qz[f]};
                for (auto d : dst) *d = mem.take<float>(n);
            }
        }
        if (nfields < 2) z_side1 = mem.off;
        z_img = mem.off;
        for (int k = 0; k < ns; k++) {
            const size_t m = (size_t)G[k].nx * nz;
            if (image) {
                S[k].mig = mem.take<float>(m);
                S[k].ill = mem.take<float>(m);
            }
            if (adcig) S[k].adcig = mem.take<float>(kAdcigAngles * m);
        }
        z_rec = mem.off;
        for (int k = 0; k < ns; k++) {
            S[k].rec_p = mem.take<float>((size_t)nt * G[k].nx);
            S[k].rec_q = edges ? mem.take<float>((size_t)nt * G[k].nx) : nullptr;
        }
        z_end = mem.off;
        for (int k = 0; k < ns; k++) {
            const int nnx = G[k].nx + 2 * npd;
            const size_t n = (size_t)nnx * nnz, L = 2 * (size_t)G[k].nx + 2 * (size_t)nz;
            ModelJob &j = jobs[k];
            j.nx = G[k].nx; j.nz = nz; j.npd = npd; j.ldz = nnz; j.col0 = G[k].col0;
            j.vp2 = var == V_MPI;   // vp <- rho*vp^2 with rho == 1 (Toa_rtm_vti_adcig_cdp.c:641)
            j.vp = mem.take<float>(n);
            j.e2 = mem.take<float>(n);
            j.d2 = kchain ? nullptr : mem.take<float>(n);
            j.rad = nullptr;
            j.kz = kchain ? mem.take<double>(n) : nullptr;
            j.kx = kchain ? mem.take<double>(n) : nullptr;
            j.pw = d_pw.as<double>();
            j.ddtx = ddtx; j.ddtz = ddtz;
            if (edges) {
                S[k].edge_p = mem.take<float>((size_t)nt * L);
                S[k].edge_q = mem.take<float>((size_t)nt * L);
            }
        }
        if (pass == 0) GEO_TRY(mem.alloc());
    }
    for (int k = 0; k < ns; k++) {
        Shot2D &h = S[k];
        h.nnx = G[k].nx + 2 * npd; h.nnz = nnz; h.npd = npd; h.nx = G[k].nx; h.nz = nz;
        h.dtx = dt / dx; h.dtz = dt / dz;
        const float **dp[8] = {&h.cx1, &h.cx2, &h.ax1, &h.ax2, &h.cz1, &h.cz2, &h.az1, &h.az2};
        for (int q = 0; q < 8; q++) *dp[q] = small.at<float>(off[k].prof[q]);
        ModelJob &j = jobs[k];
        j.ax1 = h.ax1;
        j.az1 = h.az1;
        h.vp = j.vp; h.e2 = j.e2; h.d2 = j.d2; h.kz = j.kz; h.kx = j.kx;
        if (taper) {
            h.te2 = small.at<float>(off[k].te2);
            h.td2 = small.at<float>(off[k].td2);
            if (kchain) {
                h.tkz = small.at<double>(off[k].tkz);
                h.tkx = small.at<double>(off[k].tkx);
            }
        }
        h.rec_iz = npd;
        h.rec_scale = 1.0f;
    }
    GEO_TRY(launch_model2d(raw, jobs, s));
    return clear(0, z_end, s);
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
    int by = 8, grid = 1, variant = V_CPU;
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
        return launch_vel2d(variant, d_S.as<Shot2D>(), d_items.as<int>(), (int)items.size(), by, grid, st, s);
    }
    int stress(int phase, Step2D st, cudaStream_t s) {
        return launch_stress2d(variant, phase, d_S.as<Shot2D>(), d_items.as<int>(), (int)items.size(), by, grid, st, s);
    }

    // Skewed schedule (MPI form, two or more shots): the shots are split
    // into groups A = [0, split) and B = [split, ns) of about equal tiles,
    // B half a step behind A, so that every launch pairs one group's stress
    // tiles with the other's velocity tiles (launch_mix2d).  Every shot
    // still runs velocity then stress of each step in order.  Tables, as
    // (shot | kind << 30, tile) items with the kinds interleaved:
    //   VA: velocity of A;  MX: stress of A + velocity of B;
    //   MY: velocity of A + stress of B;  SB: stress of B.
    enum { VA = 0, MX = 1, MY = 2, SB = 3 };
    DevBuf d_mix;
    int split = 0, mix_n[4] = {0, 0, 0, 0};
    size_t mix_o[4] = {0, 0, 0, 0};
    int build_mix(cudaStream_t s) {
        const int ns = (int)S.size();
        std::vector<long> tiles(ns);
        long total = 0;
        for (int k = 0; k < ns; k++) {
            tiles[k] = (long)S[k].ntz * ((S[k].nnx + by - 1) / by);
            total += tiles[k];
        }
        long acc = 0;
        split = 1;
        for (int k = 0; k < ns - 1; k++) {
            acc += tiles[k];
            split = k + 1;
            if (2 * acc >= total) break;
        }
        auto list = [&](int k0, int k1, int kind) {
            std::vector<int2> v;
            for (int k = k0; k < k1; k++)
                for (long t = 0; t < tiles[k]; t++) v.push_back(make_int2(k | (kind << 30), (int)t));
            return v;
        };
        auto merge = [](const std::vector<int2> &a, const std::vector<int2> &b) {
            std::vector<int2> v;
            v.reserve(a.size() + b.size());
            size_t i = 0, j = 0;
            while (i < a.size() || j < b.size()) {
                if (j >= b.size() || (i < a.size() && i * b.size() <= j * a.size())) v.push_back(a[i++]);
                else v.push_back(b[j++]);
            }
            return v;
        };
        const std::vector<int2> vA = list(0, split, 0), sA = list(0, split, 1), vB = list(split, ns, 0),
                                sB = list(split, ns, 1);
        const std::vector<int2> tab[4] = {vA, merge(sA, vB), merge(vA, sB), sB};
        size_t off = 0;
        for (int t = 0; t < 4; t++) {
            mix_o[t] = off;
            mix_n[t] = (int)tab[t].size();
            off += tab[t].size();
        }
        GEO_TRY(d_mix.alloc(off * sizeof(int2)));
        for (int t = 0; t < 4; t++)
            GEO_CUDA(cudaMemcpyAsync(d_mix.as<int2>() + mix_o[t], tab[t].data(), tab[t].size() * sizeof(int2),
                                     cudaMemcpyHostToDevice, s));
        GEO_CUDA(cudaStreamSynchronize(s));
        return GEO_OK;
    }
    int mix(int table, int phase, int fast, Step2D sv, Step2D ss, cudaStream_t s) {
        return launch_mix2d(phase, fast, d_S.as<Shot2D>(), d_mix.as<int2>() + mix_o[table], mix_n[table], by, grid,
                            sv, ss, s);
    }
};

// Graph of a range of steps; capture on a private stream.
struct Graph {
    cudaGraph_t g = nullptr;
    cudaGraphExec_t x = nullptr;
    long long kernels = 0;     // kernel nodes, counted once per replay
    int launch(cudaStream_t s) {
        GEO_CUDA(cudaGraphLaunch(x, s));
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
    GEO_CUDA(cudaGraphInstantiate(&G.x, g, 0));
    return GEO_OK;
}

// Autotuner: time a few forward steps for each (rows per tile, blocks per
// SM) candidate on the real batch and keep the fastest.  Results are cached
// per (grid extents, shot count, device) for the life of the process.
static std::map<std::tuple<int, int, int, int>, std::pair<int, int>> g_tune_cache;

static int autotune(Batch2D &B, int nf, int key_nx, int key_nz, cudaStream_t s, int *by_out, int *bps_out) {
    int dev = 0;
    cudaGetDevice(&dev);
    auto key = std::make_tuple(key_nx, key_nz, (int)B.S.size() * 16 + nf, dev);
    auto it = g_tune_cache.find(key);
    if (it != g_tune_cache.end()) {
        *by_out = it->second.first;
        *bps_out = it->second.second;
        return GEO_OK;
    }
    const int bys[] = {4, 8};
    const int bpss[] = {4, 8, 16};
    float best = 1e30f;
    int bb = 8, bp = 8;
    cudaEvent_t a, b;
    GEO_CUDA(cudaEventCreate(&a));
    GEO_CUDA(cudaEventCreate(&b));
    Step2D st{};
    st.nf = nf;
    for (int by : bys)
        for (int bps : bpss) {
            GEO_TRY(B.upload(by, bps, s));
            GEO_TRY(B.vel(st, s));
            GEO_TRY(B.stress(PH_BWD, st, s));
            GEO_CUDA(cudaEventRecord(a, s));
            for (int k = 0; k < 4; k++) {
                GEO_TRY(B.vel(st, s));
                GEO_TRY(B.stress(PH_BWD, st, s));
            }
            GEO_CUDA(cudaEventRecord(b, s));
            GEO_CUDA(cudaEventSynchronize(b));
            float ms = 0;
            GEO_CUDA(cudaEventElapsedTime(&ms, a, b));
            if (ms < best) {
                best = ms;
                bb = by;
                bp = bps;
            }
        }
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    g_tune_cache[key] = {bb, bp};
    *by_out = bb;
    *bps_out = bp;
    return GEO_OK;
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
    ShotSet X;
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
    GEO_TRY(X.build(raw, D.dx, D.dz, D.dt, amp, on, 1, D.nt, false, false, false, false, ss.cs));
    const float *d_amp = X.small.at<float>(X.o_amp);
    const unsigned char *d_on = X.small.at<unsigned char>(X.o_on);
    Batch2D B;
    B.variant = var;
    B.S = X.S;
    B.S[0].rec_iz = D.rec_iz;
    B.S[0].rec_scale = D.rec_scale;
    const bool persistent = !(snap && snap_every > 0);
    auto step = [&](int it) -> int {
        Step2D st{};
        st.it = it;
        st.amp = amp[it];
        st.src_on = on[it];
        st.taper = taper ? 1 : 0;
        st.nf = 1;
        GEO_TRY(B.vel(st, ss.cs));
        return B.stress(PH_FWD, st, ss.cs);
    };
    DevBuf d_sync;
    GEO_TRY(d_sync.alloc(8));
    GEO_TRY(d_sync.zero(ss.cs));
    unsigned *bar = d_sync.as<unsigned>();
    int *errw = d_sync.as<int>() + 1;
    const size_t nn = (size_t)nnx * nnz;
    Watchdog wd;
    GEO_TRY(wd.open());
    const cudaMemcpyKind ksnap = mem == GEO_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
    // CPU and GPU forms: every block keeps its tile of the fields in shared
    // memory for the run (launch_fd2d_tile), one launch per run of steps
    // between snapshots, when the grid fits on the device that way
    bool tiled = false;
    if (var == V_CPU || var == V_GPU) {
        DevBuf xch;
        GEO_TRY(xch.alloc(8 * nn * 4));
        GEO_TRY(xch.zero(ss.cs));
        for (int it0 = 0; it0 < D.nt;) {
            int it1 = it0 + 1;
            if (snap && snap_every > 0)
                while (it1 < D.nt && (it1 - 1) % snap_every != 0) it1++;
            else
                it1 = D.nt;
            bool fits = false;
            GEO_TRY(launch_fd2d_tile(var, B.S[0], xch.as<float>(), d_amp, d_on, taper ? 1 : 0, it0, it1, bar, errw, &fits, ss.cs));
            if (!fits) {   // decided by the grid alone, so on the first run of steps
                if (tiled) return fail(GEO_ERR_CUDA, "2D shot: tile-resident launch refused mid-run");
                break;
            }
            tiled = true;
            const int it = it1 - 1;
            if (snap && snap_every > 0 && it % snap_every == 0)
                GEO_CUDA(cudaMemcpyAsync(snap + (size_t)(it / snap_every) * nn, B.S[0].P[0], nn * 4, ksnap, ss.cs));
            if (wd.every > 0) {
                GEO_TRY(wd.scan(B.S[0].P[0], nn, it + 1, ss.cs));
                if (wd.tripped()) break;
            }
            it0 = it1;
        }
        if (tiled) {
            int err = 0;
            GEO_CUDA(cudaMemcpyAsync(&err, errw, 4, cudaMemcpyDeviceToHost, ss.cs));
            GEO_CUDA(cudaStreamSynchronize(ss.cs));
            if (err) return fail(GEO_ERR_CUDA, "2D shot: a grid barrier wait timed out");
            if (wd.every > 0) GEO_TRY(wd.scan(B.S[0].rec_p, (size_t)D.nx * D.nt, D.nt, ss.cs));
        }
    }
    if (!tiled) GEO_TRY(B.upload(persistent ? 16 : 8, 8, ss.cs));
    if (!tiled && snap && snap_every > 0) {
        for (int it = 0; it < D.nt; it++) {
            GEO_TRY(step(it));
            if (it % snap_every == 0)
                GEO_CUDA(cudaMemcpyAsync(snap + (size_t)(it / snap_every) * nn, B.S[0].P[0], nn * 4, ksnap, ss.cs));
            if (wd.every > 0 && ((it + 1) % wd.every == 0 || it == D.nt - 1)) {
                GEO_TRY(launch_watch_shots(B.d_S.as<Shot2D>(), 1, 1, wd.d, it + 1, ss.cs));
                if (wd.tripped()) break;
            }
        }
    } else if (!tiled) {
        // the whole shot in one cooperative launch (grid barriers between the
        // half-steps, bounded waits reported through an error word)
        Persist2D a{};
        a.nt = D.nt;
        a.taper = taper ? 1 : 0;
        a.amp = d_amp;
        a.on = d_on;
        a.bar = bar;
        a.err = errw;
        GEO_TRY(launch_fd2d_shot(var, B.d_S.as<Shot2D>(), B.d_items.as<int>(), (int)B.items.size(), B.by, a, ss.cs));
        int err = 0;
        GEO_CUDA(cudaMemcpyAsync(&err, a.err, 4, cudaMemcpyDeviceToHost, ss.cs));
        GEO_CUDA(cudaStreamSynchronize(ss.cs));
        if (err) return fail(GEO_ERR_CUDA, "2D shot: a grid barrier wait timed out");
        // the shot ran in one launch: scan its final P and its record
        if (wd.every > 0) {
            GEO_TRY(launch_watch_shots(B.d_S.as<Shot2D>(), 1, 1, wd.d, D.nt, ss.cs));
            GEO_TRY(wd.scan(B.S[0].rec_p, (size_t)D.nx * D.nt, D.nt, ss.cs));
        }
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
        GEO_TRY(launch_mute_records(B.S[0].rec_p, D.nx, D.nt, mlo.as<int>(), mhi.as<int>(), ss.cs));
    }
    const size_t rbytes = (size_t)D.nx * D.nt * 4;
    if (mem == GEO_MEM_DEVICE) {
        GEO_TRY(launch_transpose_records(B.S[0].rec_p, shot, D.nx, D.nt, ss.cs));
    } else {
        GEO_TRY(out.alloc(rbytes));
        GEO_TRY(launch_transpose_records(B.S[0].rec_p, out.as<float>(), D.nx, D.nt, ss.cs));
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
    int maxline = 0;
    for (int k = 0; k < D.ns; k++) {
        const int nxs = D.shot_nxs[k], kk = D.shot_x[k];
        // window column c <- model column c + k - nxs/2, clamped into the pad;
        // shot position inside its window: fs = nxs/2+1, ds = 0
        X.G.push_back(ShotGeom{nxs, kk - nxs / 2, (float)(nxs / 2 + 1), (float)D.zs});
        maxline = std::max(maxline, 2 * nxs + 2 * nz);
    }
    GEO_TRY(X.read(raw, ss.cs));
    GEO_TRY(check_stability(V_MPI, 2, X.st.vmin, X.st.vmax, dt, D.dx, D.dx, D.dz, D.favg));
    std::vector<float> amp;
    std::vector<uint8_t> on;
    source_amplitudes(V_MPI, nt, dt, D.favg, D.pfac, 1, amp, on);
    GEO_TRY(X.build(raw, D.dx, D.dz, dt, amp, on, 2, nt, true, true, adcig != nullptr, fast != 0, ss.cs));
    Batch2D B;
    B.variant = V_MPI;
    B.S = X.S;
    // tile shape: caller's choice or the autotuner's
    int by = D.tile_x, bps = 8;
    if (by != 4 && by != 8) GEO_TRY(autotune(B, 2, D.nx, D.nz, ss.cs, &by, &bps));
    GEO_TRY(B.upload(by, bps, ss.cs));
    // the autotuner stepped the state: start from zero again
    GEO_TRY(X.clear(X.z_side0, X.z_rec, ss.cs));
    if (adcig) GEO_TRY(load_adcig_tables(ss.cs));

    // non-finite detector: every wd.every steps (and the last) the graphs
    // scan every shot's P; the verdict follows each pass
    Watchdog wd;
    GEO_TRY(wd.open());
    auto watch = [&](int k, bool last, int nf) -> int {
        if (wd.every <= 0 || ((k + 1) % wd.every && !last)) return GEO_OK;
        return launch_watch_shots(B.d_S.as<Shot2D>(), D.ns, nf, wd.d, k + 1, ss.cs);
    };
    // forward: source side only, with records and edge lines; with two or
    // more shots on the skewed schedule (Batch2D::build_mix)
    const bool skew = D.ns >= 2;
    if (skew) GEO_TRY(B.build_mix(ss.cs));
    auto fwd_st = [&](int it) {
        Step2D st{};
        st.it = it; st.amp = amp[it]; st.src_on = on[it]; st.taper = 1; st.nf = 1; st.fast = fast;
        return st;
    };
    {
        Graph G;
        GEO_TRY(capture(G, ss.cs, [&]() -> int {
            if (skew) {
                GEO_TRY(B.mix(Batch2D::VA, PH_FWD, fast, fwd_st(0), fwd_st(0), ss.cs));
                for (int it = 0; it < nt; it++) {
                    GEO_TRY(B.mix(Batch2D::MX, PH_FWD, fast, fwd_st(it), fwd_st(it), ss.cs));
                    if (it + 1 < nt) GEO_TRY(B.mix(Batch2D::MY, PH_FWD, fast, fwd_st(it + 1), fwd_st(it), ss.cs));
                    else GEO_TRY(B.mix(Batch2D::SB, PH_FWD, fast, fwd_st(it), fwd_st(it), ss.cs));
                    GEO_TRY(watch(it, it == nt - 1, 1));
                }
                return GEO_OK;
            }
            for (int it = 0; it < nt; it++) {
                const Step2D st = fwd_st(it);
                GEO_TRY(B.vel(st, ss.cs));
                GEO_TRY(B.stress(PH_FWD, st, ss.cs));
                GEO_TRY(watch(it, it == nt - 1, 1));
            }
            return GEO_OK;
        }));
        GEO_TRY(G.launch(ss.cs));
    }
    GEO_TRY(wd.verdict(ss.cs, "batched 2D RTM forward pass"));
    // mute both records (tt = 285) and restart the source side from zero
    std::vector<int> mute;
    for (int k = 0; k < D.ns; k++) {
        const int nxs = D.shot_nxs[k];
        std::vector<int> lo, hi;
        mute_window_mpi(nxs, nt, D.dt_ms, D.favg, D.dx, D.dz, nxs / 2 + 1, 0, D.zs, k + 1, X.mu_v[k], 285, lo, hi);
        mute.insert(mute.end(), hi.begin(), hi.end());
    }
    DevBuf d_mute;
    GEO_TRY(d_mute.alloc(mute.size() * 4));
    GEO_CUDA(cudaMemcpyAsync(d_mute.p, mute.data(), mute.size() * 4, cudaMemcpyHostToDevice, ss.cs));
    for (int k = 0, o = 0; k < D.ns; o += D.shot_nxs[k++]) {
        const int *hi = d_mute.as<int>() + o;
        GEO_TRY(launch_mute_records(B.S[k].rec_p, D.shot_nxs[k], nt, nullptr, hi, ss.cs));
        GEO_TRY(launch_mute_records(B.S[k].rec_q, D.shot_nxs[k], nt, nullptr, hi, ss.cs));
    }
    GEO_TRY(X.clear(X.z_side0, X.z_side1, ss.cs));
    // backward: inject, both propagations, fused imaging
    {
        Graph G;
        auto bwd_st = [&](int it) {
            Step2D st{};
            st.it = it; st.nf = 2; st.fast = fast;
            return st;
        };
        const Shot2D *dA = B.d_S.as<Shot2D>(), *dB = dA + B.split;
        const int nA = B.split, nB = D.ns - B.split;
        GEO_TRY(capture(G, ss.cs, [&]() -> int {
            if (skew) {
                GEO_TRY(launch_inject2d(dA, nA, maxline, nt - 1, ss.cs));
                GEO_TRY(B.mix(Batch2D::VA, PH_BWD, fast, bwd_st(nt - 1), bwd_st(nt - 1), ss.cs));
                for (int it = nt - 1; it >= 0; it--) {
                    GEO_TRY(launch_inject2d(dB, nB, maxline, it, ss.cs));
                    GEO_TRY(B.mix(Batch2D::MX, PH_BWD, fast, bwd_st(it), bwd_st(it), ss.cs));
                    if (it > 0) {
                        GEO_TRY(launch_inject2d(dA, nA, maxline, it - 1, ss.cs));
                        GEO_TRY(B.mix(Batch2D::MY, PH_BWD, fast, bwd_st(it - 1), bwd_st(it), ss.cs));
                    } else {
                        GEO_TRY(B.mix(Batch2D::SB, PH_BWD, fast, bwd_st(it), bwd_st(it), ss.cs));
                    }
                    GEO_TRY(watch(nt - 1 - it, it == 0, 2));
                }
                return GEO_OK;
            }
            for (int it = nt - 1; it >= 0; it--) {
                GEO_TRY(launch_inject2d(B.d_S.as<Shot2D>(), D.ns, maxline, it, ss.cs));
                const Step2D st = bwd_st(it);
                GEO_TRY(B.vel(st, ss.cs));
                GEO_TRY(B.stress(PH_BWD, st, ss.cs));
                GEO_TRY(watch(nt - 1 - it, it == 0, 2));
            }
            return GEO_OK;
        }));
        GEO_TRY(G.launch(ss.cs));
    }
    GEO_TRY(wd.verdict(ss.cs, "batched 2D RTM backward pass"));
    // normalise per shot, stack in shot order, Laplacian
    std::vector<const float *> imgs(D.ns);
    std::vector<int> offs(D.ns), wid(D.ns);
    for (int k = 0; k < D.ns; k++) {
        GEO_TRY(launch_normalize_image(B.S[k].mig, B.S[k].ill, (size_t)D.shot_nxs[k] * nz, ss.cs));
        imgs[k] = B.S[k].mig;
        offs[k] = D.shot_x[k] - D.shot_nxs[k] / 2 - 1;
        wid[k] = D.shot_nxs[k];
    }
    DevBuf d_imgs, d_offs, d_wid, stack, lap;
    GEO_TRY(d_imgs.alloc(D.ns * sizeof(float *)));
    GEO_TRY(d_offs.alloc(D.ns * 4));
    GEO_TRY(d_wid.alloc(D.ns * 4));
    GEO_CUDA(cudaMemcpyAsync(d_imgs.p, imgs.data(), D.ns * sizeof(float *), cudaMemcpyHostToDevice, ss.cs));
    GEO_CUDA(cudaMemcpyAsync(d_offs.p, offs.data(), D.ns * 4, cudaMemcpyHostToDevice, ss.cs));
    GEO_CUDA(cudaMemcpyAsync(d_wid.p, wid.data(), D.ns * 4, cudaMemcpyHostToDevice, ss.cs));
    const size_t nimg = (size_t)D.nx * nz;
    GEO_TRY(stack.alloc(nimg * 4));
    GEO_TRY(stack.zero(ss.cs));
    GEO_TRY(launch_stack_image(stack.as<float>(), nz, d_imgs.as<const float *const>(), d_offs.as<int>(),
                               d_wid.as<int>(), D.ns, D.nx, ss.cs));
    const float *result = stack.as<float>();
    if (D.laplace) {
        GEO_TRY(lap.alloc(nimg * 4));
        GEO_TRY(launch_laplace2d(D.nx, nz, stack.as<float>(), lap.as<float>(), ss.cs));
        result = lap.as<float>();
    }
    const cudaMemcpyKind k = mem == GEO_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
    GEO_CUDA(cudaMemcpyAsync(image, result, nimg * 4, k, ss.cs));
    DevBuf gathers, d_aptr;
    if (adcig) {
        // per shot: divide by the source illumination (Toa_rtm_vti_adcig_cdp.c:1083-1090), then stack
        // every angle plane in shot order into [90][nx][nz] (adcig_ns0)
        std::vector<const float *> ap((size_t)kAdcigAngles * D.ns);
        for (int q = 0; q < D.ns; q++) {
            const size_t m = (size_t)D.shot_nxs[q] * nz;
            GEO_TRY(launch_normalize_planes(B.S[q].adcig, B.S[q].ill, m, kAdcigAngles, ss.cs));
            for (int ia = 0; ia < kAdcigAngles; ia++) ap[(size_t)ia * D.ns + q] = B.S[q].adcig + ia * m;
        }
        GEO_TRY(d_aptr.alloc(ap.size() * sizeof(float *)));
        GEO_CUDA(cudaMemcpyAsync(d_aptr.p, ap.data(), ap.size() * sizeof(float *), cudaMemcpyHostToDevice, ss.cs));
        GEO_TRY(gathers.alloc((size_t)kAdcigAngles * nimg * 4));
        GEO_TRY(gathers.zero(ss.cs));
        for (int ia = 0; ia < kAdcigAngles; ia++)
            GEO_TRY(launch_stack_image(gathers.as<float>() + ia * nimg, nz,
                                       d_aptr.as<const float *const>() + (size_t)ia * D.ns, d_offs.as<int>(),
                                       d_wid.as<int>(), D.ns, D.nx, ss.cs));
        GEO_CUDA(cudaMemcpyAsync(adcig, gathers.p, (size_t)kAdcigAngles * nimg * 4, k, ss.cs));
    }
    if (per_shot) {
        size_t o = 0;
        for (int q = 0; q < D.ns; q++) {
            const size_t m = (size_t)D.shot_nxs[q] * nz;
            GEO_CUDA(cudaMemcpyAsync(per_shot + o, B.S[q].mig, m * 4, k, ss.cs));
            o += m;
        }
    }
    GEO_CUDA(cudaStreamSynchronize(ss.cs));
    return GEO_OK;
}

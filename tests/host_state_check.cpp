// Host-side state of libgeofd against a CUDA runtime without a device
// (fake_cuda.h).  Usage: host_state_check <check>; prints what fails.
#include "fake_cuda.h"
#include "geofd.h"
#include "step2d.cuh"
#include "march2d.cuh"
#include <algorithm>
#include <cmath>
#include <vector>

extern "C" const char *geo_strerror(int);
static int failures = 0;
#define OK(call)                                                                              \
    do {                                                                                      \
        const int s_ = (call);                                                                \
        if (s_ != GEO_OK) {                                                                   \
            printf("device %d: %s: %s\n", fake::device, #call, geo_strerror(s_));             \
            failures++;                                                                       \
        }                                                                                     \
    } while (0)

static std::vector<float> filled(size_t n, float v) { return std::vector<float>(n, v); }

// Waits for the whole device are not allowed while another host thread captures
// a graph, so the calls that run beside each other in threads make none.
static int waits_of(const char *what) {
    if (fake::st().device_waits) { printf("%s: %d waits for the device\n", what, fake::st().device_waits); failures++; }
    fake::st().device_waits = 0;
    return 0;
}

static geo_fd2d_desc fd2d_desc(int variant) {
    geo_fd2d_desc d{};
    d.nx = 40; d.nz = 30; d.npd = 8; d.nt = 3;
    d.dx = d.dz = 10; d.dt = 1e-3f; d.favg = 20; d.pfac = 10; d.wtype = 1;
    d.fs = 20; d.zs = 5; d.is = 1; d.variant = variant; d.rec_iz = 12; d.rec_scale = 1;
    return d;
}

// One call of every entry point that owns kernels or tables.
static void every_entry_point() {
    const int nx = 40, nz = 30, n2 = nx * nz;
    auto v = filled(n2, 2000), e = filled(n2, 0.1f), d = filled(n2, 0.05f), th = filled(n2, 10);
    std::vector<float> out(200 * n2);
    for (int var : {GEO_VARIANT_CPU, GEO_VARIANT_GPU, GEO_VARIANT_MPI}) {
        geo_fd2d_desc D = fd2d_desc(var);
        OK(geo_fd2d_shot(&D, v.data(), e.data(), d.data(), out.data(), nullptr, 0, GEO_MEM_HOST, nullptr));
    }
    geo_fd2d_desc D = fd2d_desc(GEO_VARIANT_GPU);
    OK(geo_tti2d_shot(&D, v.data(), e.data(), d.data(), th.data(), out.data(), nullptr, 0, GEO_MEM_HOST, nullptr));
    geo_rtm2d_gpu_desc G{};
    G.nx = nx; G.nz = nz; G.npml = 8; G.nt = 3; G.dx = G.dz = 10; G.dt = 1e-3f; G.favg = 20; G.pfac = 10; G.wtype = 1;
    G.ns = 1; G.fs = 20; G.zs = 1; G.mute_tt = 20; G.nangle = 60; G.dangle = 1;
    std::vector<float> ill(n2), ag((size_t)60 * n2);
    OK(geo_rtm2d_gpu(&G, v.data(), e.data(), d.data(), nullptr, out.data(), ill.data(), ag.data(), nullptr, nullptr, GEO_MEM_HOST, nullptr));
    OK(geo_rtm2d_tti(&G, v.data(), e.data(), d.data(), th.data(), nullptr, out.data(), ill.data(), ag.data(), nullptr, GEO_MEM_HOST, nullptr));
    const int xs[2] = {18, 20}, ws[2] = {9, 11};
    for (int mode : {GEO_MODE_EXACT, GEO_MODE_FAST})
        for (int gathers = 0; gathers < 2; gathers++) {
            geo_rtm2d_desc B{};
            B.nx = nx; B.nz = nz; B.npd = 8; B.nt = 3; B.dx = B.dz = 10; B.dt_ms = 1; B.favg = 20; B.pfac = 10; B.zs = 2;
            B.ns = 2; B.shot_x = xs; B.shot_nxs = ws; B.mode = mode;
            OK(geo_rtm2d_batch_adcig(&B, v.data(), e.data(), d.data(), ill.data(), nullptr, gathers ? out.data() : nullptr, GEO_MEM_HOST, nullptr));
        }
    const int m = 20, n3 = m * m * m;
    auto v3 = filled(n3, 2000), e3 = filled(n3, 0.1f), d3 = filled(n3, 0.05f), t3 = filled(n3, 10);
    std::vector<float> o3(4 * n3);
    waits_of("2D");
    geo_ae *ae = nullptr;
    OK(geo_ae_create(&ae, 1));
    fake::st().device_waits = 0;
    for (int mode : {GEO_MODE_EXACT, GEO_MODE_FAST}) {
        geo_fd3d_desc F{};
        F.nx = F.ny = F.nz = m; F.npd = 8; F.nt = 8; F.dx = F.dy = F.dz = 10; F.dt = 1e-3f; F.favg = 20; F.pfac = 10; F.wtype = 1;
        F.mode = mode; F.fsx = F.fsy = 10; F.fsz = 2; F.rec_iz = 8; F.drx = F.dry = 1; F.nrx = F.nry = m;
        OK(geo_fd3d_shot(&F, 0, v3.data(), e3.data(), d3.data(), std::vector<float>(8 * m * m).data(), GEO_MEM_HOST, nullptr));
        for (int method = 0; method < 4; method++) {
            geo_rtm3d_desc R{};
            R.fd = F; R.ns = 1; R.mute_tt = 5; R.method = method; R.snap_every = 2; R.ae = ae;
            OK(geo_rtm3d(&R, v3.data(), e3.data(), d3.data(), o3.data(), nullptr, nullptr, GEO_MEM_HOST, nullptr));
            if (mode == GEO_MODE_EXACT || method != GEO_RTM_SNAPSHOT) continue;
            R.theta = R.phi = t3.data();
            OK(geo_rtm3d(&R, v3.data(), e3.data(), d3.data(), o3.data(), nullptr, nullptr, GEO_MEM_HOST, nullptr));
        }
    }
    std::vector<float> blk((size_t)128 * 4096, 1.0f), rec(blk), grad(geo_ae_num_params());
    double loss;
    OK(geo_ae_eval(ae, blk.data(), 128, rec.data(), &loss, grad.data(), GEO_MEM_HOST, nullptr));
    for (int side : {32, 512}) {   // few and many tiles
        std::vector<float> a((size_t)side * side * 128), b(a.size());
        OK(geo_ae_roundtrip(ae, side, side, 128, a.data(), b.data(), 1, nullptr, nullptr));
    }
    for (int w : {64, 128, 256})   // every kernel of the GEMM rule
        for (int rows : {128, 512, 152 * 128})
            for (int K : {64, 128, 192, 256, 320}) {
                std::vector<unsigned short> A((size_t)rows * K), B((size_t)w * K);
                std::vector<float> o((size_t)rows * w);
                for (int f32 = 0; f32 < 2; f32++)
                    OK(geo_tc_gemm_bf16(rows, w, K, A.data(), B.data(), nullptr, 0, o.data(), f32, nullptr));
            }
    waits_of("3D and the codec");
    OK(geo_ae_destroy(ae));
}

// Constant tables and kernel attributes belong to a device: a second device
// gets what the first did, and none of its launches is refused.
static void check_devices() {
    for (int dev : {0, 1}) {
        fake::device = dev;
        every_entry_point();
    }
    for (const auto &s : fake::st().symbols[0])
        if (!fake::st().symbols[1].count(s)) { printf("constant %s not set on device 1\n", s.c_str()); failures++; }
    for (const auto &s : fake::st().attributes[0])
        if (!fake::st().attributes[1].count(s)) { printf("attribute of %s not set on device 1\n", s.c_str()); failures++; }
    printf("%s", fake::st().refused.c_str());
    if (!fake::st().refused.empty()) failures++;
    if (fake::st().symbols[0].size() < 5 || fake::st().attributes[0].size() < 20) { printf("too few calls seen\n"); failures++; }
    printf("%zu constants, %zu kernels with attributes\n", fake::st().symbols[0].size(), fake::st().attributes[0].size());
}

// A batch that does not fit at once runs in groups of shots: it succeeds where
// only half of its shots' memory is left, and one that cannot run at all says
// so and leaves no error behind for the next call.
static void check_batch_memory() {
    const int nx = 600, nz = 150, npd = 20, n2 = nx * nz, ns = 9;
    auto v = filled(n2, 2000), e = filled(n2, 0.1f), d = filled(n2, 0.05f);
    std::vector<int> xs(ns), ws(ns, 201);
    for (int k = 0; k < ns; k++) xs[k] = 200 + 20 * k;
    std::vector<float> img(n2), ag((size_t)90 * n2), per((size_t)ns * 201 * nz);
    for (int mode : {GEO_MODE_EXACT, GEO_MODE_FAST})
        for (int gathers = 0; gathers < 2; gathers++) {
            geo_rtm2d_desc B{};
            B.nx = nx; B.nz = nz; B.npd = npd; B.nt = 4; B.dx = B.dz = 10; B.dt_ms = 1; B.favg = 20; B.pfac = 10; B.zs = 2;
            B.ns = ns; B.shot_x = xs.data(); B.shot_nxs = ws.data(); B.mode = mode;
            auto run = [&](size_t limit) {
                fake::st().limit = limit;
                fake::st().peak = fake::st().in_use;
                return geo_rtm2d_batch_adcig(&B, v.data(), e.data(), d.data(), img.data(), per.data(),
                                             gathers ? ag.data() : nullptr, GEO_MEM_HOST, nullptr);
            };
            OK(run(~size_t(0)));
            const size_t all = fake::st().peak, fixed = gathers ? (size_t)90 * n2 * 4 : 0;
            for (double share : {0.99, 0.8, 0.5, 0.25}) OK(run(fixed + (size_t)(share * (all - fixed))));
            if (run(1 << 20) != GEO_ERR_NOMEM) { printf("1 MiB was enough\n"); failures++; }
            OK(run(~size_t(0)));
            if (fake::st().in_use) { printf("%zu bytes left allocated\n", fake::st().in_use); failures++; }
        }
}

// A batch of little work spreads over the warps that it has columns for: four
// of them a block forward, two pairs a block backward.
static void check_batch_spread() {
    struct Case { int ns, w, nz; } cases[] = {{1, 61, 101}, {1, 201, 301}, {4, 201, 301}, {3, 401, 401}, {2, 3, 20}};
    for (const Case &q : cases)
        for (int gathers = 0; gathers < 2; gathers++) {
            const int nx = q.w + 40, npd = 30, n2 = nx * q.nz;
            auto v = filled(n2, 2000), e = filled(n2, 0.1f), d = filled(n2, 0.05f);
            std::vector<float> img(n2), ag((size_t)90 * n2);
            std::vector<int> xs(q.ns, q.w / 2 + 1), ws(q.ns, q.w);
            geo_rtm2d_desc B{};
            B.nx = nx; B.nz = q.nz; B.npd = npd; B.nt = 2; B.dx = B.dz = 10; B.dt_ms = 1; B.favg = 20; B.pfac = 10; B.zs = 2;
            B.ns = q.ns; B.shot_x = xs.data(); B.shot_nxs = ws.data();
            fake::st().blocks_max.clear();
            OK(geo_rtm2d_batch_adcig(&B, v.data(), e.data(), d.data(), img.data(), nullptr, gathers ? ag.data() : nullptr, GEO_MEM_HOST, nullptr));
            // columns of all strips, at most 8 a warp, at least half of the resident warps (pairs) busy
            const long cols = (long)q.ns * (q.w + 2 * npd - 8) * ((q.nz + 2 * npd - 8 + 119) / 120);
            for (const auto &kv : fake::st().blocks_max) {
                if (kv.first.find("k_march2d") == std::string::npos) continue;
                const bool fwd = kv.first.find("k_march2dILi0E") != std::string::npos;
                const long res = 152 * 2 * (fwd ? 4 : 2), per = (fwd ? 4 : 2);   // two blocks an SM (fake occupancy)
                if (kv.second * per < std::min(cols, res / 2)) {
                    printf("%d shots %dx%d: %ld blocks of %s for %ld columns\n", q.ns, q.w, q.nz, kv.second, kv.first.c_str(), cols);
                    failures++;
                }
            }
        }
}

// The detector of non-finite values sees what a backward step computed: the
// next step's lines and records go in after a scan, not before it.
static int scans, late_scans, lines_of, lines_in;
static void watch_order(const std::string &n, void **args) {
    static int inject = -1;
    auto is = [&](const char *k) { return n.find(k) != n.npos; };
    if (is("k_march2d")) {
        const auto &st = *static_cast<const geo::MarchStep *>(args[3]);
        const bool fwd = is("k_march2dILi0E");
        if (!fwd && lines_in != st.it) late_scans++;   // its own lines are in the level it reads
        lines_in = inject = fwd ? -1 : st.inject;
    } else if (is("k_march_inject")) {
        lines_in = *static_cast<const int *>(args[1]);
    } else if (is("k_march_watch")) {
        scans++;
        if (inject >= 0) late_scans++;
    } else if (is("k_step2d_restore")) {
        lines_of = *static_cast<const int *>(args[1]);
    } else if (is("k_step2dILi3E")) {   // backward: a run starts with its lines put in by the launch before
        if (lines_of != static_cast<const geo::SStep *>(args[1])->it0) late_scans++;
    }
}
static void check_watch_order() {
    const int nx = 40, nz = 30, n2 = nx * nz, xs[2] = {18, 20}, ws[2] = {9, 11};
    auto v = filled(n2, 2000), e = filled(n2, 0.1f), d = filled(n2, 0.05f), th = filled(n2, 10);
    std::vector<float> img(n2);
    setenv("GEO_WATCH_EVERY", "3", 1);
    fake::st().on_launch = watch_order;
    geo_rtm2d_desc B{};
    B.nx = nx; B.nz = nz; B.npd = 8; B.nt = 11; B.dx = B.dz = 10; B.dt_ms = 1; B.favg = 20; B.pfac = 10; B.zs = 2;
    B.ns = 2; B.shot_x = xs; B.shot_nxs = ws;
    OK(geo_rtm2d_batch(&B, v.data(), e.data(), d.data(), img.data(), nullptr, GEO_MEM_HOST, nullptr));
    geo_rtm2d_gpu_desc G{};
    G.nx = nx; G.nz = nz; G.npml = 8; G.nt = 11; G.dx = G.dz = 10; G.dt = 1e-3f; G.favg = 20; G.pfac = 10; G.wtype = 1;
    G.ns = 2; G.fs = 20; G.zs = 1; G.mute_tt = 20; G.nangle = 60; G.dangle = 1;
    OK(geo_rtm2d_gpu(&G, v.data(), e.data(), d.data(), nullptr, img.data(), nullptr, nullptr, nullptr, nullptr, GEO_MEM_HOST, nullptr));
    OK(geo_rtm2d_tti(&G, v.data(), e.data(), d.data(), th.data(), nullptr, img.data(), nullptr, nullptr, nullptr, GEO_MEM_HOST, nullptr));
    if (scans != 8 || late_scans) { printf("%d scans of the batch, %d steps or scans out of order\n", scans, late_scans); failures++; }
}

// A plan's step keeps its tensor maps while steps of other plans (here between
// its two launches, as from another thread) push the cache of maps over.
static geo_fd3d_plan *tilted_plan() {
    const int m = 12, n3 = m * m * m;
    static auto v = filled(n3, 2000), e = filled(n3, 0.1f), d = filled(n3, 0.05f), t = filled(n3, 10);
    geo_fd3d_desc F{};
    F.nx = F.ny = F.nz = m; F.npd = 5; F.nt = 8; F.dx = F.dy = F.dz = 10; F.dt = 1e-3f; F.favg = 20; F.pfac = 10; F.wtype = 1;
    F.mode = GEO_MODE_FAST; F.fsx = F.fsy = 6; F.fsz = 2; F.rec_iz = 5; F.drx = F.dry = 1; F.nrx = F.nry = m;
    geo_fd3d_plan *p = nullptr;
    OK(geo_fd3d_plan_create(&p, &F));
    OK(geo_fd3d_set_model(p, v.data(), e.data(), d.data(), GEO_MEM_HOST, nullptr));
    OK(geo_fd3d_set_tilt(p, t.data(), t.data(), GEO_MEM_HOST, nullptr));
    return p;
}
static int bad_maps, stress_seen;
static void others_step(const std::string &n, void **args) {
    if (n.find("k_tti3d_vel") != n.npos) {
        fake::st().on_launch = nullptr;
        for (int k = 0; k < 40; k++) {
            float ms;
            OK(geo_fd3d_time_steps(tilted_plan(), 2, &ms, nullptr));   // plans stay: distinct buffers
        }
        fake::st().on_launch = others_step;
    } else if (n.find("k_tti3d_stress") != n.npos && !stress_seen++) {
        for (int k = 0; k < 15; k++) {
            const CUtensorMap &m = static_cast<const CUtensorMap *>(args[0])[k];
            char *base;
            memcpy(&base, &m, sizeof base);
            auto it = fake::st().blocks.upper_bound(base);   // the allocation it lies in
            if (it == fake::st().blocks.begin() || base >= static_cast<char *>((--it)->first) + it->second) bad_maps++;
        }
    }
}
static void check_tti_maps() {
    geo_fd3d_plan *p = tilted_plan();
    fake::st().on_launch = others_step;
    float ms;
    OK(geo_fd3d_time_steps(p, 1, &ms, nullptr));
    if (!stress_seen || bad_maps) { printf("%d of 15 maps of a step are not its own\n", bad_maps); failures++; }
}

static void check_chunk_override() {
    const int nx = 60, nz = 40, n2 = nx * nz, xs[2] = {18, 20}, ws[2] = {9, 11};
    auto v = filled(n2, 2000), e = filled(n2, 0.1f), d = filled(n2, 0.05f);
    std::vector<float> img(n2);
    geo_rtm2d_desc B{};
    B.nx = nx; B.nz = nz; B.npd = 8; B.nt = 2; B.dx = B.dz = 10; B.dt_ms = 1; B.favg = 20; B.pfac = 10; B.zs = 2;
    B.ns = 2; B.shot_x = xs; B.shot_nxs = ws;
    OK(geo_rtm2d_batch(&B, v.data(), e.data(), d.data(), img.data(), nullptr, GEO_MEM_HOST, nullptr));
    long steps = 0;
    for (const auto &kv : fake::st().launches)
        if (kv.first.find("k_march2d") != std::string::npos) steps += kv.second;
    if (steps != 4) { printf("%ld of 4 steps launched\n", steps); failures++; }
}

// Scratch of the codec that could not grow: the calls after it, of any size,
// find buffers again.
static void check_codec_growth() {
    geo_ae *ae = nullptr;
    OK(geo_ae_create(&ae, 1));
    std::vector<float> a((size_t)256 * 256 * 64), b(a.size()), blk((size_t)512 * 4096, 1.0f), grad(geo_ae_num_params());
    double loss;
    auto trip = [&](int n, int escape) { return geo_ae_roundtrip(ae, n, n, 64, a.data(), b.data(), escape, nullptr, nullptr); };
    auto eval = [&](int n) { return geo_ae_eval(ae, blk.data(), n, nullptr, &loss, grad.data(), GEO_MEM_DEVICE, nullptr); };
    OK(trip(64, 1));
    OK(eval(128));
    const size_t base = fake::st().in_use;
    // stop the growth at each of its buffers in turn
    for (int mib = 2; mib < 64; mib += 3) {
        fake::st().limit = base + ((size_t)mib << 20);
        const int st[2] = {trip(256, 1), eval(512)};
        for (int s : st)
            if (s != GEO_OK && s != GEO_ERR_NOMEM) { printf("limit %d MiB: %s\n", mib, geo_strerror(s)); failures++; }
        fake::st().limit = ~size_t(0);
        OK(trip(64, 1));
        OK(eval(128));
    }
    OK(geo_ae_destroy(ae));
    printf("%s", fake::st().refused.c_str());
    if (!fake::st().refused.empty()) failures++;
}

// A plain round trip takes the scratch that its kernels use: 25604 B a block
// (E2 to E4's, D4's and D3's outputs and the scale), blocks padded to 128.
static void check_codec_memory() {
    geo_ae *ae = nullptr;
    OK(geo_ae_create(&ae, 1));
    std::vector<float> a((size_t)256 * 256 * 64), b(a.size());
    const size_t before = fake::st().in_use, blocks = a.size() / 4096;
    OK(geo_ae_roundtrip(ae, 256, 256, 64, a.data(), b.data(), 0, nullptr, nullptr));
    const size_t used = fake::st().in_use - before, want = blocks * 25604;
    if (used > want + 65536) { printf("%zu bytes of scratch, %zu used by the kernels\n", used, want); failures++; }
    OK(geo_ae_destroy(ae));
}

// Tile widths of the 2D RTM programs' passes: the grids of
// test_rtm2d_gpu_program_wide_tiles take 16 columns on 152 SMs, with a tile a
// block and with several, and a width without a kernel is refused.
static void check_plans() {
    const int grids[][4] = {{143, 443, 5, 1}, {150, 450, 5, 1}, {1665, 200, 7, 0}};   // nx, nz, sponge, a tile a block
    for (const auto &q : grids)
        for (geo::StepKind k : {geo::SK_GFWD, geo::SK_GBWD}) {
            geo::SGrid g{};
            g.nx = q[0]; g.nz = q[1]; g.npd = q[2];
            g.nnx = q[0] + 2 * q[2]; g.nnz = q[1] + 2 * q[2]; g.ldz = (g.nnz + 3) / 4 * 4;
            geo::Fused2D p;
            OK(p.plan(k, false, g));
            if (p.tx != 16 || (p.tiles == p.grid) != (q[3] == 1)) {
                printf("%dx%d kind %d: %d columns, %d tiles on %d blocks\n", q[0], q[1], k, p.tx, p.tiles, p.grid);
                failures++;
            }
            OK(p.plan(k, true, g, 8));
            if (p.plan(k, true, g, 16) == GEO_OK) { printf("kind %d: 16 columns of the tilted medium accepted\n", k); failures++; }
            OK(p.plan(k, true, g));
            if (p.tx != 8) { printf("kind %d: tilted medium, %d columns\n", k, p.tx); failures++; }
        }
}

int main(int argc, char **argv) {
    const std::string check = argc > 1 ? argv[1] : "";
    if (check == "batch_chunk_override") {
        // any length leaves every window at least one chunk
        setenv("GEO_RTM2D_CHUNK", "2147483647", 1);
        check_chunk_override();
    } else if (check == "devices") check_devices();
    else if (check == "batch_memory") check_batch_memory();
    else if (check == "plans") check_plans();
    else if (check == "codec_growth") check_codec_growth();
    else if (check == "codec_memory") check_codec_memory();
    else if (check == "batch_spread") check_batch_spread();
    else if (check == "watch_order") check_watch_order();
    else if (check == "tti_maps") check_tti_maps();
    else return 2;
    return failures ? 1 : 0;
}

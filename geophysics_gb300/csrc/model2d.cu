// Model set-up of the 2D entry points on the device: the model check, the
// edge padding (pad_vv, CPU_vti2dfd_kernels.c:221-246: columns first, then
// rows, so corners take the corner value), the stencil's model arrays and
// the few values the host's set-up formulas read.  Float for float the
// host formulas.
//
// Copying the model to the host, padding it and forming the arrays there
// with one thread and copying them back was 2.1 ms of a 17.0 ms shot at
// 401^2 (15.4 ms now), 13 of 33.9 ms at 2401x601 (21.2), 3.6 of 12.9 ms for
// the 600x300 TTI shot (9.9) and 200 of 664 ms for a 16-shot RTM batch
// (481).  The kernels are bound by the bytes they read and write (k_raw_stats
// 22 us and k_model2d 22 us at 2401x601, 144 us for the batch's 16 windows
// with their double factors); one small copy each way carries the rest.
#include "model2d.cuh"
#include <algorithm>
#include <cmath>
#include <cstring>
#include <thread>

namespace geo {

namespace {

struct RawView {
    const float *a[4];
    int nx, nz;
};

struct StatsHead {
    unsigned long long bad, badth;   // smallest failing index*4 + kind; smallest non-finite theta
    unsigned vmin, nvmax;            // bits of the minimum; inverted bits of the maximum
};

// One warp per column: check_model's conditions, velocity range, column
// maxima.  The head starts as all ones.
__global__ void __launch_bounds__(256) k_raw_stats(const RawView r, StatsHead *h, float *colmax) {
    const int lane = threadIdx.x & 31;
    unsigned lo = 0xffffffffu, hi = 0u;
    for (int ix = blockIdx.x * 8 + (threadIdx.x >> 5); ix < r.nx; ix += gridDim.x * 8) {
        unsigned cm = 0u;
        for (int iz = lane; iz < r.nz; iz += 32) {
            const size_t i = (size_t)ix * r.nz + iz;
            const float v = r.a[0][i], e = r.a[1][i], d = r.a[2][i];
            int kind = 0;
            if (!isfinite(v) || !(v > 0.0f)) kind = 1;
            else if (!isfinite(e) || !isfinite(d)) kind = 2;
            else if (1 + 2 * d < 0) kind = 3;
            if (kind) atomicMin(&h->bad, (unsigned long long)i * 4 + (kind - 1));
            if (r.a[3] && !isfinite(r.a[3][i])) atomicMin(&h->badth, (unsigned long long)i);
            const unsigned b = __float_as_uint(v);   // positive, so ordered like the floats
            lo = min(lo, b);
            cm = max(cm, b);
        }
        for (int o = 16; o; o >>= 1) cm = max(cm, __shfl_xor_sync(0xffffffffu, cm, o));
        if (lane == 0) colmax[ix] = __uint_as_float(cm);
        hi = max(hi, cm);
    }
    for (int o = 16; o; o >>= 1) lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    if (lane == 0) {
        atomicMin(&h->vmin, lo);
        atomicMin(&h->nvmax, ~hi);
    }
}

__global__ void k_pick(const RawView r, const unsigned long long *idx, int n, float *out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) out[k] = r.a[idx[k] >> 60][idx[k] & ((1ull << 60) - 1)];
}

// Jobs travel as a kernel parameter, a pack per launch: no list to allocate.
constexpr int kPack = 16;
struct JobPack {
    ModelJob j[kPack];
};

__global__ void __launch_bounds__(256) k_model2d(const RawView r, const __grid_constant__ JobPack jobs) {
    const ModelJob &j = jobs.j[blockIdx.y];
    const int nnx = j.nx + 2 * j.npd, nnz = j.nz + 2 * j.npd, lane = threadIdx.x & 31;
    for (int ix = blockIdx.x * 8 + (threadIdx.x >> 5); ix < nnx; ix += gridDim.x * 8) {
        const int sx = min(min(max(ix - j.npd, 0), j.nx - 1) + j.col0, r.nx - 1);
        const float ax1 = j.kx ? j.ax1[ix] : 0.0f;
        for (int iz = lane; iz < nnz; iz += 32) {
            const int sz = min(max(iz - j.npd, 0), j.nz - 1);
            const size_t src = (size_t)sx * r.nz + sz, o = (size_t)ix * j.ldz + iz;
            const float v = r.a[0][src], vp = j.vp2 ? v * v : v;
            j.vp[o] = vp;
            j.e2[o] = 1 + 2 * r.a[1][src];
            if (j.d2) j.d2[o] = sqrtf(1 + 2 * r.a[2][src]);
            if (j.rad) j.rad[o] = (float)((double)r.a[3][src] * (kPiGui / 180.0));
            if (j.pwd) {
                const double pw = j.pw[src];
                const float h = (float)pw;
                j.pwd[o] = pw;
                j.ph[o] = h;
                j.pl[o] = (float)(pw - (double)h);
            }
            if (j.kz) {
                const double pw = j.pw[src];
                j.kz[o] = (double)(j.az1[iz] * vp) * pw * j.ddtz;
                j.kx[o] = (double)(ax1 * vp) * pw * j.ddtx;
            }
        }
    }
}

__global__ void k_box2d(float *e2, float *d2, int nnx, int nnz, int x0, int z0, int nb, const float *te2,
                        const float *td2) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nb * nb; k += gridDim.x * blockDim.x) {
        const int ix = x0 + k / nb, iz = z0 + k % nb;
        if (ix < 0 || ix >= nnx || iz < 0 || iz >= nnz) continue;
        e2[(size_t)ix * nnz + iz] = te2[k];
        d2[(size_t)ix * nnz + iz] = td2[k];
    }
}

RawView view(const Raw2D &r) { return RawView{{r.a[0], r.a[1], r.a[2], r.a[3]}, r.nx, r.nz}; }

}  // namespace

int Raw2D::open(int nx_, int nz_, const float *v, const float *e, const float *d, const float *theta, int mem,
                cudaStream_t s) {
    if (mem != GEO_MEM_DEVICE && mem != GEO_MEM_HOST) return fail(GEO_ERR_ARG, "bad mem kind");
    nx = nx_;
    nz = nz_;
    const float *src[4] = {v, e, d, theta};
    if (mem == GEO_MEM_DEVICE) {
        for (int k = 0; k < 4; k++) a[k] = src[k];
        return GEO_OK;
    }
    const size_t n = (size_t)nx * nz;
    GEO_TRY(own.alloc((theta ? 4 : 3) * n * 4));
    for (int k = 0; k < (theta ? 4 : 3); k++) {
        GEO_CUDA(cudaMemcpyAsync(own.as<float>() + k * n, src[k], n * 4, cudaMemcpyHostToDevice, s));
        a[k] = own.as<float>() + k * n;
    }
    return GEO_OK;
}

int raw_stats(const Raw2D &r, const std::vector<unsigned long long> &pick, RawStats &out, cudaStream_t s) {
    const size_t np = pick.size(), head = 32;
    static_assert(sizeof(StatsHead) <= 32, "head");
    // head, column maxima, picked values (copied back together), then the list
    const size_t o_col = head, o_val = o_col + (size_t)r.nx * 4, back = o_val + np * 4, o_idx = (back + 15) / 16 * 16;
    DevBuf buf;
    GEO_TRY(buf.alloc(o_idx + np * 8));
    char *b = buf.as<char>();
    GEO_CUDA(cudaMemsetAsync(b, 0xff, head, s));
    if (np) GEO_CUDA(cudaMemcpyAsync(b + o_idx, pick.data(), np * 8, cudaMemcpyHostToDevice, s));
    k_raw_stats<<<std::min((r.nx + 7) / 8, 152 * 8), 256, 0, s>>>(view(r), reinterpret_cast<StatsHead *>(b),
                                                                 reinterpret_cast<float *>(b + o_col));
    GEO_TRY(check_launch("raw_stats"));
    if (np) {
        k_pick<<<(unsigned)((np + 255) / 256), 256, 0, s>>>(view(r), reinterpret_cast<unsigned long long *>(b + o_idx),
                                                            (int)np, reinterpret_cast<float *>(b + o_val));
        GEO_TRY(check_launch("pick"));
    }
    std::vector<char> h(back);
    GEO_CUDA(cudaMemcpyAsync(h.data(), b, back, cudaMemcpyDeviceToHost, s));
    GEO_CUDA(cudaStreamSynchronize(s));
    StatsHead hd;
    memcpy(&hd, h.data(), sizeof hd);
    if (hd.bad != ~0ull) {   // reported as check_model does
        const size_t i = (size_t)(hd.bad >> 2);
        float bad = 0;
        GEO_CUDA(cudaMemcpy(&bad, r.a[0] + i, 4, cudaMemcpyDeviceToHost));
        if ((hd.bad & 3) == 0) return fail(GEO_ERR_MODEL, "velocity[%zu]=%g", i, bad);
        if ((hd.bad & 3) == 1) return fail(GEO_ERR_MODEL, "eps/del[%zu] not finite", i);
        return fail(GEO_ERR_MODEL, "1+2*delta[%zu] < 0", i);
    }
    if (hd.badth != ~0ull) return fail(GEO_ERR_MODEL, "theta[%zu] not finite", (size_t)hd.badth);
    const unsigned vmax = ~hd.nvmax;
    memcpy(&out.vmin, &hd.vmin, 4);
    memcpy(&out.vmax, &vmax, 4);
    out.colmax.resize(r.nx);
    memcpy(out.colmax.data(), h.data() + o_col, (size_t)r.nx * 4);
    out.val.resize(np);
    if (np) memcpy(out.val.data(), h.data() + o_val, np * 4);
    return GEO_OK;
}

int launch_model2d(const Raw2D &r, const std::vector<ModelJob> &jobs, cudaStream_t s) {
    for (size_t k = 0; k < jobs.size(); k += kPack) {
        JobPack p{};
        const int m = (int)std::min<size_t>(kPack, jobs.size() - k);
        int nnx = 0;
        for (int q = 0; q < m; q++) {
            p.j[q] = jobs[k + q];
            nnx = std::max(nnx, p.j[q].nx + 2 * p.j[q].npd);
        }
        k_model2d<<<dim3((nnx + 7) / 8, m), 256, 0, s>>>(view(r), p);
        GEO_TRY(check_launch("model2d"));
    }
    return GEO_OK;
}

static void host_pow_half(const float *del, size_t n, double *out) {
    auto part = [&](size_t a, size_t b) {
        for (size_t k = a; k < b; k++) out[k] = std::pow((double)(1 + 2 * del[k]), 0.5);
    };
    // about 15 ns a value: threads pay from a few hundred microseconds on
    const size_t want = std::max<size_t>(1, std::min<size_t>(n / 32768, std::thread::hardware_concurrency()));
    std::vector<std::thread> th;
    size_t done = 0;
    try {
        for (size_t t = 0; t + 1 < want; t++) {
            const size_t e = done + n / want;
            th.emplace_back(part, done, e);
            done = e;
        }
    } catch (...) {   // no more threads: the rest runs here
    }
    part(done, n);
    for (std::thread &t : th) t.join();
}

int upload_pow_half(const Raw2D &r, DevBuf &out, cudaStream_t s) {
    const size_t n = (size_t)r.nx * r.nz;
    std::vector<float> hd(n);
    std::vector<double> pw(n);
    GEO_CUDA(cudaMemcpyAsync(hd.data(), r.a[2], n * 4, cudaMemcpyDeviceToHost, s));
    GEO_CUDA(cudaStreamSynchronize(s));
    host_pow_half(hd.data(), n, pw.data());
    GEO_TRY(out.alloc(n * 8));
    GEO_CUDA(cudaMemcpyAsync(out.p, pw.data(), n * 8, cudaMemcpyHostToDevice, s));
    GEO_CUDA(cudaStreamSynchronize(s));   // pw is freed on return
    return GEO_OK;
}

int launch_box2d(float *e2, float *d2, int nnx, int nnz, int x0, int z0, int nb, const float *te2, const float *td2,
                 cudaStream_t s) {
    k_box2d<<<(nb * nb + 255) / 256, 256, 0, s>>>(e2, d2, nnx, nnz, x0, z0, nb, te2, td2);
    return check_launch("box2d");
}

}  // namespace geo

// Device-side model set-up of the 2D entry points (model2d.cu).
#pragma once
#include "geo_internal.h"
#include <cstring>
#include <vector>

namespace geo {

// One device allocation carved into 256-byte aligned arrays.  The caller
// runs its carving code twice: on an empty Arena to learn the size, then
// after alloc() to get the addresses.
struct Arena {
    DevBuf buf;
    size_t off = 0;
    template <class T>
    T *take(size_t n) {
        T *p = buf.p ? reinterpret_cast<T *>(static_cast<char *>(buf.p) + off) : nullptr;
        off += (n * sizeof(T) + 255) & ~(size_t)255;
        return p;
    }
    int alloc() {
        const size_t n = off;
        off = 0;
        return buf.alloc(n);
    }
};

// A packed host image of the small arrays a run uploads (profiles, taper
// boxes, source amplitudes): one copy to the device.
struct Blob {
    std::vector<unsigned char> h;
    DevBuf d;
    size_t put(const void *p, size_t bytes) {
        const size_t o = (h.size() + 15) / 16 * 16;
        h.resize(o + bytes);
        memcpy(h.data() + o, p, bytes);
        return o;
    }
    template <class T>
    size_t put(const std::vector<T> &v) {
        return put(v.data(), v.size() * sizeof(T));
    }
    template <class T>
    T *at(size_t o) const {
        return reinterpret_cast<T *>(d.as<char>() + o);
    }
    int upload(cudaStream_t s) {
        GEO_TRY(d.alloc(h.size()));
        GEO_CUDA(cudaMemcpyAsync(d.p, h.data(), h.size(), cudaMemcpyHostToDevice, s));
        return GEO_OK;
    }
};

// The unpadded model arrays v, eps, del (and theta) on the device: the
// caller's own device arrays, or copies of its host arrays.
struct Raw2D {
    const float *a[4] = {nullptr, nullptr, nullptr, nullptr};
    int nx = 0, nz = 0;
    DevBuf own;
    int open(int nx_, int nz_, const float *v, const float *e, const float *d, const float *theta, int mem,
             cudaStream_t s);
};

// Index of array k (0 v, 1 eps, 2 del, 3 theta) at an unpadded position.
inline unsigned long long raw_at(int k, const Raw2D &r, int ix, int iz) {
    return ((unsigned long long)k << 60) | ((unsigned long long)ix * r.nz + iz);
}

// What the host set-up needs from a model, in one round trip: the check of
// check_model (plus finite theta), the velocity range, the largest velocity
// of every column, and the values at the listed raw_at positions.
struct RawStats {
    float vmin = 0, vmax = 0;
    std::vector<float> colmax, val;
};
int raw_stats(const Raw2D &r, const std::vector<unsigned long long> &pick, RawStats &out, cudaStream_t s);

// Padded propagation model of one shot window: window column c reads model
// column min(c + col0, nx_model - 1), edges replicated into the sponge.
// Arrays have nnx columns of pitch ldz.  Null outputs are left out.
struct ModelJob {
    int nx, nz, npd, ldz, col0;
    int vp2;                          // vp holds vp*vp (the MPI program's rho*vp^2, rho == 1)
    float *vp, *e2, *d2, *rad;        // vp, 1+2eps, sqrtf(1+2del), tilt in radians
    // MPI exact form: kz = ((double)(az1*vp)*pw)*ddtz and kx with ax1, ddtx,
    // pw the unpadded pow(1+2del, 0.5)
    double *kz, *kx;
    const double *pw;
    const float *ax1, *az1;
    double ddtx, ddtz;
    // pw on the padded grid and its split into two floats
    double *pwd;
    float *ph, *pl;
};
int launch_model2d(const Raw2D &r, const std::vector<ModelJob> &jobs, cudaStream_t s);

// pow(1 + 2 del, 0.5) of every model point with the host's pow (over host
// threads), on the device.
int upload_pow_half(const Raw2D &r, DevBuf &out, cudaStream_t s);

// e2, d2 on the box (x0.., z0..) of edge nb from te2, td2 (nb*nb), clipped
// to the nnx x nnz grid.
int launch_box2d(float *e2, float *d2, int nnx, int nnz, int x0, int z0, int nb, const float *te2, const float *td2,
                 cudaStream_t s);

}  // namespace geo

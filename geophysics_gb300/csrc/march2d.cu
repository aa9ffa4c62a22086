// Fused 2D VTI time step of a batch of shots (the MPI RTM program's
// arithmetic, Toa_rtm_vti_adcig_cdp.c:1200-1327): one launch per step moves
// every shot from one time level to the next.
//
// A warp owns a strip of up to 120 depths (lanes 1-30, four each, 16-byte
// accesses) and marches along x over a chunk of columns.  P of the last
// eight columns and the new u of the last eight sit in registers, so each
// column brings P once, gives the new u four columns back and the stresses
// seven back; w is rebuilt from the column's Q, the lanes either side of the
// strip recomputing the four-point halos (shuffles).  u and w therefore make
// no round trip between the half-steps and warps wait for nobody.  The rows
// of the next two columns arrive by TMA bulk copies, one lane per array, in a
// two-stage ring of the warp's own with bounded mbarrier waits.
//
// Backward, two warps march the same chunk in step, one for the source
// side, one for the receiver side; the source warp hands its new P through
// shared memory (one named barrier per column) for the image.  The lines and
// records of the next step go into the new level as it is written.
//
// Per updated point and field the step moves 16 B of u,w,P,Q and 16 B of
// split stresses each way and 16 B of model, 80 B against the 96 B of the
// velocity and stress launches this replaces; the exact form's double
// chains are decided in FP32 (ziv.cuh).  16 shots (9.5 M points), exact
// form: 182 us a forward step (367 before) and 328 us a backward step (548
// before); the fast form 157 and 288 us, 4.6 and 5.1 TB/s.  The exact form is
// bound by instruction issue at three warps per scheduler (168 registers:
// the queues take 64; capped at 128 they spill, and with the shared memory
// the ring takes the spills miss L1: 394 us forward), the fast form by memory.
// Plain loads instead of the ring took 222 and 456 us with cp.async and 329
// and 698 us from registers.
#include "march2d.cuh"
#include "ziv.cuh"
#include "tc_util.cuh"
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>

namespace geo {

__constant__ float cm_fd[4] = {1.196289f, -0.0797526f, 0.009570313f, -0.0006975447f};
__constant__ float cm_adthr[kAdcigAngles];
__constant__ double cm_adw[kAdcigAngles];
// exp(-x^2-z^2) on the 7x7 source window (ptsource), from the host's exp
__constant__ double cm_gauss[49];

namespace {

struct V4 {
    float v[4];
};

__device__ __forceinline__ V4 ldc4(const float *p, bool on) {
    float4 t = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (on) t = __ldg(reinterpret_cast<const float4 *>(p));
    return V4{{t.x, t.y, t.z, t.w}};
}
__device__ __forceinline__ V4 lds4(const float4 *p) {
    const float4 t = *p;
    return V4{{t.x, t.y, t.z, t.w}};
}
// One row of a column, global -> shared by the TMA engine, completing on bar.
__device__ __forceinline__ void row_copy(float4 *dst, const float *src, unsigned bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     tc::su32(dst)),
                 "l"(src), "r"(bytes), "r"(tc::su32(bar))
                 : "memory");
}
__device__ __forceinline__ void st4(float *p, const V4 &a) {
    *reinterpret_cast<float4 *>(p) = make_float4(a.v[0], a.v[1], a.v[2], a.v[3]);
}

// The chain in double, where neither form decides (Toa_rtm_vti_adcig_cdp.c:1300-1310).
__device__ __noinline__ float chain_double(float a, float f, const double *pw, double ddt, float z) {
    return (float)((double)a - (double)f * *pw * ddt * (double)z);
}
__device__ __noinline__ float square_add_double(float ill, float s) {
    return (float)((double)ill + (double)s * (double)s);
}

// Poynting angle bin (RTM_corr_adcig, Toa_rtm_vti_adcig_cdp.c:1004-1068).
// The program bins with (int)(float)(0.5*acosf(a1)*180/pi), a non-increasing
// function of the float a1, so the host finds, with the same libm, the
// largest a1 of every bin count (cm_adthr[k-1]: largest a1 whose bin is >=
// k) and the kernel counts thresholds instead of calling acosf.
__device__ __forceinline__ int adcig_bin(float a1) {
    if (!(a1 >= -1.0f && a1 <= 1.0f)) return 0;
    int lo = 0, hi = kAdcigAngles;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (a1 <= cm_adthr[mid - 1]) lo = mid;
        else hi = mid - 1;
    }
    return lo == kAdcigAngles ? kAdcigAngles - 1 : lo;   // ia == 90 -> 89
}

constexpr int kMarchThreads = 128;
enum MarchMode { MM_FWD = 0, MM_BWD = 1, MM_ADCIG = 2 };   // forward; backward; backward with angle gathers
constexpr int kMarchBlocks = 3;   // per SM
// A warp's prefetch stage: rows of one column, 128 depths each (float4
// units): Q with the four depths either side, then P (seven columns on), u
// (three on), w, the split stresses, the model, the image row.
enum { MB_Q = 1, MB_P = 34, MB_U = 66, MB_W = 98, MB_S = 130, MB_M = 258, MB_I = 386, MB_STAGE = 418 };
constexpr int kRows = 13;   // with the image row; the low half of pow(1+2del, 0.5) only in the exact form
constexpr int kMarchStages = 2;
constexpr size_t kMarchSmem = (size_t)(kMarchThreads / 32) * kMarchStages * (MB_STAGE * 16 + 8);   // with the barriers
// source-side values handed to the receiver warp: P, and for the gathers Q, u, w
constexpr int march_xch(int mode) { return mode == MM_FWD ? 0 : mode == MM_BWD ? 1 : 4; }
constexpr size_t march_smem(int mode) {
    return kMarchSmem + (size_t)(kMarchThreads / 64) * 2 * march_xch(mode) * 32 * 16;
}
static_assert(kMarchBlocks * (march_smem(MM_ADCIG) + 1024) <= 233472, "blocks per SM");

// I: type of element offsets, 32 bits while a shot's slots fit.
template <int MODE, bool FAST, class I>
__global__ void __launch_bounds__(kMarchThreads, kMarchBlocks)
    k_march2d(const March2D *__restrict__ shots, const int4 *__restrict__ items, int nitems, const MarchStep st) {
    constexpr bool BWD = MODE != MM_FWD;
    constexpr int XN = march_xch(MODE);
    extern __shared__ float4 ring[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int side = BWD ? (warp & 1) : 0, pair = warp >> 1;
    const int item = BWD ? blockIdx.x * (kMarchThreads / 64) + pair : blockIdx.x * (kMarchThreads / 32) + warp;
    if (item >= nitems) return;   // both warps of a pair
    const int4 wk = __ldg(items + item);
    const March2D &S = shots[wk.x & 0xffffff];
    const int own_lanes = wk.x >> 24;
    const int z0 = wk.y + 4 * lane, xa = wk.z, xb = wk.w;
    const int nnx = S.nnx, nnz = S.nnz, ldz = S.ldz, npd = S.npd, nx = S.nx, nz = S.nz;
    const bool zin = z0 < ldz, own = lane >= 1 && lane <= own_lanes && z0 < nnz - 4;
    // depths on the updated grid; lanes that hold others (the first and the
    // last of the column) restore them afterwards
    bool m[4];
#pragma unroll
    for (int j = 0; j < 4; j++) m[j] = z0 + j >= 4 && z0 + j < nnz - 4;
    const bool edge = !(m[0] && m[1] && m[2] && m[3]);
    const float dtx = S.dtx, dtz = S.dtz;
    // one base pointer; every array is a slot at an offset
    float *const F = S.f;
    float4 *const buf = ring + warp * kMarchStages * MB_STAGE;
    uint64_t *const bar = reinterpret_cast<uint64_t *>(reinterpret_cast<char *>(ring) + march_smem(MODE) -
                                                       (kMarchThreads / 32) * kMarchStages * 8) +
                          warp * kMarchStages;
    if (lane == 0) {
        for (int k = 0; k < kMarchStages; k++) tc::mbar_init(&bar[k], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    const I n = S.n, sd = (I)(side * MS_SIDE) * n, l0 = sd + (I)(st.lev * MS_LEVEL) * n,
            l1 = sd + (I)((st.lev ^ 1) * MS_LEVEL) * n;
    const float *zp = S.cz1 + z0;   // cz1, cz2, az1, az2, ldz apart: read per column (L1), not kept in registers

    V4 p[8], q[8];   // P(c-7 .. c), new u(c-11 .. c-4)
#pragma unroll
    for (int k = 0; k < 8; k++)
#pragma unroll
        for (int j = 0; j < 4; j++) p[k].v[j] = q[k].v[j] = 0.0f;
    auto push = [](V4 *r, const V4 &a) {
#pragma unroll
        for (int k = 0; k < 7; k++) r[k] = r[k + 1];
        r[7] = a;
    };
    // new u of column xu from the queue P(xu-3 .. xu+4)
    auto vel_u = [&](int xu, const V4 &uo) {
        V4 r = uo;
        if (xu >= 4 && xu < nnx - 4) {
            const float c1 = __ldg(S.cx1 + xu) * dtx, c2 = __ldg(S.cx2 + xu);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                float xx = 0.0f;
#pragma unroll
                for (int k = 0; k < 4; k++) xx += cm_fd[k] * (p[4 + k].v[j] - p[3 - k].v[j]);
                r.v[j] = c2 * uo.v[j] - c1 * xx;
            }
            if (edge) {
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (!m[j]) r.v[j] = uo.v[j];
            }
        }
        return r;
    };
    // Rows of column x into stage x & 1: lane k brings row k.  Rows cover 128
    // depths whatever the grid holds there (the depths past it are the next
    // column's, inside the allocation, and are never used); only the image
    // row depends on the column.
    const bool rows = FAST ? lane != 11 : true;
    unsigned row_slot = 0, row_bytes = 512;
    int row_dst = 0, row_off = wk.y;
    {
        const int lv = side * MS_SIDE + st.lev * MS_LEVEL, sp = side * MS_SIDE;
        const int slot[kRows] = {lv + MS_Q, lv + MS_P, lv + MS_U, lv + MS_W, sp + MS_PX, sp + MS_PZ, sp + MS_QX, sp + MS_QZ,
                                 MS_VP, MS_E2, MS_D2, MS_PL, side ? MS_MIG : MS_ILL};
        const int dst[kRows] = {MB_Q, MB_P, MB_U, MB_W, MB_S, MB_S + 32, MB_S + 64, MB_S + 96,
                                MB_M, MB_M + 32, MB_M + 64, MB_M + 96, MB_I};
#pragma unroll
        for (int k = 0; k < kRows; k++)
            if (lane == k) {
                row_slot = slot[k];
                row_dst = dst[k];
            }
        if (lane == 0) {   // Q with its neighbours; at the top edge those are not used
            const int up = wk.y >= 4 ? 4 : 0;
            row_off -= up;
            row_dst -= up / 4;
            row_bytes = 512 + 4 * up + 16;
        }
        if (lane == 1) row_off += 7 * ldz;
        if (lane == 2) row_off += 3 * ldz;
    }
    const float *const row_src = F + ((size_t)row_slot * S.n + row_off);
    const unsigned col_bytes = (wk.y >= 4 ? 544 : 528) + 512 * (FAST ? 10 : 11);
    auto fetch = [&](int x) {
        const int k = x & (kMarchStages - 1), gx = x - npd;
        const bool img = BWD && gx >= 0 && gx < nx;
        if (lane == 0) tc::mbar_expect_tx(&bar[k], col_bytes + (img ? 512 : 0));
        __syncwarp();
        if (lane < kRows - 1 ? rows : img && lane == kRows - 1) {
            tc::fence_async_smem();
            row_copy(buf + k * MB_STAGE + row_dst, row_src + (size_t)x * ldz, row_bytes, &bar[k]);
        }
    };
#pragma unroll
    for (int k = 0; k < kMarchStages; k++)
        if (xa + k < xb) fetch(xa + k);
    {
        // P of the seven columns before, then u of columns xa-4 .. xa+2 (all
        // inside the grid), each set of loads in flight together
#pragma unroll
        for (int k = 0; k < 7; k++) p[k + 1] = ldc4(F + (l0 + MS_P * n + (I)((long)(xa - 7 + k) * ldz + z0)), zin && xa - 7 + k >= 0);
        V4 pc[7], uo[7];
#pragma unroll
        for (int k = 0; k < 7; k++) {
            const I o = (I)(xa + k) * ldz + z0;
            pc[k] = ldc4(F + (l0 + MS_P * n + o), zin && xa + k < nnx);
            uo[k] = ldc4(F + (l0 + MS_U * n + o - 4 * ldz), zin);
        }
#pragma unroll
        for (int k = 0; k < 7; k++) {
            push(p, pc[k]);
            const V4 un = vel_u(xa + k - 4, uo[k]);
            push(q, un);
            if (own && k >= 4 && xa + k - 4 < xb) st4(F + (l1 + MS_U * n + ((I)(xa + k - 4) * ldz + z0)), un);
        }
    }

    bool dead = false;
    for (int x = xa; x < xb; x++) {
        const I o = (I)x * ldz + z0;
        // A stage that never completes (no healthy device shows one) is
        // reported and waited for no more; the warp walks on to its end,
        // since its partner meets it at the pair's barrier.
        if (!dead && !tc::mbar_wait(&bar[x & (kMarchStages - 1)], ((x - xa) / kMarchStages) & 1)) {
            dead = true;
            if (lane == 0) atomicExch(st.err, 1);
        }
        const float4 *d = buf + (x & (kMarchStages - 1)) * MB_STAGE + lane;
        const V4 pc = lds4(d + MB_P), uo = lds4(d + MB_U);
        const V4 qa = lds4(d + MB_Q - 1), qb = lds4(d + MB_Q), qc = lds4(d + MB_Q + 1), wo = lds4(d + MB_W);
        V4 px = lds4(d + MB_S), pz = lds4(d + MB_S + 32), qx = lds4(d + MB_S + 64), qz = lds4(d + MB_S + 96);
        const V4 vp = lds4(d + MB_M);
        V4 e2 = lds4(d + MB_M + 32), d2 = lds4(d + MB_M + 64), ph = d2, pl = d2;   // the third slot is d2 or ph
        if (!FAST) pl = lds4(d + MB_M + 96);
        V4 im = vp;
        if (BWD) im = lds4(d + MB_I);
        __syncwarp();
        if (x + kMarchStages < xb && !dead) fetch(x + kMarchStages);
        const int gx = x - npd, gz0 = z0 - npd;
        const bool img = BWD && own && gx >= 0 && gx < nx && gz0 + 3 >= 0 && gz0 < nz;
        const float ax1 = __ldg(S.ax1 + x), ax2 = __ldg(S.ax2 + x);
        if (!BWD) {
            // SV taper box (forward only)
            const int bx = x - S.tx0;
            if (bx >= 0 && bx < kTB) {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int bz = z0 + j - S.tz0;
                    if (bz < 0 || bz >= kTB) continue;
                    e2.v[j] = S.te2[bx * kTB + bz];
                    if (FAST) {
                        d2.v[j] = S.td2[bx * kTB + bz];
                    } else {
                        const float2 t = S.tpw2[bx * kTB + bz];
                        ph.v[j] = t.x;
                        pl.v[j] = t.y;
                    }
                }
            }
        }

        push(p, pc);
        const V4 un = vel_u(x + 3, uo);
        push(q, un);
        if (own && x + 3 < xb) st4(F + (l1 + MS_U * n + o + 3 * ldz), un);

        // w of this lane's four depths
        V4 wn = wo;
        {
            const V4 cz1 = ldc4(zp, zin), cz2 = ldc4(zp + ldz, zin);
            const float e[12] = {qa.v[0], qa.v[1], qa.v[2], qa.v[3], qb.v[0], qb.v[1],
                                 qb.v[2], qb.v[3], qc.v[0], qc.v[1], qc.v[2], qc.v[3]};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                float zz = 0.0f;
#pragma unroll
                for (int k = 0; k < 4; k++) zz += cm_fd[k] * (e[4 + j + k + 1] - e[4 + j - k]);
                wn.v[j] = cz2.v[j] * wo.v[j] - cz1.v[j] * dtz * zz;
            }
            if (edge) {
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (!m[j]) wn.v[j] = wo.v[j];
            }
        }
        float f[11];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            f[j] = __shfl_up_sync(0xffffffffu, wn.v[j], 1);
            f[4 + j] = wn.v[j];
            if (j < 3) f[8 + j] = __shfl_down_sync(0xffffffffu, wn.v[j], 1);
        }
        V4 Pn, Qn;
        const V4 az1 = ldc4(zp + 2 * ldz, own), az2 = ldc4(zp + 3 * ldz, own);
        V4 xx4, zz4;
        bool open = false;   // a double chain not decided in FP32
#pragma unroll
        for (int j = 0; j < 4; j++) {
            float xx = 0.0f, zz = 0.0f;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                xx += cm_fd[k] * (q[4 + k].v[j] - q[3 - k].v[j]);
                zz += cm_fd[k] * (f[4 + j + k] - f[4 + j - k - 1]);
            }
            const float avx = ax1 * vp.v[j], avz = az1.v[j] * vp.v[j];
            px.v[j] = ax2 * px.v[j] - avx * e2.v[j] * dtx * xx;
            qz.v[j] = az2.v[j] * qz.v[j] - avz * dtz * zz;
            pz.v[j] = az2.v[j] * pz.v[j];
            qx.v[j] = ax2 * qx.v[j];
            if (FAST) {
                pz.v[j] = pz.v[j] - avz * d2.v[j] * dtz * zz;
                qx.v[j] = qx.v[j] - avx * d2.v[j] * dtx * xx;
            } else {
                bool s1, s2;
                const float r1 = zv_chain(pz.v[j], avz, ph.v[j], pl.v[j], st.dhz, st.dlz, zz, s1);
                const float r2 = zv_chain(qx.v[j], avx, ph.v[j], pl.v[j], st.dhx, st.dlx, xx, s2);
                // undecided ones keep their operand, marked by the derivative
                xx4.v[j] = s2 ? 0.0f : xx;
                zz4.v[j] = s1 ? 0.0f : zz;
                if (s1) pz.v[j] = r1;
                if (s2) qx.v[j] = r2;
                open |= !(s1 && s2) && m[j];
            }
        }
        if (!FAST && __any_sync(0xffffffffu, open && own)) {
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float avx = ax1 * vp.v[j], avz = az1.v[j] * vp.v[j];
                bool s1 = true, s2 = true;
                if (zz4.v[j] != 0.0f) {
                    const float r = zv_chain_tiny(pz.v[j], avz, ph.v[j], pl.v[j], st.dhz, st.dlz, zz4.v[j], s1);
                    if (s1) pz.v[j] = r;
                }
                if (xx4.v[j] != 0.0f) {
                    const float r = zv_chain_tiny(qx.v[j], avx, ph.v[j], pl.v[j], st.dhx, st.dlx, xx4.v[j], s2);
                    if (s2) qx.v[j] = r;
                }
                if (!(s1 && s2) && own && m[j]) {
                    const double *pw = S.pw + (o + j);
                    if (!BWD) {
                        const int bx = x - S.tx0, bz = z0 + j - S.tz0;
                        if (bx >= 0 && bx < kTB && bz >= 0 && bz < kTB) pw = S.tpw + (bx * kTB + bz);
                    }
                    if (!s1) pz.v[j] = chain_double(pz.v[j], avz, pw, st.ddtz, zz4.v[j]);
                    if (!s2) qx.v[j] = chain_double(qx.v[j], avx, pw, st.ddtx, xx4.v[j]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            Pn.v[j] = px.v[j] + pz.v[j];
            Qn.v[j] = qx.v[j] + qz.v[j];
        }
        if (!BWD && st.src_on && x - S.ixs >= -3 && x - S.ixs <= 3) {
            // 7x7 Gaussian source window, added after the split sum
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int rz = z0 + j - S.izs;
                if (rz < -3 || rz > 3) continue;
                const float s = (float)((double)st.amp * cm_gauss[(x - S.ixs + 3) * 7 + rz + 3]);
                Pn.v[j] = Pn.v[j] + s;
                Qn.v[j] = Qn.v[j] + s;
            }
        }
        // points off the updated grid keep their zeros
        if (edge) {
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (!m[j]) Pn.v[j] = Qn.v[j] = px.v[j] = pz.v[j] = qx.v[j] = qz.v[j] = 0.0f;
        }

        if (BWD) {
            // image and source illumination from the new level
            // (Toa_rtm_vti_adcig_cdp.c:1067-1076), a zero illumination becomes 1
            float4(*slot)[32] = reinterpret_cast<float4(*)[32]>(ring + (kMarchThreads / 32) * kMarchStages * MB_STAGE +
                                                                (pair * 2 + (x & 1)) * XN * 32);
            if (side == 0) {
                slot[0][lane] = make_float4(Pn.v[0], Pn.v[1], Pn.v[2], Pn.v[3]);
                if (MODE == MM_ADCIG) {
                    slot[1][lane] = make_float4(Qn.v[0], Qn.v[1], Qn.v[2], Qn.v[3]);
                    slot[2][lane] = make_float4(q[4].v[0], q[4].v[1], q[4].v[2], q[4].v[3]);
                    slot[3][lane] = make_float4(wn.v[0], wn.v[1], wn.v[2], wn.v[3]);
                }
            }
            asm volatile("bar.sync %0, 64;" ::"r"(pair + 1) : "memory");
            if (img) {
                if (side == 0) {
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        if (gz0 + j < 0 || gz0 + j >= nz) continue;
                        float v;
                        if (FAST) {
                            v = im.v[j] + Pn.v[j] * Pn.v[j];
                        } else {
                            bool sure;
                            v = zv_square_add(im.v[j], Pn.v[j], sure);
                            if (!sure) v = square_add_double(im.v[j], Pn.v[j]);
                        }
                        im.v[j] = v == 0.0f ? 1.0f : v;
                    }
                    st4(F + (MS_ILL * n + o), im);
                } else {
                    const float4 s4 = slot[0][lane];
                    const float sP[4] = {s4.x, s4.y, s4.z, s4.w};
                    V4 mg = im;
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        if (gz0 + j >= 0 && gz0 + j < nz) mg.v[j] = im.v[j] + Pn.v[j] * sP[j];
                    st4(F + (MS_MIG * n + o), mg);
                    if (MODE == MM_ADCIG) {
                        // Poynting vectors from the new P,Q and u,w of both
                        // fields (RTM_corr_adcig :1004-1068)
                        const float4 a4 = slot[1][lane], b4 = slot[2][lane], c4 = slot[3][lane];
                        const float sQ[4] = {a4.x, a4.y, a4.z, a4.w}, su[4] = {b4.x, b4.y, b4.z, b4.w},
                                    sw[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            if (gz0 + j < 0 || gz0 + j >= nz) continue;
                            // a zero product changes no sum but the sign of a zero one (a negative
                            // product below 2^-150 rounds to -0 there), and the shots' stack, which
                            // starts at +0, keeps no -0
                            if (Pn.v[j] * sP[j] == 0.0f) continue;
                            const float sx = -sP[j] * su[j], sz = -sQ[j] * sw[j];
                            const float rx = Pn.v[j] * q[4].v[j], rz = Qn.v[j] * wn.v[j];
                            const float b1 = sx * sx + sz * sz, b2 = rx * rx + rz * rz, a = sx * rx + sz * rz;
                            const float a1 = (float)((double)a / ((double)sqrtf(b1 * b2) + 0.0000000000001));
                            const int ia = adcig_bin(a1);
                            float *ag = S.adcig + ((long)ia * nx + gx) * nz + gz0 + j;
                            *ag = (float)((double)*ag + (double)(Pn.v[j] * sP[j]) * cm_adw[ia]);
                        }
                    }
                }
            }
            // the next step's lines (source side) and records (receiver
            // side) replace the new level's values as it is stored
            // (Toa_rtm_vti_adcig_cdp.c:914-927, 953-957; the left and right
            // lines win at the corners)
            if (st.inject >= 0 && own && gx >= 0 && gx < nx) {
                const long L = 2L * nx + 2L * nz, eo = (long)st.inject * L;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int gz = gz0 + j;
                    if (gz < 0 || gz >= nz) continue;
                    if (side) {
                        if (gz == 0) {
                            Pn.v[j] = S.rec_p[(long)st.inject * nx + gx];
                            Qn.v[j] = S.rec_q[(long)st.inject * nx + gx];
                        }
                        continue;
                    }
                    long k = -1;
                    if (gx == nx - 1) k = 2 * nx + nz + gz;
                    else if (gx == 0) k = 2 * nx + gz;
                    else if (gz == nz - 1) k = nx + gx;
                    else if (gz == 0) k = gx;
                    if (k >= 0) {
                        Pn.v[j] = S.edge_p[eo + k];
                        Qn.v[j] = S.edge_q[eo + k];
                    }
                }
            }
        }
        if (own) {
            st4(F + (l1 + MS_W * n + o), wn);
            st4(F + (sd + MS_PX * n + o), px);
            st4(F + (sd + MS_PZ * n + o), pz);
            st4(F + (sd + MS_QX * n + o), qx);
            st4(F + (sd + MS_QZ * n + o), qz);
            st4(F + (l1 + MS_P * n + o), Pn);
            st4(F + (l1 + MS_Q * n + o), Qn);
        }
        if (!BWD && own && gx >= 0 && gx < nx) {
            // receivers and interior-edge lines (Toa_rtm_vti_adcig_cdp.c:668-683)
            const long L = 2L * nx + 2L * nz, eo = (long)st.it * L;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int gz = gz0 + j;
                if (gz < 0 || gz >= nz) continue;
                if (gz == 0) {
                    S.rec_p[(long)st.it * nx + gx] = Pn.v[j];
                    S.rec_q[(long)st.it * nx + gx] = Qn.v[j];
                    S.edge_p[eo + gx] = Pn.v[j];
                    S.edge_q[eo + gx] = Qn.v[j];
                }
                if (gz == nz - 1) {
                    S.edge_p[eo + nx + gx] = Pn.v[j];
                    S.edge_q[eo + nx + gx] = Qn.v[j];
                }
                if (gx == 0) {
                    S.edge_p[eo + 2 * nx + gz] = Pn.v[j];
                    S.edge_q[eo + 2 * nx + gz] = Qn.v[j];
                }
                if (gx == nx - 1) {
                    S.edge_p[eo + 2 * nx + nz + gz] = Pn.v[j];
                    S.edge_q[eo + 2 * nx + nz + gz] = Qn.v[j];
                }
            }
        }
    }
}

__global__ void k_march_inject(const March2D *__restrict__ shots, int it, int lev) {
    const March2D &sh = shots[blockIdx.y];
    const int nx = sh.nx, nz = sh.nz, npd = sh.npd, ldz = sh.ldz;
    const long L = 2L * nx + 2L * nz;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < L; k += gridDim.x * blockDim.x) {
        int ix, iz;
        bool corner = false;   // the rows' corners take the columns' values
        if (k < nx) { ix = npd + k; iz = npd; corner = k == 0 || k == nx - 1; }
        else if (k < 2 * nx) { ix = npd + k - nx; iz = npd + nz - 1; corner = k == nx || k == 2 * nx - 1; }
        else if (k < 2 * nx + nz) { ix = npd; iz = npd + k - 2 * nx; }
        else { ix = npd + nx - 1; iz = npd + k - 2 * nx - nz; }
        const long id = (long)ix * ldz + iz;
        if (!corner) {
            sh.f[(size_t)(lev * MS_LEVEL + MS_P) * sh.n + id] = sh.edge_p[(long)it * L + k];
            sh.f[(size_t)(lev * MS_LEVEL + MS_Q) * sh.n + id] = sh.edge_q[(long)it * L + k];
        }
        if (k < nx) {
            sh.f[(size_t)(MS_SIDE + lev * MS_LEVEL + MS_P) * sh.n + id] = sh.rec_p[(long)it * nx + k];
            sh.f[(size_t)(MS_SIDE + lev * MS_LEVEL + MS_Q) * sh.n + id] = sh.rec_q[(long)it * nx + k];
        }
    }
}

// Block row y scans shot y's P; the first writer of a non-finite value's
// tag wins.
__global__ void k_march_watch(const March2D *__restrict__ shots, int nf, int lev, int *flag, int tag) {
    const March2D &sh = shots[blockIdx.y];
    const size_t n = sh.n / 4;
    bool bad = false;
    for (int f = 0; f < nf; f++) {
        const float4 *P = reinterpret_cast<const float4 *>(sh.f + (size_t)(f * MS_SIDE + lev * MS_LEVEL + MS_P) * sh.n);
        for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x) {
            const float4 a = P[k];
            bad |= !(fabsf(a.x) <= FLT_MAX) || !(fabsf(a.y) <= FLT_MAX) || !(fabsf(a.z) <= FLT_MAX) ||
                   !(fabsf(a.w) <= FLT_MAX);
        }
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) atomicCAS(flag, 0, tag);
}

__global__ void k_march_image(const March2D *__restrict__ shots, float *const *img, float *const *ill) {
    const March2D &sh = shots[blockIdx.y];
    const long n = (long)sh.nx * sh.nz;
    for (long k = blockIdx.x * (long)blockDim.x + threadIdx.x; k < n; k += (long)gridDim.x * blockDim.x) {
        const long o = (k / sh.nz + sh.npd) * sh.ldz + k % sh.nz + sh.npd;
        const float il = sh.f[(size_t)MS_ILL * sh.n + o];
        ill[blockIdx.y][k] = il;
        img[blockIdx.y][k] = sh.f[(size_t)MS_MIG * sh.n + o] / il;
    }
}

// Kernel of a mode, form and offset width.
const void *march_fn(int mode, bool fast, bool wide) {
#define MARCH_FN(M, F) \
    (wide ? (const void *)k_march2d<M, F, unsigned long long> : (const void *)k_march2d<M, F, unsigned>)
    switch (mode) {
        case MM_FWD: return fast ? MARCH_FN(MM_FWD, true) : MARCH_FN(MM_FWD, false);
        case MM_BWD: return fast ? MARCH_FN(MM_BWD, true) : MARCH_FN(MM_BWD, false);
        default: return fast ? MARCH_FN(MM_ADCIG, true) : MARCH_FN(MM_ADCIG, false);
    }
#undef MARCH_FN
}

int march_attr(int mode, bool fast, bool wide) {
    static OncePerDevice once[3][2][2];
    return allow_smem(once[mode][fast][wide], march_fn(mode, fast, wide), march_smem(mode));
}

int march_mode(bool backward, bool adcig) { return !backward ? MM_FWD : adcig ? MM_ADCIG : MM_BWD; }

}  // namespace

int march2d_resident(bool backward, bool fast, bool adcig, int *out) {
    const int mode = march_mode(backward, adcig);
    int dev = 0, sms = 0, occ = 0;
    GEO_TRY(march_attr(mode, fast, false));
    GEO_CUDA(cudaGetDevice(&dev));
    GEO_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    GEO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, march_fn(mode, fast, false), kMarchThreads,
                                                           march_smem(mode)));
    *out = std::max(1, occ * sms * (backward ? kMarchThreads / 64 : kMarchThreads / 32));
    return GEO_OK;
}

int launch_march2d(bool backward, bool fast, bool adcig, bool wide, const March2D *d_shots, const int4 *d_items,
                   int nitems, const MarchStep &st, cudaStream_t s) {
    if (nitems < 1) return GEO_OK;
    const int mode = march_mode(backward, adcig), per = backward ? kMarchThreads / 64 : kMarchThreads / 32;
    GEO_TRY(march_attr(mode, fast, wide));
    void *args[] = {(void *)&d_shots, (void *)&d_items, (void *)&nitems, (void *)&st};
    GEO_CUDA(cudaLaunchKernel(march_fn(mode, fast, wide), dim3((nitems + per - 1) / per), dim3(kMarchThreads), args,
                              march_smem(mode), s));
    return check_launch("march2d");
}

int launch_march_inject(const March2D *d_shots, int ns, int maxline, int it, int lev, cudaStream_t s) {
    k_march_inject<<<dim3((maxline + 255) / 256, ns), 256, 0, s>>>(d_shots, it, lev);
    return check_launch("march_inject");
}

int launch_march_watch(const March2D *d_shots, int ns, int nf, int lev, int *flag, int tag, cudaStream_t s) {
    if (!flag || ns < 1) return GEO_OK;
    k_march_watch<<<dim3(64, ns), 256, 0, s>>>(d_shots, nf, lev, flag, tag);
    return check_launch("march_watch");
}

int launch_march_image(const March2D *d_shots, int ns, float *const *img, float *const *ill, cudaStream_t s) {
    k_march_image<<<dim3(256, ns), 256, 0, s>>>(d_shots, img, ill);
    return check_launch("march_image");
}

// The MPI program's bin of one cosine a1 (before its 90 -> 89 clamp).
static int ref_adcig_bin(float a1) {
    const float a2 = (float)(0.5 * std::acos(a1) * 180 / kPiMpi);
    return (int)(a2 / 1.0);
}

static uint32_t order_key(float f) {
    uint32_t b;
    memcpy(&b, &f, 4);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

static float key_float(uint32_t k) {
    const uint32_t b = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
    float f;
    memcpy(&f, &b, 4);
    return f;
}

int load_march_tables(bool adcig, cudaStream_t s) {
    double g[49];
    for (int x = -3; x <= 3; x++)
        for (int z = -3; z <= 3; z++) g[(x + 3) * 7 + (z + 3)] = std::exp((double)(-z * z - x * x));
    GEO_CUDA(cudaMemcpyToSymbolAsync(cm_gauss, g, sizeof g, 0, cudaMemcpyHostToDevice, s));
    if (!adcig) return GEO_OK;
    static float thr[kAdcigAngles];
    static double w[kAdcigAngles];
    static std::once_flag built;
    std::call_once(built, [] {
        const uint32_t lo = order_key(-1.0f), hi = order_key(1.0f);
        for (int k = 1; k <= kAdcigAngles; k++) {
            if (ref_adcig_bin(-1.0f) < k) {
                thr[k - 1] = -2.0f;   // no cosine reaches this bin
                continue;
            }
            uint32_t a = lo, b = hi;  // ref_adcig_bin(key_float(a)) >= k
            while (a < b) {
                const uint32_t m = a + (b - a + 1) / 2;
                if (ref_adcig_bin(key_float(m)) >= k) a = m;
                else b = m - 1;
            }
            thr[k - 1] = key_float(a);
        }
        for (int ia = 0; ia < kAdcigAngles; ia++) w[ia] = std::pow(std::cos(ia * kPiMpi / 180.0), 3);
    });
    GEO_CUDA(cudaMemcpyToSymbolAsync(cm_adthr, thr, sizeof thr, 0, cudaMemcpyHostToDevice, s));
    GEO_CUDA(cudaMemcpyToSymbolAsync(cm_adw, w, sizeof w, 0, cudaMemcpyHostToDevice, s));
    return GEO_OK;
}

}  // namespace geo

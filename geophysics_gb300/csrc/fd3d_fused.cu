// Fused 3D VTI time step: one kernel per step, marching along y.
//
// A block owns a 32(z) x 16(x) column of the grid and a chunk of y planes.
// Per plane it rebuilds the velocities it needs from P,Q (u with a 4-cell
// x halo, w with a 4-cell z halo, v from a register queue along y) and then
// updates the stresses, so u,v,w never make a round trip through HBM between
// the two half-steps of the reference (GPU_vti3dfd_kernels.cu:90-201).
//
// Each of the 256 threads owns two consecutive depths of one x column and
// moves them as one 8-byte vector: a tap along x is one shared-memory load
// for two points, the eight taps along z are five, and addresses, predicates
// and loop bookkeeping are paid once per two points.  The y taps come from
// two register queues (P of planes y .. y+7, the new v of planes y-4 .. y+3).
//
// Data movement: the boxes with halos and the model of a plane go through
// TMA (cp.async.bulk.tensor) into a 3-stage shared-memory pipeline, one
// mbarrier per stage; the thread's own P seven planes ahead and v three
// planes ahead are loaded into registers one plane early, the split stresses
// (sponge planes of the fast form, every plane of the exact form) at the
// start of their plane.  The rebuilt u and w tiles are double-buffered, so a
// plane has one block barrier, after which the previous plane's stage is
// refilled.  A chunk's queues are filled by plain loads, all in flight
// together, before the march.  Writes go to the next level (u,v,w,P,Q
// ping-pong between steps; split stresses in place).
//
// Measured per step against one depth and two columns per thread with every
// array in the TMA stages and two barriers a plane: 400^3 + 40 fast 1.557 ->
// 1.395 ms (8.2 GB of DRAM traffic: 5.9 TB/s), exact 1.780 -> 1.736 ms;
// 176x160x144 + 20 with imaging 0.184 -> 0.137 ms; 121x93x107 + 20 exact 83
// -> 62 us.  The fast form is bound by DRAM at the large size (halos miss L2:
// 1.21x the algorithmic bytes), by issue and latency at the small ones (240^3:
// 333 thread instructions a point, issue 58%, DRAM 64% busy).  Four depths
// per thread (128 threads, 168 registers, 12 warps an SM) took 1.53 ms, 190
// and 100 us: half the instructions' latency is exposed; capped at 128
// registers, or at 80 with two depths, it spills and the spills miss L1 (2.0
// ms and more).  32 columns a tile: 1.45 ms; two stages 1.55 ms; four 1.39.

// Arithmetic: GEO_MODE_EXACT keeps the reference's operation chain (no
// contraction) and is bit-identical to it; GEO_MODE_FAST uses fused
// multiply-adds at fixed places and the premultiplied model (A,B,C), the
// same operations as the oracle's fast mode.
#include "geo_internal.h"
#include "fd3d.cuh"
#include "fd3d_fused.cuh"
#include "tc_util.cuh"
#include <cudaTypedefs.h>

namespace geo {

__constant__ float cf_fd[4] = {1.196289f, -0.0797526f, 0.009570313f, -0.0006975447f};

// stage layout (floats)
constexpr int OFF_PH = 0;                 // P x-halo box, stress plane
constexpr int OFF_Q = OFF_PH + kPB;
constexpr int OFF_U = OFF_Q + kQB;
constexpr int OFF_W = OFF_U + kUB;
constexpr int OFF_M = OFF_W + kQB;        // vp,e2,d2 or A,B,C
static_assert(OFF_M + 3 * kOB == kStageFloats, "stage layout");
static_assert((OFF_Q * 4) % 128 == 0 && (OFF_U * 4) % 128 == 0 && (OFF_W * 4) % 128 == 0 && (OFF_M * 4) % 128 == 0 &&
                  (kStageFloats * 4) % 128 == 0,
              "TMA destinations must stay 128-byte aligned");
static_assert((kFusedSmem + 1024 + 64) * kFusedBlocks <= 233472, "blocks per SM must fit in shared memory");

// mbarrier helpers with bounded waits (2 s), shared with the codec kernels
using tc::mbar_expect_tx;
using tc::mbar_init;
using tc::mbar_wait;
using tc::su32;

__device__ __forceinline__ void tma3(float *dst, const CUtensorMap *map, int c0, int c1, int c2, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::
            "r"(su32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(su32(bar))
        : "memory");
}

namespace {

constexpr unsigned kFull = (1u << kW) - 1;

// kW consecutive depths, moved as one vector.
struct FV {
    float v[kW];
};
static_assert(kW == 2, "vectors are float2");
__device__ __forceinline__ FV unpack(const float2 &t) { return FV{{t.x, t.y}}; }
__device__ __forceinline__ FV ld_s(const float *p) { return unpack(*reinterpret_cast<const float2 *>(p)); }
// Plain loads throughout, also of arrays that this launch only reads: its
// blocks come up while the kernel before, which wrote them, still runs, and
// ld.global.nc (__ldg) is defined only for what nobody writes while a kernel
// lives and may be moved ahead of the wait for that kernel.
__device__ __forceinline__ FV ld_g(const float *p) { return unpack(*reinterpret_cast<const float2 *>(p)); }
__device__ __forceinline__ FV ld_g(const float *p, bool on) {
    float2 t{};
    if (on) t = *reinterpret_cast<const float2 *>(p);
    return unpack(t);
}
__device__ __forceinline__ void st_v(float *p, const FV &a) {
    *reinterpret_cast<float2 *>(p) = make_float2(a.v[0], a.v[1]);
}
__device__ __forceinline__ void push(FV *q, const FV &a) {
#pragma unroll
    for (int k = 0; k < 7; k++) q[k] = q[k + 1];
    q[7] = a;
}
// a where the point is updated, else b
__device__ __forceinline__ FV pick(unsigned m, const FV &a, const FV &b) {
    FV r = a;
    if (m != kFull) {
#pragma unroll
        for (int j = 0; j < kW; j++)
            if (!(m >> j & 1u)) r.v[j] = b.v[j];
    }
    return r;
}

// 8-tap staggered derivative sum_m c_m (a_m - b_m).  EXACT: the reference's
// accumulation from 0; FAST: first product, then three fused multiply-adds.
template <int MODE>
__device__ __forceinline__ float deriv(float a0, float b0, float a1, float b1, float a2, float b2, float a3,
                                       float b3) {
    if (MODE == GEO_MODE_FAST) {
        float d = cf_fd[0] * (a0 - b0);
        d = __fmaf_rn(cf_fd[1], a1 - b1, d);
        d = __fmaf_rn(cf_fd[2], a2 - b2, d);
        return __fmaf_rn(cf_fd[3], a3 - b3, d);
    }
    float d = 0.0f;
    d += cf_fd[0] * (a0 - b0);
    d += cf_fd[1] * (a1 - b1);
    d += cf_fd[2] * (a2 - b2);
    d += cf_fd[3] * (a3 - b3);
    return d;
}

// Derivative over eight vectors a(-3) .. a(+4) (forward stagger) or, shifted
// by one, a(-4) .. a(+3) (backward).
template <int MODE>
__device__ __forceinline__ FV deriv8(const FV *q) {
    FV r;
#pragma unroll
    for (int j = 0; j < kW; j++)
        r.v[j] = deriv<MODE>(q[4].v[j], q[3].v[j], q[5].v[j], q[2].v[j], q[6].v[j], q[1].v[j], q[7].v[j], q[0].v[j]);
    return r;
}

// Derivative along z of the kW depths at p; SHIFT 1: taps +1..+4 minus
// 0..-3 (forward), 0: 0..+3 minus -1..-4.  mid: the vector at p, if the
// caller has it in registers.
template <int MODE, int SHIFT>
__device__ __forceinline__ FV derivz(const float *p, const FV &mid) {
    float e[8 + kW];
#pragma unroll
    for (int k = 0; k < 8 + kW; k += kW) {
        const FV t = k == 4 ? mid : ld_s(p + k - 4);
#pragma unroll
        for (int j = 0; j < kW; j++) e[k + j] = t.v[j];
    }
    FV r;
#pragma unroll
    for (int j = 0; j < kW; j++) {
        const float *q = e + 4 + j + SHIFT;
        r.v[j] = deriv<MODE>(q[0], q[-1], q[1], q[-2], q[2], q[-3], q[3], q[-4]);
    }
    return r;
}

// Velocity update: c2*old - k1*d with k1 = c1*dt.
template <int MODE>
__device__ __forceinline__ float vel_update(float c2, float old, float k1, float d) {
    if (MODE == GEO_MODE_FAST) return __fmaf_rn(-k1, d, c2 * old);
    return c2 * old - k1 * d;
}

template <int MODE, bool RTM>
__global__ void __launch_bounds__(kFusedThreads, kFusedBlocks)
    k_fused3d(const __grid_constant__ StepMaps tm, const Fused3D g, const StepArgs3D st) {
    extern __shared__ unsigned char smem_raw[];
    float *base = reinterpret_cast<float *>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    float *stages = base;
    float *utiles = stages + kStages * kStageFloats;   // two of each tile
    float *wtiles = utiles + 2 * kUTile;
    float *zprof = wtiles + 2 * kWTile;                // cz1*dtz, cz2, az1, az2 on the tile's 32 depths
    uint64_t *bar = reinterpret_cast<uint64_t *>(zprof + 4 * kTZ);
    __shared__ int s_abort;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tile = blockIdx.x % g.ntiles, chunk = blockIdx.x / g.ntiles;
    // consecutive blocks are z neighbours
    const int z0 = (tile % g.ntz) * kTZ, x0 = (tile / g.ntz) * kFX;
    const int ylo = 4 + chunk * g.chunk;
    const int yhi = min(ylo + g.chunk, g.nny - 4);
    const int NI = yhi - ylo;
    const bool xz_inside = x0 >= g.npd && x0 + kFX <= g.npd + g.nx && z0 >= g.npd && z0 + kTZ <= g.npd + g.nz;

    if (tid == 0) {
        for (int s = 0; s < kStages; s++) mbar_init(&bar[s], 1);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < kTZ) {
        const int z = min(z0 + tid, g.nnz - 1);
        zprof[tid] = g.cz1[z] * g.dtz;
        zprof[kTZ + tid] = g.cz2[z];
        zprof[2 * kTZ + tid] = g.az1[z];
        zprof[3 * kTZ + tid] = g.az2[z];
    }
    __syncthreads();
    // Launched while the step before still runs (the profiles above are fixed
    // for the run); from here on that step's results are read.  The next step's
    // blocks may start once all of this one's have.
    tc::after_predecessor();

    // Boxes of plane ylo + i into stage s, spread over the warps'
    // first lanes.  The expected byte count may be posted after a copy
    // completes: the phase cannot finish before warp 0 arrives.
    auto issue = [&](int i, int s) {
        const int y = ylo + i;
        float *sp = stages + s * kStageFloats;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (warp == 0) {
            mbar_expect_tx(&bar[s], kStageFloats * 4);
            tma3(sp + OFF_PH, &tm.m[0], z0, x0 - 7, y, &bar[s]);
            tma3(sp + OFF_Q, &tm.m[1], z0 - 8, x0, y, &bar[s]);
        } else if (warp == 1) {
            tma3(sp + OFF_U, &tm.m[2], z0, x0 - 4, y, &bar[s]);
            tma3(sp + OFF_W, &tm.m[3], z0 - 8, x0, y, &bar[s]);
        } else if (warp == 2) {
            for (int r = 0; r < 3; r++) tma3(sp + OFF_M + r * kOB, &tm.m[4 + r], z0, x0, y, &bar[s]);
        }
    };
    if (lane == 0)
        for (int i = 0; i < kStages && i < NI; i++) issue(i, i);

    // ---- the thread's column and depths
    const int zl = tid % (kTZ / kW) * kW, c = tid / (kTZ / kW), xa = x0 + c, zo = z0 + zl;
    const bool mem = xa < g.nnx && zo < g.ldz;   // its vector exists
    unsigned um = 0;                             // updated depths
    if (xa >= 4 && xa < g.nnx - 4)
#pragma unroll
        for (int j = 0; j < kW; j++) um |= (zo + j >= 4 && zo + j < g.nnz - 4 ? 1u : 0u) << j;
    unsigned in4 = 0;                            // depths inside the physical box (x and z)
    if (xa >= g.npd && xa < g.npd + g.nx)
#pragma unroll
        for (int j = 0; j < kW; j++) in4 |= (zo + j >= g.npd && zo + j < g.npd + g.nz ? 1u : 0u) << j;
    const bool wr = um != 0;
    const int xc = min(xa, g.nnx - 1);
    const float kx = g.cx1[xc] * g.dtx, cx2 = g.cx2[xc], ax1 = g.ax1[xc], ax2 = g.ax2[xc];
    // receiver trace along x (or -1) and depth within the vector
    int rec_x = -1;
    const int rec_j = st.rec_iz - zo;
    if (st.rec && rec_j >= 0 && rec_j < kW) {
        const int r = xa - g.npd - st.rx0;
        if (r >= 0 && r % st.drx == 0 && r / st.drx < st.nrx && (um >> rec_j & 1u)) rec_x = r / st.drx;
    }
    // halo velocities: the first threads u on the 7 halo columns (4 left, 3
    // right), threads of the upper half w on the four depths above and below
    // each column
    FV hk, hc2;
    unsigned hm = 0;
    int h_tile = 0, h_src = 0;
    constexpr int kUTasks = 7 * kTZ / kW, kWGroups = 8 / kW, kHalf = kFusedThreads / 2;
    static_assert(kUTasks <= kHalf && kFX * kWGroups <= kHalf, "halo tasks");
    const bool hu = tid < kUTasks, hw = tid >= kHalf && tid < kHalf + kFX * kWGroups;
    if (hu) {
        const int hc = c, cc = hc < 4 ? hc : kFX + hc, x = x0 - 4 + cc, xcl = min(max(x, 0), g.nnx - 1);
        if (x >= 4 && x < g.nnx - 4)
            for (int j = 0; j < kW; j++) hm |= (zo + j >= 4 && zo + j < g.nnz - 4 ? 1u : 0u) << j;
        for (int j = 0; j < kW; j++) {
            hk.v[j] = g.cx1[xcl] * g.dtx;
            hc2.v[j] = g.cx2[xcl];
        }
        h_tile = cc * kTZ + zl;          // u tile and u box
        h_src = (cc + 3) * kTZ + zl;     // P halo box
    } else {
        const int t = (tid - kHalf + kFusedThreads) % (kFX * kWGroups), col = t / kWGroups, grp = t % kWGroups;
        const int zr = grp < kWGroups / 2 ? grp * kW - 4 : kTZ + (grp - kWGroups / 2) * kW, x = x0 + col, z = z0 + zr;
        for (int j = 0; j < kW; j++) {
            if (x >= 4 && x < g.nnx - 4) hm |= (z + j >= 4 && z + j < g.nnz - 4 ? 1u : 0u) << j;
            const int zcl = min(max(z + j, 0), g.nnz - 1);
            hk.v[j] = g.cz1[zcl] * g.dtz;
            hc2.v[j] = g.cz2[zcl];
        }
        h_tile = col * 40 + zr + 4;          // w tile
        h_src = col * 48 + zr + 8;           // Q and w boxes
    }
    const int sxy = (int)g.sxy, own = zo + g.ldz * xa;   // element offsets fit in 32 bits (checked on the host)
    // the step's point source, P,Q += amp before the velocity update
    // (GPU_vti3dfd_kernels.cu:135), on this thread's own copy of P
    const int src_j = st.src_on && xa == st.ixs ? st.izs - zo : -1;
    auto add_source = [&](FV &a, int plane) {
        if (src_j >= 0 && plane == st.iys)
#pragma unroll
            for (int j = 0; j < kW; j++)
                if (j == src_j) a.v[j] += st.amp;
    };

    // ---- queues: P of planes ylo-1 .. ylo+6, the new v of ylo-4 .. ylo+2
    FV p[8], q[8];
#pragma unroll
    for (int k = 0; k < 8; k++)
#pragma unroll
        for (int j = 0; j < kW; j++) p[k].v[j] = q[k].v[j] = 0.0f;
    auto ld_P = [&](int y) { return ld_g(g.P0 + own + sxy * y, mem && y >= 0 && y < g.nny); };
    auto ld_v = [&](int y) { return ld_g(g.v0 + own + sxy * y, mem && y >= 0 && y < g.nny); };
    auto new_v = [&](const FV &vo, int yv, float cy1, float cy2) {
        if (yv < 4 || yv >= g.nny - 4) return vo;
        const float ky = cy1 * g.dty;
        const FV d = deriv8<MODE>(p);
        FV r;
#pragma unroll
        for (int j = 0; j < kW; j++) r.v[j] = vel_update<MODE>(cy2, vo.v[j], ky, d.v[j]);
        return pick(um, r, vo);
    };
#pragma unroll
    for (int k = 0; k < 7; k++) p[k + 1] = ld_P(ylo - 7 + k);
    {
        FV pn[7], vn[7];
#pragma unroll
        for (int k = 0; k < 7; k++) {
            pn[k] = ld_P(ylo + k);
            vn[k] = ld_v(ylo - 4 + k);
        }
#pragma unroll
        for (int k = 0; k < 7; k++) add_source(p[k + 1], ylo - 7 + k);
#pragma unroll
        for (int k = 0; k < 7; k++) {
            const int yv = ylo - 4 + k, yc = min(max(yv, 0), g.nny - 1);
            add_source(pn[k], ylo + k);
            push(p, pn[k]);
            const FV t = new_v(vn[k], yv, g.cy1[yc], g.cy2[yc]);
            push(q, t);
            if (wr && yv >= ylo && yv < yhi) st_v(g.v1 + own + sxy * yv, t);
        }
    }
    // one plane ahead: own P and v, y-direction sponge factors
    FV nP = ld_P(ylo + 7), nv = ld_v(ylo + 3);
    auto ycoef = [&](int y, float &c1, float &c2, float &a1, float &a2) {
        const int yv = min(y + 3, g.nny - 1), ys = min(y, g.nny - 1);
        c1 = __ldg(g.cy1 + yv); c2 = __ldg(g.cy2 + yv); a1 = __ldg(g.ay1 + ys); a2 = __ldg(g.ay2 + ys);
    };
    float ncy1, ncy2, nay1, nay2;
    ycoef(ylo, ncy1, ncy2, nay1, nay2);

    int s = 0, off = own + sxy * ylo;   // stage and offset of the plane
    unsigned par = 0;                   // parity of the stage's phase
    for (int i = 0; i < NI; i++, s = s + 1 == kStages ? 0 : s + 1, par ^= s == 0, off += sxy) {
        const int y = ylo + i;
        const float cy1 = ncy1, cy2 = ncy2, ay1 = nay1, ay2 = nay2;
        const bool y_in = y >= g.npd && y < g.npd + g.ny;
        const bool split = MODE == GEO_MODE_EXACT || !xz_inside || !y_in;   // this plane of the block
        const unsigned in = y_in ? in4 : 0u;
        const bool own_split = MODE == GEO_MODE_EXACT ? wr : wr && (um & ~in) != 0;
        // own P seven and v three planes ahead, then the next plane's
        FV pc = nP;
        const FV vo = nv;
        if (i + 1 < NI) {
            nP = ld_P(y + 8);
            nv = ld_v(y + 4);
            ycoef(y + 1, ncy1, ncy2, nay1, nay2);
        }
        FV S[6];
        if (split && own_split) {
            S[0] = ld_g(g.px + off); S[1] = ld_g(g.py + off); S[2] = ld_g(g.pz + off);
            S[3] = ld_g(g.qx + off); S[4] = ld_g(g.qy + off); S[5] = ld_g(g.qz + off);
        }
        // illumination / image inputs (RTM), loaded here so that their latency
        // hides behind the plane's arithmetic
        FV ill, mig, oth;
        const unsigned im = RTM ? in & um : 0u;
        const bool imv = im == kFull && st.img_vec;
        long io = 0;
        if (RTM && im) {
            io = (long)(zo - g.npd) + (long)g.nz * ((xa - g.npd) + (long)g.nx * (y - g.npd));
            if (imv) {
                if (st.ill) ill = ld_g(st.ill + io);
                if (st.mig) mig = ld_g(st.mig + io);
            } else {
#pragma unroll
                for (int j = 0; j < kW; j++)
                    if (im >> j & 1u) {
                        if (st.ill) ill.v[j] = st.ill[io + j];
                        if (st.mig) mig.v[j] = st.mig[io + j];
                    }
            }
            if (st.mig) oth = ld_g(st.other_P + off);
        }

        add_source(pc, y + 7);
        push(p, pc);
        {
            const FV vn = new_v(vo, y + 3, cy1, cy2);
            push(q, vn);
            if (wr && y + 3 < yhi) st_v(g.v1 + off + 3 * sxy, vn);
        }

        if (!mbar_wait(&bar[s], par)) *(volatile int *)&s_abort = 1;
        float *sp = stages + s * kStageFloats;
        if (st.src_on && y == st.iys) {
            // the shared copies that hold the source cell
            const bool pH = st.izs >= z0 && st.izs < z0 + kTZ && st.ixs >= x0 - 7 && st.ixs < x0 + kFX + 7;
            const bool pQ = st.ixs >= x0 && st.ixs < x0 + kFX && st.izs >= z0 - 8 && st.izs < z0 + 40;
            if (pH || pQ) {
                if (tid == 0) {
                    if (pH) sp[OFF_PH + (st.ixs - (x0 - 7)) * kTZ + (st.izs - z0)] += st.amp;
                    if (pQ) sp[OFF_Q + (st.ixs - x0) * 48 + (st.izs - (z0 - 8))] += st.amp;
                    // these cells are later overwritten by the async proxy
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                }
                __syncthreads();
            }
        }
        float *ut = utiles + (i & 1) * kUTile, *wt = wtiles + (i & 1) * kWTile;
        // own u: taps P(x-3 .. x+4) = P box columns c+4 .. c+11
        FV un;
        {
            const float *ph = sp + OFF_PH + (c + 4) * kTZ + zl;
            FV t[8];
#pragma unroll
            for (int k = 0; k < 8; k++) t[k] = ld_s(ph + k * kTZ);
            const FV uo = ld_s(sp + OFF_U + (c + 4) * kTZ + zl), d = deriv8<MODE>(t);
#pragma unroll
            for (int j = 0; j < kW; j++) un.v[j] = vel_update<MODE>(cx2, uo.v[j], kx, d.v[j]);
            un = pick(um, un, uo);
            st_v(ut + (c + 4) * kTZ + zl, un);
            if (wr) st_v(g.u1 + off, un);
        }
        // own w
        FV wn, qo;
        {
            const float *Q = sp + OFF_Q + c * 48 + zl + 8;
            qo = ld_s(Q);
            const FV wo = ld_s(sp + OFF_W + c * 48 + zl + 8);
            const FV kz = ld_s(zprof + zl), cz2 = ld_s(zprof + kTZ + zl), d = derivz<MODE, 1>(Q, qo);
#pragma unroll
            for (int j = 0; j < kW; j++) wn.v[j] = vel_update<MODE>(cz2.v[j], wo.v[j], kz.v[j], d.v[j]);
            wn = pick(um, wn, wo);
            st_v(wt + c * 40 + zl + 4, wn);
            if (wr) st_v(g.w1 + off, wn);
        }
        // halo u and w
        if (hu) {
            FV t[8], r;
#pragma unroll
            for (int k = 0; k < 8; k++) t[k] = ld_s(sp + OFF_PH + h_src + (k - 3) * kTZ);
            const FV uo = ld_s(sp + OFF_U + h_tile), d = deriv8<MODE>(t);
#pragma unroll
            for (int j = 0; j < kW; j++) r.v[j] = vel_update<MODE>(hc2.v[j], uo.v[j], hk.v[j], d.v[j]);
            st_v(ut + h_tile, pick(hm, r, uo));
        } else if (hw) {
            const float *Q = sp + OFF_Q + h_src;
            const FV wo = ld_s(sp + OFF_W + h_src), d = derivz<MODE, 1>(Q, ld_s(Q));
            FV r;
#pragma unroll
            for (int j = 0; j < kW; j++) r.v[j] = vel_update<MODE>(hc2.v[j], wo.v[j], hk.v[j], d.v[j]);
            st_v(wt + h_tile, pick(hm, r, wo));
        }
        __syncthreads();
        if (*(volatile int *)&s_abort) {
            // a stage never completed: report, let copies in flight land
            // (bounded), and leave
            if (tid == 0) {
                atomicExch(g.err, 1);
                for (int k = 1; k < kStages; k++)
                    if (i + k < NI && i + k < (i ? i + 2 : kStages)) mbar_wait(&bar[(i + k) % kStages], ((i + k) / kStages) & 1);
            }
            return;
        }
        // every thread is past plane i-1: its stage takes plane i+2
        if (lane == 0 && i >= 1 && i - 1 + kStages < NI) issue(i - 1 + kStages, s == 0 ? kStages - 1 : s - 1);

        // stresses
        FV xx, zz;
        {
            FV t[8];
#pragma unroll
            for (int k = 0; k < 8; k++) t[k] = k == 4 ? un : ld_s(ut + (c + k) * kTZ + zl);
            xx = deriv8<MODE>(t);
            zz = derivz<MODE, 0>(wt + c * 40 + zl + 4, wn);
        }
        const FV yy = deriv8<MODE>(q);
        const float *M = sp + OFF_M + c * kTZ + zl;
        const FV m0 = ld_s(M), m1 = ld_s(M + kOB), m2 = ld_s(M + 2 * kOB);
        FV P, Q;
        if (MODE == GEO_MODE_FAST) {
            // m = A, B, C; inside the box all sponge factors are 1
            FV p0 = p[0];
            if (src_j >= 0 && src_j < kW && y == st.iys) {   // the stress update starts from the cell's own P, Q
                const float ps = g.P0[own + src_j + sxy * y], qs = g.Q0[own + src_j + sxy * y];
#pragma unroll
                for (int j = 0; j < kW; j++)
                    if (j == src_j) {
                        p0.v[j] = ps;
                        qo.v[j] = qs;
                    }
            }
#pragma unroll
            for (int j = 0; j < kW; j++) {
                const float Ax = m0.v[j] * g.dtx, Ay = m0.v[j] * g.dty, Bz = m1.v[j] * g.dtz;
                const float Bx = m1.v[j] * g.dtx, By = m1.v[j] * g.dty, Cz = m2.v[j] * g.dtz;
                P.v[j] = __fmaf_rn(-Bz, zz.v[j], __fmaf_rn(-Ay, yy.v[j], __fmaf_rn(-Ax, xx.v[j], p0.v[j])));
                Q.v[j] = __fmaf_rn(-Cz, zz.v[j], __fmaf_rn(-By, yy.v[j], __fmaf_rn(-Bx, xx.v[j], qo.v[j])));
            }
        }
        if (split && own_split) {
            const FV az1 = ld_s(zprof + 2 * kTZ + zl), az2 = ld_s(zprof + 3 * kTZ + zl);
#pragma unroll
            for (int j = 0; j < kW; j++) {
                float px, py, pz, qx, qy, qz;
                if (MODE == GEO_MODE_FAST) {
                    const float Ax = m0.v[j] * g.dtx, Ay = m0.v[j] * g.dty, Bz = m1.v[j] * g.dtz;
                    const float Bx = m1.v[j] * g.dtx, By = m1.v[j] * g.dty, Cz = m2.v[j] * g.dtz;
                    px = __fmaf_rn(-(ax1 * Ax), xx.v[j], ax2 * S[0].v[j]);
                    py = __fmaf_rn(-(ay1 * Ay), yy.v[j], ay2 * S[1].v[j]);
                    pz = __fmaf_rn(-(az1.v[j] * Bz), zz.v[j], az2.v[j] * S[2].v[j]);
                    qx = __fmaf_rn(-(ax1 * Bx), xx.v[j], ax2 * S[3].v[j]);
                    qy = __fmaf_rn(-(ay1 * By), yy.v[j], ay2 * S[4].v[j]);
                    qz = __fmaf_rn(-(az1.v[j] * Cz), zz.v[j], az2.v[j] * S[5].v[j]);
                    // points of the vector inside the box keep the unsplit form
                    if ((in & um) >> j & 1u) continue;
                } else {
                    // m = vp, 1+2eps, sqrtf(1+2del); the reference's chain
                    const float vp = m0.v[j], e2 = m1.v[j], d2 = m2.v[j];
                    px = ax2 * S[0].v[j] - ax1 * vp * vp * e2 * g.dtx * xx.v[j];
                    py = ay2 * S[1].v[j] - ay1 * vp * vp * e2 * g.dty * yy.v[j];
                    pz = az2.v[j] * S[2].v[j] - az1.v[j] * vp * vp * d2 * g.dtz * zz.v[j];
                    qx = ax2 * S[3].v[j] - ax1 * vp * vp * d2 * g.dtx * xx.v[j];
                    qy = ay2 * S[4].v[j] - ay1 * vp * vp * d2 * g.dty * yy.v[j];
                    qz = az2.v[j] * S[5].v[j] - az1.v[j] * vp * vp * g.dtz * zz.v[j];
                }
                if (um >> j & 1u) {
                    S[0].v[j] = px; S[1].v[j] = py; S[2].v[j] = pz;
                    S[3].v[j] = qx; S[4].v[j] = qy; S[5].v[j] = qz;
                }
                P.v[j] = px + py + pz;
                Q.v[j] = qx + qy + qz;
            }
            st_v(g.px + off, S[0]); st_v(g.py + off, S[1]); st_v(g.pz + off, S[2]);
            st_v(g.qx + off, S[3]); st_v(g.qy + off, S[4]); st_v(g.qz + off, S[5]);
        }
        if (!wr) continue;
        if (um != kFull) {   // points off the updated grid keep their zeros
#pragma unroll
            for (int j = 0; j < kW; j++)
                if (!(um >> j & 1u)) P.v[j] = Q.v[j] = 0.0f;
        }
        st_v(g.P1 + off, P);
        st_v(g.Q1 + off, Q);
        if (rec_x >= 0) {
            const int rr = y - g.npd - st.ry0;
            if (rr >= 0 && rr % st.dry == 0 && rr / st.dry < st.nry) {
                float a = P.v[0], b = Q.v[0];
#pragma unroll
                for (int j = 1; j < kW; j++)
                    if (j == rec_j) {
                        a = P.v[j];
                        b = Q.v[j];
                    }
                st.rec[(long)st.it * st.nrx * st.nry + rec_x + (long)st.nrx * (rr / st.dry)] = st.rec_pq ? a + b : a;
            }
        }
        // RTM imaging epilogue on the physical box
        // (cal_illumination / cal_migration, 3D RTM program :508-537)
        if (RTM && im) {
#pragma unroll
            for (int j = 0; j < kW; j++) {
                if (st.ill) ill.v[j] = ill.v[j] + (P.v[j] * P.v[j] + Q.v[j] * Q.v[j]);
                if (st.mig) mig.v[j] = mig.v[j] + oth.v[j] * P.v[j];
            }
            if (imv) {
                if (st.ill) st_v(st.ill + io, ill);
                if (st.mig) st_v(st.mig + io, mig);
            } else {
#pragma unroll
                for (int j = 0; j < kW; j++)
                    if (im >> j & 1u) {
                        if (st.ill) st.ill[io + j] = ill.v[j];
                        if (st.mig) st.mig[io + j] = mig.v[j];
                    }
            }
        }
    }
}

}  // namespace

// ------------------------------------------------------------------ host
static PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;

int encode_map(CUtensorMap *map, const float *base, int nnz, int ldz, int nnx, int nny, int boxz, int boxx) {
    if (!g_encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        GEO_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q));
        if (!fn || q != cudaDriverEntryPointSuccess) return fail(GEO_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
        g_encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
    }
    if ((ldz * 4) % 16 != 0 || (reinterpret_cast<uintptr_t>(base) & 15) != 0)
        return fail(GEO_ERR_ARG, "tensor map needs 16-byte aligned base and z stride");
    cuuint64_t dims[3] = {(cuuint64_t)nnz, (cuuint64_t)nnx, (cuuint64_t)nny};
    cuuint64_t strides[2] = {(cuuint64_t)ldz * 4, (cuuint64_t)ldz * nnx * 4};
    cuuint32_t box[3] = {(cuuint32_t)boxz, (cuuint32_t)boxx, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    // 128-byte promotion: at 400^3 + 40 the step reads 5.24 GB per launch
    // against 5.52 GB with 256-byte promotion, in the same time (1.543 ms)
    CUresult r = g_encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(base), dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(GEO_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return GEO_OK;
}

int launch_fused3d(const StepMaps &maps, const Fused3D &g, int mode, const StepArgs3D &args, cudaStream_t s) {
    static OncePerDevice once[2][2];
    StepArgs3D st = args;
    const bool rtm = st.ill || st.mig, fast = mode == GEO_MODE_FAST;
    // 16-byte image accesses need aligned rows whose first depth sits on a vector
    st.img_vec = g.npd % kW == 0 && g.nz % kW == 0 &&
                 ((reinterpret_cast<uintptr_t>(st.ill) | reinterpret_cast<uintptr_t>(st.mig)) & (4 * kW - 1)) == 0;
    const void *fn = fast ? (rtm ? (const void *)k_fused3d<GEO_MODE_FAST, true> : (const void *)k_fused3d<GEO_MODE_FAST, false>)
                          : (rtm ? (const void *)k_fused3d<GEO_MODE_EXACT, true> : (const void *)k_fused3d<GEO_MODE_EXACT, false>);
    GEO_TRY(allow_smem(once[fast][rtm], fn, kFusedSmem));
    using Fn = void (*)(const StepMaps, const Fused3D, const StepArgs3D);
    GEO_CUDA(launch_early(reinterpret_cast<Fn>(const_cast<void *>(fn)), (unsigned)g.nitems, dim3(kFusedThreads), kFusedSmem, s, maps, g, st));
    return check_launch("fused3d");
}

}  // namespace geo

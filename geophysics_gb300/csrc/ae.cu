// Learned snapshot codec: kernels, training and the geo_ae_* C ABI.
//
// Inference (snapshot encode in the forward pass of RTM, decode + imaging in
// the backward pass):
//   k_ae_e12     gather the cells of 16^3 blocks of the wavefield, scale by the
//                block's max |value|, level E1 (8 -> 16) on CUDA cores, E2 on
//                tcgen05;
//   tc_gemm x2   E3, E4 on tcgen05 (the last one writes the bf16 code);
//   tc_gemm x2   D4, D3 on tcgen05;
//   k_ae_d21     D2 on tcgen05, D1 (16 -> 8) on CUDA cores, unscale, store the
//                snapshot (a round trip); or, in an RTM run,
//   tc_gemm, k_ae_d1_vol  D2, then D1 with the product with the receiver
//                wavefield added to the image (or, for the escape check, the
//                comparison with the field).
// The snapshot kernels take E1's and D1's weights by value (a host copy kept
// per weight version), so every weight is an operand of its multiply-add.
// Training (one CUDA graph per iteration): the same forward on blocks drawn
// from a store of solver snapshots (k_ae_e1, weights read from the device
// copy that Adam updates inside the graph), the loss and the D1 backward in
// k_ae_d1, per level the input gradient (tc_gemm against the transposed
// weights, the activation derivative fused as a gate), then every level's
// weight gradient (tc_wgrad) and bias gradient (k_ae_colsum) in one launch
// each, E1's weight gradient (k_ae_e1_bwd), Adam and the bf16 repack.
#include "ae.cuh"
#include "tc_gemm.cuh"
#include "tc_util.cuh"
#include "fd3d.cuh"
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

using namespace geo;

namespace geo {

__host__ __device__ inline int morton_of(int z, int x, int y) {
    int m = 0;
#pragma unroll
    for (int l = 0; l < 4; l++)
        m |= (((z >> l) & 1) << (3 * l)) | (((x >> l) & 1) << (3 * l + 1)) | (((y >> l) & 1) << (3 * l + 2));
    return m;
}

__host__ __device__ inline unsigned long long splitmix(unsigned long long x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

__device__ __forceinline__ float bf16r(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
// leaky ReLU as max(v, kLeak v): the same value as v > 0 ? v : kLeak v for
// 0 < kLeak < 1 (signed zeros, infinities and NaN included), one
// instruction fewer
__device__ __forceinline__ float leaky_d(float v) { return fmaxf(v, kLeak * v); }

// ---------------------------------------------------------------- layout
struct AeOffsets {
    long w[kAeLayers], b[kAeLayers], total;   // fp32 parameters: W [N x K] then b [N]
    long wb[kAeLayers], nbf;                  // bf16 copies of the GEMM layers (1..6)
};

static AeOffsets ae_offsets() {
    AeOffsets o{};
    long p = 0, q = 0;
    for (int l = 0; l < kAeLayers; l++) {
        o.w[l] = p;
        p += (long)kAeNet[l].N * kAeNet[l].K;
        o.b[l] = p;
        p += kAeNet[l].N;
        if (l >= 1 && l <= 6) {
            o.wb[l] = q;
            q += (long)kAeNet[l].N * kAeNet[l].K;
        } else {
            o.wb[l] = -1;
        }
    }
    o.total = p;
    o.nbf = q;
    return o;
}

// Weights of the two CUDA-core levels, passed by value to the snapshot
// kernels (the host keeps a copy of the current ones).
// Input by input, so that the weights of two neighbouring outputs are one
// 8-byte operand of a packed multiply-add.
struct __align__(8) AeSmallW {
    float w1[128], b1[16];   // E1: W^T [8 x 16] (bf16 values), b [16]
    float v1[128], c1[8];    // D1: W^T [16 x 8] (bf16 values), b [8]
};

// Two floats side by side and Blackwell's packed arithmetic on them: each
// half rounds as its scalar instruction does.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 pair(const float *w) { return *reinterpret_cast<const f32x2 *>(w); }
// the two values of a bf16x2 word, each twice
__device__ __forceinline__ f32x2 twice_lo(uint32_t q) {
    const float f = __uint_as_float(q << 16);
    return pack2(f, f);
}
__device__ __forceinline__ f32x2 twice_hi(uint32_t q) {
    const float f = __uint_as_float(q & 0xffff0000u);
    return pack2(f, f);
}

// Where the value of Morton index m sits in a block's shared copy: bits 4 and
// 2 take up bits 6 and 9 (the depth bits whose strides are multiples of the 32
// banks: a warp's 16 depths of two rows land on 32 banks), and bit 2 takes up
// bit 5 (eight neighbouring nodes' halves are 16-byte accesses to all banks).
__device__ __forceinline__ int swz(int m) { return m ^ ((m >> 2) & 16) ^ ((m >> 3) & 4) ^ ((m >> 7) & 4); }
// Thread (z, x)'s sixteen values, one per plane y: base[f] + off, f the parity of y's low bits.
struct BlockCol {
    int base[2];
    __device__ __forceinline__ BlockCol(int z, int x) {
        base[0] = swz(morton_of(z, x, 0));
        base[1] = base[0] ^ 4;
    }
    __device__ __forceinline__ int at(int y) const {
        return base[(y ^ (y >> 1)) & 1] + (morton_of(0, 0, y) & ~4);
    }
};

// E1 of two nodes of a snapshot: x[r] the eight values of node r as bf16
// pairs, out[r] 16 bf16.  Two nodes share every weight's load.
__device__ __forceinline__ void e1_pairs(const AeSmallW &w, const uint32_t (&x)[2][4], uint4 (&out)[2][2]) {
    f32x2 acc[2][8];
#pragma unroll
    for (int c = 0; c < 8; c++) acc[0][c] = acc[1][c] = 0;
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const f32x2 k = pair(w.w1 + j * 16 + 2 * c);
#pragma unroll
            for (int r = 0; r < 2; r++) acc[r][c] = fma2(k, j & 1 ? twice_hi(x[r][j / 2]) : twice_lo(x[r][j / 2]), acc[r][c]);
        }
    const f32x2 leak = pack2(kLeak, kLeak);
#pragma unroll
    for (int c = 0; c < 8; c++)
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const f32x2 v = add2(acc[r][c], pair(w.b1 + 2 * c));
            const float2 a = unpack2(v), b = unpack2(mul2(leak, v));
            reinterpret_cast<__nv_bfloat162 *>(out[r])[c] = __floats2bfloat162_rn(fmaxf(a.x, b.x), fmaxf(a.y, b.y));
        }
}

// D1 of two nodes of a snapshot times the block's scale s: in[r] their 16 bf16,
// y[r] eight floats.
__device__ __forceinline__ void d1_pairs(const AeSmallW &w, const uint4 (&in)[2][2], float s, float4 (&y)[2][2]) {
    f32x2 acc[2][4];
#pragma unroll
    for (int c = 0; c < 4; c++) acc[0][c] = acc[1][c] = 0;
#pragma unroll
    for (int j = 0; j < 16; j++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const f32x2 k = pair(w.v1 + j * 8 + 2 * c);
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const uint32_t q = reinterpret_cast<const uint32_t *>(in[r])[j / 2];
                acc[r][c] = fma2(k, j & 1 ? twice_hi(q) : twice_lo(q), acc[r][c]);
            }
        }
    const f32x2 sc = pack2(s, s);
#pragma unroll
    for (int r = 0; r < 2; r++) {
        float2 o[4];
#pragma unroll
        for (int c = 0; c < 4; c++) o[c] = unpack2(mul2(add2(acc[r][c], pair(w.c1 + 2 * c)), sc));
        y[r][0] = make_float4(o[0].x, o[0].y, o[1].x, o[1].y);
        y[r][1] = make_float4(o[2].x, o[2].y, o[3].x, o[3].y);
    }
}

// E1 of one level-1 node: h = leaky(W1 x + b1) as 16 bf16 (32 bytes).
__device__ __forceinline__ void e1_node(const float *w1, const float *b1, const float *x8, __nv_bfloat16 *out) {
    uint4 q[2];
    __nv_bfloat16 *qb = reinterpret_cast<__nv_bfloat16 *>(q);
    float h[16];
#pragma unroll
    for (int c = 0; c < 16; c++) {
        float acc = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; j++) acc = __fmaf_rn(w1[c * 8 + j], x8[j], acc);
        h[c] = leaky_d(acc + b1[c]);
    }
    // two channels per conversion (low half = even channel)
    __nv_bfloat162 *q2 = reinterpret_cast<__nv_bfloat162 *>(qb);
#pragma unroll
    for (int c = 0; c < 8; c++) q2[c] = __floats2bfloat162_rn(h[2 * c], h[2 * c + 1]);
    uint4 *dst = reinterpret_cast<uint4 *>(out);
    dst[0] = q[0];
    dst[1] = q[1];
}

// D1 of one level-1 node: y = V1 g + c1 from its 16 bf16 inputs.
__device__ __forceinline__ void d1_node(const float *v1, const float *c1, const __nv_bfloat16 *in, float *g,
                                        float *y) {
    const uint4 *src = reinterpret_cast<const uint4 *>(in);
    uint4 q[2] = {src[0], src[1]};
    const __nv_bfloat16 *qb = reinterpret_cast<const __nv_bfloat16 *>(q);
#pragma unroll
    for (int j = 0; j < 16; j++) g[j] = __bfloat162float(qb[j]);
#pragma unroll
    for (int c = 0; c < 8; c++) {
        float acc = 0.0f;
#pragma unroll
        for (int j = 0; j < 16; j++) acc = __fmaf_rn(v1[c * 16 + j], g[j], acc);
        y[c] = acc + c1[c];
    }
}

// ---------------------------------------------------------------- kernels
struct E1Args {
    const float *direct;          // given blocks (Morton, nb x 4096), or null
    const float *store;           // training store (Morton), sampled by hash
    long nstore;
    unsigned long long seed;
    const int *step;
    int nb;                       // real blocks (grid covers the padded count)
    const float *w1, *b1;         // E1: W [16 x 8] (bf16 values), b [16]
    __nv_bfloat16 *h1;            // [nbp*512 x 16]
    float *scale;                 // [nbp]
    float *xn;                    // [nbp x 4096] normalized input (training), or null
    const float *wstore;          // training: per-block weights of the store
    float *wrow;                  // training: weight of each row's block
    float *wsum;                  // training: batch weight sums, slot *step - step0
    int step0;
};

// Blocks whose max |value| is below this are coded as zero (their inverse
// scale would overflow).
constexpr float kAeTiny = 1e-30f;

__device__ __forceinline__ float block_max(float v, float *red) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float m = red[0];
#pragma unroll
    for (int w = 1; w < 8; w++) m = fmaxf(m, red[w]);
    return m;
}

// E1 on blocks given in Morton order (evaluation) or drawn from the training
// store: scale by the block max, W1 x + b1, leaky ReLU, bf16 out.
__global__ void __launch_bounds__(256) k_ae_e1(const E1Args a) {
    __shared__ float xs[kAePts];
    __shared__ float red[8];
    tc::after_predecessor();
    const int b = blockIdx.x, t = threadIdx.x;
    float mx = 0.0f;
    if (b < a.nb) {
        const float *src;
        if (a.direct) {
            src = a.direct + (long)b * kAePts;
        } else {
            const unsigned long long h = splitmix(a.seed ^ splitmix(((unsigned long long)*a.step << 24) + b));
            const long pick = (long)(h % (unsigned long long)a.nstore);
            src = a.store + pick * kAePts;
            if (t == 0 && a.wrow) {
                const float w = a.wstore ? a.wstore[pick] : 1.0f;
                a.wrow[b] = w;
                atomicAdd(a.wsum + (*a.step - a.step0), w);
            }
        }
#pragma unroll 4
        for (int p = 0; p < 16; p++) {
            const float val = src[p * 256 + t];
            xs[p * 256 + t] = val;
            mx = fmaxf(mx, fabsf(val));
        }
    } else {
        for (int p = 0; p < 16; p++) xs[p * 256 + t] = 0.0f;
    }
    const float s = block_max(mx, red);   // includes the barrier after the fills
    const float inv = s >= kAeTiny ? 1.0f / s : 0.0f;
    if (t == 0) a.scale[b] = s >= kAeTiny ? s : 0.0f;
#pragma unroll 1
    for (int r = 0; r < 2; r++) {
        const int p = t + 256 * r;
        float x8[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const float xv = xs[p * 8 + j] * inv;
            if (a.xn) a.xn[(long)b * kAePts + p * 8 + j] = xv;
            x8[j] = bf16r(xv);
        }
        e1_node(a.w1, a.b1, x8, a.h1 + ((long)b * 512 + p) * 16);
    }
}

// A thread's place in a snapshot: row r of a tile of two blocks (128 rows) is
// one 4x4x4 cell of block 2 tile + r / 64.  Consecutive rows are Morton
// neighbours, so a warp's 16-byte accesses at one (x, y) of its cells are whole
// 64-byte runs of the field's lines.
struct CellAt {
    int b, iz, ix, iy;            // block, first point of the cell
    __device__ __forceinline__ CellAt(const AeVolume &v, int tile, int r) {
        b = 2 * tile + (r >> 6);
        const int bz = b % v.nbz, bx = (b / v.nbz) % v.nbx, by = b / (v.nbz * v.nbx);
        iz = bz * 16 + 4 * ((r & 1) | ((r >> 2) & 2));
        ix = bx * 16 + 4 * (((r >> 1) & 1) | ((r >> 3) & 2));
        iy = by * 16 + 4 * (((r >> 2) & 1) | ((r >> 4) & 2));
    }
};
// Whether four consecutive depths of every line are one aligned vector.
__device__ __forceinline__ bool lines_aligned(const AeVolume &v, const float *p) {
    return !((reinterpret_cast<uintptr_t>(p + v.oz) & 15) || (v.ldz & 3) || (v.sxy & 3));
}

// E1 and E2 of a snapshot in one launch: a group of 128 threads takes a tile
// of two blocks, a thread one cell -- 64 points, eight E1 nodes, one row of
// E2's operand.  It loads its points, scales them by the block's max, forms E1
// (packed FP32 multiply-adds, weights by value) and writes the row's 256 bytes
// as the swizzled shared-memory operand tcgen05 reads; one thread multiplies
// by E2's weights (resident), and the same threads finish E2 from TMEM and
// send 32 x 64 boxes out by TMA.  E1's output, 16 KB a block, never leaves the
// SM.  Persistent, two CTAs of two groups per SM.  Waits are bounded.
// A 512x512x384 snapshot takes 164 us; E1 and E2 one after the other took 250
// (159 + 91), E1's output costing 800 MB of traffic.  Bound by instruction
// issue and the latency of the constant loads at 16 warps per SM (2000
// instructions a cell, half of them E1's products); the next tile's points are
// loaded during this one's arithmetic (172 us without).  Weights from shared
// memory instead, 16 bytes a load: 225 us.
struct E12Args {
    AeVolume vol;
    int nb, tiles;                // blocks of the volume; tiles of two, padding included
    float *scale;                 // [nbp]
    const float *bias;            // E2's
    int *err;
    AeSmallW w;
};
constexpr int kE12Group = 32768;                             // bytes of a group's operand
constexpr size_t kE12Smem = 16384 + 2 * kE12Group + 1024;

__global__ void __launch_bounds__(256, 2) k_ae_e12(const __grid_constant__ CUtensorMap tw, const __grid_constant__ CUtensorMap to,
                                                   const __grid_constant__ E12Args a) {
    extern __shared__ unsigned char smem_raw[];
    uint8_t *sm = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int grp = threadIdx.x >> 7, r = threadIdx.x & 127, warp = r >> 5, lane = r & 31;
    uint8_t *A = sm + 16384 + grp * kE12Group;
    __shared__ __align__(8) float sbias[64];
    __shared__ float red[2][4];
    __shared__ __align__(8) uint64_t wbar, done[2];
    __shared__ uint32_t tslot;
    __shared__ int s_abort[2];   // of each group: set by its warps, read by all of them after a barrier
    if (threadIdx.x == 0) {
        tc::mbar_init(&wbar, 1);
        tc::mbar_init(&done[0], 1);
        tc::mbar_init(&done[1], 1);
        s_abort[0] = s_abort[1] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (threadIdx.x < 32) tc::tmem_alloc(&tslot, 128);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tslot + grp * 64;
    // the weights too: the kernel before may be the one that packs them
    tc::after_predecessor();
    if (threadIdx.x == 0) {
        // E2's weights, two slices of 64 inputs
        tc::mbar_expect_tx(&wbar, 16384);
        tc::tma2(sm, &tw, 0, 0, &wbar);
        tc::tma2(sm + 8192, &tw, 64, 0, &wbar);
    }
    if (threadIdx.x < 64) sbias[threadIdx.x] = a.bias[threadIdx.x];
    if (!tc::mbar_wait(&wbar, 0)) s_abort[0] = s_abort[1] = 1;
    __syncthreads();
    const AeVolume &v = a.vol;
    const bool vec = lines_aligned(v, v.src);
    // line x + 4 y of the thread's cell of tile t: plain loads, the step that
    // wrote the field may still run when this kernel starts
    float4 f[16];
    auto load = [&](int t) {
        const CellAt c(v, t, r);
        const float *p = v.src + (long)(v.oz + c.iz) + v.ldz * (v.ox + c.ix) + v.sxy * (v.oy + c.iy);
        const bool in = c.b < a.nb;
        if (vec && in && c.iz + 4 <= v.nz && c.ix + 4 <= v.nx && c.iy + 4 <= v.ny) {
#pragma unroll
            for (int q = 0; q < 16; q++) f[q] = *reinterpret_cast<const float4 *>(p + v.ldz * (q & 3) + v.sxy * (q >> 2));
        } else {
#pragma unroll
            for (int q = 0; q < 16; q++) {
                const bool l = in && c.ix + (q & 3) < v.nx && c.iy + (q >> 2) < v.ny;
                const float *s = p + v.ldz * (q & 3) + v.sxy * (q >> 2);
                f[q].x = l && c.iz < v.nz ? *s : 0.0f;
                f[q].y = l && c.iz + 1 < v.nz ? s[1] : 0.0f;
                f[q].z = l && c.iz + 2 < v.nz ? s[2] : 0.0f;
                f[q].w = l && c.iz + 3 < v.nz ? s[3] : 0.0f;
            }
        }
    };
    unsigned k = 0;
    if ((int)blockIdx.x * 2 + grp < a.tiles) load(blockIdx.x * 2 + grp);
    for (int t = blockIdx.x * 2 + grp; t < a.tiles; t += gridDim.x * 2, k++) {
        float mx = 0.0f;
#pragma unroll
        for (int q = 0; q < 16; q++) mx = fmaxf(mx, fmaxf(fmaxf(fabsf(f[q].x), fabsf(f[q].y)), fmaxf(fabsf(f[q].z), fabsf(f[q].w))));
#pragma unroll
        for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        // the last tile's boxes have left this warp's part of the operand
        if (lane == 0) {
            red[grp][warp] = mx;
            asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        }
        asm volatile("bar.sync %0, 128;" ::"r"(grp + 1) : "memory");
        if (*(volatile int *)&s_abort[grp]) break;
        const float s = fmaxf(red[grp][warp & 2], red[grp][warp | 1]);
        const float inv = s >= kAeTiny ? 1.0f / s : 0.0f;
        if ((r & 63) == 0) a.scale[2 * t + (r >> 6)] = s >= kAeTiny ? s : 0.0f;
        // the scaled points wait as bf16 in the row's second half: the two
        // nodes along z at (x1, y1) = (m & 1, m >> 1) in its chunks 2m, 2m + 1
        uint8_t *row = A + r * 128;
        const int sw = (r & 7) << 4;
#pragma unroll
        for (int m = 0; m < 4; m++) {
            uint32_t x[2][4];
#pragma unroll
            for (int q = 0; q < 4; q++) {   // line (x0, y0) = (q & 1, q >> 1) of the nodes
                const float4 l = f[2 * (m & 1) + (q & 1) + 4 * (2 * (m >> 1) + (q >> 1))];
                const __nv_bfloat162 lo = __floats2bfloat162_rn(l.x * inv, l.y * inv), hi = __floats2bfloat162_rn(l.z * inv, l.w * inv);
                x[0][q] = *reinterpret_cast<const uint32_t *>(&lo);
                x[1][q] = *reinterpret_cast<const uint32_t *>(&hi);
            }
#pragma unroll
            for (int n = 0; n < 2; n++)
                *reinterpret_cast<uint4 *>(row + 16384 + (((2 * m + n) << 4) ^ sw)) = make_uint4(x[n][0], x[n][1], x[n][2], x[n][3]);
        }
        // the next tile's points, on their way during this one's arithmetic
        if (t + (int)gridDim.x * 2 < a.tiles) load(t + gridDim.x * 2);
        // E1 of two nodes at a time; nodes 4-7 overwrite the points of pairs
        // already done
#pragma unroll 1
        for (int m = 0; m < 4; m++) {
            uint32_t x[2][4];
#pragma unroll
            for (int n = 0; n < 2; n++) {
                const uint4 q = *reinterpret_cast<const uint4 *>(row + 16384 + (((2 * m + n) << 4) ^ sw));
                x[n][0] = q.x; x[n][1] = q.y; x[n][2] = q.z; x[n][3] = q.w;
            }
            uint4 h[2][2];
            e1_pairs(a.w, x, h);
            uint8_t *half = row + (m >> 1) * 16384;
#pragma unroll
            for (int n = 0; n < 2; n++)
#pragma unroll
                for (int e = 0; e < 2; e++)
                    *reinterpret_cast<uint4 *>(half + ((((m & 1) * 4 + n * 2 + e) << 4) ^ sw)) = h[n][e];
        }
        tc::fence_async_smem();
        tc::tc_fence_before();
        asm volatile("bar.sync %0, 128;" ::"r"(grp + 1) : "memory");
        if (r == 0) {
            tc::tc_fence_after();
            constexpr uint32_t idesc = tc::idesc_bf16_f32(128, 64);
            const uint32_t a0 = tc::su32(A), b0 = tc::su32(sm);
#pragma unroll
            for (int q = 0; q < 8; q++)
                tc::mma_bf16(tmem, tc::sdesc_k128(a0 + (q >> 2) * 16384 + (q & 3) * 32),
                             tc::sdesc_k128(b0 + (q >> 2) * 8192 + (q & 3) * 32), idesc, q != 0);
            tc::mma_commit(&done[grp]);
        }
        __syncwarp();
        if (!__all_sync(0xffffffffu, tc::mbar_wait(&done[grp], k & 1))) {
            s_abort[grp] = 1;
            continue;   // the group leaves together, after its next barrier
        }
        tc::tc_fence_after();
        const uint32_t ta = tmem + ((uint32_t)(warp * 32) << 16);
        uint8_t *o = A + warp * 4096;   // this warp's rows of the first slice, read by the MMAs and free
#pragma unroll 1
        for (int e = 0; e < 2; e++) {
            uint32_t d[32];
            tc::tmem_ld32(ta + 32 * e, d);
            tc::tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 4; q++) {
                uint4 w4;
                __nv_bfloat162 *w2 = reinterpret_cast<__nv_bfloat162 *>(&w4);
#pragma unroll
                for (int n = 0; n < 4; n++) {
                    const float2 bb = *reinterpret_cast<const float2 *>(sbias + 32 * e + 8 * q + 2 * n);
                    w2[n] = __floats2bfloat162_rn(leaky_d(__uint_as_float(d[8 * q + 2 * n]) + bb.x),
                                                  leaky_d(__uint_as_float(d[8 * q + 2 * n + 1]) + bb.y));
                }
                *reinterpret_cast<uint4 *>(o + lane * 128 + (((4 * e + q) ^ (lane & 7)) << 4)) = w4;
            }
        }
        tc::fence_async_smem();
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) {
            asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                             reinterpret_cast<uint64_t>(&to)),
                         "r"(tc::su32(o)), "r"(0), "r"(t * 128 + warp * 32)
                         : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    __syncwarp();
    tc::tc_fence_before();
    __syncthreads();
    if ((s_abort[0] || s_abort[1]) && threadIdx.x == 0) atomicExch(a.err, 2);
    if (threadIdx.x < 32) tc::tmem_dealloc(tslot, 128);
}

// D2 and D1 of a snapshot in one launch, unscaled and stored to the interior
// box (dst, the box's strides) with the escaped blocks' residuals added: the
// walk of tc_gemm.cu (persistent, TMA producer, MMA issuer, two epilogue groups
// on two accumulators) over D2 with its weights resident, where an epilogue
// thread finishes a cell: D2's bias and activation, bf16, D1 of its eight
// nodes (packed FP32 multiply-adds) and 16 four-depth stores.  D2's output, 16
// KB a block, never leaves the SM.  Two CTAs per SM.  Waits are bounded.
// A 512x512x384 snapshot takes 116 us, 5.1 TB/s; D2 and D1 one after the other
// took 221 (101 + 120).  The round trip's decode; imaging and the escape check
// take D2 as a GEMM and k_ae_d1_vol.
struct D21Args {
    AeVolume vol;
    int nb, tiles;
    const float *scale;           // [nbp]
    const float *bias;            // D2's
    float *dst;
    const int *esc;               // escaped-block slot per row (-1: none), or null
    const __nv_bfloat16 *res;     // residual pool (4096 per slot, natural order)
    int *err;
    AeSmallW w;
};
constexpr int kD21Stages = 4, kD21Threads = 320;
constexpr size_t kD21Smem = 16384 + kD21Stages * 16384 + 1024;

__global__ void __launch_bounds__(kD21Threads, 2)
    k_ae_d21(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tw, const __grid_constant__ D21Args a) {
    extern __shared__ unsigned char smem_raw[];
    uint8_t *sm = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *ring = sm + 16384;
    __shared__ __align__(16) float sbias[128];
    __shared__ __align__(8) uint64_t wbar, full[kD21Stages], empty[kD21Stages], acc_full[2], acc_empty[2];
    __shared__ uint32_t tslot;
    __shared__ int s_abort;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        tc::mbar_init(&wbar, 1);
        for (int s = 0; s < kD21Stages; s++) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < 2; s++) {
            tc::mbar_init(&acc_full[s], 1);
            tc::mbar_init(&acc_empty[s], 4);
        }
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == 9) tc::tmem_alloc(&tslot, 256);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = tslot;
    tc::after_predecessor();
    if (threadIdx.x < 128) sbias[threadIdx.x] = a.bias[threadIdx.x];
    __syncthreads();

    if (warp == 8 && lane == 0) {
        unsigned it = 0;
        bool ok = true;
        tc::mbar_expect_tx(&wbar, 16384);
        tc::tma2(sm, &tw, 0, 0, &wbar);
        for (int t = blockIdx.x; t < a.tiles; t += gridDim.x, it++) {
            const unsigned s = it % kD21Stages;
            if (it >= kD21Stages && !tc::mbar_wait(&empty[s], (it / kD21Stages - 1) & 1)) {
                s_abort = 1;
                ok = false;
                break;
            }
            tc::mbar_expect_tx(&full[s], 16384);
            tc::tma2(ring + s * 16384, &ta, 0, t * 128, &full[s]);
        }
        if (!ok) {   // let the copies still in flight land (bounded)
            for (unsigned k = it > kD21Stages ? it - kD21Stages : 0; k < it; k++)
                tc::mbar_wait(&full[k % kD21Stages], (k / kD21Stages) & 1);
            tc::mbar_wait(&wbar, 0);
        }
    } else if (warp == 9 && lane == 0) {
        constexpr uint32_t idesc = tc::idesc_bf16_f32(128, 128);
        bool ok = tc::mbar_wait(&wbar, 0);
        unsigned i = 0;
        for (int t = blockIdx.x; t < a.tiles && ok; t += gridDim.x, i++) {
            const unsigned ab = i & 1, s = i % kD21Stages;
            if ((i >= 2 && !tc::mbar_wait(&acc_empty[ab], ((i >> 1) - 1) & 1)) ||
                !tc::mbar_wait(&full[s], (i / kD21Stages) & 1)) {
                ok = false;
                break;
            }
            tc::tc_fence_after();
            const uint32_t a0 = tc::su32(ring + s * 16384), b0 = tc::su32(sm);
#pragma unroll
            for (int k = 0; k < 4; k++)
                tc::mma_bf16(tmem + ab * 128, tc::sdesc_k128(a0 + k * 32), tc::sdesc_k128(b0 + k * 32), idesc, k != 0);
            tc::mma_commit(&empty[s]);
            tc::mma_commit(&acc_full[ab]);
        }
        if (!ok) s_abort = 1;
    } else if (warp < 8) {
        const int grp = warp >> 2, quad = warp & 3;
        const AeVolume &v = a.vol;
        const bool vec = lines_aligned(v, a.dst);
        unsigned i = 0;
        for (int t = blockIdx.x; t < a.tiles; t += gridDim.x, i++) {
            if ((int)(i & 1) != grp) continue;
            const CellAt c(v, t, quad * 32 + lane);
            const bool in = c.b < a.nb;
            const float s = in ? a.scale[c.b] : 0.0f;
            const int slot = in && a.esc ? a.esc[c.b] : -1;
            if (!__all_sync(0xffffffffu, tc::mbar_wait(&acc_full[grp], (i >> 1) & 1))) {
                s_abort = 1;
                break;
            }
            tc::tc_fence_after();
            const uint32_t ta0 = tmem + ((uint32_t)(quad * 32) << 16) + grp * 128;
            float *p = a.dst + (long)(v.oz + c.iz) + v.ldz * (v.ox + c.ix) + v.sxy * (v.oy + c.iy);
            const bool whole = vec && in && c.iz + 4 <= v.nz && c.ix + 4 <= v.nx && c.iy + 4 <= v.ny;
#pragma unroll 1
            for (int m = 0; m < 4; m++) {   // the two nodes along z at (x1, y1) = (m & 1, m >> 1)
                uint32_t d[32];
                tc::tmem_ld32(ta0 + m * 32, d);
                tc::tmem_ld_wait();
                if (m == 3) {
                    tc::tc_fence_before();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&acc_empty[grp]);
                }
                uint4 g[2][2];
#pragma unroll
                for (int q = 0; q < 16; q++) {
                    const float2 bb = *reinterpret_cast<const float2 *>(sbias + m * 32 + 2 * q);
                    reinterpret_cast<__nv_bfloat162 *>(g)[q] = __floats2bfloat162_rn(
                        leaky_d(__uint_as_float(d[2 * q]) + bb.x), leaky_d(__uint_as_float(d[2 * q + 1]) + bb.y));
                }
                float4 y[2][2];
                d1_pairs(a.w, g, s, y);
                if (!in) continue;
                const float *y0 = reinterpret_cast<const float *>(y[0]), *y1 = reinterpret_cast<const float *>(y[1]);
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int dx = 2 * (m & 1) + (q & 1), dy = 2 * (m >> 1) + (q >> 1);
                    float4 o = make_float4(y0[2 * q], y0[2 * q + 1], y1[2 * q], y1[2 * q + 1]);
                    if (slot >= 0) {   // escaped block: decoded + residual
                        const uint2 e = *reinterpret_cast<const uint2 *>(
                            a.res + (long)slot * kAePts + ((c.iy + dy) & 15) * 256 + ((c.ix + dx) & 15) * 16 + (c.iz & 15));
                        o.x += __uint_as_float(e.x << 16);
                        o.y += __uint_as_float(e.x & 0xffff0000u);
                        o.z += __uint_as_float(e.y << 16);
                        o.w += __uint_as_float(e.y & 0xffff0000u);
                    }
                    float *l = p + v.ldz * dx + v.sxy * dy;
                    if (whole) {
                        *reinterpret_cast<float4 *>(l) = o;
                    } else if (c.ix + dx < v.nx && c.iy + dy < v.ny) {
                        if (c.iz < v.nz) l[0] = o.x;
                        if (c.iz + 1 < v.nz) l[1] = o.y;
                        if (c.iz + 2 < v.nz) l[2] = o.z;
                        if (c.iz + 3 < v.nz) l[3] = o.w;
                    }
                }
            }
        }
    }
    __syncwarp();
    tc::tc_fence_before();
    __syncthreads();
    if (s_abort && threadIdx.x == 0) atomicExch(a.err, 2);
    if (warp == 9) tc::tmem_dealloc(tmem, 256);
}

// out[(c * SC + j * SJ)] += sum over the block's 512 nodes of a[c] b[j], and
// bias += the column sums of a (BIAS_A) or of b: the weight and bias
// gradients of D1 (a = dy, b = g) and E1 (a = x, b = dh).  The nodes' 8 and
// 16 values sit in shared memory, a node per row of an array padded so that
// the 32-byte and 64-byte rows of consecutive nodes start in different banks.
// Thread t owns a 2 x 4 tile of the 8 x 16 products (t & 15) over the nodes
// congruent to t >> 4: two loads and eight multiply-adds per node, then a
// shuffle, a pass through shared memory and one global atomic per product.
// Bound by shared-memory latency; 136 shared atomics of every thread on the
// same 136 words, which this replaces, took 675 us (D1) and 738 us (E1) for
// 256 blocks; the kernels now take 11.7 us and 5.6 us.
constexpr int kOutA = 12, kOutB = 20;   // row strides (floats)
constexpr int kOutFloats = 512 * (kOutA + kOutB);

template <bool BIAS_A, int SC, int SJ>
__device__ __forceinline__ void block_outer(float *sm, float *gw, float *gb) {
    const float *A = sm, *B = sm + 512 * kOutA;
    const int t = threadIdx.x, c0 = (t & 3) * 2, j0 = ((t >> 2) & 3) * 4, grp = t >> 4;
    float acc[2][4], sa[2] = {0.0f, 0.0f}, sb[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.0f;
#pragma unroll 4
    for (int k = 0; k < 32; k++) {
        const int p = k * 16 + grp;
        const float2 a = *reinterpret_cast<const float2 *>(A + p * kOutA + c0);
        const float4 b = *reinterpret_cast<const float4 *>(B + p * kOutB + j0);
        const float av[2] = {a.x, a.y}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = __fmaf_rn(av[i], bv[j], acc[i][j]);
        if (BIAS_A) {
            sa[0] += av[0];
            sa[1] += av[1];
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++) sb[j] += bv[j];
        }
    }
    __syncthreads();   // every thread is done with A and B
    // 16 groups -> 8 warps -> 1: slot (warp, tile) of 8 products and 4 sums
    float *red = sm;
    float v[12];
#pragma unroll
    for (int q = 0; q < 8; q++) v[q] = acc[q >> 2][q & 3];
#pragma unroll
    for (int q = 0; q < 4; q++) v[8 + q] = BIAS_A ? (q < 2 ? sa[q] : 0.0f) : sb[q];
#pragma unroll
    for (int q = 0; q < 12; q++) {
        v[q] += __shfl_xor_sync(0xffffffffu, v[q], 16);
        if (!(t & 16)) red[((t >> 5) * 16 + (t & 15)) * 13 + q] = v[q];
    }
    __syncthreads();
    for (int o = t; o < 16 * 12; o += 256) {
        const int tile = o / 12, q = o % 12;
        float s = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; w++) s += red[(w * 16 + tile) * 13 + q];
        const int c = (tile & 3) * 2, j = (tile >> 2) * 4;
        if (q < 8) atomicAdd(gw + (c + (q >> 2)) * SC + (j + (q & 3)) * SJ, s);
        else if (BIAS_A) {
            if (j == 0 && q < 10) atomicAdd(gb + c + (q - 8), s);
        } else if (c == 0) {
            atomicAdd(gb + j + (q - 8), s);
        }
    }
}

struct D1Args {
    int nb;
    const __nv_bfloat16 *g1;      // [nbp*512 x 16]
    const float *v1, *c1;         // D1: W [8 x 16] (bf16 values), b [8]
    const float *xn;              // normalized target
    float *recon;                 // normalized reconstruction, or null
    int recon16;                  // 1: recon is 16-byte aligned
    __nv_bfloat16 *dg1;           // gradient at D2's output (gated)
    float *gd1;                   // D1 gradient (W then b, 136 floats), or null: no gradients
    double *loss;                 // sum of squared errors, slot *step - step0
    const int *step;
    int step0;
    const float *wrow;            // block weights (null: all 1)
    const float *wsum;            // batch weight sum slot base (null: block count)
};

// D1 in training / evaluation: reconstruction, weighted loss, D1's weight
// and bias gradients and the gated gradient at D2's output.
// loss = sum_b w_b |e_b|^2 / (W * 4096), W = sum_b w_b.
__global__ void __launch_bounds__(256) k_ae_d1(const D1Args a) {
    extern __shared__ float sm[];
    __shared__ float red[8];
    tc::after_predecessor();
    const int b = blockIdx.x, t = threadIdx.x;
    if (b >= a.nb) return;
    float *A = sm, *B = sm + 512 * kOutA;
    float lsum = 0.0f;
    const float W = a.wsum ? a.wsum[*a.step - a.step0] : (float)gridDim.x;
    const float wb = a.wrow ? a.wrow[b] : 1.0f;
    const float gsc = wb / (W * (float)kAePts);
#pragma unroll 1
    for (int r = 0; r < 2; r++) {
        const int p = t + 256 * r;
        float g[16], y[8], x[8];
        const float4 *xp = reinterpret_cast<const float4 *>(a.xn + (long)b * kAePts + p * 8);
        *reinterpret_cast<float4 *>(x) = xp[0];
        *reinterpret_cast<float4 *>(x + 4) = xp[1];
        d1_node(a.v1, a.c1, a.g1 + ((long)b * 512 + p) * 16, g, y);
        float dy[8];
#pragma unroll
        for (int c = 0; c < 8; c++) {
            const float d = y[c] - x[c];
            lsum += d * d;
            dy[c] = 2.0f * d * gsc;
        }
        if (a.recon) {   // the caller's buffer: 4-byte aligned
            float *rp = a.recon + (long)b * kAePts + p * 8;
            if (a.recon16) {
                reinterpret_cast<float4 *>(rp)[0] = make_float4(y[0], y[1], y[2], y[3]);
                reinterpret_cast<float4 *>(rp)[1] = make_float4(y[4], y[5], y[6], y[7]);
            } else {
#pragma unroll
                for (int c = 0; c < 8; c++) rp[c] = y[c];
            }
        }
        if (a.gd1) {
#pragma unroll
            for (int c = 0; c < 2; c++)
                reinterpret_cast<float4 *>(A + p * kOutA)[c] =
                    make_float4(dy[4 * c], dy[4 * c + 1], dy[4 * c + 2], dy[4 * c + 3]);
#pragma unroll
            for (int c = 0; c < 4; c++)
                reinterpret_cast<float4 *>(B + p * kOutB)[c] =
                    make_float4(g[4 * c], g[4 * c + 1], g[4 * c + 2], g[4 * c + 3]);
            uint4 o4[2];
            __nv_bfloat16 *ob = reinterpret_cast<__nv_bfloat16 *>(o4);
#pragma unroll
            for (int j = 0; j < 16; j++) {
                float acc = 0.0f;
#pragma unroll
                for (int c = 0; c < 8; c++) acc += a.v1[c * 16 + j] * dy[c];
                ob[j] = __float2bfloat16_rn(g[j] > 0.0f ? acc : kLeak * acc);
            }
            uint4 *dst = reinterpret_cast<uint4 *>(a.dg1 + ((long)b * 512 + p) * 16);
            dst[0] = o4[0];
            dst[1] = o4[1];
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
    if ((t & 31) == 0) red[t >> 5] = lsum;
    __syncthreads();
    if (t == 0) {
        double tot = 0.0;
        for (int w = 0; w < 8; w++) tot += red[w];
        const double Wd = a.wsum ? (double)a.wsum[*a.step - a.step0] : (double)gridDim.x;
        atomicAdd(a.loss + (*a.step - a.step0), tot * wb / Wd);
    }
    if (a.gd1) block_outer<true, 16, 1>(sm, a.gd1, a.gd1 + 128);
}

// D1 of a snapshot's blocks with the weights passed by value, unscaled: mode 1
// adds wimg * snapshot * gP to the image (escaped blocks with their residual),
// mode 3 compares with the field vol.src and keeps every block's residual
// (bf16, natural order) and its squared error and norm (the escape check).
// Thread t owns nodes t and t + 256, then depth z = t & 15 of row x = t >> 4 on
// all sixteen planes; the values change hands in shared memory without bank
// conflicts (swz).
struct D1Vol {
    AeVolume vol;
    int nb;
    const __nv_bfloat16 *g1;      // [nbp*512 x 16]
    const float *scale;           // [nbp]
    const float *gP;              // mode 1: receiver field (vol's strides)
    float *mig;                   // mode 1: image, iz + nz*(ix + nx*iy)
    float wimg;                   // mode 1: weight of this snapshot
    const int *esc;               // mode 1: escaped-block slot per row (-1: none), or null
    const __nv_bfloat16 *res;     // mode 1: residual pool (4096 per slot, natural order)
    __nv_bfloat16 *resall;        // mode 3: residual of every row (natural order)
    float *err2, *norm2;          // mode 3: per-row squared error and squared norm
    AeSmallW w;
};

template <int MODE>
__global__ void __launch_bounds__(256, 4) k_ae_d1_vol(const D1Vol a) {
    __shared__ __align__(16) float ys[kAePts];
    __shared__ float red2[2][8];
    const int b = blockIdx.x, t = threadIdx.x;
    if (b >= a.nb) return;
    const float s = a.scale[b];
    uint4 g[2][2];
    float4 yv[2][2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const uint4 *src = reinterpret_cast<const uint4 *>(a.g1 + ((long)b * 512 + t + 256 * r) * 16);
        g[r][0] = src[0];
        g[r][1] = src[1];
    }
    d1_pairs(a.w, g, s, yv);
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int o = swz((t + 256 * r) * 8);
        *reinterpret_cast<float4 *>(ys + o) = yv[r][0];
        *reinterpret_cast<float4 *>(ys + (o ^ 4)) = yv[r][1];
    }
    __syncthreads();
    const AeVolume &v = a.vol;
    const int bz = b % v.nbz, bx = (b / v.nbz) % v.nbx, by = b / (v.nbz * v.nbx);
    const int z = t & 15, x = t >> 4, iz = bz * 16 + z, ix = bx * 16 + x, iy0 = by * 16;
    const bool zx = iz < v.nz && ix < v.nx;
    const long col = (long)(v.oz + iz) + v.ldz * (v.ox + ix) + v.sxy * (v.oy + iy0);
    const BlockCol c(z, x);
    if (MODE == 3) {
        float e2 = 0.0f, x2 = 0.0f;
        __nv_bfloat16 *rb = a.resall + (long)b * kAePts;
        float vals[16];
#pragma unroll
        for (int y = 0; y < 16; y++) vals[y] = zx && iy0 + y < v.ny ? __ldg(v.src + col + v.sxy * y) : 0.0f;
#pragma unroll
        for (int y = 0; y < 16; y++) {
            const float d = vals[y] - ys[c.at(y)];
            rb[y * 256 + t] = __float2bfloat16_rn(d);
            e2 += d * d;
            x2 += vals[y] * vals[y];
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            e2 += __shfl_xor_sync(0xffffffffu, e2, o);
            x2 += __shfl_xor_sync(0xffffffffu, x2, o);
        }
        if ((t & 31) == 0) {
            red2[0][t >> 5] = e2;
            red2[1][t >> 5] = x2;
        }
        __syncthreads();
        if (t == 0) {
            float E = 0.0f, X = 0.0f;
            for (int w = 0; w < 8; w++) {
                E += red2[0][w];
                X += red2[1][w];
            }
            a.err2[b] = E;
            a.norm2[b] = X;
        }
        return;
    }
    if (!zx) return;
    const int slot = a.esc ? a.esc[b] : -1;
    const __nv_bfloat16 *res = slot >= 0 ? a.res + (long)slot * kAePts : nullptr;
    // mode 1: all image and receiver-field loads in flight first
    const long o0 = iz + (long)v.nz * (ix + (long)v.nx * iy0), so = (long)v.nz * v.nx;
    float gp[16], mg[16];
#pragma unroll
    for (int y = 0; y < 16; y++) {
        const bool in = iy0 + y < v.ny;
        gp[y] = in ? __ldg(a.gP + col + v.sxy * y) : 0.0f;
        mg[y] = in ? a.mig[o0 + so * y] : 0.0f;
    }
#pragma unroll
    for (int y = 0; y < 16; y++) {
        if (iy0 + y >= v.ny) break;
        float val = ys[c.at(y)];
        if (res) val += __bfloat162float(res[y * 256 + t]);
        a.mig[o0 + so * y] = mg[y] + a.wimg * val * gp[y];
    }
}

// Escape pass 1 is k_ae_d1_vol in mode 3: decode, compare with the field, keep
// every block's residual (bf16, natural order) and its squared error and norm.

// Escape pass 2 (one block of 1024 threads): the cap blocks with the
// largest squared error, among those with err2 > tau2 * norm2, get residual
// slots: a binary search on the float bits of err2 finds the threshold.
__global__ void __launch_bounds__(1024) k_ae_select(const float *err2, const float *norm2, int nb, float tau2, int cap,
                                                    int *esc, int *count) {
    __shared__ int cnt;
    __shared__ int next;
    auto eligible = [&](int b) { return err2[b] > 0.0f && err2[b] > tau2 * norm2[b]; };
    // smallest threshold bits T with #{eligible, bits(err2) > T} <= cap
    unsigned lo = 0u, hi = 0x7f800000u;   // error bits of non-negative floats
    while (lo < hi) {
        const unsigned mid = lo + (hi - lo) / 2;
        if (threadIdx.x == 0) cnt = 0;
        __syncthreads();
        int c = 0;
        for (int b = threadIdx.x; b < nb; b += blockDim.x) c += eligible(b) && __float_as_uint(err2[b]) > mid;
        atomicAdd(&cnt, c);
        __syncthreads();
        const int total = cnt;
        __syncthreads();
        if (total <= cap) hi = mid;
        else lo = mid + 1;
    }
    if (threadIdx.x == 0) next = 0;
    __syncthreads();
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
        int sl = -1;
        if (eligible(b) && __float_as_uint(err2[b]) > lo) sl = atomicAdd(&next, 1);
        esc[b] = sl < cap ? sl : -1;
    }
    __syncthreads();
    if (threadIdx.x == 0) *count = min(next, cap);
}

// Escape pass 3: copy the selected residuals into their slots.
__global__ void __launch_bounds__(256) k_ae_escape_copy(const int *esc, const __nv_bfloat16 *resall,
                                                        __nv_bfloat16 *res, int nb) {
    const int b = blockIdx.x;
    if (b >= nb) return;
    const int sl = esc[b];
    if (sl < 0) return;
    const uint4 *src = reinterpret_cast<const uint4 *>(resall + (long)b * kAePts);
    uint4 *dst = reinterpret_cast<uint4 *>(res + (long)sl * kAePts);
    for (int i = threadIdx.x; i < kAePts / 8; i += 256) dst[i] = src[i];
}

// E1 weight and bias gradients from the normalized input and the gated
// gradient at E1's output.
__global__ void __launch_bounds__(256) k_ae_e1_bwd(const float *xn, const __nv_bfloat16 *dh1, float *ge1, int nb) {
    extern __shared__ float sm[];
    tc::after_predecessor();
    const int b = blockIdx.x, t = threadIdx.x;
    if (b >= nb) return;
    float *A = sm, *B = sm + 512 * kOutA;
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int p = t + 256 * r;
        const float4 *xp = reinterpret_cast<const float4 *>(xn + (long)b * kAePts + p * 8);
        const float4 x0 = xp[0], x1 = xp[1];
        float4 *ap = reinterpret_cast<float4 *>(A + p * kOutA);
        ap[0] = make_float4(bf16r(x0.x), bf16r(x0.y), bf16r(x0.z), bf16r(x0.w));
        ap[1] = make_float4(bf16r(x1.x), bf16r(x1.y), bf16r(x1.z), bf16r(x1.w));
        const uint4 *src = reinterpret_cast<const uint4 *>(dh1 + ((long)b * 512 + p) * 16);
        const uint4 q[2] = {src[0], src[1]};
        const __nv_bfloat16 *qb = reinterpret_cast<const __nv_bfloat16 *>(q);
        float4 *bp = reinterpret_cast<float4 *>(B + p * kOutB);
#pragma unroll
        for (int c = 0; c < 4; c++)
            bp[c] = make_float4(__bfloat162float(qb[4 * c]), __bfloat162float(qb[4 * c + 1]),
                                __bfloat162float(qb[4 * c + 2]), __bfloat162float(qb[4 * c + 3]));
    }
    __syncthreads();
    block_outer<false, 1, 8>(sm, ge1, ge1 + 128);   // W1[j * 8 + c]
}

// Bias gradients of the GEMM levels in one launch: gb[n] += sum over the
// rows of dy[m*N + n].  A thread sums 8 columns (one 16-byte load per row)
// over every (256 / (N/8))-th row of its block's range, the block reduces
// through shared memory and adds N values.  Latency-bound (4 MB of reads at
// 256 blocks); one launch for the six levels instead of one each.
struct ColsumLevel {
    const __nv_bfloat16 *dy;
    float *gb;
    int M, N, base, ctas;
};
struct ColsumArgs {
    ColsumLevel it[6];
};

__global__ void __launch_bounds__(256) k_ae_colsum(const ColsumArgs g) {
    __shared__ float red[256 * 8];
    tc::after_predecessor();
    int l = 0;
    while (l < 5 && (int)blockIdx.x >= g.it[l + 1].base) l++;
    const ColsumLevel &w = g.it[l];
    const int rel = (int)blockIdx.x - w.base, t = threadIdx.x;
    const int m0 = (int)((long)w.M * rel / w.ctas), m1 = (int)((long)w.M * (rel + 1) / w.ctas);
    const int cg = w.N / 8, per = 256 / cg, col = t % cg, r0 = t / cg;   // N <= 2048, a multiple of 64
    float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int m = m0 + r0; m < m1; m += per) {
        const uint4 q = *reinterpret_cast<const uint4 *>(w.dy + (long)m * w.N + col * 8);
        const __nv_bfloat16 *h = reinterpret_cast<const __nv_bfloat16 *>(&q);
#pragma unroll
        for (int j = 0; j < 8; j++) s[j] += __bfloat162float(h[j]);
    }
#pragma unroll
    for (int j = 0; j < 8; j++) red[t * 8 + j] = s[j];
    __syncthreads();
    for (int n = t; n < w.N; n += 256) {
        float v = 0.0f;
        for (int r = 0; r < per; r++) v += red[r * w.N + n];
        atomicAdd(w.gb + n, v);
    }
}

// Adam (bias-corrected) with the step's learning rate from lrs[*step - step0].
__global__ void k_ae_adam(float *p, const float *g, float *m1, float *m2, long n, const int *step, int step0,
                          const float *lrs) {
    const int t = *step + 1;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float bc1 = 1.0f - powf(b1, (float)t), bc2 = 1.0f - powf(b2, (float)t);
    const float lr = lrs[*step - step0];
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float a = b1 * m1[i] + (1.0f - b1) * gi;
        const float v = b2 * m2[i] + (1.0f - b2) * gi * gi;
        m1[i] = a;
        m2[i] = v;
        p[i] -= lr * (a / bc1) / (sqrtf(v / bc2) + eps);
    }
}

// bf16 copies of the GEMM weights ([N x K] and transposed [K x N]) and the
// bf16-valued fp32 copies of E1 and D1; then step += inc.
struct PackArgs {
    const float *params;
    __nv_bfloat16 *wb, *wtb;
    float *small;                 // E1 W (128) then D1 W (128)
    long w[kAeLayers], wb_off[kAeLayers];
    int N[kAeLayers], K[kAeLayers];
    int *step, inc;
};

__global__ void k_ae_pack(const PackArgs a) {
    const long tid = blockIdx.x * (long)blockDim.x + threadIdx.x, nth = (long)gridDim.x * blockDim.x;
    for (int l = 1; l <= 6; l++) {
        const int N = a.N[l], K = a.K[l];
        const long n = (long)N * K;
        for (long i = tid; i < n; i += nth) {
            const int r = (int)(i / K), c = (int)(i % K);
            const __nv_bfloat16 v = __float2bfloat16_rn(a.params[a.w[l] + i]);
            a.wb[a.wb_off[l] + i] = v;
            a.wtb[a.wb_off[l] + (long)c * N + r] = v;
        }
    }
    for (long i = tid; i < 128; i += nth) {
        a.small[i] = bf16r(a.params[a.w[0] + i]);
        a.small[128 + i] = bf16r(a.params[a.w[7] + i]);
    }
    if (tid == 0 && a.inc) *a.step += a.inc;
}

// Per-snapshot max |value| of an interior box (as ordered int bits).
__global__ void k_ae_absmax(const AeVolume v, unsigned *out) {
    float mx = 0.0f;
    const long n = (long)v.nz * v.nx * v.ny;
    for (long k = blockIdx.x * (long)blockDim.x + threadIdx.x; k < n; k += (long)gridDim.x * blockDim.x) {
        const int iz = (int)(k % v.nz), ix = (int)((k / v.nz) % v.nx), iy = (int)(k / ((long)v.nz * v.nx));
        mx = fmaxf(mx, fabsf(v.src[(long)(v.oz + iz) + v.ldz * (v.ox + ix) + v.sxy * (v.oy + iy)]));
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(mx));
}

// Append the full blocks of a snapshot whose max |value| exceeds
// rel * (snapshot max) to the training store (Morton order).
__global__ void __launch_bounds__(256) k_ae_collect(const AeVolume v, const unsigned *snapmax, float rel, float *store,
                                                    float *wstore, long cap, unsigned long long *count) {
    __shared__ float xs[kAePts];
    __shared__ float red[8];
    __shared__ long slot;
    const int b = blockIdx.x, t = threadIdx.x;
    const int bz = b % v.nbz, bx = (b / v.nbz) % v.nbx, by = b / (v.nbz * v.nbx);
    if ((bz + 1) * 16 > v.nz || (bx + 1) * 16 > v.nx || (by + 1) * 16 > v.ny) return;  // full blocks only
    float mx = 0.0f;
    for (int p = 0; p < 16; p++) {
        const int idx = p * 256 + t, z = idx & 15, x = (idx >> 4) & 15, y = idx >> 8;
        const float val = v.src[(long)(v.oz + bz * 16 + z) + v.ldz * (v.ox + bx * 16 + x) + v.sxy * (v.oy + by * 16 + y)];
        xs[morton_of(z, x, y)] = val;
        mx = fmaxf(mx, fabsf(val));
    }
    const float s = block_max(mx, red);
    if (!(s > rel * __uint_as_float(*snapmax))) return;
    if (t == 0) slot = (long)atomicAdd(count, 1ull);
    __syncthreads();
    if (slot >= cap) return;
    if (t == 0) {
        const float r = s / __uint_as_float(*snapmax);
        wstore[slot] = r * r;   // the block's share of its snapshot's energy scale
    }
    for (int p = 0; p < 16; p++) store[slot * kAePts + p * 256 + t] = xs[p * 256 + t];
}

}  // namespace geo

// ---------------------------------------------------------------- host state
struct geo_ae {
    AeOffsets off;
    unsigned long long seed = 0;
    DevBuf params, grad, m1, m2, wb, wtb, small, step, err;
    int h_step = 0;
    // block store for training
    DevBuf store, wstore, count, snapmax;
    long cap = 0;
    // forward scratch (rows = padded blocks)
    DevBuf h1, h2, h3, z, g3, g2, g1, scale;
    // training scratch
    DevBuf xn, dg1, dg2, dg3, dz, dh3, dh2, dh1, wrow;
    DevBuf ev;                                 // evaluation: loss (double), zero step counter
    // escape settings
    float tau = 0.05f, frac = 0.03f;
    DevBuf resall, err2, norm2;
    long long st_blocks = 0, st_escaped = 0;   // totals over RTM shots
    // host copy of the CUDA-core levels' weights for the snapshot kernels:
    // wver counts weight updates (packs), hver the version copied
    geo::AeSmallW hw{};
    long wver = 1, hver = 0;
};

namespace geo {

static int pad128(long n) { return (int)((n + 127) / 128 * 128); }

static int ae_pack(geo_ae *ae, int inc, cudaStream_t s) {
    PackArgs a{};
    a.params = ae->params.as<float>();
    a.wb = ae->wb.as<__nv_bfloat16>();
    a.wtb = ae->wtb.as<__nv_bfloat16>();
    a.small = ae->small.as<float>();
    for (int l = 0; l < kAeLayers; l++) {
        a.w[l] = ae->off.w[l];
        a.wb_off[l] = ae->off.wb[l];
        a.N[l] = kAeNet[l].N;
        a.K[l] = kAeNet[l].K;
    }
    a.step = ae->step.as<int>();
    a.inc = inc;
    ae->wver++;
    k_ae_pack<<<152 * 4, 256, 0, s>>>(a);
    return check_launch("ae_pack");
}

// A scratch buffer of at least n bytes.  A buffer that could not grow is empty
// and is asked for again by the next call.
static int at_least(DevBuf &b, size_t n) { return b.bytes >= n ? GEO_OK : b.alloc(n); }

static int ensure_rows(geo_ae *ae, int rows) {
    const size_t r = (size_t)rows;
    GEO_TRY(at_least(ae->h2, r * 64 * 64 * 2));
    GEO_TRY(at_least(ae->h3, r * 8 * 256 * 2));
    GEO_TRY(at_least(ae->z, r * 512 * 2));
    GEO_TRY(at_least(ae->g3, r * 2048 * 2));
    GEO_TRY(at_least(ae->g2, r * 8 * 512 * 2));
    return at_least(ae->scale, r * 4);
}
// E1's output: training only (snapshots have E1 and E2 in one kernel).
static int ensure_h1(geo_ae *ae, int rows) { return at_least(ae->h1, (size_t)rows * 512 * 16 * 2); }
// D2's output: training, imaging and the escape check (a plain decode has D2 and D1 in one kernel).
static int ensure_g1(geo_ae *ae, int rows) { return at_least(ae->g1, (size_t)rows * 64 * 128 * 2); }

static int ensure_train(geo_ae *ae, int rows) {
    GEO_TRY(ensure_rows(ae, rows));
    GEO_TRY(ensure_h1(ae, rows));
    GEO_TRY(ensure_g1(ae, rows));
    const size_t r = (size_t)rows;
    GEO_TRY(at_least(ae->xn, r * kAePts * 4));
    GEO_TRY(at_least(ae->dg1, r * 8192 * 2));
    GEO_TRY(at_least(ae->dg2, r * 4096 * 2));
    GEO_TRY(at_least(ae->dg3, r * 2048 * 2));
    GEO_TRY(at_least(ae->dz, r * 512 * 2));
    GEO_TRY(at_least(ae->dh3, r * 2048 * 2));
    GEO_TRY(at_least(ae->dh2, r * 4096 * 2));
    GEO_TRY(at_least(ae->dh1, r * 8192 * 2));
    return at_least(ae->wrow, r * 4);
}

static __nv_bfloat16 *bf(const DevBuf &b) { return b.as<__nv_bfloat16>(); }

// One GEMM level: out = act(in * W^T + b) for `rows` blocks.
static int level(geo_ae *ae, int l, int rows, const __nv_bfloat16 *in, __nv_bfloat16 *out, cudaStream_t s) {
    const AeLayer &L = kAeNet[l];
    TcGemm g{};
    g.M = rows * L.rows;
    g.N = L.N;
    g.K = L.K;
    g.A = in;
    g.B = bf(ae->wb) + ae->off.wb[l];
    g.bias = ae->params.as<float>() + ae->off.b[l];
    g.act = L.act;
    g.out = out;
    g.err = ae->err.as<int>();
    return tc_gemm(g, s);
}

// Input gradient of GEMM level l, gated by the input activation (null gate:
// linear).
static int level_bwd(geo_ae *ae, int l, int rows, const __nv_bfloat16 *dout, __nv_bfloat16 *din,
                     const __nv_bfloat16 *gate, cudaStream_t s) {
    const AeLayer &L = kAeNet[l];
    TcGemm g{};
    g.M = rows * L.rows;
    g.N = L.K;
    g.K = L.N;
    g.A = dout;
    g.B = bf(ae->wtb) + ae->off.wb[l];
    g.gate = gate;
    g.out = din;
    g.err = ae->err.as<int>();
    return tc_gemm(g, s);
}

// Weight and bias gradients of the GEMM levels 1..6 from their output
// gradients dout[l] and inputs in[l]: one launch each.
static int wgrads(geo_ae *ae, int rows, const __nv_bfloat16 *const *dout, const __nv_bfloat16 *const *in,
                  cudaStream_t s) {
    TcWgradLevel lv[6];
    ColsumArgs c{};
    int base = 0;
    for (int q = 0; q < 6; q++) {
        const int l = q + 1;
        const AeLayer &L = kAeNet[l];
        const int M = rows * L.rows;
        float *gw = ae->grad.as<float>() + ae->off.w[l];
        // the 128-row operand is dY, or X where dY has only 64 columns
        const bool xa = L.N % 128 != 0;
        lv[q] = TcWgradLevel{M, xa ? in[l] : dout[l], xa ? dout[l] : in[l], xa ? L.K : L.N, xa ? L.N : L.K, gw,
                             xa ? 1L : (long)L.K, xa ? (long)L.K : 1L};
        ColsumLevel &k = c.it[q];
        k.dy = dout[l];
        k.gb = ae->grad.as<float>() + ae->off.b[l];
        k.M = M;
        k.N = L.N;
        k.base = base;
        k.ctas = std::max(1, std::min(M / 16, 64));
        base += k.ctas;
    }
    GEO_TRY(tc_wgrad(lv, 6, ae->err.as<int>(), s));
    GEO_CUDA(launch_early(k_ae_colsum, base, 256, 0, s, c));
    return check_launch("ae_colsum");
}

// Encoder levels E2..E4 from h1 into `code` (rows x 512 bf16).
static int encode_rows(geo_ae *ae, int rows, __nv_bfloat16 *code, cudaStream_t s) {
    GEO_TRY(level(ae, 1, rows, bf(ae->h1), bf(ae->h2), s));
    GEO_TRY(level(ae, 2, rows, bf(ae->h2), bf(ae->h3), s));
    return level(ae, 3, rows, bf(ae->h3), code, s);
}

// Decoder levels D4..D2 from `code` into g1.
static int decode_rows(geo_ae *ae, int rows, const __nv_bfloat16 *code, cudaStream_t s) {
    GEO_TRY(level(ae, 4, rows, code, bf(ae->g3), s));
    GEO_TRY(level(ae, 5, rows, bf(ae->g3), bf(ae->g2), s));
    return level(ae, 6, rows, bf(ae->g2), bf(ae->g1), s);
}

static E1Args e1_args(geo_ae *ae, int nb) {
    E1Args a{};
    a.nb = nb;
    a.w1 = ae->small.as<float>();
    a.b1 = ae->params.as<float>() + ae->off.b[0];
    a.h1 = bf(ae->h1);
    a.scale = ae->scale.as<float>();
    a.step = ae->step.as<int>();
    a.seed = ae->seed;
    return a;
}

static D1Args d1_args(geo_ae *ae, int nb) {
    D1Args a{};
    a.nb = nb;
    a.g1 = bf(ae->g1);
    a.v1 = ae->small.as<float>() + 128;
    a.c1 = ae->params.as<float>() + ae->off.b[7];
    return a;
}

// The host copy of the E1/D1 weights, refreshed when a pack changed them
// (a 1 KB read and a wait on the stream, once per weight version).
static int ae_mirror(geo_ae *ae, cudaStream_t s) {
    if (ae->hver == ae->wver) return GEO_OK;
    AeSmallW &h = ae->hw;
    const float *sm = ae->small.as<float>(), *pr = ae->params.as<float>();
    float w[256];
    GEO_CUDA(cudaMemcpyAsync(w, sm, sizeof w, cudaMemcpyDeviceToHost, s));
    GEO_CUDA(cudaMemcpyAsync(h.b1, pr + ae->off.b[0], sizeof h.b1, cudaMemcpyDeviceToHost, s));
    GEO_CUDA(cudaMemcpyAsync(h.c1, pr + ae->off.b[7], sizeof h.c1, cudaMemcpyDeviceToHost, s));
    GEO_CUDA(cudaStreamSynchronize(s));
    for (int c = 0; c < 16; c++)
        for (int j = 0; j < 8; j++) {
            h.w1[j * 16 + c] = w[c * 8 + j];
            h.v1[c * 8 + j] = w[128 + j * 16 + c];
        }
    ae->hver = ae->wver;
    return GEO_OK;
}

int ae_check_err(geo_ae *ae, cudaStream_t s) {
    int e = 0;
    GEO_CUDA(cudaMemcpyAsync(&e, ae->err.p, 4, cudaMemcpyDeviceToHost, s));
    GEO_CUDA(cudaStreamSynchronize(s));
    if (e) return fail(GEO_ERR_CUDA, "snapshot codec: a tensor-core pipeline wait timed out");
    return GEO_OK;
}

static int blocks_of(const AeVolume &v) { return v.nbz * v.nbx * v.nby; }

AeVolume ae_volume(const float *src, long ldz, long sxy, int oz, int ox, int oy, int nz, int nx, int ny) {
    AeVolume v{};
    v.src = src;
    v.ldz = ldz;
    v.sxy = sxy;
    v.oz = oz; v.ox = ox; v.oy = oy;
    v.nz = nz; v.nx = nx; v.ny = ny;
    v.nbz = (nz + 15) / 16;
    v.nbx = (nx + 15) / 16;
    v.nby = (ny + 15) / 16;
    return v;
}

int ae_code_rows(const AeVolume &v) { return pad128(blocks_of(v)); }

int ae_escape_cap(geo_ae *ae, const AeVolume &v) {
    const int nb = blocks_of(v);
    return std::min(nb, (int)std::ceil(ae->frac * nb));
}

static int ae_smem() {
    static OncePerDevice e12, d21;
    GEO_TRY(allow_smem(e12, (const void *)k_ae_e12, kE12Smem));
    return allow_smem(d21, (const void *)k_ae_d21, kD21Smem);
}

// Encode the interior box v into code[rows x 512] (bf16) and scale[rows];
// with esc != null also decode, and keep the residuals of the blocks the
// code misses (esc[rows], res[cap x 4096] bf16, *count escaped blocks).
int ae_encode_volume(geo_ae *ae, const AeVolume &v, void *code, float *scale, int *esc, void *res, int *count,
                     cudaStream_t s) {
    const int nb = blocks_of(v), rows = pad128(nb);
    GEO_TRY(ensure_rows(ae, rows));
    if (esc) GEO_TRY(ensure_g1(ae, rows));   // before a run, not at its first decode
    GEO_TRY(ae_mirror(ae, s));
    E12Args a{};
    a.vol = v;
    a.nb = nb;
    a.tiles = rows / 2;
    a.scale = scale;
    a.bias = ae->params.as<float>() + ae->off.b[1];
    a.err = ae->err.as<int>();
    a.w = ae->hw;
    CUtensorMap tw, to;
    GEO_TRY(tc_map_bf16(&tw, bf(ae->wb) + ae->off.wb[1], 64, 128, 64));
    GEO_TRY(tc_map_bf16(&to, ae->h2.p, rows * 64, 64, 32));
    GEO_TRY(ae_smem());
    GEO_CUDA(launch_early(k_ae_e12, std::min((a.tiles + 1) / 2, 2 * sm_count()), 256, kE12Smem, s, tw, to, a));
    GEO_TRY(check_launch("ae_e12"));
    GEO_TRY(level(ae, 2, rows, bf(ae->h2), bf(ae->h3), s));
    GEO_TRY(level(ae, 3, rows, bf(ae->h3), static_cast<__nv_bfloat16 *>(code), s));
    if (!esc) return GEO_OK;
    if (ae_escape_cap(ae, v) == 0) {   // no escape budget: no re-decode
        GEO_CUDA(cudaMemsetAsync(esc, 0xff, (size_t)rows * 4, s));
        if (count) GEO_CUDA(cudaMemsetAsync(count, 0, 4, s));
        return GEO_OK;
    }
    GEO_TRY(at_least(ae->resall, (size_t)rows * kAePts * 2));
    GEO_TRY(at_least(ae->err2, (size_t)rows * 4));
    GEO_TRY(at_least(ae->norm2, (size_t)rows * 4));
    GEO_TRY(decode_rows(ae, rows, static_cast<const __nv_bfloat16 *>(code), s));
    D1Vol c{};
    c.vol = v;
    c.nb = nb;
    c.g1 = bf(ae->g1);
    c.scale = scale;
    c.resall = bf(ae->resall);
    c.err2 = ae->err2.as<float>();
    c.norm2 = ae->norm2.as<float>();
    c.w = ae->hw;
    k_ae_d1_vol<3><<<rows, 256, 0, s>>>(c);
    GEO_TRY(check_launch("ae_check"));
    k_ae_select<<<1, 1024, 0, s>>>(ae->err2.as<float>(), ae->norm2.as<float>(), nb, ae->tau * ae->tau,
                                   ae_escape_cap(ae, v), esc, count);
    GEO_TRY(check_launch("ae_select"));
    k_ae_escape_copy<<<nb, 256, 0, s>>>(esc, bf(ae->resall), static_cast<__nv_bfloat16 *>(res), nb);
    return check_launch("ae_escape_copy");
}

// Decode code/scale (and escaped residuals) of box geometry v: mode 0
// writes the snapshot into dst (v's strides), mode 1 adds w * snapshot * gP
// to mig.
int ae_decode_volume(geo_ae *ae, const AeVolume &v, const void *code, const float *scale, const int *esc,
                     const void *res, int mode, float *dst, const float *gP, float *mig, float w, cudaStream_t s) {
    const int nb = blocks_of(v), rows = pad128(nb);
    GEO_TRY(ensure_rows(ae, rows));
    GEO_TRY(ae_mirror(ae, s));
    if (mode == 0) {
        GEO_TRY(level(ae, 4, rows, static_cast<const __nv_bfloat16 *>(code), bf(ae->g3), s));
        GEO_TRY(level(ae, 5, rows, bf(ae->g3), bf(ae->g2), s));
        D21Args a{};
        a.vol = v;
        a.nb = nb;
        a.tiles = (nb + 1) / 2;
        a.scale = scale;
        a.bias = ae->params.as<float>() + ae->off.b[6];
        a.dst = dst;
        a.esc = esc;
        a.res = static_cast<const __nv_bfloat16 *>(res);
        a.err = ae->err.as<int>();
        a.w = ae->hw;
        CUtensorMap ta, tw;
        GEO_TRY(tc_map_bf16(&ta, ae->g2.p, rows * 64, 64, 128));
        GEO_TRY(tc_map_bf16(&tw, bf(ae->wb) + ae->off.wb[6], 128, 64, 128));
        GEO_TRY(ae_smem());
        GEO_CUDA(launch_early(k_ae_d21, std::min(a.tiles, 2 * sm_count()), kD21Threads, kD21Smem, s, ta, tw, a));
        return check_launch("ae_d21");
    }
    GEO_TRY(ensure_g1(ae, rows));
    GEO_TRY(decode_rows(ae, rows, static_cast<const __nv_bfloat16 *>(code), s));
    D1Vol a{};
    a.vol = v;
    a.nb = nb;
    a.g1 = bf(ae->g1);
    a.scale = scale;
    a.gP = gP;
    a.mig = mig;
    a.wimg = w;
    a.esc = esc;
    a.res = static_cast<const __nv_bfloat16 *>(res);
    a.w = ae->hw;
    k_ae_d1_vol<1><<<rows, 256, 0, s>>>(a);
    return check_launch("ae_d1");
}

// Dynamic shared memory of the kernels that end in block_outer (64 KB).
static int outer_smem() {
    static OncePerDevice d1, e1;
    GEO_TRY(allow_smem(d1, (const void *)k_ae_d1, kOutFloats * 4));
    return allow_smem(e1, (const void *)k_ae_e1_bwd, kOutFloats * 4);
}

// Forward (+ backward when grads are wanted) over `rows` blocks already
// loaded by k_ae_e1 (xn filled); loss slot *step - step0.
static int train_pass(geo_ae *ae, int rows, double *loss, const float *wsum, const int *step, int step0, float *recon,
                      bool backward, cudaStream_t s) {
    GEO_TRY(encode_rows(ae, rows, bf(ae->z), s));
    GEO_TRY(decode_rows(ae, rows, bf(ae->z), s));
    D1Args a = d1_args(ae, rows);
    a.xn = ae->xn.as<float>();
    a.recon = recon;
    a.recon16 = (reinterpret_cast<uintptr_t>(recon) & 15) == 0;
    if (backward) {
        a.dg1 = bf(ae->dg1);
        a.gd1 = ae->grad.as<float>() + ae->off.w[7];
    }
    a.loss = loss;
    a.step = step;
    a.step0 = step0;
    a.wrow = wsum ? ae->wrow.as<float>() : nullptr;
    a.wsum = wsum;
    GEO_TRY(outer_smem());
    GEO_CUDA(launch_early(k_ae_d1, rows, 256, kOutFloats * 4, s, a));
    GEO_TRY(check_launch("ae_d1_train"));
    if (!backward) return GEO_OK;
    GEO_TRY(level_bwd(ae, 6, rows, bf(ae->dg1), bf(ae->dg2), bf(ae->g2), s));   // D2
    GEO_TRY(level_bwd(ae, 5, rows, bf(ae->dg2), bf(ae->dg3), bf(ae->g3), s));   // D3
    GEO_TRY(level_bwd(ae, 4, rows, bf(ae->dg3), bf(ae->dz), nullptr, s));       // D4
    GEO_TRY(level_bwd(ae, 3, rows, bf(ae->dz), bf(ae->dh3), bf(ae->h3), s));    // E4
    GEO_TRY(level_bwd(ae, 2, rows, bf(ae->dh3), bf(ae->dh2), bf(ae->h2), s));   // E3
    GEO_TRY(level_bwd(ae, 1, rows, bf(ae->dh2), bf(ae->dh1), bf(ae->h1), s));   // E2
    const __nv_bfloat16 *dout[7] = {nullptr, bf(ae->dh2), bf(ae->dh3), bf(ae->dz), bf(ae->dg3), bf(ae->dg2), bf(ae->dg1)};
    const __nv_bfloat16 *in[7] = {nullptr, bf(ae->h1), bf(ae->h2), bf(ae->h3), bf(ae->z), bf(ae->g3), bf(ae->g2)};
    GEO_TRY(wgrads(ae, rows, dout, in, s));
    GEO_CUDA(launch_early(k_ae_e1_bwd, rows, 256, kOutFloats * 4, s, ae->xn.as<float>(), bf(ae->dh1),
                          ae->grad.as<float>() + ae->off.w[0], rows));
    return check_launch("ae_e1_bwd");
}

// He-normal initial weights (own generator, identical on every host), zero biases.
static void init_params(const AeOffsets &o, unsigned long long seed, std::vector<float> &p) {
    p.assign(o.total, 0.0f);
    unsigned long long st = seed;
    auto uni = [&]() {
        st = splitmix(st);
        return ((st >> 11) + 0.5) * (1.0 / 9007199254740992.0);
    };
    for (int l = 0; l < kAeLayers; l++) {
        const double sd = std::sqrt((kAeNet[l].act || l == 3 ? 2.0 : 1.0) / kAeNet[l].K);
        const long n = (long)kAeNet[l].N * kAeNet[l].K;
        for (long i = 0; i < n; i += 2) {
            const double u1 = uni(), u2 = uni(), r = std::sqrt(-2.0 * std::log(u1));
            p[o.w[l] + i] = (float)(sd * r * std::cos(6.283185307179586 * u2));
            if (i + 1 < n) p[o.w[l] + i + 1] = (float)(sd * r * std::sin(6.283185307179586 * u2));
        }
    }
}

}  // namespace geo

// ---------------------------------------------------------------- C ABI
extern "C" size_t geo_ae_num_params(void) { return (size_t)ae_offsets().total; }

extern "C" int geo_ae_create(geo_ae **out, unsigned long long seed) {
    if (!out) return fail(GEO_ERR_ARG, "null argument");
    geo_ae *ae = new geo_ae();
    ae->off = ae_offsets();
    ae->seed = seed;
    const size_t P = ae->off.total;
    int st = GEO_OK;
    DevBuf *f32[4] = {&ae->params, &ae->grad, &ae->m1, &ae->m2};
    for (DevBuf *b : f32)
        if (st == GEO_OK) st = b->alloc(P * 4);
    if (st == GEO_OK) st = ae->wb.alloc(ae->off.nbf * 2);
    if (st == GEO_OK) st = ae->wtb.alloc(ae->off.nbf * 2);
    if (st == GEO_OK) st = ae->small.alloc(256 * 4);
    if (st == GEO_OK) st = ae->step.alloc(16);
    if (st == GEO_OK) st = ae->err.alloc(16);
    if (st == GEO_OK) st = ae->count.alloc(16);
    if (st == GEO_OK) st = ae->snapmax.alloc(16);
    if (st != GEO_OK) {
        delete ae;
        return st;
    }
    std::vector<float> p;
    init_params(ae->off, seed, p);
    int e = GEO_OK;
    if (cudaMemcpy(ae->params.p, p.data(), P * 4, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(ae->m1.p, 0, P * 4) != cudaSuccess || cudaMemset(ae->m2.p, 0, P * 4) != cudaSuccess ||
        cudaMemset(ae->step.p, 0, 16) != cudaSuccess || cudaMemset(ae->err.p, 0, 16) != cudaSuccess ||
        cudaMemset(ae->count.p, 0, 16) != cudaSuccess)
        e = fail(GEO_ERR_CUDA, "codec initialisation copy failed");
    if (e == GEO_OK) e = ae_pack(ae, 0, nullptr);
    if (e == GEO_OK && cudaDeviceSynchronize() != cudaSuccess) e = fail(GEO_ERR_CUDA, "codec initialisation failed");
    if (e != GEO_OK) {
        delete ae;
        return e;
    }
    *out = ae;
    return GEO_OK;
}

extern "C" int geo_ae_destroy(geo_ae *ae) {
    delete ae;
    return GEO_OK;
}

extern "C" int geo_ae_get_params(geo_ae *ae, float *host) {
    if (!ae || !host) return fail(GEO_ERR_ARG, "null argument");
    GEO_CUDA(cudaMemcpy(host, ae->params.p, ae->off.total * 4, cudaMemcpyDeviceToHost));
    return GEO_OK;
}

extern "C" int geo_ae_set_params(geo_ae *ae, const float *host) {
    if (!ae || !host) return fail(GEO_ERR_ARG, "null argument");
    GEO_CUDA(cudaMemcpy(ae->params.p, host, ae->off.total * 4, cudaMemcpyHostToDevice));
    GEO_TRY(ae_pack(ae, 0, nullptr));
    GEO_CUDA(cudaDeviceSynchronize());
    return GEO_OK;
}

extern "C" long long geo_ae_num_blocks(geo_ae *ae) {
    if (!ae || !ae->cap) return 0;
    unsigned long long n = 0;
    if (cudaMemcpy(&n, ae->count.p, 8, cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    return (long long)std::min<unsigned long long>(n, (unsigned long long)ae->cap);
}

extern "C" int geo_ae_reserve(geo_ae *ae, long long max_blocks) {
    if (!ae || max_blocks < 1) return fail(GEO_ERR_ARG, "bad argument");
    ae->cap = 0;   // no store until both buffers stand
    GEO_TRY(ae->store.alloc((size_t)max_blocks * kAePts * 4));
    GEO_TRY(ae->wstore.alloc((size_t)max_blocks * 4));
    ae->cap = max_blocks;
    GEO_CUDA(cudaMemset(ae->count.p, 0, 16));
    return GEO_OK;
}

extern "C" int geo_ae_add_blocks(geo_ae *ae, const float *blocks, long long n, int mem) {
    if (!ae || !blocks || n < 0) return fail(GEO_ERR_ARG, "bad argument");
    const long long have = geo_ae_num_blocks(ae);
    if (have < 0 || have + n > ae->cap) return fail(GEO_ERR_ARG, "block store full (reserve more)");
    GEO_CUDA(cudaMemcpy(ae->store.as<float>() + have * kAePts, blocks, (size_t)n * kAePts * 4,
                        mem == GEO_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice));
    std::vector<float> ones((size_t)n, 1.0f);
    GEO_CUDA(cudaMemcpy(ae->wstore.as<float>() + have, ones.data(), (size_t)n * 4, cudaMemcpyHostToDevice));
    const unsigned long long c = (unsigned long long)(have + n);
    GEO_CUDA(cudaMemcpy(ae->count.p, &c, 8, cudaMemcpyHostToDevice));
    return GEO_OK;
}

struct CollectCtx {
    geo_ae *ae;
    geo_fd3d_plan *plan;
    int snap_every, t_first;
    float rel;
    cudaStream_t s;
};

static int collect_step(void *ctx, int it) {
    CollectCtx *c = static_cast<CollectCtx *>(ctx);
    if (it < c->t_first || (it - c->t_first) % c->snap_every) return GEO_OK;
    const Grid3D g = make_grid(c->plan);
    const AeVolume v = ae_volume(g.P, g.ldz, g.sxy, g.npd, g.npd, g.npd, g.nz, g.nx, g.ny);
    GEO_CUDA(cudaMemsetAsync(c->ae->snapmax.p, 0, 4, c->s));
    k_ae_absmax<<<152 * 8, 256, 0, c->s>>>(v, c->ae->snapmax.as<unsigned>());
    GEO_TRY(check_launch("ae_absmax"));
    k_ae_collect<<<v.nbz * v.nbx * v.nby, 256, 0, c->s>>>(v, c->ae->snapmax.as<unsigned>(), c->rel,
                                                          c->ae->store.as<float>(), c->ae->wstore.as<float>(),
                                                          c->ae->cap,
                                                          c->ae->count.as<unsigned long long>());
    return check_launch("ae_collect");
}

extern "C" int geo_ae_add_shot(geo_ae *ae, geo_fd3d_plan *plan, int is, int snap_every, int t_first, float rel,
                               void *stream) {
    if (!ae || !plan || snap_every < 1 || t_first < 0) return fail(GEO_ERR_ARG, "bad argument");
    if (!ae->cap) return fail(GEO_ERR_ARG, "reserve the block store first");
    CollectCtx c{ae, plan, snap_every, t_first, rel, (cudaStream_t)stream};
    GEO_TRY(run_shot_3d(plan, is, c.s, collect_step, &c));
    GEO_CUDA(cudaStreamSynchronize(c.s));
    return GEO_OK;
}

// Forward (and backward) of the network on given blocks (Morton order, raw
// amplitudes): recon = normalized reconstruction, loss = mean squared error
// in normalized units, grad = d loss / d params (flat, like the params).
extern "C" int geo_ae_eval(geo_ae *ae, const float *blocks, int nb, float *recon, double *loss, float *grad,
                           int mem, void *stream) {
    if (!ae || !blocks || nb < 1) return fail(GEO_ERR_ARG, "bad argument");
    if (nb % 128) return fail(GEO_ERR_ARG, "block count must be a multiple of 128");
    cudaStream_t s = (cudaStream_t)stream;
    GEO_TRY(ensure_train(ae, nb));
    DevBuf in, rec;
    const float *src = blocks;
    if (mem != GEO_MEM_DEVICE) {
        GEO_TRY(in.alloc((size_t)nb * kAePts * 4));
        GEO_CUDA(cudaMemcpyAsync(in.p, blocks, (size_t)nb * kAePts * 4, cudaMemcpyHostToDevice, s));
        src = in.as<float>();
    }
    // device callers take the reconstruction straight from D1; the loss and
    // a zero step counter (the loss slot) share one small buffer
    float *prec = mem == GEO_MEM_DEVICE ? recon : nullptr;
    if (recon && !prec) {
        GEO_TRY(rec.alloc((size_t)nb * kAePts * 4));
        prec = rec.as<float>();
    }
    if (!ae->ev.p) GEO_TRY(ae->ev.alloc(16));
    GEO_TRY(ae->ev.zero(s));
    GEO_CUDA(cudaMemsetAsync(ae->grad.p, 0, ae->off.total * 4, s));
    GEO_CUDA(cudaMemsetAsync(ae->err.p, 0, 4, s));
    E1Args a = e1_args(ae, nb);
    a.direct = src;
    a.xn = ae->xn.as<float>();
    k_ae_e1<<<nb, 256, 0, s>>>(a);
    GEO_TRY(check_launch("ae_e1"));
    GEO_TRY(train_pass(ae, nb, ae->ev.as<double>(), nullptr, ae->ev.as<int>() + 2, 0, prec, grad != nullptr, s));
    const cudaMemcpyKind k = mem == GEO_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost;
    double l = 0;
    GEO_CUDA(cudaMemcpyAsync(&l, ae->ev.p, 8, cudaMemcpyDeviceToHost, s));
    GEO_TRY(ae_check_err(ae, s));
    if (recon && prec != recon) GEO_CUDA(cudaMemcpyAsync(recon, prec, (size_t)nb * kAePts * 4, k, s));
    if (grad) GEO_CUDA(cudaMemcpyAsync(grad, ae->grad.p, ae->off.total * 4, k, s));
    GEO_CUDA(cudaStreamSynchronize(s));
    if (loss) *loss = l / kAePts;
    return GEO_OK;
}

// iters Adam steps on batches of `batch` blocks drawn from the store;
// learning rate lr with a cosine decay to lr/20; loss[i] = the batch's mean
// squared error with each block weighted by (its max / its snapshot's max)^2.
extern "C" int geo_ae_train(geo_ae *ae, int iters, int batch, float lr, float *loss, void *stream) {
    if (!ae || iters < 1 || batch < 128 || batch % 128) return fail(GEO_ERR_ARG, "bad argument (batch %% 128)");
    const long long nstore = geo_ae_num_blocks(ae);
    if (nstore < 1) return fail(GEO_ERR_ARG, "the block store is empty");
    cudaStream_t s = nullptr;
    GEO_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    struct SG {
        cudaStream_t s;
        ~SG() { cudaStreamDestroy(s); }
    } sg{s};
    (void)stream;
    GEO_CUDA(cudaDeviceSynchronize());
    GEO_TRY(ensure_train(ae, batch));
    int step0 = 0;
    GEO_CUDA(cudaMemcpy(&step0, ae->step.p, 4, cudaMemcpyDeviceToHost));
    std::vector<float> lrs(iters);
    for (int i = 0; i < iters; i++)
        lrs[i] = (float)(lr * (0.05 + 0.95 * 0.5 * (1.0 + std::cos(3.141592653589793 * i / iters))));
    DevBuf dlr, dloss, dwsum;
    GEO_TRY(dlr.alloc((size_t)iters * 4));
    GEO_TRY(dloss.alloc((size_t)iters * 8));
    GEO_TRY(dwsum.alloc((size_t)iters * 4));
    GEO_TRY(dwsum.zero(s));
    GEO_CUDA(cudaMemcpyAsync(dlr.p, lrs.data(), (size_t)iters * 4, cudaMemcpyHostToDevice, s));
    GEO_TRY(dloss.zero(s));
    GEO_CUDA(cudaMemsetAsync(ae->err.p, 0, 4, s));
    auto iteration = [&]() -> int {
        GEO_CUDA(cudaMemsetAsync(ae->grad.p, 0, ae->off.total * 4, s));
        E1Args a = e1_args(ae, batch);
        a.store = ae->store.as<float>();
        a.nstore = nstore;
        a.xn = ae->xn.as<float>();
        a.wstore = ae->wstore.as<float>();
        a.wrow = ae->wrow.as<float>();
        a.wsum = dwsum.as<float>();
        a.step0 = step0;
        k_ae_e1<<<batch, 256, 0, s>>>(a);
        GEO_TRY(check_launch("ae_e1"));
        GEO_TRY(train_pass(ae, batch, dloss.as<double>(), dwsum.as<float>(), ae->step.as<int>(), step0, nullptr, true,
                           s));
        k_ae_adam<<<152 * 4, 256, 0, s>>>(ae->params.as<float>(), ae->grad.as<float>(), ae->m1.as<float>(),
                                          ae->m2.as<float>(), ae->off.total, ae->step.as<int>(), step0,
                                          dlr.as<float>());
        GEO_TRY(check_launch("ae_adam"));
        return ae_pack(ae, 1, s);
    };
    // first iteration eagerly (sets kernel attributes), the rest from a graph
    GEO_TRY(iteration());
    if (iters > 1) {
        const long long before = launches_so_far();
        cudaGraph_t graph = nullptr;
        GEO_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
        const int st = iteration();
        cudaError_t ce = cudaStreamEndCapture(s, &graph);
        if (st != GEO_OK) {
            if (graph) cudaGraphDestroy(graph);
            return st;
        }
        if (ce != cudaSuccess) return fail(GEO_ERR_CUDA, "graph capture: %s", cudaGetErrorString(ce));
        const long long per = launches_so_far() - before;
        count_launch(-per);
        cudaGraphExec_t exec = nullptr;
        ce = cudaGraphInstantiate(&exec, graph, 0);
        cudaGraphDestroy(graph);
        if (ce != cudaSuccess) return fail(GEO_ERR_CUDA, "graph instantiate: %s", cudaGetErrorString(ce));
        for (int i = 1; i < iters && ce == cudaSuccess; i++) {
            ce = cudaGraphLaunch(exec, s);
            count_launch(per);
        }
        cudaGraphExecDestroy(exec);
        if (ce != cudaSuccess) return fail(GEO_ERR_CUDA, "graph launch: %s", cudaGetErrorString(ce));
    }
    ae->wver++;   // the graph's packs changed the weights
    GEO_TRY(ae_check_err(ae, s));
    std::vector<double> l(iters);
    GEO_CUDA(cudaMemcpyAsync(l.data(), dloss.p, (size_t)iters * 8, cudaMemcpyDeviceToHost, s));
    GEO_CUDA(cudaStreamSynchronize(s));
    if (loss)
        for (int i = 0; i < iters; i++) loss[i] = (float)(l[i] / kAePts);
    return GEO_OK;
}

void geo::ae_note_run(geo_ae *ae, long long blocks, long long escaped) {
    ae->st_blocks += blocks;
    ae->st_escaped += escaped;
}

// Coded and escaped blocks over the RTM shots run with this codec.
extern "C" int geo_ae_stats(geo_ae *ae, long long *blocks, long long *escaped) {
    if (!ae) return fail(GEO_ERR_ARG, "null codec");
    if (blocks) *blocks = ae->st_blocks;
    if (escaped) *escaped = ae->st_escaped;
    return GEO_OK;
}

// Escape settings: per snapshot, the (at most frac of all) blocks with the
// largest squared decoding error, among those whose error exceeds tau times
// their norm, keep their residual.
extern "C" int geo_ae_set_escape(geo_ae *ae, float tau, float frac) {
    if (!ae || !(tau >= 0) || !(frac >= 0) || frac > 1) return fail(GEO_ERR_ARG, "bad argument");
    ae->tau = tau;
    ae->frac = frac;
    return GEO_OK;
}

// Encode + decode a dense nz-fastest volume (nx*ny*nz, layout
// iz + nz*(ix + nx*iy), device pointers): out = the codec's reconstruction
// (with escapes when `escape`); *nesc (optional) = escaped blocks.
extern "C" int geo_ae_roundtrip(geo_ae *ae, int nx, int ny, int nz, const float *vol, float *out, int escape,
                                int *nesc, void *stream) {
    if (!ae || !vol || !out || nx < 1 || ny < 1 || nz < 1) return fail(GEO_ERR_ARG, "bad argument");
    cudaStream_t s = (cudaStream_t)stream;
    const AeVolume v = ae_volume(vol, nz, (long)nz * nx, 0, 0, 0, nz, nx, ny);
    const int rows = ae_code_rows(v), cap = ae_escape_cap(ae, v);
    DevBuf esc, res, cnt;
    // the code and its scales stay in the codec's own scratch
    GEO_TRY(ensure_rows(ae, rows));
    void *code = ae->z.p;
    float *scale = ae->scale.as<float>();
    if (escape) {
        GEO_TRY(esc.alloc((size_t)rows * 4));
        GEO_TRY(res.alloc((size_t)std::max(cap, 1) * kAePts * 2));
        GEO_TRY(cnt.alloc(16));
        GEO_TRY(cnt.zero(s));
    }
    GEO_CUDA(cudaMemsetAsync(ae->err.p, 0, 4, s));
    GEO_TRY(ae_encode_volume(ae, v, code, scale, esc.as<int>(), res.p, cnt.as<int>(), s));
    GEO_TRY(ae_decode_volume(ae, v, code, scale, esc.as<int>(), res.p, 0, out, nullptr, nullptr, 0.0f,
                             s));
    if (nesc) {
        *nesc = 0;
        if (escape) GEO_CUDA(cudaMemcpyAsync(nesc, cnt.p, 4, cudaMemcpyDeviceToHost, s));
    }
    return ae_check_err(ae, s);
}

// tcgen05 BF16 GEMM with FP32 accumulation in tensor memory.
//
// One CTA computes a 128 x BN tile of C = A * B^T.  Four warps:
//   warp 0 lane 0  TMA producer: per 64-wide K slice, one 128x64 tile of A
//                  and one BNx64 tile of B (128-byte swizzle) into a
//                  2- to 4-stage ring, one "full" mbarrier per stage;
//   warp 1 lane 0  MMA issuer: four tcgen05.mma (K = 16 each) per slice
//                  into a 128 x BN fp32 accumulator in TMEM; tcgen05.commit
//                  to the stage's "empty" mbarrier releases it to the
//                  producer, a final commit signals the epilogue;
//   all 4 warps    epilogue: warp w reads TMEM lanes 32w..32w+31 (rows) with
//                  tcgen05.ld, adds the bias, applies the activation or the
//                  activation-derivative gate, and stores fp32, or bf16
//                  staged in the freed ring and written back as whole rows.
// Every wait is bounded (2 s): on timeout the CTA sets the error word, lets
// its copies in flight land (bounded), frees its TMEM and returns.
#include "geo_internal.h"
#include "tc_util.cuh"
#include "tc_gemm.cuh"
#include <algorithm>
#include <cudaTypedefs.h>

namespace geo {
using namespace tc;

constexpr int kGM = 128, kGK = 64;

// Stage ring sized so two CTAs fit on an SM (one's epilogue overlaps the
// other's main loop): 2 stages for BN 256, 3 for 128, 4 for 64.  A GEMM
// with fewer K slices than that gets as many stages as slices (ST), so that
// more CTAs share an SM and more tiles are in flight: the skinny codec
// levels (K = 64, 128) have one or two slices per tile.  The shared memory
// is then padded so that no more of a launch's CTAs fit than tensor memory
// holds accumulators for (512 columns per SM), so none of them waits for
// another.  A CTA launched early can find its predecessor's CTAs still holding
// columns and wait in its allocation; that ends, since every predecessor CTA
// has allocated before it lets a successor come and needs nothing of it.
constexpr int default_stages(int bn) { return bn >= 256 ? 2 : (bn >= 128 ? 3 : 4); }
// GEMMs of few tiles take narrow ones with a deep ring instead (launch_bn_k).
constexpr int kDeepStages = 8;
constexpr size_t kSmSmem = 233472;      // shared memory per SM
constexpr size_t kCtaReserve = 1024;    // reserved per resident CTA

template <int BN, int ST = default_stages(BN)>
struct GemmShape {
    static constexpr int kA = kGM * kGK * 2;
    static constexpr int kB = BN * kGK * 2;
    static constexpr int kStage = kA + kB;
    static constexpr int kStages = ST;
    static constexpr uint32_t kCols = BN < 32 ? 32 : BN;
    // the ring, reused after the last MMA as the bf16 output tile
    static constexpr size_t kOut = (size_t)kGM * BN * 2;
    static constexpr size_t kData = (size_t)kStages * kStage > kOut ? (size_t)kStages * kStage : kOut;
    static constexpr size_t kRing = kData + 1024 + 256;
    // fewest bytes with which at most 512 / kCols CTAs fit on an SM
    static constexpr size_t kFloor = kSmSmem / (512 / kCols + 1) + 1 - kCtaReserve;
    static constexpr size_t kSmem = kRing > kFloor ? kRing : kFloor;
    static_assert(kA % 1024 == 0 && kB % 1024 == 0, "swizzle atoms stay 1024-byte aligned");
    static_assert(BN % 16 == 0 && BN >= 16 && BN <= 256, "UMMA N for M = 128");
    static_assert(ST >= 1 && (ST <= default_stages(BN) || ST == kDeepStages), "stage count");
    static_assert((ST == kDeepStages ? 1 : 2) * kSmem <= 232448, "two CTAs per SM, or one with the deep ring");
    static_assert((kSmSmem / (kSmem + kCtaReserve)) * kCols <= 512, "resident CTAs' accumulators fit in TMEM");
};

// max(v, kLeak v) = (v > 0 ? v : kLeak v) for 0 < kLeak < 1, one instruction fewer
__device__ __forceinline__ float leaky(float v) { return fmaxf(v, kLeak * v); }

template <int BN, int ST>
__global__ void __launch_bounds__(128, 2)
    k_tc_gemm(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, const TcGemm g) {
    using S = GemmShape<BN, ST>;
    extern __shared__ unsigned char smem_raw[];
    uint8_t *sm = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr int kGStages = S::kStages;
    uint64_t *full = reinterpret_cast<uint64_t *>(sm + S::kData);
    uint64_t *empty = full + kGStages;
    uint64_t *done = empty + kGStages;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(done + 1);
    __shared__ int s_abort;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // consecutive CTAs share a row tile of A (its second and later reads hit L2)
    const int ntn = g.N / BN;
    const int m0 = (int)(blockIdx.x / ntn) * kGM, n0 = (int)(blockIdx.x % ntn) * BN;
    const int nk = g.K / kGK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kGStages; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(done, 1);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(tslot, S::kCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    after_predecessor();

    if (warp == 0 && lane == 0) {
        // producer
        int issued = 0;
        for (int kb = 0; kb < nk; kb++) {
            const int s = kb % kGStages;
            if (kb >= kGStages && !mbar_wait(&empty[s], ((kb / kGStages) - 1) & 1)) {
                s_abort = 1;
                break;
            }
            uint8_t *st = sm + s * S::kStage;
            mbar_expect_tx(&full[s], S::kStage);
            tma2(st, &ta, kb * kGK, m0, &full[s]);
            tma2(st + S::kA, &tb, kb * kGK, n0, &full[s]);
            issued = kb + 1;
        }
        // after a failure, let the copies still in flight land (bounded)
        if (*(volatile int *)&s_abort)
            for (int kb = issued > kGStages ? issued - kGStages : 0; kb < issued; kb++)
                mbar_wait(&full[kb % kGStages], (kb / kGStages) & 1);
    } else if (warp == 1 && lane == 0) {
        // MMA issuer
        constexpr uint32_t idesc = idesc_bf16_f32(kGM, BN);
        for (int kb = 0; kb < nk; kb++) {
            const int s = kb % kGStages;
            if (!mbar_wait(&full[s], (kb / kGStages) & 1)) {
                s_abort = 1;
                break;
            }
            tc_fence_after();
            const uint32_t a0 = su32(sm + s * S::kStage), b0 = a0 + S::kA;
#pragma unroll
            for (int k = 0; k < kGK / 16; k++)
                mma_bf16(tmem, sdesc_k128(a0 + k * 32), sdesc_k128(b0 + k * 32), idesc, (kb | k) != 0);
            mma_commit(&empty[s]);
        }
        mma_commit(done);  // arrives once every MMA issued above has completed
    }
    __syncwarp();

    // epilogue.  bf16 output goes through shared memory (the ring is free
    // once every MMA has completed): each warp stages its 32 rows with the
    // 16-byte chunks of a row XOR-swizzled by the row (conflict-free in both
    // directions), then writes them back as whole rows, consecutive lanes on
    // consecutive 16-byte chunks.
    if (!mbar_wait(done, 0)) s_abort = 1;
    tc_fence_after();
    const int row = m0 + warp * 32 + lane;
    const bool ok = !*(volatile int *)&s_abort;
    uint4 *stg = reinterpret_cast<uint4 *>(sm + (size_t)warp * 32 * BN * 2);
    constexpr int CPR = BN / 8;   // 16-byte chunks per output row
#pragma unroll 1
    for (int c0 = 0; c0 < BN; c0 += 16) {
        uint32_t r[16];
        tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, r);
        if (!ok) continue;
        const int n = n0 + c0;
        float v[16];
#pragma unroll
        for (int j = 0; j < 16; j++) v[j] = __uint_as_float(r[j]);
        if (g.bias) {
#pragma unroll
            for (int j = 0; j < 16; j++) v[j] += g.bias[n + j];
        }
        if (g.act) {
#pragma unroll
            for (int j = 0; j < 16; j++) v[j] = leaky(v[j]);
        }
        const long o = (long)row * g.N + n;
        if (g.gate) {
            const uint4 *gp = reinterpret_cast<const uint4 *>(g.gate + o);
            uint4 q[2] = {gp[0], gp[1]};
            const __nv_bfloat16 *gb = reinterpret_cast<const __nv_bfloat16 *>(q);
#pragma unroll
            for (int j = 0; j < 16; j++) v[j] = __bfloat162float(gb[j]) > 0.0f ? v[j] : kLeak * v[j];
        }
        if (g.out_f32) {
            float4 *op = reinterpret_cast<float4 *>(static_cast<float *>(g.out) + o);
#pragma unroll
            for (int j = 0; j < 4; j++) op[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        } else {
            uint4 q[2];
            __nv_bfloat162 *q2 = reinterpret_cast<__nv_bfloat162 *>(q);
#pragma unroll
            for (int j = 0; j < 8; j++) q2[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
            const int q0 = c0 / 8;
            stg[lane * CPR + (q0 ^ (lane & 7))] = q[0];
            stg[lane * CPR + ((q0 + 1) ^ (lane & 7))] = q[1];
        }
    }
    if (ok && !g.out_f32) {
        __syncwarp();
        __nv_bfloat16 *out = static_cast<__nv_bfloat16 *>(g.out) + (long)(m0 + warp * 32) * g.N + n0;
#pragma unroll 4
        for (int it = 0; it < CPR; it++) {
            const int idx = it * 32 + lane, rl = idx / CPR, q = idx % CPR;
            reinterpret_cast<uint4 *>(out + (long)rl * g.N)[q] = stg[rl * CPR + (q ^ (rl & 7))];
        }
    }
    tc_fence_before();
    __syncthreads();
    if (s_abort && threadIdx.x == 0) atomicExch(g.err, 2);
    if (warp == 0) tmem_dealloc(tmem, S::kCols);
}

// ------------------------------------------------------------- many tiles
// The same product with bf16 output, a bias and an activation, for GEMMs of
// more tiles than SMs: one persistent CTA per SM walks 128 x BN tiles with ten
// warps of fixed roles, so that loads, MMAs and epilogues of consecutive tiles
// overlap:
//   warp 8 lane 0  TMA producer over a ring of K slices that runs on across
//                  tiles;
//   warp 9 lane 0  MMA issuer into two TMEM accumulators in turn;
//   warps 0-3, 4-7 epilogues of the even and of the odd tiles: warp w reads
//                  lanes 32(w & 3).. of its accumulator 64 columns at a time,
//                  adds the bias, applies the activation, and sends 32 x 64
//                  bf16 boxes out by TMA stores from two buffers of its own.
// RB: B (one tile wide, up to 32 KB) stays in shared memory for the run.
// Bound by memory where K is small and by the ring's L2 reads (48 KB a slice)
// where it is large.  A 512x512x384 snapshot's levels (24 576 blocks): the four
// 256-wide ones 213 us against 357 with a CTA per tile, whose epilogue two
// resident CTAs hid only in part; D2 101 against 128; E2 91 against 105 (6.6
// TB/s).
// Every wait is bounded; a role that gives up sets the error word and ends,
// after which the others' waits run out too.
template <int BN, bool RB>
struct WalkShape {
    static constexpr int kA = kGM * kGK * 2, kB = BN * kGK * 2;
    static constexpr int kStage = kA + (RB ? 0 : kB);
    static constexpr int kStages = RB ? 6 : 3;
    static constexpr int kRes = RB ? 32768 : 0;          // resident B
    static constexpr int kStg = 8 * 2 * 4096;            // two store buffers a warp
    static constexpr int kMaxN = 2048;                   // bias floats
    static constexpr size_t kData = (size_t)kRes + (size_t)kStages * kStage + kStg;
    static constexpr size_t kSmem = kData + kMaxN * 4 + 256 + 1024;
    static_assert(kSmem <= 232448, "one CTA per SM");
    static_assert(2 * BN <= 512, "two accumulators fit in TMEM");
};
constexpr int kWalkThreads = 320;

template <int BN, bool RB>
__global__ void __launch_bounds__(kWalkThreads, 1)
    k_tc_walk(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb,
              const __grid_constant__ CUtensorMap to, const TcGemm g, int tiles) {
    using S = WalkShape<BN, RB>;
    constexpr int ST = S::kStages;
    extern __shared__ unsigned char smem_raw[];
    uint8_t *sm = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *ring = sm + S::kRes, *stg = ring + (size_t)ST * S::kStage;
    float *sbias = reinterpret_cast<float *>(sm + S::kData);
    uint64_t *full = reinterpret_cast<uint64_t *>(sbias + S::kMaxN), *empty = full + ST;
    uint64_t *acc_full = empty + ST, *acc_empty = acc_full + 2, *b_full = acc_empty + 2;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(b_full + 1);
    __shared__ int s_abort;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ntn = g.N / BN, nk = g.K / kGK;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], 4);
        }
        mbar_init(b_full, 1);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == 9) tmem_alloc(tslot, 2 * BN < 32 ? 32 : 2 * BN);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    after_predecessor();
    for (int n = threadIdx.x; n < g.N; n += kWalkThreads) sbias[n] = g.bias ? g.bias[n] : 0.0f;
    __syncthreads();

    if (warp == 8 && lane == 0) {
        bool ok = true;
        unsigned it = 0;   // slices issued
        if (RB) {
            mbar_expect_tx(b_full, nk * S::kB);
            for (int kb = 0; kb < nk; kb++) tma2(sm + kb * S::kB, &tb, kb * kGK, 0, b_full);
        }
        for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
            const int m0 = t / ntn * kGM, n0 = t % ntn * BN;
            for (int kb = 0; kb < nk && ok; kb++, it++) {
                const unsigned s = it % ST;
                if (it >= ST && !mbar_wait(&empty[s], (it / ST - 1) & 1)) {
                    s_abort = 1;
                    ok = false;
                    break;
                }
                uint8_t *st = ring + s * S::kStage;
                mbar_expect_tx(&full[s], S::kStage);
                tma2(st, &ta, kb * kGK, m0, &full[s]);
                if (!RB) tma2(st + S::kA, &tb, kb * kGK, n0, &full[s]);
            }
        }
        // after a failure, let the copies still in flight land (bounded)
        if (!ok)
            for (unsigned k = it > ST ? it - ST : 0; k < it; k++) mbar_wait(&full[k % ST], (k / ST) & 1);
        if (RB && !ok) mbar_wait(b_full, 0);
    } else if (warp == 9 && lane == 0) {
        constexpr uint32_t idesc = idesc_bf16_f32(kGM, BN);
        bool ok = true;
        unsigned it = 0, i = 0;
        if (RB && !mbar_wait(b_full, 0)) ok = false;
        for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, i++) {
            const unsigned ab = i & 1, use = i >> 1;
            if (use && !mbar_wait(&acc_empty[ab], (use - 1) & 1)) {
                ok = false;
                break;
            }
            tc_fence_after();
            for (int kb = 0; kb < nk; kb++, it++) {
                const unsigned s = it % ST;
                if (!mbar_wait(&full[s], (it / ST) & 1)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
                const uint32_t a0 = su32(ring + s * S::kStage), b0 = RB ? su32(sm + kb * S::kB) : a0 + S::kA;
#pragma unroll
                for (int k = 0; k < kGK / 16; k++)
                    mma_bf16(tmem + ab * BN, sdesc_k128(a0 + k * 32), sdesc_k128(b0 + k * 32), idesc, (kb | k) != 0);
                mma_commit(&empty[s]);
            }
            mma_commit(&acc_full[ab]);
        }
        if (!ok) s_abort = 1;
    } else if (warp < 8) {
        const int grp = warp >> 2, quad = warp & 3;
        uint8_t *buf = stg + warp * 8192;
        unsigned i = 0, stores = 0;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x, i++) {
            if ((int)(i & 1) != grp) continue;
            const int m0 = t / ntn * kGM + quad * 32, n0 = t % ntn * BN;
            if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[grp], (i >> 1) & 1))) {
                s_abort = 1;
                break;
            }
            tc_fence_after();
            const uint32_t ta0 = tmem + ((uint32_t)(quad * 32) << 16) + grp * BN;
#pragma unroll 1
            for (int c = 0; c < BN; c += 64, stores++) {
                uint32_t r[64];
                tmem_ld32(ta0 + c, r);
                tmem_ld32(ta0 + c + 32, r + 32);
                tmem_ld_wait();
                if (c + 64 == BN) {   // the accumulator is in registers: the issuer may have it
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[grp]);
                }
                uint8_t *b = buf + (stores & 1) * 4096;
                // this buffer's store, two back, has left
                if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                __syncwarp();
                const float4 *bp = reinterpret_cast<const float4 *>(sbias + n0 + c);
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    const float4 u = bp[2 * q], w = bp[2 * q + 1];
                    const float bb[8] = {u.x, u.y, u.z, u.w, w.x, w.y, w.z, w.w};
                    uint4 o;
                    __nv_bfloat162 *o2 = reinterpret_cast<__nv_bfloat162 *>(&o);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        float v0 = __uint_as_float(r[8 * q + 2 * j]), v1 = __uint_as_float(r[8 * q + 2 * j + 1]);
                        if (g.bias) {
                            v0 += bb[2 * j];
                            v1 += bb[2 * j + 1];
                        }
                        if (g.act) {
                            v0 = leaky(v0);
                            v1 = leaky(v1);
                        }
                        o2[j] = __floats2bfloat162_rn(v0, v1);
                    }
                    *reinterpret_cast<uint4 *>(b + lane * 128 + ((q ^ (lane & 7)) << 4)) = o;
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) {
                    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                                     reinterpret_cast<uint64_t>(&to)),
                                 "r"(su32(b)), "r"(n0 + c), "r"(m0)
                                 : "memory");
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                }
            }
        }
        if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (s_abort && threadIdx.x == 0) atomicExch(g.err, 2);
    if (warp == 9) tmem_dealloc(tmem, 2 * BN < 32 ? 32 : 2 * BN);
}

static PFN_cuTensorMapEncodeTiled_v12000 g_enc2 = nullptr;

int tc_map_bf16(CUtensorMap *map, const void *base, int rows, int cols, int box_rows) {
    if (!g_enc2) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        GEO_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q));
        if (!fn || q != cudaDriverEntryPointSuccess) return fail(GEO_ERR_CUDA, "cuTensorMapEncodeTiled unavailable");
        g_enc2 = (PFN_cuTensorMapEncodeTiled_v12000)fn;
    }
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = g_enc2(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(GEO_ERR_CUDA, "cuTensorMapEncodeTiled (bf16) failed (%d)", (int)r);
    return GEO_OK;
}

template <int BN, int ST>
static int launch_bn(const TcGemm &g, cudaStream_t s) {
    using S = GemmShape<BN, ST>;
    static OncePerDevice once;
    GEO_TRY(allow_smem(once, (const void *)k_tc_gemm<BN, ST>, S::kSmem));
    CUtensorMap ta, tb;
    GEO_TRY(tc_map_bf16(&ta, g.A, g.M, g.K, kGM));
    GEO_TRY(tc_map_bf16(&tb, g.B, g.N, g.K, BN));
    const dim3 grid((unsigned)(g.M / kGM) * (unsigned)(g.N / BN));
    GEO_CUDA(launch_early(k_tc_gemm<BN, ST>, grid.x, 128, S::kSmem, s, ta, tb, g));
    return check_launch("tc_gemm");
}

template <int BN, bool RB>
static int launch_walk(const TcGemm &g, cudaStream_t s) {
    using S = WalkShape<BN, RB>;
    static OncePerDevice once;
    GEO_TRY(allow_smem(once, (const void *)k_tc_walk<BN, RB>, S::kSmem));
    CUtensorMap ta, tb, to;
    GEO_TRY(tc_map_bf16(&ta, g.A, g.M, g.K, kGM));
    GEO_TRY(tc_map_bf16(&tb, g.B, g.N, g.K, BN));
    GEO_TRY(tc_map_bf16(&to, g.out, g.M, g.N, 32));
    const int tiles = (g.M / kGM) * (g.N / BN);
    GEO_CUDA(launch_early(k_tc_walk<BN, RB>, std::min(tiles, sm_count()), kWalkThreads, S::kSmem, s, ta, tb, to, g, tiles));
    return check_launch("tc_walk");
}

// Tile width: the widest that divides N and leaves a tile for every SM,
// else 64.  A training batch of 256 blocks has 4 to 32 tiles of width 256
// (E4: 4 CTAs walking 32 K slices each behind a two-slot ring), so the chip
// idles and a slice costs a full memory latency; with width 64 and, where
// no more than one CTA lands on an SM anyway, an eight-slot ring, the ten
// input and output GEMMs of such an evaluation take 80 us instead of
// 145 us.  From 152 tiles on the wide tile's fewer operand reads win, and
// k_tc_walk takes what it handles (bf16 out, no gate).
constexpr long kFewTiles = 152;

// stages = K slices, up to the tile width's default
template <int BN>
static int launch_bn_k(const TcGemm &g, cudaStream_t s) {
    const int nk = g.K / kGK;
    if constexpr (BN == 64)
        if (nk > 4 && (long)(g.M / kGM) * (g.N / BN) <= kFewTiles) return launch_bn<BN, kDeepStages>(g, s);
    if constexpr (default_stages(BN) >= 4)
        if (nk >= 4) return launch_bn<BN, 4>(g, s);
    if constexpr (default_stages(BN) >= 3)
        if (nk >= 3) return launch_bn<BN, (default_stages(BN) >= 3 ? 3 : 1)>(g, s);
    if (nk >= 2) return launch_bn<BN, 2>(g, s);
    return launch_bn<BN, 1>(g, s);
}

int tc_gemm(const TcGemm &g, cudaStream_t s) {
    if (g.M <= 0 || g.N <= 0 || g.K <= 0 || g.M % kGM || g.N % 64 || g.K % kGK)
        return fail(GEO_ERR_ARG, "tc_gemm: M %% 128, N %% 64 and K %% 64 must be 0 (M=%d N=%d K=%d)", g.M, g.N, g.K);
    if (!g.A || !g.B || !g.out || !g.err) return fail(GEO_ERR_ARG, "tc_gemm: null pointer");
    const uintptr_t al = reinterpret_cast<uintptr_t>(g.A) | reinterpret_cast<uintptr_t>(g.B) |
                         reinterpret_cast<uintptr_t>(g.out) | reinterpret_cast<uintptr_t>(g.gate);
    if (al & 15) return fail(GEO_ERR_ARG, "tc_gemm: operands must be 16-byte aligned");
    const long mt = g.M / kGM;
    if (!g.gate && !g.out_f32 && g.N <= WalkShape<256, false>::kMaxN) {
        if (g.N % 256 == 0 && mt * (g.N / 256) >= kFewTiles) return launch_walk<256, false>(g, s);
        if (g.N == 128 && g.K <= 128 && mt >= kFewTiles) return launch_walk<128, true>(g, s);
        if (g.N == 64 && g.K <= 256 && mt >= kFewTiles) return launch_walk<64, true>(g, s);
    }
    if (g.N % 256 == 0 && mt * (g.N / 256) >= kFewTiles) return launch_bn_k<256>(g, s);
    if (g.N % 128 == 0 && mt * (g.N / 128) >= kFewTiles) return launch_bn_k<128>(g, s);
    return launch_bn_k<64>(g, s);
}

// ---------------------------------------------------------- weight gradients
// dW = dY^T X of every codec level in one launch.  The contraction runs over
// the rows, which are the slow dimension of both operands in memory, so both
// are handed to tcgen05.mma MN-major: a TMA box of 64 rows x 64 columns is a
// swizzled operand slice as it lies.  A CTA owns a 128 x (64 or 128) tile of
// one level's dW and a range of 64-row slices (three-stage TMA ring, the same
// roles and bounded waits as k_tc_gemm) and adds its tile to the gradient
// with vector reductions.  The levels have 1 to 64 tiles and 4 to 256 slices
// at 256 blocks; the slices of a tile are split so that each level fills the
// chip once (kWgradCtas), and all levels share the launch, which leaves one
// partial wave instead of six.  Bound by latency and by the reductions (a
// few MB into L2), not by the tensor cores (7 GFLOP, 4 us at peak).
// 256 blocks: 19.7 us, against 197 us for six CUDA-core launches.
struct WgradItem {
    float *out;
    long sa, sb;
    int base, tb, splits, slices, bn;   // first CTA, tiles along b, splits, slices in all, tile width
};
struct WgradArgs {
    CUtensorMap ta[kWgradMax], tb[kWgradMax];
    WgradItem it[kWgradMax];
    int n;
    int *err;
};

constexpr int kWgStages = 3, kWgBox = 64 * 128, kWgA = 2 * kWgBox, kWgStage = 4 * kWgBox;
constexpr size_t kWgSmem = (size_t)kWgStages * kWgStage + 1024 + 128;
constexpr int kWgradCtas = 128;
static_assert(2 * kWgSmem <= 232448 && 2 * 128 <= 512, "two CTAs per SM");

__device__ __forceinline__ void red_add4(float *p, float a, float b, float c, float d) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c), "f"(d)
                 : "memory");
}

__global__ void __launch_bounds__(128, 2) k_tc_wgrad(const __grid_constant__ WgradArgs g) {
    extern __shared__ unsigned char smem_raw[];
    uint8_t *sm = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(sm + (size_t)kWgStages * kWgStage);
    uint64_t *empty = full + kWgStages;
    uint64_t *done = empty + kWgStages;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(done + 1);
    __shared__ int s_abort;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int l = 0;
    while (l + 1 < g.n && (int)blockIdx.x >= g.it[l + 1].base) l++;
    const WgradItem &w = g.it[l];
    const int rel = (int)blockIdx.x - w.base, tile = rel / w.splits, sp = rel % w.splits;
    const int a0 = (tile / w.tb) * 128, b0 = (tile % w.tb) * w.bn;
    const int s0 = (int)((long)w.slices * sp / w.splits), nk = (int)((long)w.slices * (sp + 1) / w.splits) - s0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kWgStages; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(done, 1);
        s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(tslot, 128);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;
    after_predecessor();
    const int nbox = w.bn / 64;

    if (warp == 0 && lane == 0) {
        int issued = 0;
        for (int kb = 0; kb < nk; kb++) {
            const int s = kb % kWgStages;
            if (kb >= kWgStages && !mbar_wait(&empty[s], ((kb / kWgStages) - 1) & 1)) {
                s_abort = 1;
                break;
            }
            uint8_t *st = sm + s * kWgStage;
            const int m = (s0 + kb) * 64;
            mbar_expect_tx(&full[s], (2 + nbox) * kWgBox);
            tma2(st, &g.ta[l], a0, m, &full[s]);
            tma2(st + kWgBox, &g.ta[l], a0 + 64, m, &full[s]);
            for (int q = 0; q < nbox; q++) tma2(st + kWgA + q * kWgBox, &g.tb[l], b0 + 64 * q, m, &full[s]);
            issued = kb + 1;
        }
        if (*(volatile int *)&s_abort)
            for (int kb = issued > kWgStages ? issued - kWgStages : 0; kb < issued; kb++)
                mbar_wait(&full[kb % kWgStages], (kb / kWgStages) & 1);
    } else if (warp == 1 && lane == 0) {
        const uint32_t idesc = idesc_bf16_f32_mn(128, w.bn);
        for (int kb = 0; kb < nk; kb++) {
            const int s = kb % kWgStages;
            if (!mbar_wait(&full[s], (kb / kWgStages) & 1)) {
                s_abort = 1;
                break;
            }
            tc_fence_after();
            const uint32_t pa = su32(sm + s * kWgStage), pb = pa + kWgA;
#pragma unroll
            for (int k = 0; k < 4; k++)
                mma_bf16(tmem, sdesc_mn128(pa + k * 2048, kWgBox), sdesc_mn128(pb + k * 2048, kWgBox), idesc,
                         (kb | k) != 0);
            mma_commit(&empty[s]);
        }
        mma_commit(done);
    }
    __syncwarp();

    if (!mbar_wait(done, 0)) s_abort = 1;
    tc_fence_after();
    const bool ok = !*(volatile int *)&s_abort;
    float *row = w.out + (long)(a0 + warp * 32 + lane) * w.sa + (long)b0 * w.sb;
#pragma unroll 1
    for (int c0 = 0; c0 < w.bn; c0 += 16) {
        uint32_t r[16];
        tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, r);
        if (!ok) continue;
        if (w.sb == 1) {
#pragma unroll
            for (int j = 0; j < 16; j += 4)
                red_add4(row + c0 + j, __uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]),
                         __uint_as_float(r[j + 3]));
        } else {
#pragma unroll
            for (int j = 0; j < 16; j++) atomicAdd(row + (long)(c0 + j) * w.sb, __uint_as_float(r[j]));
        }
    }
    tc_fence_before();
    __syncthreads();
    if (s_abort && threadIdx.x == 0) atomicExch(g.err, 2);
    if (warp == 0) tmem_dealloc(tmem, 128);
}

int tc_wgrad(const TcWgradLevel *lv, int n, int *err, cudaStream_t s) {
    if (n < 1 || n > kWgradMax || !err) return fail(GEO_ERR_ARG, "tc_wgrad: 1 to %d levels", kWgradMax);
    WgradArgs g;
    int base = 0;
    for (int l = 0; l < n; l++) {
        const TcWgradLevel &L = lv[l];
        if (L.M <= 0 || L.M % 64 || L.wa % 128 || (L.wb != 64 && L.wb % 128) || !L.A || !L.B || !L.out ||
            (L.sa != 1 && L.sb != 1) || (L.sa * L.sb) % 4)
            return fail(GEO_ERR_ARG, "tc_wgrad: bad level (M=%d wa=%d wb=%d)", L.M, L.wa, L.wb);
        if ((reinterpret_cast<uintptr_t>(L.A) | reinterpret_cast<uintptr_t>(L.B) |
             reinterpret_cast<uintptr_t>(L.out)) & 15)
            return fail(GEO_ERR_ARG, "tc_wgrad: operands must be 16-byte aligned");
        GEO_TRY(tc_map_bf16(&g.ta[l], L.A, L.M, L.wa, 64));
        GEO_TRY(tc_map_bf16(&g.tb[l], L.B, L.M, L.wb, 64));
        WgradItem &w = g.it[l];
        w.out = L.out;
        w.sa = L.sa;
        w.sb = L.sb;
        w.bn = L.wb == 64 ? 64 : 128;
        w.tb = L.wb / w.bn;
        w.slices = L.M / 64;
        const int tiles = (L.wa / 128) * w.tb;
        w.splits = (kWgradCtas + tiles - 1) / tiles;
        if (w.splits > w.slices) w.splits = w.slices;
        w.base = base;
        base += tiles * w.splits;
    }
    g.n = n;
    g.err = err;
    static OncePerDevice once;
    GEO_TRY(allow_smem(once, (const void *)k_tc_wgrad, kWgSmem));
    GEO_CUDA(launch_early(k_tc_wgrad, base, 128, kWgSmem, s, g));
    return check_launch("tc_wgrad");
}

}  // namespace geo

// C-ABI entry for tests and callers with their own bf16 operands (device
// pointers): out[M x N] = A[M x K] * B[N x K]^T (+bias, leaky ReLU).
extern "C" int geo_tc_gemm_bf16(int M, int N, int K, const void *A, const void *B, const float *bias, int act,
                                void *out, int out_f32, void *stream) {
    using namespace geo;
    DevBuf err;
    GEO_TRY(err.alloc(16));
    cudaStream_t s = (cudaStream_t)stream;
    GEO_TRY(err.zero(s));
    TcGemm g{};
    g.M = M; g.N = N; g.K = K;
    g.A = static_cast<const __nv_bfloat16 *>(A);
    g.B = static_cast<const __nv_bfloat16 *>(B);
    g.bias = bias;
    g.act = act;
    g.out = out;
    g.out_f32 = out_f32;
    g.err = err.as<int>();
    GEO_TRY(tc_gemm(g, s));
    int e = 0;
    GEO_CUDA(cudaMemcpyAsync(&e, err.p, 4, cudaMemcpyDeviceToHost, s));
    GEO_CUDA(cudaStreamSynchronize(s));
    if (e) return fail(GEO_ERR_CUDA, "tc_gemm: a pipeline wait timed out");
    return GEO_OK;
}

// BF16 tensor-core GEMM (tcgen05, TMEM accumulator, TMA-fed) used by the
// snapshot codec: C[M x N] = A[M x K] * B[N x K]^T with a fused epilogue.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>

namespace geo {

struct TcGemm {
    int M, N, K;                      // M % 128 == 0, N % 64 == 0, K % 64 == 0
    const __nv_bfloat16 *A;           // [M x K] row-major (K contiguous)
    const __nv_bfloat16 *B;           // [N x K] row-major
    const float *bias;                // [N] or null
    int act;                          // 1: leaky ReLU (slope kLeak) after the bias
    const __nv_bfloat16 *gate;        // [M x N] or null: multiply by the leaky-ReLU
                                      // derivative taken at gate's sign
    void *out;                        // [M x N] row-major
    int out_f32;                      // 1: fp32 output, 0: bf16 (round to nearest even)
    int *err;                         // device error word (wait timeouts)
};

constexpr float kLeak = 0.1f;

int tc_gemm(const TcGemm &g, cudaStream_t s);

// TMA map over a row-major [rows x cols] bf16 matrix, boxes of box_rows x 64
// columns (128 bytes), 128-byte swizzle.
int tc_map_bf16(CUtensorMap *map, const void *base, int rows, int cols, int box_rows);

// Weight gradients of up to kWgradMax levels in one launch: for each,
// out[a*sa + b*sb] += sum over m < M of A[m*wa + a] * B[m*wb + b].
struct TcWgradLevel {
    int M;                            // rows, M % 64 == 0
    const __nv_bfloat16 *A, *B;       // [M x wa], [M x wb] row-major
    int wa, wb;                       // wa % 128 == 0, wb == 64 or wb % 128 == 0
    float *out;                       // fp32, accumulated into; 16-byte aligned
    long sa, sb;                      // one of them 1
};
constexpr int kWgradMax = 6;

int tc_wgrad(const TcWgradLevel *lv, int n, int *err, cudaStream_t s);

}  // namespace geo

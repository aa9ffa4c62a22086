// Fused 3D VTI time step: shared declarations between the plan (fd3d.cu)
// and the y-marching TMA kernel (fd3d_fused.cu).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace geo {

// Tensor maps of one step's boxes: per time level 0 P x-halo box, 1 Q z-halo
// box, 2 u x-halo box, 3 w z-halo box; then the model's own boxes 4-6.
constexpr int kNumMaps = 7;
struct StepMaps {
    CUtensorMap m[kNumMaps];
};

struct Fused3D {
    int nnx, nny, nnz, ldz;
    long sxy;
    int npd, nx, ny, nz;
    float dtx, dty, dtz;
    const float *cx1, *cx2, *ax1, *ax2, *cy1, *cy2, *ay1, *ay2, *cz1, *cz2, *az1, *az2;
    const float *m0, *m1, *m2;             // model: (vp, 1+2eps, sqrtf(1+2del)) exact,
                                           //        (A, B, C) fast
    const float *P0, *Q0, *v0;             // current level
    float *u1, *v1, *w1, *P1, *Q1;         // next level
    float *px, *py, *pz, *qx, *qy, *qz;    // split stresses (in place)
    int ntz, ntx, ntiles, chunk, nitems;   // work decomposition
    int *err;                              // device error word (wait timeouts)
};

// Tile and pipeline geometry.
constexpr int kTZ = 32;                 // z points per tile
constexpr int kTXF = 16;                // x columns per tile of the TTI kernels
constexpr int kFX = 16;                 // x columns per tile of the fused step
constexpr int kW = 2;                   // depths per thread (one vector)
constexpr int kFusedThreads = kTZ / kW * kFX, kFusedBlocks = 2;   // blocks per SM
constexpr int kStages = 3;              // TMA pipeline depth (planes)
constexpr int kPB = kTZ * (kFX + 14);  // P x-halo box (z 32, x TX+14 from x0-7)
constexpr int kQB = 48 * kFX;          // Q / w box (z 48 from z0-8, x TX)
constexpr int kUB = kTZ * (kFX + 8);   // u box (z 32, x TX+8 from x0-4)
constexpr int kOB = kTZ * kFX;         // own box (z 32, x TX)
// stage: the plane's P halo, Q, u, w and model (3)
constexpr int kStageFloats = kPB + kQB + kUB + kQB + 3 * kOB;
constexpr int kUTile = (kFX + 7) * kTZ;
constexpr int kWTile = kFX * 40;
constexpr size_t kFusedSmem = (size_t)(kStages * kStageFloats + 2 * (kUTile + kWTile) + 4 * kTZ) * 4 + 256;

struct StepArgs3D;
int launch_fused3d(const StepMaps &maps, const Fused3D &g, int mode, const StepArgs3D &st, cudaStream_t s);
int encode_map(CUtensorMap *map, const float *base, int nnz, int ldz, int nnx, int nny, int boxz, int boxx);

}  // namespace geo

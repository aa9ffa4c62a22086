// Fused 2D VTI steps of a single shot: shared declarations (step2d.cu).
#pragma once
#include "geo_internal.h"
#include <cuda.h>

namespace geo {

// A shot's grid, profiles and model.  Arrays are nnx columns of pitch ldz (a
// multiple of 4 floats, 16-byte aligned); zp holds cz1, cz2, az1, az2, ldz
// floats each.
struct SGrid {
    int nnx, nnz, ldz, npd, nx, nz;
    float dtx, dtz;
    const float *cx1, *cx2, *ax1, *ax2, *zp;
};

// One side's wavefields: P, Q, u, w at two time levels, split stresses in
// place, and the tensor maps of both levels' boxes.
struct SField {
    float *u[2], *w[2], *P[2], *Q[2], *px, *pz, *qx, *qz;
};
struct SMaps {
    CUtensorMap P, Q, u, w, S;
};

enum StepKind { SK_CPU = 0, SK_GPU = 1, SK_GFWD = 2, SK_GBWD = 3 };

struct SStep {
    SGrid g;
    SField f[2];                     // side 0 source (or only), 1 receiver
    int lev;                         // level the launch's first step reads
    int it0, it1;                    // forward: steps it0 .. it1-1; backward: it0 down to it1
    const float *amp;                // source of every step
    const unsigned char *on;
    int ixs, izs;
    // forward modelling: P at row rec_iz, time-major
    float *rec;
    int rec_iz;
    float rec_scale;
    int nt;                          // TTI: trace-major record, nt samples a trace
    // GPU RTM program: ring of P and Q (L entries a step), illumination,
    // image, angle gathers
    float *bp, *bq, *ill, *mig, *adcig;
    int L, nangle, dcdp;             // gathers at every dcdp-th CDP
    unsigned *bar;                   // grid-barrier counter
    int *err;                        // set when a wait gave up
};

// A run's launch shape and tensor maps: plan() for its kind and grid, maps()
// of each side (the receiver side backward only) and model() (vp, 1+2eps,
// sqrtf(1+2del), one array behind the other), then run() any number of times.
struct Fused2D {
    StepKind kind = SK_CPU;
    bool tti = false;
    int tx = 0, tiles = 0, stages = 0, grid = 0;   // columns per tile
    SMaps m[2][2];                                 // side, level
    CUtensorMap mm, mt;
    // fixed: columns per tile (8 or 16) whatever the grid; 0: by the grid
    int plan(StepKind k, bool tti, const SGrid &g, int fixed = 0);
    int maps(const SGrid &g, const SField &f, int side);
    int model(const SGrid &g, const float *p, const float *trig = nullptr);
    int run(const SStep &a, cudaStream_t s) const;
};
// The 12 arrays of a side, n floats each, from p.
void step2d_fields(float *p, size_t n, SField &f);
// Ring and record of step it into level lev (before a backward run that starts with it).
int launch_step2d_restore(const SStep &a, int it, int lev, cudaStream_t s);
// angle tables (device), and the source window of SK_CPU
int load_step2d_angles(const float *thr, const float *cs, cudaStream_t s);
int load_step2d_gauss();

}  // namespace geo

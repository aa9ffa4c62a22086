// Fused 2D VTI step of whole batches: shared declarations (march2d.cu).
#pragma once
#include "geo_internal.h"

namespace geo {

// One shot's descriptor (device memory).  Arrays are nnx columns of pitch
// ldz (a multiple of 4 floats, 16-byte aligned), z-profiles ldz long.
// P, Q, u, w exist at two time levels: neighbours read the old one while
// the new one is written; the split stresses are updated in place.
struct March2D {
    int nnx, nnz, ldz, npd, nx, nz;
    float dtx, dtz;
    const float *cx1, *cx2, *ax1, *ax2;
    const float *cz1;                // cz1, cz2, az1, az2, ldz floats each
    // field and model arrays, n floats each, slot k at f + k * n: MarchSlot
    float *f;
    unsigned n;                      // nnx * ldz
    // exact form: pow(1+2del, 0.5) as the program holds it, read where
    // ziv.cuh cannot decide
    const double *pw;
    int tx0, tz0;                    // taper box origin; box arrays kTB*kTB
    const float *te2, *td2;
    const float2 *tpw2;
    const double *tpw;
    int ixs, izs;
    float *rec_p, *rec_q, *edge_p, *edge_q;         // as Shot2D
    float *adcig;                    // [90][nx][nz], or null
};

// Slots of March2D::f.  A side has P, Q, u, w of level 0, the same of level
// 1, then px, pz, qx, qz; after both sides the image and the illumination
// (padded layout), then the model: rho*vp^2, 1+2eps and sqrtf(1+2del) (fast
// form) or the high and low floats of pow(1+2del, 0.5) (exact form).
enum MarchSlot {
    MS_P = 0, MS_Q = 1, MS_U = 2, MS_W = 3, MS_LEVEL = 4,
    MS_PX = 8, MS_PZ = 9, MS_QX = 10, MS_QZ = 11, MS_SIDE = 12,
    MS_MIG = 24, MS_ILL = 25, MS_STATE = 26,
    MS_VP = 26, MS_E2 = 27, MS_D2 = 28, MS_PL = 29, MS_SLOTS = 30
};

struct MarchStep {
    int it, lev;       // step, level read (lev ^ 1 is written)
    float amp;
    int src_on, inject;   // forward source; backward: step whose lines go into the new level (-1: none, also
                          // ahead of a scan of that level)
    float dhx, dlx, dhz, dlz;   // two-float (double)(dt/dx), (double)(dt/dz)
    double ddtx, ddtz;
    int *err;             // set when a pipeline wait gave up
};

// Source window and, for the gathers, angle thresholds and cos^3 weights.
int load_march_tables(bool adcig, cudaStream_t s);
// Work items of one launch: (shot | strip lanes << 24, z of lane 0, first and
// end column); lanes 1 .. strip lanes own four depths each.
// wide: a shot's slots exceed 2^32 floats.
int launch_march2d(bool backward, bool fast, bool adcig, bool wide, const March2D *d_shots, const int4 *d_items,
                   int nitems, const MarchStep &st, cudaStream_t s);
// Warps (forward) or warp pairs (backward) of the kernel resident at once.
int march2d_resident(bool backward, bool fast, bool adcig, int *out);
// The lines of step it into level lev of the source side, the records into the receiver side.
int launch_march_inject(const March2D *d_shots, int ns, int maxline, int it, int lev, cudaStream_t s);
// Watchdog over P of level lev, sides 0..nf-1.
int launch_march_watch(const March2D *d_shots, int ns, int nf, int lev, int *flag, int tag, cudaStream_t s);
// Compact image mig/ill and illumination of every shot (nx*nz each).
int launch_march_image(const March2D *d_shots, int ns, float *const *img, float *const *ill, cudaStream_t s);

}  // namespace geo

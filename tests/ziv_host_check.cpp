// Host build of ziv.cuh against the double chains it stands for: random
// operands over the ranges a run meets, cancellation, values next to float
// rounding boundaries, and values next to underflow.  Prints the number of
// decided values whose bits differ, the values, the undecided and the total of
// the plain kind, of the second stage, and the undecided squares.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include "../geophysics_gb300/csrc/ziv.cuh"

static uint32_t bits(float f) {
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
}

int main() {
    std::mt19937_64 g(12345);
    std::uniform_real_distribution<double> u(-1, 1);
    long bad = 0, n = 0, usual_open = 0, usual = 0, tiny = 0, tiny_open = 0, sq_open = 0;
    for (int it = 0; it < 6000000; it++) {
        const int kind = it % 6;
        const float vp = 4e6f * (float)(1 + u(g)) * 4 + 1e6f, az = it & 1 ? 1.0f : (float)(1 - 0.5 * fabs(u(g)));
        const float f = az * vp, del = 0.3f * (float)(u(g) * u(g));
        const double pw = std::pow((double)(1 + 2 * del), 0.5), ddt = (double)(float)(1e-3f / 10.0f);
        const float ph = (float)pw, pl = (float)(pw - (double)ph), dh = (float)ddt, dl = (float)(ddt - (double)dh);
        const double K = (double)f * pw * ddt;
        float a = (float)(u(g) * exp(20 * u(g))), z = (float)(u(g) * exp(20 * u(g)) / K);
        if (kind == 1) z = (float)(a / K);                                     // cancellation
        if (kind == 2) a = (float)((double)z * K * (1 + 1e-6 * u(g)));
        if (kind == 3) {                                                        // result near a boundary
            const float t = (float)u(g);
            const double mid = 0.5 * ((double)t + (double)std::nextafter(t, 2.0f));
            a = (float)(mid + K * (double)z);
        }
        if (kind == 4) { a = ldexpf(a, -95 - (int)(g() % 60)); z = ldexpf(z, -95 - (int)(g() % 60)); }
        if (kind == 5) { if (g() % 2) z = g() % 2 ? 0.0f : -0.0f; if (g() % 2) a = g() % 2 ? 0.0f : -0.0f; }
        bool sure;
        float r = geo::zv_chain(a, f, ph, pl, dh, dl, z, sure);
        float ref = (float)((double)a - K * (double)z);
        n++;
        if (sure && bits(r) != bits(ref)) bad++;
        if (kind == 0) {
            usual++;
            usual_open += !sure;
        }
        if (!sure) {   // second stage
            r = geo::zv_chain_tiny(a, f, ph, pl, dh, dl, z, sure);
            if (kind == 4) {
                tiny++;
                tiny_open += !sure;
            }
            if (sure && bits(r) != bits(ref)) { if(bad<10) fprintf(stderr,"kind %d a=%a z=%a K=%a r=%a ref=%a\n",kind,a,z,K,r,ref); bad++; }
        }
        const float ill = kind == 5 ? 0.0f : (float)fabs(u(g) * exp(20 * u(g))), s = z;
        r = geo::zv_square_add(ill, s, sure);
        ref = (float)((double)ill + (double)s * (double)s);
        n++;
        if (!sure) sq_open++;
        else if (bits(r) != bits(ref)) bad++;
    }
    printf("%ld %ld %ld %ld %ld %ld %ld\n", bad, n, usual_open, usual, tiny_open, tiny, sq_open);
}

// Host build of adcig.cuh against the programs' double quotient and bin:
// random pairs over all float exponents, subnormal and zero denominators,
// quotients next to the thresholds and to +-1, infinities and NaN.  Prints
// the number of differing bins, the pairs, and those with |S||G| below 1e-30.
#define __device__
#define __forceinline__ inline
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include "../geophysics_gb300/csrc/adcig.cuh"

static int bin_double(float dot, float b1, float b2, const float *thr, int na) {
    const float den = sqrtf(b1 * b2);
    const float a = (float)((double)dot / ((double)den * (1 - 0.1)));
    if (!(a >= -1.0f && a <= 1.0f)) return -1;
    int k = 0;
    while (k < na && a <= thr[k]) k++;
    return k < na ? k : -1;
}

int main() {
    std::mt19937_64 g(7);
    std::uniform_real_distribution<double> u(-1, 1);
    const int na = 70;
    float thr[na];
    for (int k = 0; k < na; k++) thr[k] = (float)std::cos(2 * (k + 1) * 3.14159265358979 / 180);
    thr[44] = 0.0f;   // 45 degrees: a threshold at zero
    const float inf = std::numeric_limits<float>::infinity(), nan = std::numeric_limits<float>::quiet_NaN();
    const float odd[] = {0.0f, -0.0f, inf, -inf, nan, 1.4e-45f, 1.1754944e-38f, 1e-30f, 3.4e38f};
    long bad = 0, n = 0, small = 0;
    for (int it = 0; it < 4000000; it++) {
        const int kind = it % 4;
        float b1 = ldexpf((float)(1 + std::fabs(u(g))), (int)(g() % 270) - 148);
        float b2 = kind == 0 ? ldexpf((float)(1 + std::fabs(u(g))), (int)(g() % 270) - 148) : b1 * (float)(0.5 + std::fabs(u(g)));
        const double den = (double)sqrtf(b1 * b2) * 0.9;
        float dot = (float)(den * 1.3 * u(g));
        if (kind == 1) {
            const double t = g() % 3 ? thr[g() % na] : (g() % 2 ? 1.0 : -1.0);
            dot = (float)(den * t * (1 + 3e-7 * u(g)));
        }
        if (kind == 2) dot = ldexpf((float)u(g), (int)(g() % 276) - 149);
        if (kind == 3 && it % 5 == 0) {
            if (g() % 2) dot = odd[g() % 9];
            if (g() % 2) b1 = std::fabs(odd[g() % 9]);
            if (g() % 2) b2 = std::fabs(odd[g() % 9]);
        }
        small += sqrtf(b1 * b2) < 1e-30f;
        n++;
        bad += geo::poynting_bin(dot, b1, b2, thr, na) != bin_double(dot, b1, b2, thr, na);
    }
    printf("%ld %ld %ld\n", bad, n, small);
}

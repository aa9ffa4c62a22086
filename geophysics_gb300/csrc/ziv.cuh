// Double-precision chains of the MPI RTM program decided in FP32.
//
// The program forms two stress chains and its illumination sum in double and
// rounds the result to float:
//   chain:  (float)((double)a - K * (double)z),  K = ((double)f * pw) * ddt
//   illum:  (float)((double)ill + (double)s * s)
// GB300 issues FP64 at 1/64 of the FP32 rate and its float<->double
// conversions on the same pipe, so the same bits are obtained from FP32 as
// Ziv's strategy does for correctly rounded functions (A. Ziv, "Fast
// evaluation of elementary mathematical functions with correctly rounded
// last bit", ACM TOMS 17(3), 1991): evaluate in unevaluated sums of two
// floats (error-free products by FMA, Knuth's two-sum), with an error bound
// E; if every value within E rounds to the same float, that float is the
// double chain's result too, since rounding is monotone.  Otherwise (about
// one value in 2^19, and values next to underflow) the caller evaluates the
// chain in double.
//
// Bounds.  pw = ph + pl leaves 2^-48 |pw|; each later operation on a low
// part rounds at 2^-24 of a quantity below 2^-23 of the leading one, six of
// them in all, so the two-float value is within 2^-44 (|a| + |th|) of the
// exact a - K z; the double chain is within 2^-51 of it.  E = 2^-43
// (|a| + |th|) covers both and the rounding of lo +- E below.  Where products
// underflow the error is below 2^-148 each; the absolute term 2^-140 covers
// those.  z = 0 (s = 0) is exact at once: K * 0 is a zero.
//
// Ahead of a wavefront the fields fall through the subnormals within a few
// cells, and every warp on that rim meets values the above cannot decide.
// zv_chain_tiny takes those: the operands scaled by 2^64 (exact), and a sum
// below the scaled normals rounded to the scaled subnormal spacing by adding
// 2^-62 of its sign, whose binade has that spacing.
#pragma once

#include <cmath>

#if defined(__CUDACC__)
#define GEO_ZV_FN __host__ __device__ __forceinline__
#else
#define GEO_ZV_FN inline
#endif

namespace geo {

GEO_ZV_FN float zv_fma(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
    return __fmaf_rn(a, b, c);
#else
    return std::fma(a, b, c);
#endif
}

// r = fl(x + y) and the exact remainder (Knuth).
GEO_ZV_FN float zv_two_sum(float x, float y, float &rem) {
    const float r = x + y, b = r - x;
    rem = (x - (r - b)) + (y - b);
    return r;
}

constexpr float kZvTiny = 7.17464814e-43f;   // 2^-140

// a - K z with K = (f * (ph + pl)) * (dh + dl); sure = false: not decided.
// s + (lo - e) and s + (lo + e) bracket every value within E of s + lo (the
// rounding of lo +- e is inside E), so their agreement decides.
GEO_ZV_FN float zv_chain(float a, float f, float ph, float pl, float dh, float dl, float z, bool &sure) {
    const float p = f * ph, pe = zv_fma(f, pl, zv_fma(f, ph, -p));
    const float k = p * dh, ke = zv_fma(pe, dh, zv_fma(p, dl, zv_fma(p, dh, -k)));
    const float th = k * z, tl = zv_fma(ke, z, zv_fma(k, z, -th));
    float e1;
    const float s = zv_two_sum(a, -th, e1), lo = e1 - tl;
    const float e = zv_fma(1.13686838e-13f, fabsf(a) + fabsf(th), kZvTiny);   // 2^-43
    const float r = s + (lo + e), r2 = s + (lo - e);
    const bool zero = z == 0.0f;
    sure = zero || r == r2;
    return zero ? s : r;
}

// The same chain where zv_chain was not sure, down to subnormal results.
GEO_ZV_FN float zv_chain_tiny(float a, float f, float ph, float pl, float dh, float dl, float z, bool &sure) {
    constexpr float up = 18446744073709551616.0f, down = 5.42101086e-20f;   // 2^64, 2^-64
    constexpr float norm = 2.16840434e-19f;                                  // 2^-62, the scaled least normal
    a *= up;
    z *= up;
    const float p = f * ph, pe = zv_fma(f, pl, zv_fma(f, ph, -p));
    const float k = p * dh, ke = zv_fma(pe, dh, zv_fma(p, dl, zv_fma(p, dh, -k)));
    const float th = k * z, tl = zv_fma(ke, z, zv_fma(k, z, -th));
    float e1, e2;
    const float s = zv_two_sum(a, -th, e1), lo = e1 - tl;
    const float sg = s == 0.0f ? lo : s;
    const float c = fabsf(s) < norm ? (sg < 0.0f ? -norm : norm) : 0.0f;
    const float s2 = zv_two_sum(c, s, e2);
    // 2^-43 of the operands, and 2^-108 for the rounding of lo + e2
    const float e = zv_fma(1.13686838e-13f, fabsf(a) + fabsf(th), 3.08148791e-33f), l2 = lo + e2;
    const float r = s2 + (l2 + e);
    const float out = (r - c) * down;
    // sums at the ends of the binade have two spacings: left to the double chain
    sure = r == s2 + (l2 - e) && fabsf(r) >= norm && (c == 0.0f || fabsf(r) < 2.0f * norm);
    return out == 0.0f && sg < 0.0f ? -0.0f : out;
}

// ill + s * s
GEO_ZV_FN float zv_square_add(float ill, float s, bool &sure) {
    const float h = s * s, l = zv_fma(s, s, -h);
    float e1;
    const float t = zv_two_sum(ill, h, e1), lo = e1 + l;
    const float e = zv_fma(1.13686838e-13f, fabsf(t), kZvTiny);
    const float r = t + (lo + e);
    const bool zero = s == 0.0f;
    sure = zero || r == t + (lo - e);
    return zero ? ill : r;
}

}  // namespace geo

// Branch decisions of the Godunov / PPM passes in the arithmetic type of the
// pass: FP64 operands are compared on the integer pipe (ks_common.cuh), FP32
// operands with plain compares.  The forward kernels and their reverse
// (adjoint) kernels take every decision through these functions, so a reverse
// kernel re-evaluates exactly the branch its forward took.
#pragma once

#include "ks_common.cuh"

namespace ks {

#ifdef __CUDACC__
__device__ inline bool same_sign(double a, double b) { return isame_sign(a, b); }
__device__ inline bool same_sign(float a, float b) { return a * b > 0.0f; }
__device__ inline bool abs_lt(double a, double b) { return iabs_lt2(a, b); }  // |a| < |b|
__device__ inline bool abs_lt(float a, float b) { return fabsf(a) < fabsf(b); }
__device__ inline double mag_sign(double m, double s) { return isign(m, s); }  // |m| with the sign of s
__device__ inline float mag_sign(float m, float s) { return copysignf(fabsf(m), s); }
__device__ inline double clip2(double e, double a, double b) { return imin(imax(e, imin(a, b)), imax(a, b)); }
__device__ inline float clip2(float e, float a, float b) { return fminf(fmaxf(e, fminf(a, b)), fmaxf(a, b)); }
__device__ inline bool gt0(double x) { return igt0(x); }
__device__ inline bool gt0(float x) { return x > 0.0f; }
__device__ inline bool le0(double x) { return ile0(x); }
__device__ inline bool le0(float x) { return x <= 0.0f; }
__device__ inline bool ge0(double x) { return ige0(x); }
__device__ inline bool ge0(float x) { return x >= 0.0f; }
__device__ inline bool above_small(double u) { return dbits(u) > dbits(kSmallVel); }          // u > small_vel
__device__ inline bool above_small(float u) { return u > (float)kSmallVel; }
__device__ inline bool below_msmall(double u) { return okey(u) < okey(-kSmallVel); }      // u < -small_vel
__device__ inline bool below_msmall(float u) { return u < -(float)kSmallVel; }
__device__ inline bool below_small_abs(double u) { return iabs_lt(u, kSmallVel); }        // |u| < small_vel
__device__ inline bool below_small_abs(float u) { return fabsf(u) < (float)kSmallVel; }
__device__ inline double absv(double x) { return iabs(x); }
__device__ inline float absv(float x) { return fabsf(x); }
__device__ inline double neg_if(bool c, double x) { return hiword(x, __double2hiint(x) ^ (c ? (int)0x80000000 : 0)); }
__device__ inline float neg_if(bool c, float x) { return c ? -x : x; }
__device__ inline double min2(double a, double b) { return imin(a, b); }
__device__ inline float min2(float a, float b) { return fminf(a, b); }
__device__ inline double max2(double a, double b) { return imax(a, b); }
__device__ inline float max2(float a, float b) { return fmaxf(a, b); }
__device__ inline bool lt(double a, double b) { return ilt(a, b); }  // a < b
__device__ inline bool lt(float a, float b) { return a < b; }
__device__ inline bool nonzero(double x) { return (dbits(x) & kMag) != 0; }
__device__ inline bool nonzero(float x) { return x != 0.0f; }

// The FP64 forms below spend fewer FP64 instructions: scaling by a power of two
// is an addition to the exponent field, and a choice is made before the
// arithmetic it selects, for an instruction that is predicated off still takes
// its FP64 issue slot.  At the ends of the range a half below the normal numbers
// becomes zero, twice a subnormal a normal number of at most 2^-1021, and twice
// 2^1023 or more no infinity.
constexpr long long kExp1 = 1LL << 52;
__device__ inline double twice(double x) { return hiword(x, __double2hiint(x) + 0x00100000); }  // x normal, below 2^1023
__device__ inline double half_fin(double x) {  // x finite
    const int h = __double2hiint(x);
    return (h & 0x7fffffff) >= 0x00200000 ? hiword(x, h - 0x00100000) : 0.0;
}
__device__ inline double half_of(double x) {  // infinities and NaN are kept
    return (__double2hiint(x) & 0x7ff00000) == 0x7ff00000 ? x : half_fin(x);
}

// van Leer (monotonized-central) limited slope of the middle cell of (a, b, c)
// from l = b - a, r = c - b and d = c - a: copysign(min(|d / 2|, |2 l|, |2 r|), d)
// where l r > 0, else 0.  (A non-finite neighbour reaches the edge through its
// value and difference, whatever the slope.)
__device__ inline double vls3(double l, double r, double d) {
    if (!same_sign(l, r)) return 0.0;
    const double m = abs_lt(l, r) ? l : r;
    if ((dbits(d) & kMag) < (dbits(m) & kMag) + 2 * kExp1) return half_fin(d);
    return mag_sign(twice(m), d);
}
__device__ inline float vls3(float l, float r, float d) {
    const float dsc = 0.5f * d, dsl = 2.0f * l, dsr = 2.0f * r;
    if (!same_sign(dsl, dsr)) return 0.0f;
    float m = abs_lt(dsl, dsr) ? dsl : dsr;
    m = abs_lt(dsc, m) ? dsc : m;
    return mag_sign(m, dsc);
}

// unlimited PPM edge value between cells with values a0, a1 = a0 + l and
// slopes s0, s1 (before the clip to the two cells)
__device__ inline double edge_value(double a0, double, double l, double s0, double s1) { return fma(-1.0 / 6.0, s1 - s0, fma(0.5, l, a0)); }
__device__ inline float edge_value(float a0, float a1, float, float s0, float s1) { return 0.5f * (a0 + a1) - float(1.0 / 6.0) * (s1 - s0); }

#endif

}  // namespace ks

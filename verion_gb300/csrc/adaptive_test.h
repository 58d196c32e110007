// The adaptive sampling test of a pixel in single precision, where that is certain of the answer in double.
#pragma once

#if defined(__CUDACC__)
#define VG_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#define VG_HD inline
#endif

namespace vgd {

// Whether a pixel with n samples, their sum s1 and sum of squares s2 takes more: 1 yes, 0 no, -1 for the caller to find
// out in double. Variance of the mean against its square, (s2 / n - mean^2) / (n - 1) > (threshold m)^2: `e` bounds the
// left side's rounding (2^-19 of its terms, some 30 ulps), the factors the right side's, and the double test's own
// rounding is far inside that margin. Both bounds are relative, so a yes asks for a left side, a no for a right
// side, whose terms are far from underflow. Not finite, or a negative threshold: no comparison holds, or none is
// made. (GB300 has few FP64 units: four divisions and a root per finished path kept them 61% busy in the
// resolve stage.)
VG_HD int adaptive_certain(double n, double s1, double s2, float threshold)
{
    float nf = (float)n, mf = (float)s1 / nf, q = (float)s2 / nf, m2 = mf * mf;
    float left = q - m2, e = 1.9073486e-6f * (q + m2);
    float right = threshold * fmaxf(mf, 0.05f);
    right = right * right * (nf - 1.0f);
    if (threshold >= 0.0f && q >= 1.0e-30f && left - e > right * 1.00001f)
        return 1;
    if (threshold >= 0.0f && right >= 1.0e-30f && left + e < right * 0.99999f)
        return 0;
    return -1;
}

} // namespace vgd

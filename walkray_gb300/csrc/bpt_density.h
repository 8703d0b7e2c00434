// bpt_density.h — direction densities of the bidirectional weights (bpt.cu).
//
// The reference computes them in double and rounds to float.  The FP64 unit
// does some two operations per SM and clock, conversions included, so the
// cosine density, which every diffuse vertex of a weight asks for, has a float
// form where that gives the same float; the Phong lobe's stays in double.
// Compiled without contraction, on the device and by the host test.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define WR_HD __host__ __device__ __forceinline__
#else
#define WR_HD inline
#endif

namespace wr {

constexpr double INV_PI_D = 0.31830988618379067153776752674503;

// x / pi, the double product rounded to float.  The constant in two floats
// gives the same result for every 24-bit significand as long as no partial
// product leaves the normal range; the few arguments beyond take the product
// itself (all 2^23 significands and every exponent: tests/test_densities.py).
constexpr float OVER_PI_HI = (float)INV_PI_D, OVER_PI_LO = (float)(INV_PI_D - (double)OVER_PI_HI);
WR_HD float over_pi(float x) {
    if (!(x > 1e-26f && x < 1e30f)) return (float)((double)x * INV_PI_D);
    const float p = x * OVER_PI_HI;
    return p + fmaf(x, OVER_PI_LO, fmaf(x, OVER_PI_HI, -p));
}

// (power + 1) * c / (2 pi), c the cosine's power (a pair of floats for each
// product kept some 46 bits, lost them below 1e-30 and made a NaN of an
// infinite c)
WR_HD float lobe_density(float power, float c) { return (float)(((double)power + 1.0) * (double)c * (INV_PI_D * 0.5)); }

}  // namespace wr

// bpt_density.h — direction densities of the bidirectional weights (bpt.cu):
// the reference's double products rounded to float.  Float forms of them cost
// bits where their partial products underflow (the cosine's below 1e-30, two
// floats for 1 / pi; the lobe's also by its 46 bits), and guarding the cosine's
// with a branch is slower than the product (bidirectional Cornell box 8.85 ms,
// 8.81 this way, 8.73 unguarded).  Compiled without contraction, on the device
// and by the host test.
#pragma once

#ifdef __CUDACC__
#define WR_HD __host__ __device__ __forceinline__
#else
#define WR_HD inline
#endif

namespace wr {

constexpr double INV_PI_D = 0.31830988618379067153776752674503;

WR_HD float over_pi(float x) { return (float)((double)x * INV_PI_D); }

// (power + 1) * c / (2 pi), c the cosine's power
WR_HD float lobe_density(float power, float c) { return (float)(((double)power + 1.0) * (double)c * (INV_PI_D * 0.5)); }

}  // namespace wr

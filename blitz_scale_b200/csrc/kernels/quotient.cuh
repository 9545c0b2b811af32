// A quotient without a branch, from an approximate reciprocal of the denominator (P. Markstein, IBM J. Res. Dev. 34, 1990: the reciprocal
// refined by one residual, then the quotient by its own).  Nothing here needs a GPU, so that a program for the host can check it.
#pragma once
#include <math.h>

#ifdef __CUDACC__
#define BLITZ_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define BLITZ_HOST_DEVICE inline
#endif

namespace blitz {

// x / d for a finite x and 1 <= d, both below 8e37, where r is 1 / d to a unit of the last place: the IEEE quotient, the sign of zero
// included, wherever that is no smaller than 2^-100 (below, the residual is no longer exact: the last bits may differ).
BLITZ_HOST_DEVICE float refined_quotient(float x, float d, float r) {
  r = fmaf(fmaf(-d, r, 1.f), r, r);
  const float q = x * r;
  return copysignf(fmaf(fmaf(-d, q, x), r, q), x);  // (the residual of -0 is +0, and so would be the sum)
}

}  // namespace blitz

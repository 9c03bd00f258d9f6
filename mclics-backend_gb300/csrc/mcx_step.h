// mcx_step.h -- the step-size rule (src/evolve.cpp:169-178 of the reference)
// in FP32 operations, bit for bit the reference's float/double expression.
//
// The reference multiplies or divides the float step by the double 0.99 and
// stores a float.  A product of two floats plus a correction term (the
// constant split into two floats, the product's rounding error by fmaf) gives
// the same float for every mantissa in the range below (tested over all of
// them), without double-precision arithmetic on the path from a sweep's last
// acceptance to the next sweep's first move.  The acceptance ratio is compared
// with 1/2 as integers.
#pragma once
#include <math.h>

#if defined(__CUDACC__)
#define MCX_HD __host__ __device__ __forceinline__
#else
#define MCX_HD static inline
#endif

namespace mcx {

// The step after a sweep with acc accepted moves of valid active sites.
MCX_HD float next_step(float av, unsigned acc, unsigned valid) {
  const unsigned long long two = 2ull * acc;
  if (two == valid) return av;
  const bool less = two < valid;
  if (!(av > 1e-6f && av < 1e6f)) {  // far from any step the rule reaches by itself
    if (less) {
      av = (float)((double)av * 0.99);
      if ((double)av < 0.01) av = (float)0.01;
    } else {
      av = (float)((double)av / 0.99);
      if ((double)av > 1.0) av = (float)((double)av - 0.5);
    }
    return av;
  }
  const float h = less ? (float)0.99 : (float)(1.0 / 0.99);
  const float l = less ? (float)(0.99 - (double)(float)0.99) : (float)(1.0 / 0.99 - (double)(float)(1.0 / 0.99));
#if defined(__CUDA_ARCH__)
  const float p = __fmul_rn(av, h);
  const float r = __fadd_rn(p, fmaf(av, l, fmaf(av, h, -p)));
#else
  const float p = av * h;  // host: compiled without contraction
  const float r = p + fmaf(av, l, fmaf(av, h, -p));
#endif
  if (less) return r <= (float)0.01 ? (float)0.01 : r;  // the float below 0.01: r < 0.01 in double
  return r > 1.f ? r - 0.5f : r;                        // exact: r is in (1, 2), or its ulp divides 0.5
}

}  // namespace mcx

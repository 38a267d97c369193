// fastmath.cuh -- the FP64 reciprocal square root and decaying exponential of
// the panel-pair kernels, written for their arguments (finite positive squared
// distances, non-positive exponents).
//
// Per pair the library's rsqrt and exp cost about as many FP64 instructions as
// all the rest of the one-point kernel; here they take 5 and 10.
#pragma once
#include <cuda_runtime.h>

#include <cmath>

#include "common.cuh"

namespace fb {

// 1/sqrt(x) for normal x > 0: one third-order Householder step
//   y (1 + e/2 + 3 e^2 / 8),  e = 1 - x y^2,
// from the hardware's approximation, whose relative error of at most about
// 2^-20 makes |e| 2^-19 and leaves a truncation of 5/16 e^3 = 2^-58.7.  With the
// roundings within 1.6 * 2^-53 of the exact value (1.24 measured, 1.01 for the library).
__device__ __forceinline__ double rsqrt_pos(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// e^t by a table of 2^(j/64) and a short polynomial (the table method of
// P. T. P. Tang, ACM TOMS 15, 1989): with s = 64 t / ln 2 = 64 m + j + f,
// |f| <= 1/2, e^t = 2^m 2^(j/64) e^(f ln2/64), the last factor by its Taylor
// polynomial of degree 5 (truncation below 4e-17).  The caller passes s, whose
// rounding is the argument's own.  s <= 0; below -64 * 1021 the result is
// 2^-1021 (about 1e-308) instead of a denormal or zero.  Within 2.4 * 2^-53 of
// e^t (2.03 measured, 1.23 for the library).  tab: the 64 values, in shared memory (load_exp_tab).
constexpr int kExpTab = 64;
constexpr double kExpScale = 92.332482616893656877;   // 64 / ln 2
__device__ double g_expTab[kExpTab];

__device__ __forceinline__ double exp_tab(double s, const double *tab) {
  constexpr double c1 = 1.0 / kExpScale, c2 = c1 * c1 / 2, c3 = c2 * c1 / 3, c4 = c3 * c1 / 4, c5 = c4 * c1 / 5;
  const double magic = 6755399441055744.0;   // 3 * 2^51: the sum's low word is s rounded to an integer
  const double n = s + magic;
  double f = s - (n - magic);
  int k = __double2loint(n);
  if ((unsigned)__double2hiint(s) > 0xC0EFE800u) {   // s < -65344
    k = -64 * 1021;
    f = 0.0;
  }
  const double p = fma(fma(fma(fma(c5, f, c4), f, c3), f, c2), f, c1);
  const double t0 = tab[k & (kExpTab - 1)];
  const double t = __hiloint2double(__double2hiint(t0) + ((k >> 6) << 20), __double2loint(t0));
  return fma(t, p * f, t);
}

// the block's copy of the table; the caller synchronises before its first use
__device__ __forceinline__ void load_exp_tab(double *tab) {
  for (int i = threadIdx.x; i < kExpTab; i += blockDim.x) tab[i] = g_expTab[i];
}

inline bool init_exp_tab() {
  double h[kExpTab];
  for (int j = 0; j < kExpTab; j++) h[j] = std::exp2(j / 64.0);
  FB_CUDA(cudaMemcpyToSymbol(g_expTab, h, sizeof(h)));
  return true;
}

}  // namespace fb

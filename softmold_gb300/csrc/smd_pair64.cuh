// FP64 pair terms of the plain form and of smd_pair_forces_static.
//
// On GB300 an FP64 instruction costs about a hundred FP32 ones, so what counts
// here is the number of FP64 instructions per pair within the cutoff.
#pragma once

#include <cuda_runtime.h>

namespace smd {

// 1 / sqrt(r2) and sqrt(r2): the reciprocal root is CUDA's rsqrt (1 ulp); the
// root is r2 / sqrt(r2) with one residual step (r <- r + (r2 - r^2) / (2 r)),
// which rounds it as sqrt does but for rare last-bit cases.  The two together
// take about half the FP64 instructions of sqrt and a division.
__device__ __forceinline__ double root64(double r2, double& rinv) {
  rinv = rsqrt(r2);
  const double r = r2 * rinv;
  return __double_as_longlong(r2) != 0 ? fma(fma(-r, r, r2), 0.5 * rinv, r) : 0.0;  // coincident beads
}

// a / r for r = root64(r2) from the reciprocal root: one residual step
// (Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", 1990) rounds it as the division does but for rare last-bit cases.
__device__ __forceinline__ double div64(double a, double r, double rinv) {
  const double q = a * rinv;
  return fma(fma(-q, r, a), rinv, q);
}

// Which of a table row's two segments holds r >= 0: the reference's index
// int(r / C0) * 3, capped at 3 (include/MD.h:811-825), is 0 for r < C0 and 3
// from there on.  Compared by the bits, in the integer pipe: non-negative
// doubles order like unsigned integers, and a negative C0 stays above every r,
// as r / C0 < 1 does.
__device__ __forceinline__ int segment64(double r, double c0) {
  return (unsigned long long)__double_as_longlong(r) < (unsigned long long)__double_as_longlong(c0) ? 0 : 3;
}

// Pair force magnitude (include/MD.h:811-825) from the squared distance: force
// on i = mag * d.
__device__ __forceinline__ double pair_mag64(const double* c, double r2) {
  double rinv;
  const double r = root64(r2, rinv);
  const double* s = c + segment64(r, c[0]);
  const double m = s[0] - r;
  return ((s[1] - s[2] * m) * m) * rinv;
}

// x_i - x_j with the minimum image applied to the neighbour first, as CellOpt
// shifts the neighbour cell's positions (cellOpt.h:810-840).  half_hi is the
// high word of box / 2: the high words decide, since a separation that agrees
// with half the box edge in its leading 20 bits lies far beyond the cutoff
// (at most a third of the edge) with either image.
__device__ __forceinline__ double image64(double xi, double xj, double box, int half_hi) {
  const double d = xi - xj;
  if ((__double2hiint(d) & 0x7fffffff) <= half_hi) return d;
  return xi - (xj + copysign(box, d));
}

}  // namespace smd

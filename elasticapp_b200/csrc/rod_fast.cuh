// Cheaper forms of the FP64 rod arithmetic for the resident and streaming
// kernels and the contact search, each with the result of the plain expression
// it stands for.
//
// The resident kernel is bound by FP64 issue and by the latency of dependent FP64
// operations, and a library division or square root is ten or more of them
// with a branch of its own.  Stiff rods amplify any difference in rounding
// (two correct evaluations part by 1e-9 in the angular velocities within a
// few hundred steps), so the forms below are not merely accurate: they round
// correctly, as IEEE division and square root do.  Each takes a hardware
// approximation (20 bits or more), one Householder iteration of third order
// (error e -> O(e^3), below an ulp) and a correction by the exact residual
// (Markstein's theorem), without branches, so that independent chains
// interleave.
//
// What a correction leaves out, the residual's square, is below 2^-100 of the
// result, so only a reciprocal or root that near to a tie could round wrongly.
// Those can be listed: with 53-bit significands D and midpoints M / 2^54,
// 1 / D is near one where D M = 2^106 - k for a small k (126 significands for
// |k| <= 20, by factoring), a root where M^2 is as near to a multiple of a power
// of two (only three squares are near enough to matter), a quotient where D M
// is.  Every such reciprocal and root, and ten thousand such quotients, are
// compared with the exact result (tests/test_gpu_rod_fast.py).  Of a quotient
// -0 the sign is lost.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "rod_math.cuh"

namespace eb {

// an approximation of 1 / d within an ulp, for a normal d whose reciprocal is
// normal: with e = 1 - d y0, 1 / d = y0 (1 + e + e^2 + O(e^3))
__device__ __forceinline__ double rcp_near(double d) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double e = fma(-d, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// 1 / d from an approximation y of it that is off by little more than its own
// rounding (half an ulp; rcp_near's is).  The residual r = 1 - d y gives
// y + y r, short of 1 / d by its square, which matters only where a tie lies
// between the two: where r > 0, y with its last bit set in y's place makes up
// for it (where r < 0 no such tie is passed).
__device__ __forceinline__ double rcp_from(double d, double y) {
  const double r = fma(-d, y, 1.0);
  const int up = ~(__double2hiint(r) >> 31) & 1;
  return fma(r, __hiloint2double(__double2hiint(y), __double2loint(y) | up), y);
}

// 1 / d from an approximation y of it within 16 ulps.  (From a start of up to
// three ulps, one step alone rounds dozens of significands wrongly.  The second
// takes 2000 steps of a 100-element rod 3.83 -> 3.85 ms, 128 steps of 8192 rods
// 13.00 -> 13.01.)
__device__ __forceinline__ double rcp_from_rough(double d, double y) { return rcp_from(d, fma(fma(-d, y, 1.0), y, y)); }

// a / d from y, the rounded 1 / d
__device__ __forceinline__ double div_from(double a, double d, double y) {
  const double q = a * y;
  return fma(fma(-q, d, a), y, q);
}

// an approximation of 1 / sqrt(z) within an ulp, for a normal z > 0: with
// e = 1 - z y0^2, 1 / sqrt(z) = y0 (1 + e / 2 + 3 e^2 / 8 + O(e^3))
__device__ __forceinline__ double rsqrt_near(double z) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(z));
  const double e = fma(-(z * y), y, 1.0);
  return fma(y, e * fma(0.375, e, 0.5), y);
}

// sqrt(z) from y, 1 / sqrt(z) within an ulp
__device__ __forceinline__ double sqrt_from(double z, double y) {
  const double g = z * y;
  return fma(fma(-g, g, z), 0.5 * y, g);
}

// whether d lies in [2^-400, 2^400]: there the forms above and the products
// around them stay clear of underflow and overflow; other values (zero, not
// finite) take the plain operations
__device__ __forceinline__ bool ordinary(double d) {
  return static_cast<uint32_t>(__double2hiint(d)) - (623u << 20) < (800u << 20);
}

// 1 / d and a / d for any d
__device__ __forceinline__ double reciprocal(double d) { return ordinary(d) ? rcp_from(d, rcp_near(d)) : 1.0 / d; }
__device__ __forceinline__ double quotient(double a, double d) {
  return ordinary(d) ? div_from(a, d, rcp_from(d, rcp_near(d))) : a / d;
}

// The rod kernels take the rest lengths, dilatations and Voronoi lengths
// without the test.  Outside the range these are those of a rod that has
// collapsed, blown up or was given no usable length, whose state is no longer
// finite either way: it turns NaN at once instead of by way of an infinity.
// (The tests took the resident kernel 4 to 11 % longer: a 100-element rod 3.86
// -> 4.24 ms, 8192 rods 13.0 -> 13.6.)  Masses are not left so: an infinite
// one holds its node.

// length and reciprocal length from the squared length
struct Length {
  double l, il;
};
__device__ __forceinline__ Length length_of(double l2) {
  if (ordinary(l2)) {
    const double y = rsqrt_near(l2);
    const double l = sqrt_from(l2, y);
    // y is within 2 ulps of 1 / l.  The residual's square is taken along, by a
    // multiplicand that is corrected too (y with its last bit set, which needs
    // no wait for the residual): 2000 steps of a 100-element rod 3.83 ms,
    // where a multiplicand chosen by the residual's sign takes 3.86.
    const double r = fma(-l, y, 1.0);
    return {l, fma(r, fma(r, __hiloint2double(__double2hiint(y), __double2loint(y) | 1), y), y)};
  }
  const double l = sqrt(l2);
  return {l, 1.0 / l};
}

// The coefficients of exp(-[u]x): sin(theta) and 1 - cos(theta) from their
// Taylor series for theta < 0.1 (truncation below 1e-21 relative), which also
// avoids the cancellation of 1 - cos(theta) at small angles, and one
// reciprocal for the axis.  The rotation is applied to a slot's directors
// twice a step (the closing half drift of one step and the first of the next
// have the same angle), so they are formed once.
struct Rotation {
  double c, s;      // cos, sin of the angle
  double u[3];      // guarded axis
  double au[3];     // (1 - cos) times the axis
};

__device__ __forceinline__ Rotation rotation(double u0, double u1, double u2) {
  const double z = u0 * u0 + u1 * u1 + u2 * u2;
  double theta, r;
  if (z > 1e-30 && z < 1e30) {
    // |u| > 1e-15: the guard of 1e-14 changes the sum by at most a factor of
    // eleven, far from the ends of the range
    theta = sqrt_from(z, rsqrt_near(z));
    const double d = theta + 1e-14;
    r = rcp_from(d, rcp_near(d));
  } else {
    theta = sqrt(z);
    r = 1.0 / (theta + 1e-14);
  }
  double s, alpha;
  if (theta < 0.1) {
    s = theta * (1.0 + z * (-1.0 / 6.0 + z * (1.0 / 120.0 + z * (-1.0 / 5040.0 +
                                                           z * (1.0 / 362880.0 - z * (1.0 / 39916800.0))))));
    alpha = z * (0.5 + z * (-1.0 / 24.0 + z * (1.0 / 720.0 + z * (-1.0 / 40320.0 + z * (1.0 / 3628800.0)))));
  } else {
    double c;
    sincos(theta, &s, &c);
    alpha = 1.0 - c;
  }
  u0 *= r;
  u1 *= r;
  u2 *= r;
  return {1.0 - alpha, s, {u0, u1, u2}, {alpha * u0, alpha * u1, alpha * u2}};
}

// Q <- R Q; which products are fused is written out, so that every kernel
// rounds alike
__device__ __forceinline__ void rotate(double q[9], const Rotation& R) {
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const double q0 = q[j], q1 = q[3 + j], q2 = q[6 + j];
    const double com = fma(q2, R.u[2], fma(q0, R.u[0], q1 * R.u[1]));
    q[j] = fma(R.s, fma(q1, R.u[2], -(q2 * R.u[1])), fma(R.c, q0, R.au[0] * com));
    q[3 + j] = fma(R.s, fma(q2, R.u[0], -(q0 * R.u[2])), fma(R.au[1], com, R.c * q1));
    q[6 + j] = fma(R.s, fma(q0, R.u[1], -(q1 * R.u[0])), fma(R.au[2], com, R.c * q2));
  }
}

// Curvature (inv_rotate_divide in rod_math.cuh) with sin(acos(c) + d) =
// sqrt((1 - c)(1 + c)) cos d + c sin d, d = 1e-14 (cos d rounds to 1, sin d to
// d), and the square root and the quotient in the forms above (a 1 - cos(theta)
// outside (1e-12, 2) takes the plain operations).
__device__ __forceinline__ Vec3<double> curvature(const double qc[9], const double qn[9], double span) {
  const double tr = qc[0] * qn[0] + qc[1] * qn[1] + qc[2] * qn[2] + qc[3] * qn[3] + qc[4] * qn[4] +
                    qc[5] * qn[5] + qc[6] * qn[6] + qc[7] * qn[7] + qc[8] * qn[8];
  const double cth = 0.5 * tr - (0.5 + 1e-10);
  const double theta = acos(cth);
  const double w = (1.0 - cth) * (1.0 + cth);
  const bool fine = w > 1e-12 && ordinary(span);
  const double root = fine ? sqrt_from(w, rsqrt_near(w)) : sqrt(w);
  const double den = (root + cth * 1e-14) * span;
  const double half = 0.5 * theta;
  double st;
  if (fine)
    st = div_from(half, den, rcp_from(den, rcp_near(den)));
  else
    st = half / den;
  return {st * (-qc[3] * qn[6] - qc[4] * qn[7] - qc[5] * qn[8] + qc[6] * qn[3] + qc[7] * qn[4] +
                qc[8] * qn[5]),
          st * (qc[0] * qn[6] + qc[1] * qn[7] + qc[2] * qn[8] - qc[6] * qn[0] - qc[7] * qn[1] -
                qc[8] * qn[2]),
          st * (-qc[0] * qn[3] - qc[1] * qn[4] - qc[2] * qn[5] + qc[3] * qn[0] + qc[4] * qn[1] +
                qc[5] * qn[2])};
}

}  // namespace eb

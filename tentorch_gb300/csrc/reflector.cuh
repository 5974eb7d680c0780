// The scalars of a Householder reflector as LAPACK's dlarfg / zlarfg make them (R_jj = beta, with its signs), for
// the QR factorisations of qr.cu and svd.cu.
#pragma once

#include <cuda_runtime.h>

#include <cmath>

namespace ttg
{
  namespace
  {
    // A column whose squared norm is below this is scaled up by a power of two before its reflector is made: its
    // squares are subnormal or zero, and a norm, tau and v made from them no longer belong together (a column
    // 1e-158 of the block's largest entry left Q^H Q - I at 1e-8, 1e-161 at 4e-3; 1e-170 lost what was below the diagonal).
    constexpr double kTinySquare = 1e-290;

    // sqrt(x) and its reciprocal, each to half an ulp or so: an ulp of rsqrt in the first, largest columns
    // doubled the error of Q R
    __device__ __forceinline__ void root(double x, double &norm, double &inv)
    {
      inv = rsqrt(x);
      norm = x * inv;
      norm = fma(0.5 * inv, fma(-norm, norm, x), norm);
      inv = fma(inv, fma(-norm, inv, 1.0), inv);
    }

    // H = I - tau v v^H with v_0 = 1 takes (alpha, x) to (beta, 0), beta real; v's rest is x scale, xn = |x|^2 and
    // square = |alpha|^2 + xn.
    __device__ __forceinline__ void make_reflector(double alpha, double xn, double square, double &beta, double &tau, double &scale)
    {
      beta = alpha;
      tau = scale = 0.0;
      if (!(xn == 0.0))  // (a NaN goes on into R and Q)
      {
        double norm, inv;
        root(square, norm, inv);
        const double d = alpha + copysign(norm, alpha);  // alpha - beta, without cancellation
        beta = -copysign(norm, alpha);
        tau = fabs(d) * inv;                             // (beta - alpha) / beta
        scale = 1.0 / d;
      }
    }
    __device__ __forceinline__ void make_reflector(double2 alpha, double xn, double square, double2 &beta, double2 &tau,
                                                   double2 &scale)
    {
      beta = alpha;
      tau = scale = make_double2(0.0, 0.0);
      if (!(xn == 0.0 && alpha.y == 0.0))
      {
        double norm, inv;
        root(square, norm, inv);
        const double re = alpha.x + copysign(norm, alpha.x);  // alpha - beta, without cancellation
        const double side = copysign(inv, alpha.x);           // -1 / beta
        beta = make_double2(-copysign(norm, alpha.x), 0.0);
        tau = make_double2(fabs(re) * inv, alpha.y * side);   // (beta - alpha) / beta
        const double over = 1.0 / fma(re, re, alpha.y * alpha.y);
        scale = make_double2(re * over, -alpha.y * over);     // 1 / (alpha - beta)
      }
    }
  } // namespace
} // namespace ttg

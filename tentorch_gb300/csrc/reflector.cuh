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
    // (2^-963, by its exponent field: an integer comparison, on the chain of every column.)
    constexpr int kTinyField = 1023 - 963;

    __device__ __forceinline__ double scaled_by(double a, double s) { return a * s; }
    __device__ __forceinline__ double2 scaled_by(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
    __device__ __forceinline__ double square(double a, double c) { return fma(a, a, c); }
    __device__ __forceinline__ double square(double2 a, double c) { return fma(a.x, a.x, fma(a.y, a.y, c)); }
    __device__ __forceinline__ double largest(double a) { return fabs(a); }
    __device__ __forceinline__ double largest(double2 a) { return fmax(fabs(a.x), fabs(a.y)); }

    template <int G>
    __device__ __forceinline__ double lanes_sum(double v)
    {
#pragma unroll
      for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, G);
      return v;
    }
    template <int G>
    __device__ __forceinline__ double2 lanes_sum(double2 v) { return make_double2(lanes_sum<G>(v.x), lanes_sum<G>(v.y)); }

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

    // The power of two for a tiny column (1 when it is zero); `xn` becomes the squared norm below entry j at that scale.
    template <typename T>
    __device__ __forceinline__ double tiny_column(const T *col, int j, int len, double &xn)
    {
      const int lane = threadIdx.x & 31;
      double big = 0.0;
      for (int i = j + lane; i < len; i += 32) big = fmax(big, largest(col[i]));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
      if (!(big > 0.0)) return 1.0;
      int ex;
      frexp(big, &ex);
      const double up = ldexp(1.0, min(-ex, 1000));
      double sum = 0.0;
      for (int i = j + 1 + lane; i < len; i += 32) sum = square(scaled_by(col[i], up), sum);
      xn = lanes_sum<32>(sum);
      return up;
    }

    // The reflector of column j (entries j .. len - 1 of `col`, xn the squared norm below entry j) by one warp, whose
    // lanes all hold the results.
    template <typename T>
    __device__ __forceinline__ void column_reflector(const T *col, int j, int len, double xn, T &beta, T &tau, T &scale)
    {
      const T head = col[j];
      const double norm2 = square(head, xn);
      if (__double2hiint(norm2) >> 20 >= kTinyField)  // (also a NaN)
      {
        make_reflector(head, xn, norm2, beta, tau, scale);
        return;
      }
      const double up = tiny_column(col, j, len, xn);
      const T raised = scaled_by(head, up);
      make_reflector(raised, xn, square(raised, xn), beta, tau, scale);
      beta = scaled_by(beta, 1.0 / up);
      scale = scaled_by(scale, up);
    }
  } // namespace
} // namespace ttg

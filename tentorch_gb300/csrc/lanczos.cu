// The Lanczos eigensolver of a DMRG window (tentorch/linalg/lanczos.py:8-64) as one host loop over
// device work: every Krylov step executes the window's compiled einsum on the current basis vector and
// then one kernel that projects the image against the whole basis three times (the first projection
// holds alpha and replaces the three-term step; then the reference's two full reorthogonalisation
// passes), takes its norm and scales it into the next basis vector, with no host synchronisation.
// The device then applies the reference's early stop (a beta below `tol` ends the space), solves the
// small eigenproblem and forms the normalised Ritz vector: the whole call is stream-ordered work
// with no host wait, and its energy and Krylov size stay in device memory until the caller reads them.
//
// Per step that is the plan's launches plus one.  As thirteen launches (dot products, their sums and
// the projections, three times, the norm and the scaling) the vector algebra of a step took longer
// than a split-precision matvec at bond 256.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <vector>

#include "executor.h"
#include "launch.h"

namespace ttg
{
  namespace
  {
    constexpr int kOrthoThreads = 512;
    constexpr int kOrthoMaxRows = 64;              // basis vectors (n_iter <= 60)
    constexpr int64_t kOrthoSmem = 160 * 1024;     // of a CTA's part of the vector
    constexpr unsigned long long kOrthoWaitNs = 2000000000ull;  // two seconds

    // What one launch does to a vector of `n` doubles, its parts dealt to the CTAs:
    //   - the vector is `from` (passes 3: projected three times against the `rows` basis vectors), or the
    //     combination of the first *size basis vectors with coefficients `c`;
    //   - it goes to `to` over its norm; the norm to `beta`, the last coefficient of the first pass to
    //     `alpha` (where given).
    struct OrthoArgs
    {
      const double *from, *basis, *c;
      const int32_t *size;
      double *to, *work;   // work: `n` doubles for parts that do not fit in shared memory
      double *alpha, *beta;
      double *partial;     // rows + 1 sums (complex: two doubles each) of every CTA, for each of four passes
      unsigned *arrived;   // four counters, zero
      int *error;
      int64_t n, part;     // part: doubles a CTA holds, even
      int32_t rows, passes;
    };

    __device__ __forceinline__ unsigned long long ortho_now()
    {
      unsigned long long t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      return t;
    }

    __device__ __forceinline__ double lane_sum(double v)
    {
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
      return v;
    }

    // The vector's part stays in shared memory through the passes.  A pass: a group of warps per basis
    // vector takes its dot product with the part; the CTAs' sums meet in global memory behind a counter
    // (the grid is launched cooperatively, all CTAs resident; a wait gives up after two seconds and
    // raises the error flag); every CTA adds the sums in the same order, so that all hold the same
    // coefficients; then the part is updated.  The norm comes with the last pass's sums: what that pass
    // removes is the round-off the two before left, so |y|^2 - sum |c|^2 is exact to round-off; when it
    // removes more than that, the norm is summed again.  FP64 issues one warp instruction in 64 clocks
    // a quarter of an SM, which bounds small vectors by the lanes' sums and large ones by the
    // multiply-adds; reading the basis twice a pass bounds neither.
    template <bool Complex>
    __global__ void __launch_bounds__(kOrthoThreads) ortho_kernel(const OrthoArgs a)
    {
      extern __shared__ double held[];
      __shared__ double sub[2 * kOrthoThreads / 32], coeff[2 * (kOrthoMaxRows + 1)];
      constexpr int W = Complex ? 2 : 1;
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
      const int64_t lo = min(a.n, static_cast<int64_t>(blockIdx.x) * a.part), len = min(a.part, a.n - lo);
      const int parts = gridDim.x;
      double *y = a.part * 8 <= kOrthoSmem ? held : a.work + lo;
      dependent_entry();
      const auto meet = [&](int pass) {
        __syncthreads();
        if (threadIdx.x == 0 && parts > 1)
        {
          __threadfence();
          atomicAdd(a.arrived + pass, 1u);
          const unsigned long long start = ortho_now();
          unsigned seen = 0;
          while (true)
          {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.arrived + pass) : "memory");
            if (seen >= static_cast<unsigned>(parts) || *static_cast<volatile int *>(a.error)) break;
            if (ortho_now() - start > kOrthoWaitNs)
            {
              atomicExch(a.error, 1);
              break;
            }
          }
          __threadfence();
        }
        __syncthreads();
      };
      // coeff[0 .. W count) = the sums over all CTAs of <b_j, y> for j < rows, then of |y|^2 (`square`)
      const auto sums = [&](int pass, int rows, bool square) {
        const int count = rows + (square ? 1 : 0);
        double *out = a.partial + static_cast<int64_t>(pass) * (a.rows + 1) * parts * W;
        // the warps of one dot product: more than one while the part is long and the vectors few
        int group = 1;
        while (group * 2 * count <= warps && len / W >= static_cast<int64_t>(group) * 512) group *= 2;
        const int each = warps / group, slice = warp % group;
        for (int j0 = 0; j0 < count; j0 += each)
        {
          const int j = j0 + warp / group;
          double re = 0.0, im = 0.0;
          if (j < count)
          {
            const double *b = j < rows ? a.basis + j * a.n + lo : y;
            if constexpr (Complex)
            {
#pragma unroll 4
              for (int64_t i = (static_cast<int64_t>(slice) * 32 + lane) * 2; i < len; i += group * 64)
              {
                const double br = b[i], bi = b[i + 1], yr = y[i], yi = y[i + 1];
                re = fma(br, yr, fma(bi, yi, re));
                im = fma(br, yi, fma(-bi, yr, im));
              }
              im = lane_sum(im);
            }
            else
            {
#pragma unroll 4
              for (int64_t i = static_cast<int64_t>(slice) * 32 + lane; i < len; i += group * 32) re = fma(b[i], y[i], re);
            }
            re = lane_sum(re);
          }
          if (group > 1)
          {
            if (lane == 0)
            {
              sub[2 * warp] = re;
              sub[2 * warp + 1] = im;
            }
            __syncthreads();
            if (slice == 0)
            {
              re = im = 0.0;
              for (int s = 0; s < group; ++s)
              {
                re += sub[2 * (warp + s)];
                im += sub[2 * (warp + s) + 1];
              }
            }
            __syncthreads();
          }
          if (j < count && slice == 0 && lane == 0)
          {
            const int64_t at = (static_cast<int64_t>(j) * parts + blockIdx.x) * W;
            __stcg(out + at, re);
            if constexpr (Complex) __stcg(out + at + 1, im);
          }
        }
        meet(pass);
        for (int j = warp; j < count; j += warps)
        {
          double re = 0.0, im = 0.0;
          for (int p = lane; p < parts; p += 32)
          {
            const int64_t at = (static_cast<int64_t>(j) * parts + p) * W;
            re += __ldcg(out + at);
            if constexpr (Complex) im += __ldcg(out + at + 1);
          }
          re = lane_sum(re);
          if constexpr (Complex) im = lane_sum(im);
          if (lane == 0)
          {
            coeff[W * j] = re;
            if constexpr (Complex) coeff[W * j + 1] = im;
          }
        }
        __syncthreads();
      };

      if (a.c)
      {
        // real coefficients act on both parts of a complex vector alike
        const int32_t used = *a.size;
        for (int64_t i = threadIdx.x; i < len; i += blockDim.x)
        {
          double v = 0.0;
          for (int32_t j = 0; j < used; ++j) v = fma(a.c[j], a.basis[j * a.n + lo + i], v);
          y[i] = v;
        }
      }
      else
        for (int64_t i = threadIdx.x; i < len; i += blockDim.x) y[i] = a.from[lo + i];
      __syncthreads();
      double norm2 = 0.0;
      bool known = false;
      for (int pass = 0; pass < a.passes; ++pass)
      {
        const bool last = pass + 1 == a.passes;
        sums(pass, a.rows, last);
        if (pass == 0 && a.alpha && blockIdx.x == 0 && threadIdx.x == 0) *a.alpha = coeff[W * (a.rows - 1)];
        for (int64_t i = static_cast<int64_t>(threadIdx.x) * W; i < len; i += static_cast<int64_t>(blockDim.x) * W)
        {
          if constexpr (Complex)
          {
            double re = y[i], im = y[i + 1];
#pragma unroll 4
            for (int32_t j = 0; j < a.rows; ++j)
            {
              const double br = a.basis[j * a.n + lo + i], bi = a.basis[j * a.n + lo + i + 1];
              const double cr = coeff[2 * j], ci = coeff[2 * j + 1];
              re = fma(-cr, br, fma(ci, bi, re));
              im = fma(-cr, bi, fma(-ci, br, im));
            }
            y[i] = re;
            y[i + 1] = im;
          }
          else
          {
            double v = y[i];
#pragma unroll 4
            for (int32_t j = 0; j < a.rows; ++j) v = fma(-coeff[j], a.basis[j * a.n + lo + i], v);
            y[i] = v;
          }
        }
        if (last)
        {
          double removed = 0.0;
          for (int32_t j = 0; j < W * a.rows; ++j) removed = fma(coeff[j], coeff[j], removed);
          const double before = coeff[W * a.rows];
          norm2 = before - removed;
          known = removed <= 1e-8 * before;
        }
        __syncthreads();
      }
      if (!known)
      {
        sums(3, 0, true);
        norm2 = coeff[0];
      }
      const double norm = sqrt(fmax(norm2, 0.0)), inv = 1.0 / fmax(norm, 1e-300);
      if (a.beta && blockIdx.x == 0 && threadIdx.x == 0) *a.beta = norm;
      for (int64_t i = threadIdx.x; i < len; i += blockDim.x) a.to[lo + i] = y[i] * inv;
    }

    // The counters and the error flag of a call's launches, zero.
    __global__ void clear_kernel(unsigned *counters, int count)
    {
      dependent_entry();
      for (int i = threadIdx.x; i < count; i += blockDim.x) counters[i] = 0;
    }

    // The number of eigenvalues of the symmetric tridiagonal (diagonal a, off-diagonal b) below x: the
    // negative pivots of the LDL^T factorisation of T - x I (Sturm's sequence); a zero pivot is taken
    // as a tiny negative one.
    __device__ int below(const double *a, const double *b, int n, double x, double pivmin)
    {
      int count = 0;
      double d = a[0] - x;
      for (int i = 0;; ++i)
      {
        if (fabs(d) < pivmin) d = -pivmin;
        if (d < 0.0) ++count;
        if (i + 1 == n) break;
        d = (a[i + 1] - x) - b[i] * b[i] / d;
      }
      return count;
    }

    // The same count in FP32, on values scaled to at most one.
    __device__ int below32(const float *a, const float *b, int n, float x)
    {
      int count = 0;
      float d = a[0] - x;
      for (int i = 0;; ++i)
      {
        if (fabsf(d) < 1e-30f) d = -1e-30f;
        if (d < 0.0f) ++count;
        if (i + 1 == n) break;
        d = (a[i + 1] - x) - __fdividef(b[i] * b[i], d);
      }
      return count;
    }

    // One solve (T - shift I) y = v in place, by elimination with partial pivoting (the tridiagonal's
    // upper factor has two superdiagonals), by one thread; one reciprocal a row.  A pivot below `tiny`
    // is taken as it.
    template <typename T>
    __device__ void shifted_solve(const T *a, const T *b, int n, T shift, T tiny, T *v, T *d, T *du, T *du2)
    {
      T dnext = a[0] - shift, unext = n > 1 ? b[0] : T(0);
      T vi = v[0];
      for (int i = 0; i + 1 < n; ++i)
      {
        // row i is (dnext, unext, 0) with right side vi, row i + 1 (dl, dd, uu) with v[i + 1]
        const T dl = b[i], dd = a[i + 1] - shift, uu = i + 2 < n ? b[i + 1] : T(0), vn = v[i + 1];
        if (fabs(dnext) >= fabs(dl))
        {
          const T piv = fabs(dnext) < tiny ? tiny : dnext;
          const T r = T(1) / piv, f = dl * r;
          d[i] = r;
          du[i] = unext;
          du2[i] = T(0);
          v[i] = vi;
          dnext = dd - f * unext;
          vi = vn - f * vi;
          unext = uu;
        }
        else
        {
          // rows i and i + 1 swapped
          const T r = T(1) / dl, f = dnext * r;
          d[i] = r;
          du[i] = dd;
          du2[i] = uu;
          v[i] = vn;
          dnext = unext - f * dd;
          vi = vi - f * vn;
          unext = -f * uu;
        }
      }
      d[n - 1] = T(1) / (fabs(dnext) < tiny ? tiny : dnext);
      T x1 = vi * d[n - 1], x2 = T(0);
      v[n - 1] = x1;
      for (int i = n - 2; i >= 0; --i)
      {
        const T x = (v[i] - du[i] * x1 - du2[i] * x2) * d[i];
        x2 = x1;
        x1 = x;
        v[i] = x;
      }
    }

    // v over its largest component and then its norm, that component positive.
    template <typename T>
    __device__ void unit(T *v, int n)
    {
      int big = 0;
      for (int i = 1; i < n; ++i)
        if (fabs(v[i]) > fabs(v[big])) big = i;
      const T top = T(1) / v[big];
      T norm2 = T(0);
      for (int i = 0; i < n; ++i)
      {
        v[i] *= top;
        norm2 = fma(v[i], v[i], norm2);
      }
      const T inv = T(1) / sqrt(norm2);
      for (int i = 0; i < n; ++i) v[i] *= inv;
    }

    // The Krylov space's lowest Ritz pair on the device, one warp: the size of the space (the steps
    // before the first beta below `tol`, as the reference stops) and the tridiagonal's lowest
    // eigenpair.  An FP64 division chain costs this GPU some hundred nanoseconds a link (the FP64
    // multisection alone took most of 117 us for ten steps), so the pair is found in FP32 (multisection
    // of the Sturm count, the 32 lanes counting below 32 points of the bracket each round, then inverse
    // iteration) and refined in FP64 by Rayleigh quotient iteration, which converges cubically: one or
    // two solves.  It is kept when its residual is at round-off and the FP32 counts show one eigenvalue
    // around it and none below; otherwise (Ritz values closer than FP32 resolves) the FP64 multisection
    // from Gershgorin's bounds and inverse iteration find it (W. Kahan, "Accurate eigenvalues of a
    // symmetric tri-diagonal matrix", 1966; J. H. Wilkinson, "The Algebraic Eigenvalue Problem", 1965).
    __global__ void ritz_kernel(const double *tri, int32_t n_iter, double tol, const int *error, double *ritz, double *energy,
                                int32_t *size_out)
    {
      dependent_entry();
      __shared__ double a[kOrthoMaxRows], b[kOrthoMaxRows], v[kOrthoMaxRows], d[kOrthoMaxRows], du[kOrthoMaxRows],
        du2[kOrthoMaxRows], bracket[2], found, scale_of;
      __shared__ float a32[kOrthoMaxRows], b32[kOrthoMaxRows], v32[kOrthoMaxRows], d32[kOrthoMaxRows], du32[kOrthoMaxRows],
        du232[kOrthoMaxRows], bracket32[2];
      __shared__ int32_t shared_size, settled;
      const int lane = threadIdx.x;
      if (lane == 0)
      {
        int32_t size = n_iter;
        for (int32_t k = 0; k < n_iter; ++k)
          if (tri[n_iter + k] < tol)
          {
            size = k + 1;
            break;
          }
        shared_size = size;
      }
      __syncwarp();
      const int n = shared_size;
      for (int i = lane; i < n; i += 32)
      {
        a[i] = tri[i];
        b[i] = i + 1 < n ? tri[n_iter + i] : 0.0;
      }
      __syncwarp();
      if (lane == 0)
      {
        double scale = 0.0, lo = a[0], hi = a[0];
        for (int i = 0; i < n; ++i)
        {
          const double r = (i > 0 ? fabs(b[i - 1]) : 0.0) + fabs(b[i]);
          scale = fmax(scale, fabs(a[i]) + r);
          lo = fmin(lo, a[i] - r);
          hi = fmax(hi, a[i] + r);
        }
        scale_of = scale;
        bracket[0] = lo;
        bracket[1] = hi;
        settled = 0;
      }
      __syncwarp();
      const double scale = scale_of, pivmin = fmax(scale, 1.0) * 1e-290;
      if (scale > 0.0 && scale < 1e300)
      {
        const double inv = 1.0 / scale;
        for (int i = lane; i < n; i += 32)
        {
          a32[i] = static_cast<float>(a[i] * inv);
          b32[i] = static_cast<float>(b[i] * inv);
        }
        if (lane == 0)
        {
          bracket32[0] = static_cast<float>(bracket[0] * inv) - 1e-6f;
          bracket32[1] = static_cast<float>(bracket[1] * inv) + 1e-6f;
        }
        __syncwarp();
        for (int round = 0; round < 8; ++round)
        {
          const float lo = bracket32[0], hi = bracket32[1];
          if (!(hi - lo > 2.4e-7f * fmaxf(fabsf(lo), fabsf(hi))) || !(hi > lo)) break;
          const float x = lo + (hi - lo) * static_cast<float>(lane + 1) / 33.0f;
          const unsigned hits = __ballot_sync(0xffffffffu, below32(a32, b32, n, x) >= 1);
          __syncwarp();
          if (lane == 0)
          {
            const int first = hits ? __ffs(hits) - 1 : 32;
            const float step = (hi - lo) / 33.0f;
            bracket32[0] = first == 0 ? lo : lo + step * first;
            bracket32[1] = first == 32 ? hi : lo + step * (first + 1);
          }
          __syncwarp();
        }
        const float at = 0.5f * (bracket32[0] + bracket32[1]);
        // one eigenvalue within the FP32 resolution of `at`, none below
        const float near = 1e-6f * static_cast<float>(n);
        const int count = below32(a32, b32, n, lane == 0 ? at - near : at + near);
        const bool alone = __shfl_sync(0xffffffffu, count, 0) == 0 && __shfl_sync(0xffffffffu, count, 1) == 1;
        if (alone && lane == 0)
        {
          for (int i = 0; i < n; ++i) v32[i] = 1.0f;
          for (int it = 0; it < 3; ++it)
          {
            shifted_solve<float>(a32, b32, n, at, 1e-12f, v32, d32, du32, du232);
            unit(v32, n);
          }
        }
        __syncwarp();
        if (alone)
        {
          for (int i = lane; i < n; i += 32) v[i] = v32[i];
          __syncwarp();
          for (int it = 0; it < 5; ++it)
          {
            // the Rayleigh quotient and the residual of v, the lanes sharing the rows
            double vv = 0.0, vtv = 0.0;
            for (int i = lane; i < n; i += 32)
            {
              const double t = a[i] * v[i] + (i > 0 ? b[i - 1] * v[i - 1] : 0.0) + (i + 1 < n ? b[i] * v[i + 1] : 0.0);
              vv = fma(v[i], v[i], vv);
              vtv = fma(v[i], t, vtv);
            }
            vv = lane_sum(vv);
            const double rho = lane_sum(vtv) / vv;
            double worst = 0.0;
            for (int i = lane; i < n; i += 32)
            {
              const double t = (a[i] - rho) * v[i] + (i > 0 ? b[i - 1] * v[i - 1] : 0.0) + (i + 1 < n ? b[i] * v[i + 1] : 0.0);
              worst = fmax(worst, fabs(t));
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) worst = fmax(worst, __shfl_xor_sync(0xffffffffu, worst, off));
            if (worst <= 4.0 * 2.220446049250313e-16 * scale * sqrt(vv))
            {
              if (lane == 0)
              {
                found = rho;
                settled = fabs(rho * inv - static_cast<double>(at)) <= static_cast<double>(near);
              }
              break;
            }
            if (lane == 0)
            {
              shifted_solve<double>(a, b, n, rho, scale * 1e-290, v, d, du, du2);
              unit(v, n);
            }
            __syncwarp();
          }
          __syncwarp();
        }
      }
      __syncwarp();
      if (!settled)
      {
        for (int round = 0; round < 64; ++round)
        {
          const double lo = bracket[0], hi = bracket[1];
          if (!(hi - lo > 4.0 * 2.220446049250313e-16 * fmax(fabs(lo), fabs(hi))) || !(hi > lo)) break;
          const double x = lo + (hi - lo) * static_cast<double>(lane + 1) / 33.0;
          const bool any = below(a, b, n, x, pivmin) >= 1;
          const unsigned hits = __ballot_sync(0xffffffffu, any);
          __syncwarp();
          if (lane == 0)
          {
            // the first point with an eigenvalue below it closes the bracket of the lowest one
            const int first = hits ? __ffs(hits) - 1 : 32;
            const double step = (hi - lo) / 33.0;
            bracket[0] = first == 0 ? lo : lo + step * first;
            bracket[1] = first == 32 ? hi : lo + step * (first + 1);
          }
          __syncwarp();
        }
        if (lane == 0)
        {
          found = 0.5 * (bracket[0] + bracket[1]);
          for (int i = 0; i < n; ++i) v[i] = 1.0;
          for (int it = 0; it < 3; ++it)
          {
            shifted_solve<double>(a, b, n, found, pivmin, v, d, du, du2);
            unit(v, n);
          }
        }
      }
      __syncwarp();
      // a wait that gave up shows in the energy
      const bool failed = *error != 0;
      if (lane == 0)
      {
        *energy = failed ? __longlong_as_double(0x7ff8000000000000ll) : found;
        *size_out = n;
      }
      // the largest component positive
      double top = 0.0;
      for (int i = 0; i < n; ++i)
        if (fabs(v[i]) > fabs(top)) top = v[i];
      for (int k = lane; k < n; k += 32) ritz[k] = top < 0.0 ? -v[k] : v[k];
    }

    int64_t up32(int64_t x) { return (x + 31) / 32 * 32; }

    // CTAs of an ortho launch: one per SM at most, each with at least a warp's worth of work a lane
    int ortho_parts(int64_t n_doubles) { return static_cast<int>(std::clamp<int64_t>((n_doubles + 191) / 192, 1, device_sms())); }

    cudaError_t launch_ortho(const OrthoArgs &args, bool complex, int parts, cudaStream_t stream)
    {
      static std::once_flag once;
      static cudaError_t configured = cudaSuccess;
      std::call_once(once, [] {
        configured = cudaFuncSetAttribute(ortho_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kOrthoSmem));
        if (configured == cudaSuccess)
          configured = cudaFuncSetAttribute(ortho_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kOrthoSmem));
      });
      if (configured != cudaSuccess) return configured;
      cudaLaunchConfig_t config = {};
      config.gridDim = dim3(static_cast<unsigned>(parts));
      config.blockDim = dim3(kOrthoThreads);
      config.dynamicSmemBytes = args.part * 8 <= kOrthoSmem ? static_cast<size_t>(args.part * 8) : 0;
      config.stream = stream;
      // its CTAs wait on one another: all resident together
      cudaLaunchAttribute attribute[2];
      attribute[0].id = cudaLaunchAttributeCooperative;
      attribute[0].val.cooperative = 1;
      attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attribute[1].val.programmaticStreamSerializationAllowed = 1;
      config.attrs = attribute;
      config.numAttrs = 2;
      return complex ? cudaLaunchKernelEx(&config, ortho_kernel<true>, args) : cudaLaunchKernelEx(&config, ortho_kernel<false>, args);
    }
  } // namespace

  int64_t lanczos_scratch_doubles(int64_t n_doubles, int32_t n_iter)
  {
    const int64_t rows = n_iter + 1;
    // basis, image, the CTAs' sums, alpha and beta, Ritz coefficients with the energy and the size after
    // them, a vector's work space, counters
    return up32(rows * n_doubles) + up32(n_doubles) + up32(8 * (rows + 1) * ortho_parts(n_doubles)) + up32(2 * rows) +
           up32(rows + 2) + up32(n_doubles) + up32(2 * (n_iter + 3));
  }

  cudaError_t lanczos(const Program &p, DeviceTables &t, const ExecArgs &base, int32_t vector_operand,
                      const double *start, int64_t n_doubles, int32_t n_iter, double tol, double *scratch,
                      double *result, double *energy_dev, int32_t *size_dev)
  {
    const bool complex = base.complex;
    const int64_t rows = n_iter + 1;
    const int parts = ortho_parts(n_doubles);
    double *basis = scratch;
    double *image = basis + up32(rows * n_doubles);
    double *partial = image + up32(n_doubles);
    double *tri = partial + up32(8 * (rows + 1) * parts);  // alpha[0..n_iter), beta[n_iter..2 n_iter)
    double *ritz = tri + up32(2 * rows);
    double *work = ritz + up32(rows + 2);
    unsigned *counters = reinterpret_cast<unsigned *>(work + up32(n_doubles));  // four a launch, n_iter + 2 launches, the flag
    int *error = reinterpret_cast<int *>(counters + 4 * (n_iter + 2));
    cudaStream_t stream = base.stream;
    cudaError_t e;
    if ((e = launch_dependent(clear_kernel, 1, 128, 0, stream, counters, 4 * (n_iter + 2) + 1)) != cudaSuccess) return e;
    OrthoArgs args{};
    args.basis = basis;
    args.work = work;
    args.partial = partial;
    args.error = error;
    args.n = n_doubles;
    args.part = ((n_doubles + parts - 1) / parts + 1) / 2 * 2;
    // basis[0] = start / |start|
    args.from = start;
    args.to = basis;
    args.arrived = counters;
    if ((e = launch_ortho(args, complex, parts, stream)) != cudaSuccess) return e;
    std::vector<const void *> inputs(base.inputs, base.inputs + p.n_inputs);
    args.from = image;
    args.passes = 3;
    for (int32_t k = 0; k < n_iter; ++k)
    {
      double *row = basis + static_cast<int64_t>(k) * n_doubles;
      ExecArgs exec = base;
      inputs[static_cast<size_t>(vector_operand)] = row;
      exec.inputs = inputs.data();
      exec.output = image;
      if ((e = execute(p, t, exec)) != cudaSuccess) return e;
      args.rows = k + 1;
      args.to = row + n_doubles;
      args.alpha = tri + k;
      args.beta = tri + n_iter + k;
      args.arrived = counters + 4 * (k + 1);
      if ((e = launch_ortho(args, complex, parts, stream)) != cudaSuccess) return e;
    }
    // the lowest Ritz pair of the tridiagonal (the steps after the first beta below tol dropped, as
    // the reference stops there), then the normalised Ritz vector
    if ((e = launch_dependent(ritz_kernel, 1, 32, 0, stream, static_cast<const double *>(tri), n_iter, tol,
                              static_cast<const int *>(error), ritz, energy_dev, size_dev)) != cudaSuccess)
      return e;
    args.from = nullptr;
    args.c = ritz;
    args.size = size_dev;
    args.to = result;
    args.alpha = args.beta = nullptr;
    args.rows = args.passes = 0;
    args.arrived = counters + 4 * (n_iter + 1);
    if ((e = launch_ortho(args, complex, parts, stream)) != cudaSuccess) return e;
    return cudaGetLastError();
  }

  double *lanczos_energy_slot(double *scratch, int64_t n_doubles, int32_t n_iter)
  {
    const int64_t rows = n_iter + 1;
    return scratch + up32(rows * n_doubles) + up32(n_doubles) + up32(8 * (rows + 1) * ortho_parts(n_doubles)) + up32(2 * rows) + rows;
  }

} // namespace ttg

// Thin SVDs of the blocks of a tensor in one launch, for the truncating splittings
// (tentorch/linalg/graded/svd.cpp:41-177, which calls at::linalg_svd once per block).
//
// Method: one-sided Jacobi (Hestenes 1958; the rotation of Rutishauser as in Demmel & Veselic,
// "Jacobi's method is more accurate than QR", SIAM J. Matrix Anal. Appl. 13 (1992)).  The columns
// of W (the block, or its transpose when it is wider than tall, so that W has k = min(m, n)
// columns) are rotated in pairs until every pair is orthogonal to working precision; then the
// column norms are the singular values, the normalised columns one set of singular vectors and
// the accumulated rotations V the other.  U and V come out orthonormal to round-off, which a
// truncating DMRG needs for the kept vectors however small their values.
//
// FP64 on this GPU runs at about 1/64 of the FP32 rate (about two FP64 multiply-adds per clock
// per SM), so the rotations run in FP32 and FP64 only refines what they leave:
//   0. the columns sorted by norm and factored A P = Q R; the rest works on the graded X = R^T, and
//      U = Q J at the end (Drmac & Veselic 2008).
//   1. FP32 sweeps on a scaled copy until its columns are orthogonal to ~1e-5; they give a rotation
//      close to the right singular vectors, small columns included (their cosines are formed without
//      squares that underflow).  Blocks of four columns at a time (blocked_sweeps), or column by column
//      for columns beyond 320.
//   2. V refined in FP64 by matrix products: from the Gram matrices of W = X V and of V, all pairs' angles
//      at once and V's orthonormality, quadratically (1e-5 -> 1e-9 -> round-off), three or four times.
//   3. where the refinement does not settle (singular values closer than FP32 separates): V made
//      orthonormal by two Newton-Schulz steps, W = X V, and FP64 sweeps on W with V accumulated; a
//      sweep whose cosines were all below sqrt(tol) is the last (the cosines it leaves are below ~tol).
// In the FP64 sweeps only the dot product of the pair is taken (the squared column norms are
// carried along with the exact update of a rotation and recomputed at each sweep's start), and the
// angle is found in FP32 and then made exactly orthogonal in FP64 (c^2 + s^2 = 1 by a second-order
// correction): an angle good to 1e-7 still shrinks the pair's cosine by that factor each rotation.
//
// One launch, one block of 148 x 148 / 92 x 92 / 31 x 31 with singular values over twelve decades: 2782 / 1378 /
// 466 us; with FP32 sweeps column by column that skipped the small columns and 3 to 6 FP64 sweeps 7557 /
// 3783 / 2152 us.  Factors orthonormal to 1e-15 (3e-15 before; clusters of values 1e-9 apart 1e-11, 1e-7
// before).  At 148 columns now: QR 0.56 ms, FP32 sweeps 1.16 (eight), refinement 0.7, U = Q J 0.27.
//
// A thread-block cluster of up to 16 CTAs per block, which shares every step: QR by columns, FP32 sweeps
// by pairs of column blocks in distributed shared memory, the products by tiles, the FP64 sweeps with
// the rows of W and V dealt to the ranks and the dot products of each round summed over the cluster.
// Each sweep runs the pairs in the round-robin (circle) order.  Working sets sit in shared memory
// when they fit (227 KB per CTA), else in the global workspace (L2 resident).  At most kMaxSweeps
// sweeps per phase; a block whose FP64 phase did not converge, or with a value that is not finite or
// below 1e-128 of the block, reports -1 in `info` (the host hands it to at::linalg_svd, or raises on a NaN).
// All loops are bounded and every CTA of a cluster passes the same sequence of cluster barriers: what
// ends a loop is the same on every rank.
//
// A second kernel writes the kept part of each block's factors into the two output arenas, with
// the singular values absorbed as the caller asks, so that a whole truncating split is two
// launches and one read of the singular values.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>

#include "executor.h"
#include "reflector.cuh"

namespace ttg
{
  namespace
  {
    namespace cg = cooperative_groups;

    constexpr int kSvdThreads = 512;
    constexpr int kBlockExp = 200;              // blocks are worked on with their largest entry at about 2^200
    constexpr double kLeastSquare = 0x1p-450;   // there: columns whose squared norm is below have no direction to be trusted
    constexpr int kMaxSweeps = 40;
    constexpr int kMaxCols = 1024;              // k = min(rows, cols) of a block
    constexpr int kSvdSmemBytes = 227 * 1024;
    constexpr int kStaticBytes = 21 * 1024;     // the norms, their shares, ranks and flags of the kernel
    constexpr int64_t kDynamicBytes = kSvdSmemBytes - kStaticBytes - 1024;
    constexpr int kTile = 32;                   // tiles of the Newton-Schulz and W = A V products
    constexpr int64_t kStageBytes = 2 * kTile * (kTile + 1) * 8;
    // the end of the dynamic shared memory holds the tile stages (Newton-Schulz, W = A V) or, during
    // sweeps over a cluster, the dot-product shares every rank pushes to every rank
    __host__ __device__ inline int64_t exchange_bytes(int64_t k, int64_t ranks, int64_t size)
    {
      const int64_t pairs = (k + (k & 1)) / 2;
      return ranks > 1 ? (2 * ranks * pairs * size + 15) / 16 * 16 : 0;
    }
    constexpr int kMaxCluster = 16;
    constexpr int kNper = 12;                   // entries of a column each lane of a pair holds

    // per block: a_off, rows, cols, u_off, s_off, vh_off, ws_off (doubles)
    struct SvdEntry
    {
      int64_t a_off, rows, cols, u_off, s_off, vh_off, ws_off;
    };

    // One block's global workspace, in doubles: V and its next iterate (k x k each) and G = V^T V
    // for the Newton-Schulz steps; W (len x k) and V (k x k) by rank for working sets that do not
    // fit in shared memory (up to kMaxCluster - 1 padding rows each), in FP64 and again in FP32.
    // For a block preconditioned by QR: its columns in their sorted order factored in place (R on
    // and above the diagonal, the Householder vectors below it; len x k, column-major), the
    // Householder scalars, the sorted order (k indices), and the product Q [J; 0] (len x k).
    struct SvdLayout
    {
      int64_t v0, v1, g, w_slices, v_slices, w32_slices, v32_slices, f, tau, order, b, total;
    };
    __host__ __device__ inline SvdLayout svd_layout(int64_t len, int64_t k)
    {
      SvdLayout l;
      l.v0 = 0;
      l.v1 = k * k;
      l.g = 2 * k * k;
      l.w_slices = 3 * k * k;
      l.v_slices = l.w_slices + (len + kMaxCluster) * k;
      l.w32_slices = l.v_slices + (k + kMaxCluster) * k;
      l.v32_slices = l.w32_slices + ((len + kMaxCluster) * k + 1) / 2;  // (together k^2 doubles and more)
      l.f = l.v32_slices + ((k + kMaxCluster) * k + 1) / 2;
      l.tau = l.f + len * k;
      l.order = l.tau + k;
      l.b = l.order + k;
      l.total = l.b + len * k;
      l.total = (l.total + 31) / 32 * 32;
      return l;
    }
    // Blocks of at least this many columns are preconditioned by QR (below 32 columns, on one CTA, it
    // costs little, and the refinement needs the graded columns it leaves).
    constexpr int64_t kQrMinCols = 2;
    // The longest columns whose reflectors one warp makes ahead of the step; longer ones are made by their CTA (one
    // block, us, one warp against the CTA: 148 x 148 2729 and 2954, 300 x 150 3344 and 3467, 600 x 100 both 2929,
    // 1000 x 100 4060 and 3814, 1500 x 60 2827 and 2421).
    constexpr int64_t kAheadRows = 600;

    // The circle method's pair t of a round (players even, round < players - 1, t < players / 2):
    // player players - 1 stays, the others turn; p < q.  In 32-bit arithmetic with one conditional
    // subtraction each instead of a 64-bit remainder, which costs a long instruction sequence.
    __device__ __forceinline__ void circle_pair(int64_t round, int64_t t, int64_t players, int64_t &p, int64_t &q)
    {
      const int32_t n = static_cast<int32_t>(players - 1), r = static_cast<int32_t>(round), u = static_cast<int32_t>(t);
      int32_t a, b;
      if (u == 0)
      {
        a = r;
        b = n;
      }
      else
      {
        a = r + u;
        if (a >= n) a -= n;
        b = r - u + n;
        if (b >= n) b -= n;
      }
      p = a < b ? a : b;
      q = a < b ? b : a;
    }

    template <typename T>
    __device__ __forceinline__ T warp_sum(T v)
    {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      return v;
    }

    // The rotation that makes the pair (alpha = |w_p|^2, beta = |w_q|^2, gamma = w_p . w_q)
    // orthogonal: w_p' = c w_p - s w_q, w_q' = s w_p + c w_q with t = s / c the smaller root of
    // t^2 + 2 zeta t - 1 = 0, zeta = (beta - alpha) / (2 gamma).  Found in FP32 on values scaled
    // by a power of two; false when gamma is negligible at that scale.
    // (`diff` is b - a: in FP64 taken before the rounding to FP32, so that close norms keep their
    // difference.)
    __device__ __forceinline__ bool angle_of(float diff, float g, float &c, float &s)
    {
      if (g == 0.0f) return false;
      const float zeta = diff / (2.0f * g);
      const float t = fabsf(zeta) > 1e15f ? 0.5f / zeta : copysignf(1.0f, zeta) / (fabsf(zeta) + sqrtf(1.0f + zeta * zeta));
      c = rsqrtf(1.0f + t * t);
      s = c * t;
      return true;
    }

    // The same with the hardware's approximate reciprocal and reciprocal root (a few units in the last
    // place, like the rotations' own rounding; V is made orthonormal afterwards).
    __device__ __forceinline__ bool angle_fast(float diff, float g, float &c, float &s)
    {
      if (g == 0.0f) return false;
      const float zeta = __fdividef(diff, 2.0f * g), one = fmaf(zeta, zeta, 1.0f);
      const float t = fabsf(zeta) > 1e15f ? __fdividef(0.5f, zeta)
                                          : copysignf(__fdividef(1.0f, fabsf(zeta) + one * rsqrtf(one)), zeta);
      c = rsqrtf(fmaf(t, t, 1.0f));
      s = c * t;
      return true;
    }

    // FP32 columns are scaled to |entries| <= 1, so their squared norms neither overflow nor lose
    // the angle; FP64 ones are brought to that scale by a power of two first
    __device__ __forceinline__ bool angle(float alpha, float beta, float gamma, float &c, float &s)
    {
      return angle_of(beta - alpha, gamma, c, s);
    }
    __device__ __forceinline__ bool angle(double alpha, double beta, double gamma, float &c, float &s)
    {
      int ex;
      frexp(fmax(alpha, beta), &ex);
      return angle_of(static_cast<float>(ldexp(beta - alpha, -ex)), static_cast<float>(ldexp(gamma, -ex)), c, s);
    }

    // Whether the pair's cosine is above `limit`.  In FP32 the squares of the smaller columns' products
    // would underflow (columns 1e-10 of the largest and below were never rotated so, and were left to
    // the FP64 sweeps), so the cosine itself is formed.
    __device__ __forceinline__ bool above(float gamma, float alpha, float beta, float limit)
    {
      return fabsf(gamma) * rsqrtf(alpha) * rsqrtf(beta) > limit;
    }
    __device__ __forceinline__ bool above(double gamma, double alpha, double beta, double limit)
    {
      return gamma * gamma > limit * limit * alpha * beta;
    }

    template <typename T, int G>
    __device__ __forceinline__ T group_sum(T v)
    {
      if constexpr (G > 1)
      {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, G);
      }
      return v;
    }

    // A pair's columns as a group of G lanes holds them: lane gl has entries gl, gl + G, ... of
    // each, the first kNper in registers (loads issued together, one latency), any further ones
    // read again where needed.  Register slots past the column's length are skipped whole (the
    // count is the same for every lane), so no FP64 instruction is spent on padding.
    template <typename T, int G>
    __device__ __forceinline__ T pair_dot(const T *wp, const T *wq, int64_t n, int gl, T (&x)[kNper], T (&y)[kNper])
    {
      const int64_t slots = (n + G - 1) / G;
#pragma unroll
      for (int u = 0; u < kNper; ++u)
      {
        const int64_t i = gl + static_cast<int64_t>(u) * G;
        x[u] = u < slots && i < n ? wp[i] : T(0);
        y[u] = u < slots && i < n ? wq[i] : T(0);
      }
      T sum = 0;
#pragma unroll
      for (int u = 0; u < kNper; ++u)
        if (u < slots) sum = fma(x[u], y[u], sum);
      for (int64_t i = static_cast<int64_t>(G) * kNper + gl; i < n; i += G) sum = fma(wp[i], wq[i], sum);
      return sum;
    }

    template <typename T, int G>
    __device__ __forceinline__ void pair_rotate(T *wp, T *wq, int64_t n, int gl, const T (&x)[kNper], const T (&y)[kNper],
                                                T c, T sn)
    {
      const int64_t slots = (n + G - 1) / G;
#pragma unroll
      for (int u = 0; u < kNper; ++u)
      {
        const int64_t i = gl + static_cast<int64_t>(u) * G;
        if (u < slots && i < n)
        {
          wp[i] = fma(c, x[u], -sn * y[u]);
          wq[i] = fma(sn, x[u], c * y[u]);
        }
      }
      for (int64_t i = static_cast<int64_t>(G) * kNper + gl; i < n; i += G)
      {
        const T a = wp[i], b = wq[i];
        wp[i] = fma(c, a, -sn * b);
        wq[i] = fma(sn, a, c * b);
      }
    }

    // rotate two columns in chunks of kNper entries per lane (each chunk's loads issued together)
    template <typename T, int G>
    __device__ __forceinline__ void cols_rotate(T *vp, T *vq, int64_t n, int gl, T c, T sn)
    {
      for (int64_t base = 0; base < n; base += static_cast<int64_t>(G) * kNper)
      {
        const int64_t slots = (n - base + G - 1) / G;
        T x[kNper], y[kNper];
#pragma unroll
        for (int u = 0; u < kNper; ++u)
        {
          const int64_t i = base + gl + static_cast<int64_t>(u) * G;
          x[u] = u < slots && i < n ? vp[i] : T(0);
          y[u] = u < slots && i < n ? vq[i] : T(0);
        }
#pragma unroll
        for (int u = 0; u < kNper; ++u)
        {
          const int64_t i = base + gl + static_cast<int64_t>(u) * G;
          if (u < slots && i < n)
          {
            vp[i] = fma(c, x[u], -sn * y[u]);
            vq[i] = fma(sn, x[u], c * y[u]);
          }
        }
      }
    }

    // The rotation of a pair as FP64 values with c^2 + s^2 = 1 to FP64 precision, from the FP32
    // angle: with c, s exact in FP64, d = c^2 + s^2 - 1 (~1e-7) is exact to FP64 rounding and
    // 1 / sqrt(1 + d) = 1 - d/2 + 3 d^2/8 to below 1e-20.
    __device__ __forceinline__ void exact_rotation(float cf, float sf, double &c, double &sn)
    {
      c = cf;
      sn = sf;
      const double d = fma(sn, sn, fma(c, c, -1.0));
      const double f = fma(d, fma(0.375, d, -0.5), 1.0);
      c *= f;
      sn *= f;
    }
    __device__ __forceinline__ void exact_rotation(float cf, float sf, float &c, float &sn)
    {
      c = cf;
      sn = sf;
    }

    // Jacobi sweeps over W (column-major, `rows` rows) with the rotations accumulated into V
    // (`vrows` rows), until a sweep rotates no pair whose cosine is above sqrt(tol) (or
    // kMaxSweeps); pairs below tol are not rotated.  Alone, one CTA holds every
    // row; otherwise the rows are dealt to the CTAs of the cluster: per round each CTA takes its
    // rows' share of every pair's dot product, the shares cross the cluster through distributed
    // shared memory and every CTA adds them in the same order, so that all hold the same dot
    // products, angles and norms, and rotates its own rows.  One cluster barrier per round (shares
    // double-buffered) and two per sweep; whether a sweep ended the phase is read from rank 0, so
    // every CTA leaves the loop together.  FP32: everything in FP32; FP64: the angle in FP32 made
    // exactly orthogonal in FP64 (exact_rotation; an angle good to 1e-7 still shrinks the pair's
    // cosine by that factor each rotation).  Only the pair's dot product is taken: the squared norms are
    // recomputed at each sweep's start and carried with each rotation's exact update.
    template <typename T, int G>
    __device__ int sweeps(const cg::cluster_group &cluster, bool alone, T *w, int64_t rows, T *v, int64_t vrows, int64_t k,
                          double tol, T *norms, T *exchange, T *partial, int *flags, int *list)
    {
      const unsigned ranks = alone ? 1u : cluster.num_blocks(), me = alone ? 0u : cluster.block_rank();
      const auto sync = [&] {
        if (alone) __syncthreads();
        else cluster.sync();
      };
      const auto at_rank = [&](T *local, unsigned r) -> const T * { return alone ? local : cluster.map_shared_rank(local, r); };
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
      const int group = lane / G, gl = lane % G;
      constexpr int per_warp = 32 / G;
      const int64_t players = k + (k & 1), pairs = players / 2;
      const T least = static_cast<T>(tol);
      // a sweep whose rotations all had cosines below sqrt(tol) ends the phase: Jacobi converges
      // quadratically there, so the cosines it leaves are below ~tol and a further sweep (which
      // would find nothing above tol to rotate) is not run
      const T settled = static_cast<T>(sqrt(tol));
      // FP64 over a cluster: after the barrier a group of lanes per pair finds the rotation (the
      // scalar part) and lists it, then the whole CTA rotates the listed pairs' entries, so that
      // the FP64 instructions of the rotations spread over every warp instead of the few that hold
      // the pairs (FP64 issue is the bound of a round).  The rotations of a round are listed in
      // `list` and `partial` (free during the rounds: the other ranks read `partial` only at the
      // sweep's start, before the first round's barrier); flags[4] counts them.
      constexpr bool kSpread = std::is_same_v<T, double>;
      for (int sweep = 0; sweep < kMaxSweeps; ++sweep)
      {
        for (int64_t j = warp; j < k; j += warps)
        {
          const T *wj = w + j * rows;
          T sum = 0;
          for (int64_t i = lane; i < rows; i += 32) sum = fma(wj[i], wj[i], sum);
          sum = warp_sum(sum);
          if (lane == 0) partial[j] = sum;
        }
        if (threadIdx.x == 0) flags[sweep & 1] = 0;
        sync();
        for (int64_t j = threadIdx.x; j < k; j += blockDim.x)
        {
          T sum = 0;
          for (unsigned r = 0; r < ranks; ++r) sum += at_rank(partial, r)[j];
          norms[j] = sum;
        }
        __syncthreads();
        for (int64_t round = 0; round + 1 < players; ++round)
        {
          // this round's shares: [rank][pair], double-buffered by rounds
          T *share = exchange + (round & 1) * static_cast<int64_t>(ranks) * pairs;
          // every group of a warp walks the same number of turns, so the shuffles stay converged
          for (int64_t t0 = static_cast<int64_t>(warp) * per_warp; t0 < pairs; t0 += static_cast<int64_t>(warps) * per_warp)
          {
            const int64_t t = t0 + group;
            int64_t p, q;
            circle_pair(round, t, players, p, q);
            const bool pair = t < pairs && q < k;
            T x[kNper], y[kNper];
            T *wp = w + (pair ? p : 0) * rows, *wq = w + (pair ? q : 0) * rows;
            T gamma = pair_dot<T, G>(wp, wq, pair ? rows : 0, gl, x, y);
            gamma = group_sum<T, G>(gamma);
            if (!alone && t < pairs)
            {
              // this CTA's share goes to every rank (remote stores do not wait); after the barrier
              // each rank holds every share in its own memory
              for (unsigned r = gl; r < ranks; r += G) cluster.map_shared_rank(share + static_cast<int64_t>(me) * pairs + t, r)[0] = gamma;
            }
            if (alone)
            {
              if (!pair) continue;
              const T alpha = norms[p], beta = norms[q];
              if (!above(gamma, alpha, beta, least)) continue;
              float cf, sf;
              if (!angle(alpha, beta, gamma, cf, sf)) continue;
              T c, sn;
              exact_rotation(cf, sf, c, sn);
              pair_rotate<T, G>(wp, wq, rows, gl, x, y, c, sn);
              cols_rotate<T, G>(v + p * vrows, v + q * vrows, vrows, gl, c, sn);
              if (gl == 0)
              {
                const T cc = c * c, ss = sn * sn, cs2 = 2 * c * sn * gamma;
                norms[p] = cc * alpha - cs2 + ss * beta;
                norms[q] = ss * alpha + cs2 + cc * beta;
                if (above(gamma, alpha, beta, settled)) flags[sweep & 1] = 1;
              }
            }
          }
          if (!alone)
          {
            cluster.sync();
            if constexpr (kSpread)
            {
              T *lc = partial, *ls = partial + pairs;
              if (threadIdx.x == 0) flags[4] = 0;
              __syncthreads();
              for (int64_t t0 = static_cast<int64_t>(warp) * per_warp; t0 < pairs; t0 += static_cast<int64_t>(warps) * per_warp)
              {
                const int64_t t = t0 + group;
                int64_t p, q;
                circle_pair(round, t, players, p, q);
                const bool pair = t < pairs && q < k;
                T gamma = 0;
                if (pair)
                  for (unsigned r = gl; r < ranks; r += G) gamma += share[static_cast<int64_t>(r) * pairs + t];
                gamma = group_sum<T, G>(gamma);
                if (!pair || gl != 0) continue;
                const T alpha = norms[p], beta = norms[q];
                if (!above(gamma, alpha, beta, least)) continue;
                float cf, sf;
                if (!angle(alpha, beta, gamma, cf, sf)) continue;
                T c, sn;
                exact_rotation(cf, sf, c, sn);
                const T cc = c * c, ss = sn * sn, cs2 = 2 * c * sn * gamma;
                norms[p] = cc * alpha - cs2 + ss * beta;
                norms[q] = ss * alpha + cs2 + cc * beta;
                if (above(gamma, alpha, beta, settled)) flags[sweep & 1] = 1;
                const int at = atomicAdd(flags + 4, 1);
                list[at] = static_cast<int>(t);
                lc[at] = c;
                ls[at] = sn;
              }
              __syncthreads();
              // entry i of a listed pair: row i of W (i < rows), else row i - rows of V
              const int span = static_cast<int>(rows + vrows), items = flags[4] * span;
              for (int it = threadIdx.x; it < items; it += blockDim.x)
              {
                const int at = it / span, i = it - at * span;
                int64_t p, q;
                circle_pair(round, list[at], players, p, q);
                const T c = lc[at], sn = ls[at];
                T *x = i < rows ? w + p * rows + i : v + p * vrows + (i - rows);
                T *y = i < rows ? w + q * rows + i : v + q * vrows + (i - rows);
                const T a = *x, b = *y;
                *x = fma(c, a, -sn * b);
                *y = fma(sn, a, c * b);
              }
            }
            else
            {
              for (int64_t t0 = static_cast<int64_t>(warp) * per_warp; t0 < pairs; t0 += static_cast<int64_t>(warps) * per_warp)
              {
                const int64_t t = t0 + group;
                int64_t p, q;
                circle_pair(round, t, players, p, q);
                const bool pair = t < pairs && q < k;
                // lane gl adds ranks gl, gl + G, ...; the group's butterfly sum then gives every lane
                // of every CTA the same value
                T gamma = 0;
                if (pair)
                  for (unsigned r = gl; r < ranks; r += G) gamma += share[static_cast<int64_t>(r) * pairs + t];
                gamma = group_sum<T, G>(gamma);
                if (!pair) continue;
                const T alpha = norms[p], beta = norms[q];
                if (!above(gamma, alpha, beta, least)) continue;
                float cf, sf;
                if (!angle(alpha, beta, gamma, cf, sf)) continue;
                T c, sn;
                exact_rotation(cf, sf, c, sn);
                cols_rotate<T, G>(w + p * rows, w + q * rows, rows, gl, c, sn);
                cols_rotate<T, G>(v + p * vrows, v + q * vrows, vrows, gl, c, sn);
                if (gl == 0)
                {
                  const T cc = c * c, ss = sn * sn, cs2 = 2 * c * sn * gamma;
                  norms[p] = cc * alpha - cs2 + ss * beta;
                  norms[q] = ss * alpha + cs2 + cc * beta;
                  if (above(gamma, alpha, beta, settled)) flags[sweep & 1] = 1;
                }
              }
            }
          }
          __syncthreads();
        }
        sync();
        const int any = alone ? flags[sweep & 1] : cluster.map_shared_rank(flags, 0)[sweep & 1];
        if (!any) return sweep + 1;
      }
      return -1;
    }

    template <typename T>
    __device__ int sweeps(const cg::cluster_group &cluster, bool alone, T *w, int64_t rows, T *v, int64_t vrows, int64_t k,
                          double tol, T *norms, T *exchange, T *partial, int *flags, int *list)
    {
      const int64_t most = rows > vrows ? rows : vrows;
      // the fewest lanes per pair that hold its rows in registers (measured faster than more lanes
      // with shorter chains, in FP32 as in FP64, where the per-pair scalar work also runs once per
      // lane of the group on the narrow FP64 pipe)
      if (most <= kNper) return sweeps<T, 1>(cluster, alone, w, rows, v, vrows, k, tol, norms, exchange, partial, flags, list);
      if (most <= 2 * kNper) return sweeps<T, 2>(cluster, alone, w, rows, v, vrows, k, tol, norms, exchange, partial, flags, list);
      if (most <= 4 * kNper) return sweeps<T, 4>(cluster, alone, w, rows, v, vrows, k, tol, norms, exchange, partial, flags, list);
      if (most <= 8 * kNper) return sweeps<T, 8>(cluster, alone, w, rows, v, vrows, k, tol, norms, exchange, partial, flags, list);
      if (most <= 16 * kNper) return sweeps<T, 16>(cluster, alone, w, rows, v, vrows, k, tol, norms, exchange, partial, flags, list);
      return sweeps<T, 32>(cluster, alone, w, rows, v, vrows, k, tol, norms, exchange, partial, flags, list);
    }

    // FP32 sweeps in blocks of four columns.  W (k columns of at most 32 NR rows) and V (k x k) lie in the
    // cluster's shared memory, block b with rank b % ranks, columns 32 NR apart and zero-padded, k padded
    // to whole pairs of blocks with zero columns.  A warp takes a pair of blocks into registers (a lane
    // holds NR rows of each of the eight columns), rotates the sixteen pairs across the blocks four
    // disjoint ones at a time (the first round also the pairs within each block), and puts the columns
    // back; the rotations are accumulated as an 8 x 8 matrix (lane i its row i) and applied to the
    // block's columns of V as one product.  A sweep is one cluster barrier per round of block pairs, a
    // quarter as many rounds as columns, and the pairs of a round are dealt to all ranks.  The four dot
    // products of a step are reduced together, each lane group of eight ending with one of them and
    // finding its angle.  Returns the sweeps, -1 beyond kMaxSweeps.
    template <int NR>
    __device__ int blocked_sweeps(const cg::cluster_group &cluster, float *w, float *v, int k, float tol, float *jbuf, int *flags)
    {
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
      const int ranks = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
      const int blocks = (k + 7) / 8 * 2;
      const float settled = sqrtf(tol);
      float *jm = jbuf + warp * 64;
      const auto sync = [&] {
        if (ranks == 1) __syncthreads();
        else cluster.sync();
      };
      const auto at_home = [&](float *base, int b) -> float * {
        float *here = base + static_cast<int64_t>(b / ranks) * 4 * 32 * NR;
        return ranks == 1 ? here : cluster.map_shared_rank(here, static_cast<unsigned>(b % ranks));
      };
      for (int sweep = 0; sweep < kMaxSweeps; ++sweep)
      {
        if (threadIdx.x == 0) flags[sweep & 1] = 0;
        sync();
        for (int round = 0; round + 1 < blocks; ++round)
        {
          for (int bp = rank + warp * ranks; bp < blocks / 2; bp += warps * ranks)
          {
            int64_t bl, br;
            circle_pair(round, bp, blocks, bl, br);
            float *left = at_home(w, static_cast<int>(bl)), *right = at_home(w, static_cast<int>(br));
            float x[8][NR + 1];
#pragma unroll
            for (int c = 0; c < 8; ++c)
            {
              const float *from = (c < 4 ? left + c * 32 * NR : right + (c - 4) * 32 * NR) + lane;
#pragma unroll
              for (int r = 0; r < NR; ++r) x[c][r] = from[r * 32];
              x[c][NR] = lane == c ? 1.0f : 0.0f;
            }
            // the columns of V on their way meanwhile, where registers allow
            constexpr bool kAhead = NR <= 3;
            float *vl = at_home(v, static_cast<int>(bl)) + lane, *vr = at_home(v, static_cast<int>(br)) + lane;
            float held[kAhead ? NR : 1][8];
            if constexpr (kAhead)
            {
#pragma unroll
              for (int r = 0; r < NR; ++r)
#pragma unroll
                for (int i = 0; i < 8; ++i) held[r][i] = (i < 4 ? vl + i * 32 * NR : vr + (i - 4) * 32 * NR)[r * 32];
            }
            // squared norms: eight sums reduced together (lane bits 4..2 end with column 4 b4 + 2 b3 + b2)
            float n2[8];
            {
              float p[8];
#pragma unroll
              for (int c = 0; c < 8; ++c)
              {
                p[c] = 0.0f;
#pragma unroll
                for (int r = 0; r < NR; ++r) p[c] = fmaf(x[c][r], x[c][r], p[c]);
              }
#pragma unroll
              for (int half = 4, bit = 16; half > 0; half >>= 1, bit >>= 1)
#pragma unroll
                for (int c = 0; c < half; ++c)
                {
                  const bool high = lane & bit;
                  const float give = high ? p[c] : p[c + half], keep = high ? p[c + half] : p[c];
                  p[c] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
                }
              p[0] += __shfl_xor_sync(0xffffffffu, p[0], 2);
              p[0] += __shfl_xor_sync(0xffffffffu, p[0], 1);
#pragma unroll
              for (int c = 0; c < 8; ++c) n2[c] = __shfl_sync(0xffffffffu, p[0], c * 4);
            }
            bool any = false, large = false;
            // four disjoint pairs (pc[i], qc[i])
            const auto rotate4 = [&](const int (&pc)[4], const int (&qc)[4]) {
              float g[4];
#pragma unroll
              for (int i = 0; i < 4; ++i)
              {
                g[i] = 0.0f;
#pragma unroll
                for (int r = 0; r < NR; ++r) g[i] = fmaf(x[pc[i]][r], x[qc[i]][r], g[i]);
              }
#pragma unroll
              for (int half = 2, bit = 16; half > 0; half >>= 1, bit >>= 1)
#pragma unroll
                for (int i = 0; i < half; ++i)
                {
                  const bool high = lane & bit;
                  const float give = high ? g[i] : g[i + half], keep = high ? g[i + half] : g[i];
                  g[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
                }
#pragma unroll
              for (int off = 4; off > 0; off >>= 1) g[0] += __shfl_xor_sync(0xffffffffu, g[0], off);
              // lanes 8 i .. 8 i + 7 hold pair i's product
              const int mine = lane >> 3;
              float alpha = n2[pc[0]], beta = n2[qc[0]];
#pragma unroll
              for (int i = 1; i < 4; ++i)
              {
                alpha = mine == i ? n2[pc[i]] : alpha;
                beta = mine == i ? n2[qc[i]] : beta;
              }
              const float cosine = fabsf(g[0]) * rsqrtf(alpha) * rsqrtf(beta);
              float c = 1.0f, sn = 0.0f;
              const bool turn = cosine > tol && angle_fast(beta - alpha, g[0], c, sn);
              if (!turn)
              {
                c = 1.0f;
                sn = 0.0f;
              }
              const float cc = c * c, ss = sn * sn, cs2 = 2.0f * c * sn * g[0];
              const float na = turn ? cc * alpha - cs2 + ss * beta : alpha, nb = turn ? ss * alpha + cs2 + cc * beta : beta;
              if (!__any_sync(0xffffffffu, turn)) return;
              any = true;
              large = large || cosine > settled;
#pragma unroll
              for (int i = 0; i < 4; ++i)
              {
                const float ci = __shfl_sync(0xffffffffu, c, 8 * i), si = __shfl_sync(0xffffffffu, sn, 8 * i);
                n2[pc[i]] = __shfl_sync(0xffffffffu, na, 8 * i);
                n2[qc[i]] = __shfl_sync(0xffffffffu, nb, 8 * i);
#pragma unroll
                for (int r = 0; r <= NR; ++r)
                {
                  const float p = x[pc[i]][r], q = x[qc[i]][r];
                  x[pc[i]][r] = fmaf(ci, p, -si * q);
                  x[qc[i]][r] = fmaf(si, p, ci * q);
                }
              }
            };
            if (round == 0)
            {
              rotate4({0, 2, 4, 6}, {1, 3, 5, 7});
              rotate4({0, 1, 4, 5}, {2, 3, 6, 7});
              rotate4({0, 1, 4, 5}, {3, 2, 7, 6});
            }
            rotate4({0, 1, 2, 3}, {4, 5, 6, 7});
            rotate4({0, 1, 2, 3}, {5, 6, 7, 4});
            rotate4({0, 1, 2, 3}, {6, 7, 4, 5});
            rotate4({0, 1, 2, 3}, {7, 4, 5, 6});
            if (__any_sync(0xffffffffu, large) && lane == 0) flags[sweep & 1] = 1;
            if (!any) continue;
#pragma unroll
            for (int c = 0; c < 8; ++c)
            {
              float *to = (c < 4 ? left + c * 32 * NR : right + (c - 4) * 32 * NR) + lane;
#pragma unroll
              for (int r = 0; r < NR; ++r) to[r * 32] = x[c][r];
              if (lane < 8) jm[lane * 8 + c] = x[c][NR];
            }
            __syncwarp();
#pragma unroll
            for (int r = 0; r < NR; ++r)
            {
              float out[8] = {};
#pragma unroll
              for (int i = 0; i < 8; ++i)
              {
                float in;
                if constexpr (kAhead) in = held[r][i];
                else in = (i < 4 ? vl + i * 32 * NR : vr + (i - 4) * 32 * NR)[r * 32];
                const float4 lo = *reinterpret_cast<const float4 *>(jm + i * 8), hi = *reinterpret_cast<const float4 *>(jm + i * 8 + 4);
                out[0] = fmaf(in, lo.x, out[0]);
                out[1] = fmaf(in, lo.y, out[1]);
                out[2] = fmaf(in, lo.z, out[2]);
                out[3] = fmaf(in, lo.w, out[3]);
                out[4] = fmaf(in, hi.x, out[4]);
                out[5] = fmaf(in, hi.y, out[5]);
                out[6] = fmaf(in, hi.z, out[6]);
                out[7] = fmaf(in, hi.w, out[7]);
              }
#pragma unroll
              for (int i = 0; i < 8; ++i) (i < 4 ? vl + i * 32 * NR : vr + (i - 4) * 32 * NR)[r * 32] = out[i];
            }
            __syncwarp();
          }
          sync();
        }
        int more = threadIdx.x < ranks ? *cluster.map_shared_rank(flags + (sweep & 1), threadIdx.x) : 0;
        if (!__syncthreads_or(more)) return sweep + 1;
      }
      return -1;
    }
    constexpr int kBlockedRows = 320;  // the longest columns of blocked_sweeps

    __device__ int blocked_sweeps(const cg::cluster_group &cluster, float *w, float *v, int k, int nr, float tol, float *jbuf, int *flags)
    {
      switch (nr)
      {
      case 1: return blocked_sweeps<1>(cluster, w, v, k, tol, jbuf, flags);
      case 2: return blocked_sweeps<2>(cluster, w, v, k, tol, jbuf, flags);
      case 3: return blocked_sweeps<3>(cluster, w, v, k, tol, jbuf, flags);
      case 4: return blocked_sweeps<4>(cluster, w, v, k, tol, jbuf, flags);
      case 5: return blocked_sweeps<5>(cluster, w, v, k, tol, jbuf, flags);
      case 6: return blocked_sweeps<6>(cluster, w, v, k, tol, jbuf, flags);
      case 8: return blocked_sweeps<8>(cluster, w, v, k, tol, jbuf, flags);
      default: return blocked_sweeps<10>(cluster, w, v, k, tol, jbuf, flags);
      }
    }

    // out(i, j) = sum_x a(x, i) b(x, j) over a 16 x 16 tile, x < depth, staged 32 of x at a time (the next
    // stage's reads in flight during this one's products), each thread half the depth of one entry.
    // Small tiles deal evenly over a cluster; FP64 issue is the bound.  The loaders are called with x
    // fastest across the threads when `x_fast`, else i (or j) fastest.
    constexpr int kSmallTile = 16, kSmallDepth = 32, kSmallPitch = kSmallTile + 1;
    constexpr int64_t kSmallBytes = 2 * kSmallDepth * kSmallPitch * 8;
    template <typename Acc, typename FA, typename FB, typename Out>
    __device__ void small_product(int64_t depth, FA fa, bool a_x_fast, FB fb, bool b_x_fast, void *stage, Out out)
    {
      Acc *sa = static_cast<Acc *>(stage), *sb = sa + kSmallDepth * kSmallPitch;
      const int t = threadIdx.x, i = t & 15, j = (t >> 4) & 15, half = t >> 8;
      const int xa = a_x_fast ? t & 31 : t >> 4, ia = a_x_fast ? t >> 5 : t & 15;
      const int xb = b_x_fast ? t & 31 : t >> 4, jb = b_x_fast ? t >> 5 : t & 15;
      Acc acc = 0;
      Acc na = xa < depth ? static_cast<Acc>(fa(xa, ia)) : Acc(0), nb = xb < depth ? static_cast<Acc>(fb(xb, jb)) : Acc(0);
      for (int64_t x0 = 0; x0 < depth; x0 += kSmallDepth)
      {
        sa[xa * kSmallPitch + ia] = na;
        sb[xb * kSmallPitch + jb] = nb;
        __syncthreads();
        const int64_t x1 = x0 + kSmallDepth;
        if (x1 < depth)
        {
          na = x1 + xa < depth ? static_cast<Acc>(fa(x1 + xa, ia)) : Acc(0);
          nb = x1 + xb < depth ? static_cast<Acc>(fb(x1 + xb, jb)) : Acc(0);
        }
#pragma unroll
        for (int x = 0; x < kSmallDepth / 2; ++x)
          acc = fma(sa[(half * 16 + x) * kSmallPitch + i], sb[(half * 16 + x) * kSmallPitch + j], acc);
        __syncthreads();
      }
      if (half == 1) sa[j * kSmallPitch + i] = acc;
      __syncthreads();
      if (half == 0) out(i, j, acc + sa[j * kSmallPitch + i]);
      __syncthreads();
    }

    // out(i, j) = sum_x a(x, i) b(x, j) + c(i, j) over a kTile x kTile tile, x < depth, staged
    // kTile at a time in shared memory (a(x, i) from fa(x, i), b from fb; zero outside), with Acc
    // accumulation; each of the 512 threads takes two entries (i, j) and (i, j + 16).  The loaders
    // are called with x fastest across the threads when `x_fast`, else i (or j) fastest, to follow
    // the memory order of the operand.
    template <typename Acc, typename FA, typename FB, typename Out>
    __device__ void tile_product(int64_t depth, FA fa, bool a_x_fast, FB fb, bool b_x_fast, Acc *sa, Acc *sb, Out out)
    {
      constexpr int P = kTile + 1;
      const int t = threadIdx.x, i = t % kTile, j = t / kTile;
      Acc acc0 = 0, acc1 = 0;
      for (int64_t x0 = 0; x0 < depth; x0 += kTile)
      {
        for (int e = t; e < kTile * kTile; e += blockDim.x)
        {
          const int fast = e % kTile, slow = e / kTile;
          const int xa = a_x_fast ? fast : slow, ia = a_x_fast ? slow : fast;
          sa[xa * P + ia] = x0 + xa < depth ? static_cast<Acc>(fa(x0 + xa, ia)) : Acc(0);
          const int xb = b_x_fast ? fast : slow, jb = b_x_fast ? slow : fast;
          sb[xb * P + jb] = x0 + xb < depth ? static_cast<Acc>(fb(x0 + xb, jb)) : Acc(0);
        }
        __syncthreads();
#pragma unroll 8
        for (int x = 0; x < kTile; ++x)
        {
          const Acc ax = sa[x * P + i];
          acc0 = fma(ax, sb[x * P + j], acc0);
          acc1 = fma(ax, sb[x * P + j + 16], acc1);
        }
        __syncthreads();
      }
      out(i, j, acc0);
      out(i, j + 16, acc1);
    }

    // A thread-block cluster of up to 16 CTAs per block (grid = blocks x cluster size, the largest
    // blocks first).  The FP64 sweeps, when they run, run over the cluster for blocks of 32 columns or
    // more, on rank 0 alone for smaller ones.
    __global__ void __launch_bounds__(kSvdThreads, 1)
      jacobi_svd_kernel(const SvdEntry *__restrict__ table, const double *__restrict__ a, double *__restrict__ u,
                        double *__restrict__ s, double *__restrict__ vh, double *__restrict__ workspace,
                        int32_t *__restrict__ info)
    {
      extern __shared__ __align__(16) unsigned char dynamic[];
      __shared__ double norms_raw[kMaxCols];
      __shared__ double partial_raw[kMaxCols];
      __shared__ int rank_of[kMaxCols];
      __shared__ int flags[5];  // [0], [1]: a sweep rotated above sqrt(tol), by sweep parity; [4]: the rotations listed in a round
      __shared__ double big;
      __shared__ double taus[2];
      const cg::cluster_group cluster = cg::this_cluster();
      const unsigned ranks = cluster.num_blocks(), rank = cluster.block_rank();
      const int64_t block = blockIdx.x / ranks;
      const SvdEntry e = table[block];
      const int64_t m = e.rows, n = e.cols;
      const bool wide = n > m;
      const int64_t len = wide ? n : m, k = wide ? m : n;  // W is len x k, column-major
      if (k == 0)
      {
        if (threadIdx.x == 0 && rank == 0) info[block] = 0;
        return;
      }
      const SvdLayout lay = svd_layout(len, k);
      double *ws = workspace + e.ws_off;
      double *v_cur = ws + lay.v0, *v_next = ws + lay.v1, *g = ws + lay.g;
      double *stage = reinterpret_cast<double *>(dynamic + kDynamicBytes - kStageBytes);
      const double *src = a + e.a_off;
      const auto raw = [&](int64_t row, int64_t col) -> double
      { return wide ? src[col * n + row] : src[row * n + col]; };  // row < len, col < k
      // The block is worked on times the power of two that brings its largest entry to about 2^kBlockExp, so that the
      // products of four of its values that decide whether a pair is orthogonal neither overflow nor vanish for
      // values down to 1e-128 of the largest.  From `high`, the largest of the high words this thread has seen
      // (integers: exponents are compared).
      int shift = 0;
      double unit = 1.0;
      const auto find_unit = [&](int high) {
        high = __reduce_max_sync(0xffffffffu, high);
        if ((threadIdx.x & 31) == 0) rank_of[threadIdx.x >> 5] = high;
        __syncthreads();
        for (int w = 0; w < kSvdThreads / 32; ++w) high = max(high, rank_of[w]);
        __syncthreads();
        const int ex = (high >> 20) - 1022;  // the largest entry is below 2^ex; not finite from 1025 on
        if (ex > 1024) return 0;
        shift = max(ex - kBlockExp, -1000);
        unit = ldexp(1.0, -shift);
        return ex;
      };
      const auto entry_a = [&](int64_t row, int64_t col) -> double { return raw(row, col) * unit; };

      // 0. Preconditioning: the columns sorted by norm, largest
      // first, and factored A P = Q R by Householder reflections; the sweeps then run on X = R^T
      // (k x k), whose graded columns the FP32 sweeps orthogonalise in about a third of the
      // sweeps the block itself takes (Drmac & Veselic, "New fast and accurate Jacobi SVD
      // algorithm", SIAM J. Matrix Anal. Appl. 29 (2008), with the pivoting of their QR replaced by
      // the one sort).  The factors of X give those of A: A P = (Q J) S (U_x)^T with X J = U_x S.
      // The columns are dealt to the ranks in turn while they are factored; at the end rank r transforms
      // columns [q0, q1) of the left factor.
      const bool precond = k >= kQrMinCols;
      double *qf = ws + lay.f, *qtau = ws + lay.tau, *qb = ws + lay.b;
      int64_t *qorder = reinterpret_cast<int64_t *>(ws + lay.order);
      const int64_t cpr = (k + ranks - 1) / ranks;
      const int64_t q0 = min(k, static_cast<int64_t>(rank) * cpr), q1 = min(k, q0 + cpr);
      if (precond)
      {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
        // squared column norms in FP32 (the same on every rank) and the order they give
        float *cn = reinterpret_cast<float *>(partial_raw);
        int high = 0;
        for (int64_t j = threadIdx.x; j < k; j += blockDim.x)
        {
          float sum = 0.0f;
#pragma unroll 8
          for (int64_t i = 0; i < len; ++i)
          {
            const double entry = raw(i, j);
            high = max(high, __double2hiint(entry) & 0x7fffffff);
            const float x = static_cast<float>(entry);
            sum = fmaf(x, x, sum);
          }
          cn[j] = sum >= 0.0f ? sum : INFINITY;  // a NaN sorts like an infinity: the order is a permutation
        }
        const int ex = find_unit(high);
        if ((ex < -30 && ex > -1022) || ex > 30)
        {
          // again with the squares in FP32's range
          const double by = ldexp(1.0, -max(ex, -1000));
          for (int64_t j = threadIdx.x; j < k; j += blockDim.x)
          {
            float sum = 0.0f;
            for (int64_t i = 0; i < len; ++i)
            {
              const float x = static_cast<float>(raw(i, j) * by);
              sum = fmaf(x, x, sum);
            }
            cn[j] = sum >= 0.0f ? sum : INFINITY;
          }
        }
        __syncthreads();
        for (int64_t j = threadIdx.x; j < k; j += blockDim.x)
        {
          const float nj = cn[j];
          int r = 0;
          for (int64_t i = 0; i < k; ++i) r += (cn[i] > nj || (cn[i] == nj && i < j)) ? 1 : 0;
          rank_of[r] = static_cast<int>(j);
        }
        __syncthreads();
        // this rank's columns in shared memory while they are factored when they fit (else in the
        // global factored matrix); each reflector goes to the global one as it is made
        const bool qr_smem = (cpr + 2) * len * 8 <= kDynamicBytes;
        double *own = reinterpret_cast<double *>(dynamic);
        double *vst = qr_smem ? own + cpr * len : own;  // the reflectors of two steps in turn; one when columns are global
        const bool staged = len * 8 <= kDynamicBytes;
        const bool ahead = qr_smem && len <= kAheadRows;
        const auto colp = [&](int64_t c) -> double * { return qr_smem ? own + (c / ranks) * len : qf + c * len; };
        for (int64_t c = rank; c < k; c += ranks)
        {
          const int64_t from = rank_of[c];
          double *to = colp(c);
          for (int64_t i = threadIdx.x; i < len; i += blockDim.x) to[i] = entry_a(i, from);
          if (threadIdx.x == 0) qorder[c] = from;
        }
        cluster.sync();
        if (!ahead)
        {
          // Long columns, or too long for shared memory: the CTA that owns column j makes its reflector with all its
          // threads and the others read it from L2; a warp per column applies it.  (A block of 5000 x 64 takes 8.7 ms
          // so, 20.5 by the chain of one warp below, 10.0 with no QR ahead at all.)
          for (int64_t j = 0; j < k; ++j)
          {
            if (j % ranks == rank)
            {
              double *col = colp(j);
              double part = 0.0;
              for (int64_t i = j + 1 + threadIdx.x; i < len; i += blockDim.x) part = fma(col[i], col[i], part);
              part = warp_sum(part);
              if (lane == 0) norms_raw[warp] = part;
              __syncthreads();
              if (warp == 0)
              {
                double beta, tau, scale;
                column_reflector(col, static_cast<int>(j), static_cast<int>(len), warp_sum(lane < warps ? norms_raw[lane] : 0.0), beta, tau, scale);
                __syncwarp();
                if (lane == 0)
                {
                  col[j] = beta;
                  qtau[j] = tau;
                  big = scale;
                }
              }
              __syncthreads();
              const double scale = big;
              if (scale != 0.0)
                for (int64_t i = j + 1 + threadIdx.x; i < len; i += blockDim.x) qf[j * len + i] = col[i] * scale;
            }
            cluster.sync();
            const double tau = __ldcg(qtau + j);
            const double *v = qf + j * len;
            if (staged && tau != 0.0)
            {
              for (int64_t i = j + 1 + threadIdx.x; i < len; i += blockDim.x) vst[i] = __ldcg(v + i);
              __syncthreads();
            }
            const auto vi = [&](int64_t i) { return staged ? vst[i] : __ldcg(v + i); };
            if (tau != 0.0)
              for (int64_t c = rank + ((j + ranks - rank) / ranks + warp) * ranks; c < k; c += warps * ranks)
              {
                double *fc = colp(c), dot = 0.0;
                for (int64_t i = j + 1 + lane; i < len; i += 32) dot = fma(vi(i), fc[i], dot);
                dot = warp_sum(dot);
                const double wt = tau * (fc[j] + dot);
                for (int64_t i = j + 1 + lane; i < len; i += 32) fc[i] = fma(-wt, vi(i), fc[i]);
                __syncwarp();
                if (lane == 0) fc[j] -= wt;
              }
            __syncthreads();
          }
        }
        // Step j: the owner of column j has made its reflector (reflector.cuh) and pushed it into every rank's
        // shared memory; a warp per column right of j applies it.  The warp that holds column j + 1 does that
        // column first and makes its reflector at once, so a step is one cluster barrier and one warp's chain of a
        // dot product, the update, the norm and the scalars (the columns are dealt in turn, so that every rank has
        // columns to the end).
        const auto reflect = [&](int64_t j, double xn) {
          // by one warp, xn the squared norm of column j below its diagonal
          double *col = colp(j);
          double beta, tau, scale;
          column_reflector(col, static_cast<int>(j), static_cast<int>(len), xn, beta, tau, scale);
          __syncwarp();
          double *slot = vst + (j & 1) * len;
          for (int64_t i = j + 1 + lane; tau != 0.0 && i < len; i += 32)
          {
            const double x = col[i] * scale;
            qf[j * len + i] = x;
            for (unsigned r = 0; r < ranks; ++r) cluster.map_shared_rank(slot, r)[i] = x;
          }
          if (lane == 0)
          {
            col[j] = beta;
            qf[j * len + j] = beta;
            qtau[j] = tau;
            for (unsigned r = 0; r < ranks; ++r) cluster.map_shared_rank(taus, r)[j & 1] = tau;
          }
        };
        if (ahead && rank == 0 && warp == 0)
        {
          const double *col = colp(0);
          double xn = 0.0;
          for (int64_t i = 1 + lane; i < len; i += 32) xn = fma(col[i], col[i], xn);
          reflect(0, warp_sum(xn));
        }
        for (int64_t j = 0; ahead && j < k; ++j)
        {
          cluster.sync();
          const double *v = vst + (j & 1) * len;
          const double tau = taus[j & 1];
          // FP64 issue is what a step is made of (a warp instruction in 64 clocks a quarter of the SM): column
          // j + 1 has warp 0 and its quarter to itself, the others go four to a warp, eight lanes a column
          // (three shuffled additions for the four dot products instead of five each), on the other quarters.
          const int64_t first = (j + 1 + ranks - 1 - rank) / ranks;  // the first local column c with c ranks + rank > j
          const bool next = (j + 1) % ranks == rank;                 // it is column j + 1
          if (warp == 0)
          {
            if (next && j + 1 < k)
            {
              double *fc = colp(j + 1), xn = 0.0;
              if (tau != 0.0)
              {
                double dot = 0.0;
                for (int64_t i = j + 1 + lane; i < len; i += 32) dot = fma(v[i], fc[i], dot);
                dot = warp_sum(dot);
                const double wt = tau * (fc[j] + dot);
                for (int64_t i = j + 1 + lane; i < len; i += 32)
                {
                  const double x = fma(-wt, v[i], fc[i]);
                  fc[i] = x;
                  if (i > j + 1) xn = fma(x, x, xn);
                }
                __syncwarp();
                if (lane == 0) fc[j] -= wt;
              }
              else
                for (int64_t i = j + 2 + lane; i < len; i += 32) xn = fma(fc[i], fc[i], xn);
              __syncwarp();
              reflect(j + 1, warp_sum(xn));
            }
          }
          else if ((warp & 3) != 0 && tau != 0.0)
          {
            const int slot = (warp >> 2) * 3 + (warp & 3) - 1, lanes = lane & 7;
            for (int64_t l0 = first + (next ? 1 : 0) + slot * 4; l0 * ranks + rank < k; l0 += (warps >> 2) * 12)
            {
              const int64_t c = (l0 + (lane >> 3)) * ranks + rank;
              const bool live = c < k;
              double *fc = colp(live ? c : l0 * ranks + rank), dot = 0.0;
              for (int64_t i = j + 1 + lanes; i < len; i += 8) dot = fma(v[i], fc[i], dot);
              dot = group_sum<double, 8>(dot);
              const double head = fc[j], wt = tau * (head + dot);
              __syncwarp();
              if (!live) continue;
              for (int64_t i = j + 1 + lanes; i < len; i += 8) fc[i] = fma(-wt, v[i], fc[i]);
              if (lanes == 0) fc[j] = head - wt;
            }
          }
        }
        __syncthreads();
        // R's part of this rank's columns to the global factored matrix
        if (qr_smem)
          for (int64_t c = rank; c < k; c += ranks)
            for (int64_t i = threadIdx.x; i <= c && i < len; i += blockDim.x) qf[c * len + i] = colp(c)[i];
        cluster.sync();
      }
      // rows of the swept matrix, and its entries: the block (W orientation) or X = R^T
      const int64_t xl = precond ? k : len;
      if (!precond)
      {
        int high = 0;
        for (int64_t i = threadIdx.x; i < m * n; i += blockDim.x) high = max(high, __double2hiint(src[i]) & 0x7fffffff);
        find_unit(high);
      }
      const auto entry = [&](int64_t row, int64_t col) -> double
      { return precond ? (col <= row ? __ldcg(qf + row * len + col) : 0.0) : entry_a(row, col); };  // row < xl

      // 1. FP32 sweeps on the block scaled to |entries| <= 1, from V = I; V goes out in FP64.
      // In blocks of columns over the cluster when W and V fit in its shared memory (columns of up to
      // 320), else column by column with the rows dealt over the cluster.
      const int rows32 = static_cast<int>((max(xl, k) + 31) / 32), nr = rows32 <= 6 ? rows32 : rows32 <= 8 ? 8 : 10;
      const int64_t column_blocks = (k + 7) / 8 * 2, mine = (column_blocks + ranks - 1) / ranks, ld32 = 32 * nr;
      const bool blocked = max(xl, k) <= kBlockedRows && (2 * mine * 4 * ld32 + 64 * (kSvdThreads / 32)) * 4 <= kDynamicBytes;
      if (blocked)
      {
        float *w32 = reinterpret_cast<float *>(dynamic), *v32 = w32 + mine * 4 * ld32, *jbuf = v32 + mine * 4 * ld32;
        if (threadIdx.x == 0) big = 0.0;
        __syncthreads();
        double local = 0.0;
        for (int64_t i = threadIdx.x; i < xl * k; i += blockDim.x) local = fmax(local, fabs(entry(i % xl, i / xl)));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) local = fmax(local, __shfl_xor_sync(0xffffffffu, local, o));
        if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<unsigned long long *>(&big), __double_as_longlong(local));
        __syncthreads();
        const double scale = big > 0.0 ? 1.0 / big : 1.0;
        // place i of this rank's columns: column 4 (rank + ranks b) + c of block b here
        const auto column_of = [&](int64_t i) { return ((i / ld32 / 4) * ranks + rank) * 4 + i / ld32 % 4; };
        for (int64_t i = threadIdx.x; i < mine * 4 * ld32; i += blockDim.x)
        {
          const int64_t row = i % ld32, col = column_of(i);
          w32[i] = row < xl && col < k ? static_cast<float>(entry(row, col) * scale) : 0.0f;
          v32[i] = row == col && col < k ? 1.0f : 0.0f;
        }
        blocked_sweeps(cluster, w32, v32, static_cast<int>(k), nr, 1e-5f, jbuf, flags);
        for (int64_t i = threadIdx.x; i < mine * 4 * ld32; i += blockDim.x)
        {
          const int64_t row = i % ld32, col = column_of(i);
          if (row < k && col < k) v_cur[col * k + row] = static_cast<double>(v32[i]);
        }
      }
      else
      {
        const bool alone = ranks == 1 || (k < 32 && (xl * k + k * k) * 4 <= kDynamicBytes);
        const int64_t rows = alone ? xl : (xl + ranks - 1) / ranks, vrows = alone ? k : (k + ranks - 1) / ranks;
        const int64_t r0 = alone ? 0 : min(xl, static_cast<int64_t>(rank) * rows), r1 = alone ? xl : min(xl, r0 + rows);
        const int64_t c0 = alone ? 0 : min(k, static_cast<int64_t>(rank) * vrows), c1 = alone ? k : min(k, c0 + vrows);
        const int64_t swap32 = exchange_bytes(k, alone ? 1 : ranks, 4);
        const bool in_smem = (rows + vrows) * k * 4 + swap32 <= kDynamicBytes;
        float *w32 = in_smem ? reinterpret_cast<float *>(dynamic)
                             : reinterpret_cast<float *>(ws + lay.w32_slices) + static_cast<int64_t>(rank) * rows * k;
        float *v32 = in_smem ? w32 + rows * k : reinterpret_cast<float *>(ws + lay.v32_slices) + static_cast<int64_t>(rank) * vrows * k;
        if (alone ? rank == 0 : true)
        {
          // the largest |entry| of the block (of this rank's rows, then over the cluster)
          if (threadIdx.x == 0) big = 0.0;
          __syncthreads();
          double local = 0.0;
          for (int64_t i = threadIdx.x; i < (r1 - r0) * k; i += blockDim.x)
            local = fmax(local, fabs(entry(r0 + i % (r1 - r0), i / (r1 - r0))));
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) local = fmax(local, __shfl_xor_sync(0xffffffffu, local, o));
          if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<unsigned long long *>(&big), __double_as_longlong(local));
          __syncthreads();
        }
        if (!alone)
        {
          if (threadIdx.x == 0) partial_raw[0] = big;
          cluster.sync();
          if (threadIdx.x == 0)
          {
            double most = 0.0;
            for (unsigned r = 0; r < ranks; ++r) most = fmax(most, cluster.map_shared_rank(partial_raw, r)[0]);
            big = most;
          }
          __syncthreads();
        }
        if (alone ? rank == 0 : true)
        {
          const double scale = big > 0.0 ? 1.0 / big : 1.0;
          for (int64_t i = threadIdx.x; i < rows * k; i += blockDim.x)
          {
            const int64_t row = r0 + i % rows;
            w32[i] = row < r1 ? static_cast<float>(entry(row, i / rows) * scale) : 0.0f;
          }
          for (int64_t i = threadIdx.x; i < vrows * k; i += blockDim.x)
            v32[i] = (c0 + i % vrows == i / vrows && c0 + i % vrows < c1) ? 1.0f : 0.0f;
          __syncthreads();
        }
        if (!alone) cluster.sync();  // every rank's partial_raw read before it holds norms
        if (alone ? rank == 0 : true)
        {
          sweeps<float>(cluster, alone, w32, rows, v32, vrows, k, 1e-5, reinterpret_cast<float *>(norms_raw),
                        reinterpret_cast<float *>(dynamic + kDynamicBytes - swap32), reinterpret_cast<float *>(partial_raw),
                        flags, rank_of);
          for (int64_t i = threadIdx.x; i < vrows * k; i += blockDim.x)
          {
            const int64_t row = c0 + i % vrows;
            if (row < c1) v_cur[(i / vrows) * k + row] = static_cast<double>(v32[i]);
          }
        }
      }
      cluster.sync();

      // 2. V refined in FP64 with matrix products: W = X V, its Gram matrix G = W^T W and H = V^T V say how
      // far every pair of columns is from orthogonal; V <- V + V E with E_rc = t_rc - h_rc / 2, t the tangent
      // of the pair's Jacobi angle (from G with V's own non-orthogonality taken out) and the rest the
      // Newton-Schulz step, takes cosines of 1e-5 to 1e-9 and then to round-off (all pairs at once, the
      // idea of T. Ogita and K. Aishima, "Iterative refinement for symmetric eigenvalue decomposition",
      // Japan J. Indust. Appl. Math. 35 (2018), on the one-sided form, whose graded columns keep their
      // relative accuracy).  E has to be good only to FP32, so V E is an FP32 product.  Done when no
      // cosine is above tol and V is orthonormal to it; once both are within four times that, a last step of
      // that size leaves V as orthonormal as its rounding, and W = X V is formed again.  Pairs whose angle is not small (close singular values
      // that FP32 left mixed) are left out; when there are some after the first time, or it does not
      // settle, the FP64 sweeps below take over.  Against the 3 to 6 FP64 sweeps of 0.7 ms each that it
      // replaces, a step is about 0.1 ms at 148 columns.
      const double tol = 2.220446049250313e-16 * sqrt(static_cast<double>(xl));
      double *wg = qb, *hm = ws + lay.w_slices;
      float *em = reinterpret_cast<float *>(ws + lay.v_slices);
      void *small_stage = dynamic + kDynamicBytes - kSmallBytes;
      double *v_start = ws + lay.w32_slices;  // V as FP32 left it, for the sweeps should they run (k x k)
      bool refined = false, last = false;
      int refinements = 0;
      for (int64_t i = static_cast<int64_t>(rank) * blockDim.x + threadIdx.x; i < k * k; i += static_cast<int64_t>(ranks) * blockDim.x)
        v_start[i] = __ldcg(v_cur + i);
      for (int it = 0; it < 8 && !refined; ++it)
      {
        const double *vc = v_cur;
        const int64_t nrow = (xl + kSmallTile - 1) / kSmallTile, ncol = (k + kSmallTile - 1) / kSmallTile;
        for (int64_t tile = rank; tile < nrow * ncol; tile += ranks)
        {
          // the deepest tiles of the triangular X first
          const int64_t tr = nrow - 1 - tile / ncol, tc = tile % ncol;
          small_product<double>(
            precond ? min(k, (tr + 1) * kSmallTile) : k,
            [&](int64_t x, int i) { const int64_t row = tr * kSmallTile + i; return row < xl ? entry(row, x) : 0.0; }, precond || !wide,
            [&](int64_t x, int j) { return tc * kSmallTile + j < k ? __ldcg(vc + (tc * kSmallTile + j) * k + x) : 0.0; }, true, small_stage,
            [&](int i, int j, double sum) {
              const int64_t row = tr * kSmallTile + i, c = tc * kSmallTile + j;
              if (row < xl && c < k) wg[c * xl + row] = sum;
            });
        }
        cluster.sync();
        if (last)
        {
          refined = true;
          break;
        }
        int64_t turn = 0;
        for (int which = 0; which < 2; ++which)
          for (int64_t tr = 0; tr < ncol; ++tr)
            for (int64_t tc = tr; tc < ncol; ++tc, ++turn)
            {
              if (turn % ranks != rank) continue;
              const double *m = which == 0 ? wg : vc;
              double *to = which == 0 ? g : hm;
              const int64_t ld = which == 0 ? xl : k;
              small_product<double>(
                ld, [&](int64_t x, int i) { return tr * kSmallTile + i < k ? __ldcg(m + (tr * kSmallTile + i) * ld + x) : 0.0; }, true,
                [&](int64_t x, int j) { return tc * kSmallTile + j < k ? __ldcg(m + (tc * kSmallTile + j) * ld + x) : 0.0; }, true, small_stage,
                [&](int i, int j, double sum) {
                  const int64_t r = tr * kSmallTile + i, c = tc * kSmallTile + j;
                  if (r < k && c < k && r <= c) to[c * k + r] = sum;
                });
            }
        cluster.sync();
        for (int64_t j = threadIdx.x; j < k; j += blockDim.x) norms_raw[j] = __ldcg(g + j * k + j);
        __syncthreads();
        int status = 0;  // above four times tol: 1 a cosine, 2 V^T V - I; 8: either above tol; 4: an angle that is not small
        for (int64_t i = static_cast<int64_t>(rank) * blockDim.x + threadIdx.x; i < k * k; i += static_cast<int64_t>(ranks) * blockDim.x)
        {
          const int64_t c = i / k, r = i - c * k;
          if (r > c) continue;
          const double h = __ldcg(hm + i);
          if (r == c)
          {
            const double off = 1.0 - h;
            em[i] = static_cast<float>(0.5 * off);
            if (!(fabs(off) <= tol)) status |= fabs(off) <= 4.0 * tol ? 8 : 10;
            continue;
          }
          const double gamma = __ldcg(g + i), lr = norms_raw[r], lc = norms_raw[c];
          const double limit = tol * tol * lr * lc, square = gamma * gamma;
          const bool open = !(square <= 16.0 * limit);
          if (!(square <= limit)) status |= open ? 9 : 8;
          if (!(fabs(h) <= tol)) status |= fabs(h) <= 4.0 * tol ? 8 : 10;
          const double st = fma(-0.5 * h, lr + lc, gamma);
          float cf, sf;
          double tangent = 0.0;
          if (angle(lr, lc, st, cf, sf))
          {
            const float tf = sf / cf;
            // (at round-off the angle of a pair of equal values is noise)
            if (open && fabsf(tf) > 0.1f) status |= 4;
            if (fabsf(tf) <= (open ? 0.1f : 1e-8f)) tangent = tf;
          }
          em[c * k + r] = static_cast<float>(fma(-0.5, h, tangent));
          em[r * k + c] = static_cast<float>(fma(-0.5, h, -tangent));
        }
        status = (__syncthreads_or(status & 1) ? 1 : 0) | (__syncthreads_or(status & 2) ? 2 : 0) | (__syncthreads_or(status & 4) ? 4 : 0) |
                 (__syncthreads_or(status & 8) ? 8 : 0);
        if (threadIdx.x == 0) flags[2] = status;
        cluster.sync();
        status = 0;
        for (unsigned r = 0; r < ranks; ++r) status |= cluster.map_shared_rank(flags, r)[2];
        refinements = it + 1;
        refined = !(status & 8);
        if (refined) break;
        last = !(status & 3);
        if (!last && ((it >= 1 && (status & 4)) || it >= 6)) break;
        for (int64_t tile = rank; tile < ncol * ncol; tile += ranks)
        {
          const int64_t tr = tile / ncol, tc = tile % ncol;
          small_product<float>(
            k, [&](int64_t x, int i) { return tr * kSmallTile + i < k ? static_cast<float>(__ldcg(vc + x * k + tr * kSmallTile + i)) : 0.0f; }, false,
            [&](int64_t x, int j) { return tc * kSmallTile + j < k ? __ldcg(em + (tc * kSmallTile + j) * k + x) : 0.0f; }, true, small_stage,
            [&](int i, int j, float sum) {
              const int64_t row = tr * kSmallTile + i, c = tc * kSmallTile + j;
              if (row < k && c < k) v_next[c * k + row] = __ldcg(vc + c * k + row) + static_cast<double>(sum);
            });
        }
        cluster.sync();
        double *t = v_cur;
        v_cur = v_next;
        v_next = t;
      }
      // no rank writes over what another still reads of the statuses
      cluster.sync();
      if (!refined)
      {
        for (int64_t i = static_cast<int64_t>(rank) * blockDim.x + threadIdx.x; i < k * k; i += static_cast<int64_t>(ranks) * blockDim.x)
          v_cur[i] = __ldcg(v_start + i);
        cluster.sync();
      }

      // 3. (when the refinement did not settle) V orthonormal to FP64 precision by two Newton-Schulz steps V <- V + V (I - V^T V) / 2:
      // G = V^T V in FP64 (the tiles on and above the diagonal), the correction V E, E = I - G of
      // size ~1e-6 and then ~1e-12, in FP32 accumulation (its rounding, ~1e-7 of E, is below FP64
      // precision of V after the second step).  Tiles are dealt to the ranks; V and G pass between
      // the CTAs through the workspace, read past L1 (__ldcg) so that no CTA sees an earlier value.
      const int64_t nt = (k + kTile - 1) / kTile;
      for (int step = 0; step < (refined ? 0 : 2); ++step)
      {
        for (int64_t tile = rank; tile < nt * nt; tile += ranks)
        {
          const int64_t tr = tile % nt, tc = tile / nt;
          if (tr > tc) continue;
          const double *vc = v_cur;
          tile_product<double>(
            k, [&](int64_t x, int i) { return tr * kTile + i < k ? __ldcg(vc + (tr * kTile + i) * k + x) : 0.0; }, true,
            [&](int64_t x, int j) { return tc * kTile + j < k ? __ldcg(vc + (tc * kTile + j) * k + x) : 0.0; }, true,
            stage, stage + kTile * (kTile + 1),
            [&](int i, int j, double sum) {
              const int64_t r = tr * kTile + i, c = tc * kTile + j;
              if (r < k && c < k)
              {
                g[c * k + r] = sum;
                g[r * k + c] = sum;
              }
            });
        }
        cluster.sync();
        for (int64_t tile = rank; tile < nt * nt; tile += ranks)
        {
          const int64_t tr = tile % nt, tc = tile / nt;  // rows tr, columns tc of V'
          const double *vc = v_cur, *gc = g;
          float *sa = reinterpret_cast<float *>(stage), *sb = sa + kTile * (kTile + 1);
          tile_product<float>(
            k, [&](int64_t x, int i) { return tr * kTile + i < k ? static_cast<float>(__ldcg(vc + x * k + tr * kTile + i)) : 0.0f; },
            false,
            [&](int64_t x, int j) {
              const int64_t c = tc * kTile + j;
              return c < k ? static_cast<float>((x == c ? 1.0 : 0.0) - __ldcg(gc + c * k + x)) : 0.0f;
            },
            true, sa, sb,
            [&](int i, int j, float sum) {
              const int64_t row = tr * kTile + i, c = tc * kTile + j;
              if (row < k && c < k) v_next[c * k + row] = fma(0.5, static_cast<double>(sum), __ldcg(vc + c * k + row));
            });
        }
        cluster.sync();
        double *t = v_cur;
        v_cur = v_next;
        v_next = t;
      }

      // this rank's rows of W = A V (FP64) and of V.  FP64 sweeps over the cluster for 32 columns or
      // more, on rank 0 alone below that.
      const bool alone = ranks == 1 || k < 32;
      const int64_t rows = alone ? (rank == 0 ? xl : 0) : (xl + ranks - 1) / ranks;
      const int64_t vrows = alone ? (rank == 0 ? k : 0) : (k + ranks - 1) / ranks;
      const int64_t r0 = alone ? 0 : min(xl, static_cast<int64_t>(rank) * rows), r1 = min(xl, r0 + rows);
      const int64_t c0 = alone ? 0 : min(k, static_cast<int64_t>(rank) * vrows), c1 = min(k, c0 + vrows);
      const int64_t swap64 = exchange_bytes(k, alone ? 1 : ranks, 8);
      const bool slices_in_smem = (rows + vrows) * k * 8 + (swap64 > kStageBytes ? swap64 : kStageBytes) <= kDynamicBytes;
      double *w = slices_in_smem ? reinterpret_cast<double *>(dynamic) : ws + lay.w_slices + static_cast<int64_t>(rank) * rows * k;
      double *v = slices_in_smem ? w + rows * k : ws + lay.v_slices + static_cast<int64_t>(rank) * vrows * k;
      {
        const double *vc = v_cur;
        if (refined)
          for (int64_t i = threadIdx.x; i < rows * k; i += blockDim.x)
          {
            const int64_t row = r0 + i % rows;
            w[i] = row < r1 ? __ldcg(wg + (i / rows) * xl + row) : 0.0;
          }
        const int64_t row_tiles = refined ? 0 : (rows + kTile - 1) / kTile;
        for (int64_t tile = 0; tile < row_tiles * nt; ++tile)
        {
          const int64_t tr = tile % row_tiles, tc = tile / row_tiles;
          tile_product<double>(
            k, [&](int64_t x, int i) { const int64_t row = r0 + tr * kTile + i; return row < r1 ? entry(row, x) : 0.0; }, precond || !wide,
            [&](int64_t x, int j) { return tc * kTile + j < k ? __ldcg(vc + (tc * kTile + j) * k + x) : 0.0; }, true,
            stage, stage + kTile * (kTile + 1),
            [&](int i, int j, double sum) {
              const int64_t row = tr * kTile + i, c = tc * kTile + j;
              if (row < rows && c < k) w[c * rows + row] = r0 + row < r1 ? sum : 0.0;
            });
        }
        for (int64_t i = threadIdx.x; i < vrows * k; i += blockDim.x)
        {
          const int64_t row = c0 + i % vrows, j = i / vrows;
          v[i] = row < c1 ? __ldcg(vc + j * k + row) : 0.0;
        }
        __syncthreads();
      }

      // 4. FP64 sweeps
      int sweeps_taken = refinements;
      if (!refined && (!alone || rank == 0))
        sweeps_taken = sweeps<double>(cluster, alone, w, rows, v, vrows, k, tol, norms_raw,
                                      reinterpret_cast<double *>(dynamic + kDynamicBytes - swap64), partial_raw, flags, rank_of);

      // singular values (column norms over the cluster), their ranks, and this rank's rows of the
      // factors in descending order
      double *norms = norms_raw, *partial = partial_raw;
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
      for (int64_t j = warp; j < k; j += warps)
      {
        const double *wj = w + j * rows;
        double sum = 0;
        for (int64_t i = lane; i < rows; i += 32) sum = fma(wj[i], wj[i], sum);
        sum = warp_sum(sum);
        if (lane == 0) partial[j] = sum;
      }
      cluster.sync();
      bool sound = true;
      for (int64_t j = threadIdx.x; j < k; j += blockDim.x)
      {
        double sum = 0;
        for (unsigned r = 0; r < ranks; ++r) sum += cluster.map_shared_rank(partial, r)[j];
        norms[j] = sqrt(sum);
        // (a NaN or an infinity in the block is in every column of W; zeros need no direction)
        sound = sound && sum < INFINITY && (sum == 0.0 || sum >= kLeastSquare);
      }
      if (!__syncthreads_and(sound)) sweeps_taken = -1;
      for (int64_t j = threadIdx.x; j < k; j += blockDim.x)
      {
        int r = 0;
        const double sj = norms[j];
        for (int64_t i = 0; i < k; ++i) r += (norms[i] > sj || (norms[i] == sj && i < j)) ? 1 : 0;
        rank_of[j] = r;
        if (rank == 0) s[e.s_off + r] = sj * ldexp(1.0, shift);
      }
      __syncthreads();
      double *uo = u + e.u_off, *vo = vh + e.vh_off;
      if (!precond)
      {
        // tall: U = W / sigma (m x k), Vh = V^T; wide: U = V (m x m), Vh = (W / sigma)^T
        for (int64_t i = threadIdx.x; i < rows * k; i += blockDim.x)
        {
          const int64_t j = i / rows, row = r0 + i % rows;
          if (row >= r1) continue;
          const double sj = norms[j];
          const double x = sj > 0 ? w[i] / sj : 0.0;
          if (wide)
            vo[static_cast<int64_t>(rank_of[j]) * n + row] = x;
          else
            uo[row * k + rank_of[j]] = x;
        }
        for (int64_t i = threadIdx.x; i < vrows * k; i += blockDim.x)
        {
          const int64_t j = i / vrows, row = c0 + i % vrows;  // entry row of column j of V
          if (row >= c1) continue;
          if (wide)
            uo[row * k + rank_of[j]] = v[i];
          else
            vo[static_cast<int64_t>(rank_of[j]) * n + row] = v[i];
        }
      }
      else
      {
        // the right factor P (W / sigma): row `row` of W is row order[row] of it (tall: Vh is its
        // transpose; wide: U is it)
        for (int64_t i = threadIdx.x; i < rows * k; i += blockDim.x)
        {
          const int64_t j = i / rows, row = r0 + i % rows;
          if (row >= r1) continue;
          const double sj = norms[j];
          const double x = sj > 0 ? w[i] / sj : 0.0;
          const int64_t to = __ldcg(qorder + row);
          if (wide)
            uo[to * k + rank_of[j]] = x;
          else
            vo[static_cast<int64_t>(rank_of[j]) * n + to] = x;
        }
        // the left factor Q [J; 0], J = V: V's rows to the workspace (column-major), then each rank
        // applies the reflectors, the last first, to its columns [q0, q1), a warp per column (tall:
        // U is it; wide: Vh is its transpose)
        for (int64_t i = threadIdx.x; i < vrows * k; i += blockDim.x)
        {
          const int64_t j = i / vrows, row = c0 + i % vrows;
          if (row < c1) g[j * k + row] = v[i];
        }
        cluster.sync();
        // the reflectors pass through shared memory in batches, and this rank's columns of B stay
        // there while they are transformed, when both fit (W and V there are no longer read)
        constexpr int64_t kBatch = 16;
        if (((cpr + kBatch) * len + kBatch) * 8 <= kDynamicBytes)
        {
          double *bcols = reinterpret_cast<double *>(dynamic), *stage = bcols + cpr * len, *stau = stage + kBatch * len;
          for (int64_t i = threadIdx.x; i < (q1 - q0) * len; i += blockDim.x)
          {
            const int64_t c = q0 + i / len, r = i % len;
            bcols[i] = r < k ? __ldcg(g + c * k + r) : 0.0;
          }
          for (int64_t top = k - 1; top >= 0; top -= kBatch)
          {
            const int64_t low = max(top - kBatch + 1, static_cast<int64_t>(0));  // reflectors top down to low
            __syncthreads();
            for (int64_t i = threadIdx.x; i < (top - low + 1) * len; i += blockDim.x)
            {
              const int64_t t = top - i / len, r = i % len;
              stage[i] = r > t ? __ldcg(qf + t * len + r) : 0.0;
            }
            if (threadIdx.x < top - low + 1) stau[threadIdx.x] = __ldcg(qtau + top - threadIdx.x);
            __syncthreads();
            // eight lanes a column, four columns a warp (as in the factorisation)
            for (int64_t c0 = q0 + warp * 4; c0 < q1; c0 += warps * 4)
            {
              const int64_t c = c0 + (lane >> 3);
              const bool live = c < q1;
              const int lanes = lane & 7;
              double *bc = bcols + ((live ? c : c0) - q0) * len;
              for (int64_t t = top; t >= low; --t)
              {
                const double tau = stau[top - t];
                if (tau == 0.0) continue;
                const double *vt = stage + (top - t) * len;
                double dot = 0.0;
                for (int64_t i = t + 1 + lanes; i < len; i += 8) dot = fma(vt[i], bc[i], dot);
                dot = group_sum<double, 8>(dot);
                const double head = bc[t], wt = tau * (head + dot);
                __syncwarp();
                if (live)
                {
                  for (int64_t i = t + 1 + lanes; i < len; i += 8) bc[i] = fma(-wt, vt[i], bc[i]);
                  if (lanes == 0) bc[t] = head - wt;
                }
                __syncwarp();
              }
            }
          }
          __syncthreads();
          for (int64_t i = threadIdx.x; i < (q1 - q0) * len; i += blockDim.x)
          {
            const int64_t c = q0 + i / len, r = i % len;
            const int64_t to = rank_of[c];
            if (wide)
              vo[to * n + r] = bcols[i];
            else
              uo[r * k + to] = bcols[i];
          }
        }
        else
        {
          for (int64_t c = q0 + warp; c < q1; c += warps)
          {
            double *bc = qb + c * len;
            for (int64_t i = lane; i < len; i += 32) bc[i] = i < k ? __ldcg(g + c * k + i) : 0.0;
            __syncwarp();
            for (int64_t t = k - 1; t >= 0; --t)
            {
              const double tau = __ldcg(qtau + t);
              if (tau == 0.0) continue;
              const double *vt = qf + t * len;
              double dot = 0.0;
              for (int64_t i = t + 1 + lane; i < len; i += 32) dot = fma(__ldcg(vt + i), bc[i], dot);
              dot = warp_sum(dot);
              const double wt = tau * (bc[t] + dot);
              for (int64_t i = t + 1 + lane; i < len; i += 32) bc[i] = fma(-wt, __ldcg(vt + i), bc[i]);
              __syncwarp();
              if (lane == 0) bc[t] -= wt;
              __syncwarp();
            }
            const int64_t to = rank_of[c];
            for (int64_t i = lane; i < len; i += 32)
            {
              if (wide)
                vo[to * n + i] = bc[i];
              else
                uo[i * k + to] = bc[i];
            }
          }
        }
      }
      if (threadIdx.x == 0 && rank == 0) info[block] = sweeps_taken;
      // no CTA leaves while another may still read its shared memory
      cluster.sync();
    }

    // per kept block: where its factors sit in the packed output of the SVD and where their kept
    // part lands in the two arenas
    struct KeepEntry
    {
      int64_t u_off, s_off, vh_off;      // packed factors: U rows x k, s k, Vh k x cols
      int64_t first_off, second_off;     // output blocks: first (rows x first_ld), second (second_rows x cols)
      int64_t values_off;                // where the kept values go in the bond array
      int32_t rows, cols, k, kept, first_ld, column, row, absorb;
    };

    // eight CTAs per kept block: first[:, column:column+kept] = U[:, :kept] (times s or sqrt(s)),
    // second[row:row+kept, :] = Vh[:kept, :] (times s or sqrt(s)), values[...] = s[:kept]
    __global__ void keep_kernel(const KeepEntry *__restrict__ table, const double *__restrict__ u,
                                const double *__restrict__ s, const double *__restrict__ vh,
                                double *__restrict__ first, double *__restrict__ second, double *__restrict__ values)
    {
      const KeepEntry e = table[blockIdx.x];
      const double *sv = s + e.s_off;
      // the pads after blocks of odd size (the bond's sector has first_ld multiplets)
      if (blockIdx.y == 0 && threadIdx.x == 0)
      {
        const int64_t one = static_cast<int64_t>(e.rows) * e.first_ld, two = static_cast<int64_t>(e.first_ld) * e.cols;
        if (e.column == 0 && (one & 1)) first[e.first_off + one] = 0.0;
        if (e.row == 0 && (two & 1)) second[e.second_off + two] = 0.0;
      }
      const int32_t at = static_cast<int32_t>(blockIdx.y * blockDim.x + threadIdx.x), step = static_cast<int32_t>(gridDim.y * blockDim.x);
      for (int32_t i = at; i < e.rows * e.kept; i += step)
      {
        const int32_t r = i / e.kept, j = i - r * e.kept;
        double x = u[e.u_off + static_cast<int64_t>(r) * e.k + j];
        if (e.absorb == 1) x *= sv[j];
        else if (e.absorb == 3) x *= sqrt(sv[j]);
        first[e.first_off + static_cast<int64_t>(r) * e.first_ld + e.column + j] = x;
      }
      for (int32_t i = at; i < e.kept * e.cols; i += step)
      {
        const int32_t j = i / e.cols, c = i - j * e.cols;
        double x = vh[e.vh_off + static_cast<int64_t>(j) * e.cols + c];
        if (e.absorb == 2) x *= sv[j];
        else if (e.absorb == 3) x *= sqrt(sv[j]);
        second[e.second_off + (e.row + j) * static_cast<int64_t>(e.cols) + c] = x;
      }
      for (int32_t j = at; j < e.kept; j += step) values[e.values_off + j] = sv[j];
    }
  } // namespace

  cudaError_t svd_blocks(int32_t count, int64_t largest, const void *table, const double *a, double *u, double *s,
                         double *vh, void *workspace, int32_t *info, cudaStream_t stream)
  {
    if (count <= 0) return cudaSuccess;
    static std::once_flag once;
    static cudaError_t configured = cudaSuccess;
    static int cluster_for[kMaxCluster + 1] = {};  // clusters of each size that fit on the GPU at once
    std::call_once(once, [] {
      configured = cudaFuncSetAttribute(jacobi_svd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(kDynamicBytes));
      if (configured == cudaSuccess)
        configured = cudaFuncSetAttribute(jacobi_svd_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      for (int size = 1; size <= kMaxCluster && configured == cudaSuccess; size *= 2)
      {
        cudaLaunchConfig_t config = {};
        cudaLaunchAttribute attribute[1];
        attribute[0].id = cudaLaunchAttributeClusterDimension;
        attribute[0].val.clusterDim.x = static_cast<unsigned>(size);
        attribute[0].val.clusterDim.y = 1;
        attribute[0].val.clusterDim.z = 1;
        config.gridDim = dim3(static_cast<unsigned>(size));
        config.blockDim = dim3(kSvdThreads);
        config.dynamicSmemBytes = kDynamicBytes;
        config.attrs = attribute;
        config.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, jacobi_svd_kernel, &config) != cudaSuccess)
        {
          cudaGetLastError();
          clusters = 0;
        }
        cluster_for[size] = clusters;
      }
    });
    if (configured != cudaSuccess) return configured;
    // the cluster the largest block wants (16 CTAs from 128 columns, 8 from 16, one CTA below that), or
    // the largest the GPU can hold; blocks come largest first, so a second wave of clusters only
    // holds small blocks
    const int want = largest >= 128 ? 16 : largest >= 16 ? 8 : 1;
    int size = 1;
    for (int c = want; c > 1; c /= 2)
      if (cluster_for[c] >= 1)
      {
        size = c;
        break;
      }
    cudaLaunchConfig_t config = {};
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = static_cast<unsigned>(size);
    attribute[0].val.clusterDim.y = 1;
    attribute[0].val.clusterDim.z = 1;
    config.gridDim = dim3(static_cast<unsigned>(count) * static_cast<unsigned>(size));
    config.blockDim = dim3(kSvdThreads);
    config.dynamicSmemBytes = kDynamicBytes;
    config.stream = stream;
    config.attrs = attribute;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, jacobi_svd_kernel, static_cast<const SvdEntry *>(table), a, u, s, vh,
                              static_cast<double *>(workspace), info);
  }

  int64_t svd_workspace_doubles(int64_t rows, int64_t cols)
  {
    const int64_t len = std::max(rows, cols), k = std::min(rows, cols);
    return k == 0 ? 0 : svd_layout(len, k).total;
  }

  cudaError_t svd_keep(int32_t count, const void *table, const double *u, const double *s, const double *vh,
                       double *first, double *second, double *values, cudaStream_t stream)
  {
    if (count <= 0) return cudaSuccess;
    keep_kernel<<<dim3(static_cast<unsigned>(count), 8), 256, 0, stream>>>(static_cast<const KeepEntry *>(table), u, s, vh, first, second, values);
    return cudaGetLastError();
  }

} // namespace ttg

// ------------------------------------------------------------------------------------------
// the ranking of a split's singular values on the device
// ------------------------------------------------------------------------------------------

namespace ttg
{
  namespace
  {
    // Every singular value of a split (block after block, each block's in descending order) sorted
    // by (value descending, position ascending) — the order of the host's stable sort — by a bitonic
    // sort in shared memory; then, the threads sharing the sorted values: the cut (values above `tol`,
    // at most `max_bond`), the values each block keeps, and the +-q pairing of the bond (a domain
    // sector keeps at most as many as its dual, the first ones in the sorted order; a sector whose
    // dual keeps nothing drops out), as tentorch/linalg/graded/svd.cpp:68-118 ranks them on the host.
    __global__ void rank_kernel(const double *__restrict__ values, int32_t n_values, const int32_t *__restrict__ block_k,
                                const int32_t *__restrict__ block_sector, int32_t n_blocks, const int32_t *__restrict__ dual,
                                int32_t n_sectors, double tol, int64_t max_bond, int32_t *__restrict__ kept_out)
    {
      extern __shared__ __align__(16) unsigned char smem_raw[];
      int n = 1;
      while (n < n_values) n <<= 1;
      unsigned long long *key = reinterpret_cast<unsigned long long *>(smem_raw);  // [n]
      int32_t *pos = reinterpret_cast<int32_t *>(key + n);                          // [n]
      int32_t *block_of = pos + n;                                                  // [n_values]
      int32_t *kept = block_of + n_values;                                          // [n_blocks]
      int32_t *mult = kept + n_blocks;                                              // [n_sectors] x 3
      int32_t *paired = mult + n_sectors;
      __shared__ int32_t cut, any, differs;
      // keys: the complement of |value|'s bits (ascending keys = descending values); padding last
      for (int i = threadIdx.x; i < n; i += blockDim.x)
      {
        if (i < n_values)
        {
          key[i] = ~(static_cast<unsigned long long>(__double_as_longlong(values[i])) & 0x7fffffffffffffffull);
          pos[i] = i;
        }
        else
        {
          key[i] = ~0ull;
          pos[i] = 0x7fffffff;
        }
      }
      for (int32_t b = threadIdx.x; b < n_blocks; b += blockDim.x)
      {
        int32_t at = 0;
        for (int32_t i = 0; i < b; ++i) at += block_k[i];
        for (int32_t j = 0; j < block_k[b]; ++j) block_of[at + j] = b;
        kept[b] = 0;
      }
      for (int32_t s = threadIdx.x; s < n_sectors; s += blockDim.x) mult[s] = 0;
      if (threadIdx.x == 0)
      {
        cut = n_values;
        any = differs = 0;
      }
      __syncthreads();
      for (int size = 2; size <= n; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1)
        {
          for (int i = threadIdx.x; i < n; i += blockDim.x)
          {
            const int j = i ^ stride;
            if (j > i)
            {
              const bool ascending = (i & size) == 0;
              const bool greater = key[i] > key[j] || (key[i] == key[j] && pos[i] > pos[j]);
              if (greater == ascending)
              {
                const unsigned long long tk = key[i];
                key[i] = key[j];
                key[j] = tk;
                const int32_t tp = pos[i];
                pos[i] = pos[j];
                pos[j] = tp;
              }
            }
          }
          __syncthreads();
        }
      // the cut: the first of the sorted values that is not above tol
      for (int32_t r = threadIdx.x; r < n_values; r += blockDim.x)
        if (!(values[pos[r]] > tol)) atomicMin(&cut, r);
      __syncthreads();
      const int32_t last = max_bond >= 0 && cut > max_bond ? static_cast<int32_t>(max_bond) : cut;
      for (int32_t r = threadIdx.x; r < last; r += blockDim.x) atomicAdd(kept + block_of[pos[r]], 1);
      __syncthreads();
      for (int32_t b = threadIdx.x; b < n_blocks; b += blockDim.x) atomicAdd(mult + block_sector[b], kept[b]);
      __syncthreads();
      for (int32_t s = threadIdx.x; s < n_sectors; s += blockDim.x)
      {
        paired[s] = -1;
        if (mult[s] == 0) continue;
        if (mult[dual[s]] > 0)
        {
          paired[s] = min(mult[s], mult[dual[s]]);
          any = 1;
          if (paired[s] != mult[s]) differs = 1;
        }
        else
          differs = 1;
      }
      __syncthreads();
      if (any && differs)
      {
        for (int32_t b = threadIdx.x; b < n_blocks; b += blockDim.x) kept[b] = 0;
        __syncthreads();
        // a warp per sector walks the sorted values 32 at a time and keeps the sector's first ones
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
        for (int32_t s = warp; s < n_sectors; s += warps)
        {
          int32_t used = 0;
          for (int32_t r0 = 0; r0 < last && used < paired[s]; r0 += 32)
          {
            const int32_t r = r0 + lane, b = r < last ? block_of[pos[r]] : -1;
            const bool in = b >= 0 && block_sector[b] == s;
            const unsigned mask = __ballot_sync(0xffffffffu, in);
            if (in && used + __popc(mask & ((1u << lane) - 1u)) < paired[s]) atomicAdd(kept + b, 1);
            used += __popc(mask);
          }
        }
        __syncthreads();
      }
      for (int32_t b = threadIdx.x; b < n_blocks; b += blockDim.x) kept_out[b] = kept[b];
    }
  } // namespace

  int64_t rank_bytes(int32_t n_values, int32_t n_blocks, int32_t n_sectors)
  {
    int64_t n = 1;
    while (n < n_values) n <<= 1;
    return n * 12 + static_cast<int64_t>(n_values) * 4 + static_cast<int64_t>(n_blocks) * 4 + static_cast<int64_t>(n_sectors) * 12;
  }

  cudaError_t svd_rank(const double *values, int32_t n_values, const int32_t *block_k, const int32_t *block_sector,
                       int32_t n_blocks, const int32_t *dual, int32_t n_sectors, double tol, int64_t max_bond, int32_t *kept,
                       cudaStream_t stream)
  {
    const int64_t bytes = rank_bytes(n_values, n_blocks, n_sectors);
    cudaError_t e = cudaFuncSetAttribute(rank_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
    if (e != cudaSuccess) return e;
    rank_kernel<<<1, 1024, bytes, stream>>>(values, n_values, block_k, block_sector, n_blocks, dual, n_sectors, tol, max_bond,
                                            kept);
    return cudaGetLastError();
  }
} // namespace ttg

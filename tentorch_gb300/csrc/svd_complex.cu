// Thin SVDs of complex128 blocks in one call, for the truncating splittings
// (tentorch/linalg/graded/svd.cpp:41-177, which calls at::linalg_svd once per block).  The method of svd.cu in
// complex arithmetic, as three launches for all blocks:
//   1. the block (its conjugate transpose when it is wider than tall), len x k, its columns sorted by norm;
//   2. its QR factorisation B P = Q R (qr.cu);
//   3. one-sided Jacobi on X = R^H: FP32 sweeps in blocks of four columns over the cluster's shared memory
//      (a pair's product gamma is brought to |gamma| by a phase on its second column, then the real
//      rotation applies), V refined in FP64 by matrix products to cosines at round-off, and the factors:
//      X V = W = U_x S, so B P = (Q V) S U_x^H.
// Pairs that the refinement leaves open (columns at the block's round-off) go through FP64 sweeps.  A block
// that does not settle or has a singular value below 1e-128 of its largest entry reports -1 in `info`, and -2 where all
// is well but for values that are zero and have no direction on one side; the caller factors the first by itself, the
// second only when it keeps zeros.  See svd.cu for each step's reasons.
//
// Bound by latency: the QR's chain (a column at a time), the rounds of the sweeps, and FP64 multiply-adds (64
// clocks a warp instruction on a quarter of an SM), so a block has a cluster even where one CTA could
// hold it: with all of a 24 x 24 block in one CTA nine of them took 818 us, with eight CTAs for the FP64 products
// 491.  The two-site tensor of bond 64 (10 blocks, the largest 23 x 23), the whole call: 456 us, 9.4 ms
// with one cuSOLVER call per block; of it the QR 137 us and the Jacobi kernel 280.  Nine 48 x 48 blocks 1.1 ms (40),
// two of 150 x 150 6.7 ms (48).  |A - U S V^H| is 5e-16 of |A| where cuSOLVER's bidiagonal iteration leaves 4e-15.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>

#include "executor.h"
#include "launch.h"

namespace ttg
{
  namespace
  {
    namespace cg = cooperative_groups;

    constexpr int kThreads = 512;
    constexpr int kMaxSweeps = 40;
    // Blocks are worked on with their largest entry at about 2^200, and columns whose squared norm is then below
    // kLeastSquare (1e-128 of the block) have no direction to be trusted: products of four values neither overflow
    // nor vanish (svd.cu).
    constexpr int kBlockExp = 200;
    constexpr double kLeastSquare = 0x1p-450;
    // Up to so many columns one CTA does the FP32 sweeps, without cluster barriers and remote columns, while the
    // others wait: nine 48 x 48 blocks 1144 -> 1119 us, four 64 x 64 1497 -> 1484.
    constexpr int kOneSweeper = 64;
    constexpr int kMaxCols = 160;                      // columns (and rows of X) of a block
    constexpr int64_t kDynamic = 212 * 1024;
    constexpr int kTile = 16, kDepth = 32, kPitch = kTile + 1;
    constexpr int64_t kStageBytes = 2 * kDepth * kPitch * 16;

    // a_off, rows, cols, u_off, s_off, vh_off, ws_off in elements (complex numbers; s in doubles)
    struct Entry
    {
      int64_t a_off, rows, cols, u_off, s_off, vh_off, ws_off;
    };
    // One block's workspace, in complex elements: B P (len x k, row-major), Q (the same), R, V and its next
    // iterate, W, G, H (k x k each), E (k x k of float2: half), the QR's workspace and the sorted order.
    struct Places
    {
      int64_t b, q, r, v0, v1, w, g, h, e, qr, order, total;
    };
    __host__ __device__ inline Places layout_of(int64_t len, int64_t k)
    {
      Places l;
      l.b = 0;
      l.q = len * k;
      l.r = 2 * len * k;
      l.v0 = l.r + k * k;
      l.v1 = l.v0 + k * k;
      l.w = l.v1 + k * k;
      l.g = l.w + k * k;
      l.h = l.g + k * k;
      l.e = l.h + k * k;
      l.qr = l.e + (k * k + 1) / 2;
      l.order = l.qr + k * (len + 1);
      l.total = (l.order + (k + 3) / 4 + 15) / 16 * 16;
      return l;
    }

    __device__ __forceinline__ double2 cmul_add(double2 a, double2 b, double2 c)
    {
      return make_double2(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
    }
    __device__ __forceinline__ float2 cmul_add(float2 a, float2 b, float2 c)
    {
      return make_float2(fmaf(a.x, b.x, fmaf(-a.y, b.y, c.x)), fmaf(a.x, b.y, fmaf(a.y, b.x, c.y)));
    }
    __device__ __forceinline__ double2 conj2(double2 a) { return make_double2(a.x, -a.y); }
    __device__ __forceinline__ float2 to_float(double2 a) { return make_float2(static_cast<float>(a.x), static_cast<float>(a.y)); }
    __device__ __forceinline__ double2 load2(const double2 *p) { return __ldcg(p); }
    __device__ __forceinline__ float2 load2(const float2 *p) { return __ldcg(p); }

    // 1. the columns of the block (wide: of its conjugate transpose) sorted by norm, largest first
    __global__ void __launch_bounds__(256) sort_kernel(const Entry *__restrict__ table, const double2 *__restrict__ a, double2 *__restrict__ workspace)
    {
      __shared__ float norms[kMaxCols];
      __shared__ int order[kMaxCols];
      dependent_entry();
      const Entry e = table[blockIdx.x];
      const bool wide = e.cols > e.rows;
      const int len = static_cast<int>(wide ? e.cols : e.rows), k = static_cast<int>(wide ? e.rows : e.cols);
      const Places l = layout_of(len, k);
      double2 *ws = workspace + e.ws_off;
      const auto entry = [&](int i, int j) {
        const double2 x = a[e.a_off + (wide ? static_cast<int64_t>(j) * len + i : static_cast<int64_t>(i) * k + j)];
        return wide ? conj2(x) : x;
      };
      // the largest entry, so that the FP32 sums of squares neither overflow nor vanish
      __shared__ unsigned long long big;
      if (threadIdx.x == 0) big = 0;
      __syncthreads();
      double most = 0.0;
      for (int64_t i = threadIdx.x; i < static_cast<int64_t>(len) * k; i += blockDim.x)
      {
        const double2 x = a[e.a_off + i];
        most = fmax(most, fmax(fabs(x.x), fabs(x.y)));
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) most = fmax(most, __shfl_xor_sync(0xffffffffu, most, o));
      if ((threadIdx.x & 31) == 0) atomicMax(&big, static_cast<unsigned long long>(__double_as_longlong(most)));
      __syncthreads();
      const double top = __longlong_as_double(static_cast<long long>(big)), inv = top > 0.0 && top < 1.7976931348623157e308 ? 1.0 / top : 1.0;
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
      for (int j = warp; j < k; j += warps)
      {
        float sum = 0.0f;
        for (int i = lane; i < len; i += 32)
        {
          const double2 x = entry(i, j);
          const float re = static_cast<float>(x.x * inv), im = static_cast<float>(x.y * inv);
          sum = fmaf(re, re, fmaf(im, im, sum));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) norms[j] = sum >= 0.0f ? sum : INFINITY;  // a NaN sorts like an infinity
      }
      __syncthreads();
      for (int j = threadIdx.x; j < k; j += blockDim.x)
      {
        int r = 0;
        for (int i = 0; i < k; ++i) r += (norms[i] > norms[j] || (norms[i] == norms[j] && i < j)) ? 1 : 0;
        order[r] = j;
      }
      __syncthreads();
      int32_t *out = reinterpret_cast<int32_t *>(ws + l.order);
      for (int j = threadIdx.x; j < k; j += blockDim.x) out[j] = order[j];
      for (int64_t i = threadIdx.x; i < static_cast<int64_t>(len) * k; i += blockDim.x)
        ws[l.b + i] = entry(static_cast<int>(i / k), order[static_cast<int>(i % k)]);
    }

    __device__ __forceinline__ void circle_pair(int round, int t, int players, int &p, int &q)
    {
      const int n = players - 1;
      int a = round, b = n;
      if (t != 0)
      {
        a = round + t;
        if (a >= n) a -= n;
        b = round - t + n;
        if (b >= n) b -= n;
      }
      p = a < b ? a : b;
      q = a < b ? b : a;
    }

    // c, s of the rotation for norms alpha, beta (diff = beta - alpha) and a real product g > 0 (svd.cu angle_fast)
    __device__ __forceinline__ void angle(float diff, float g, float &c, float &s)
    {
      const float zeta = __fdividef(diff, 2.0f * g), one = fmaf(zeta, zeta, 1.0f);
      const float t = fabsf(zeta) > 1e15f ? __fdividef(0.5f, zeta)
                                          : copysignf(__fdividef(1.0f, fabsf(zeta) + one * rsqrtf(one)), zeta);
      c = rsqrtf(fmaf(t, t, 1.0f));
      s = c * t;
    }

    // The FP32 sweeps (svd.cu blocked_sweeps) on complex columns, by the first `ranks` CTAs of the cluster: 1 or all.
    template <int NR>
    __device__ int sweeps(const cg::cluster_group &cluster, int ranks, float2 *w, float2 *v, int k, float tol, float2 *jbuf, int *flags)
    {
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
      const int rank = static_cast<int>(cluster.block_rank());
      const int blocks = (k + 7) / 8 * 2;
      const float settled = sqrtf(tol);
      float2 *jm = jbuf + warp * 64;
      const auto sync = [&] {
        if (ranks == 1) __syncthreads();
        else cluster.sync();
      };
      const auto at_home = [&](float2 *base, int b) -> float2 * {
        float2 *here = base + static_cast<int64_t>(b / ranks) * 4 * 32 * NR;
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
            int bl, br;
            circle_pair(round, bp, blocks, bl, br);
            float2 *left = at_home(w, bl), *right = at_home(w, br);
            float2 x[8][NR + 1];
#pragma unroll
            for (int c = 0; c < 8; ++c)
            {
              const float2 *from = (c < 4 ? left + c * 32 * NR : right + (c - 4) * 32 * NR) + lane;
#pragma unroll
              for (int r = 0; r < NR; ++r) x[c][r] = from[r * 32];
              x[c][NR] = make_float2(lane == c ? 1.0f : 0.0f, 0.0f);
            }
            // eight sums reduced together: lane bits 4..2 end with value 4 b4 + 2 b3 + b2
            const auto reduce8 = [&](float (&p)[8]) {
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
              return p[0];
            };
            float n2[8];
            {
              float p[8];
#pragma unroll
              for (int c = 0; c < 8; ++c)
              {
                p[c] = 0.0f;
#pragma unroll
                for (int r = 0; r < NR; ++r) p[c] = fmaf(x[c][r].x, x[c][r].x, fmaf(x[c][r].y, x[c][r].y, p[c]));
              }
              const float sum = reduce8(p);
#pragma unroll
              for (int c = 0; c < 8; ++c) n2[c] = __shfl_sync(0xffffffffu, sum, c * 4);
            }
            bool any = false, large = false;
            const auto rotate4 = [&](const int (&pc)[4], const int (&qc)[4]) {
              // gamma_i = x_p^H x_q: real parts first, then imaginary ones
              float g[8];
#pragma unroll
              for (int i = 0; i < 4; ++i)
              {
                g[i] = g[i + 4] = 0.0f;
#pragma unroll
                for (int r = 0; r < NR; ++r)
                {
                  const float2 p = x[pc[i]][r], q = x[qc[i]][r];
                  g[i] = fmaf(p.x, q.x, fmaf(p.y, q.y, g[i]));
                  g[i + 4] = fmaf(p.x, q.y, fmaf(-p.y, q.x, g[i + 4]));
                }
              }
              const float part = reduce8(g), other = __shfl_xor_sync(0xffffffffu, part, 16);
              const float re = lane & 16 ? other : part, im = lane & 16 ? part : other;
              // lanes 4 i .. 4 i + 3 (and 16 on) hold pair i's product; its size without squares that underflow
              const float most = fmaxf(fabsf(re), fabsf(im)), ratio = most > 0.0f ? __fdividef(fminf(fabsf(re), fabsf(im)), most) : 0.0f;
              const float one = fmaf(ratio, ratio, 1.0f), size = most * one * rsqrtf(one);
              const int mine = (lane >> 2) & 3;
              float alpha = n2[pc[0]], beta = n2[qc[0]];
#pragma unroll
              for (int i = 1; i < 4; ++i)
              {
                alpha = mine == i ? n2[pc[i]] : alpha;
                beta = mine == i ? n2[qc[i]] : beta;
              }
              const float cosine = size * rsqrtf(alpha) * rsqrtf(beta);
              float c = 1.0f, sn = 0.0f, fr = 1.0f, fi = 0.0f;
              const bool turn = cosine > tol && size > 0.0f;
              if (turn)
              {
                angle(beta - alpha, size, c, sn);
                fr = __fdividef(re, size);
                fi = __fdividef(im, size);
              }
              const float cc = c * c, ss = sn * sn, cs2 = 2.0f * c * sn * size;
              const float na = turn ? cc * alpha - cs2 + ss * beta : alpha, nb = turn ? ss * alpha + cs2 + cc * beta : beta;
              if (!__any_sync(0xffffffffu, turn)) return;
              any = true;
              large = large || cosine > settled;
#pragma unroll
              for (int i = 0; i < 4; ++i)
              {
                const float ci = __shfl_sync(0xffffffffu, c, 4 * i), si = __shfl_sync(0xffffffffu, sn, 4 * i);
                const float pr = __shfl_sync(0xffffffffu, fr, 4 * i), pm = __shfl_sync(0xffffffffu, fi, 4 * i);
                n2[pc[i]] = __shfl_sync(0xffffffffu, na, 4 * i);
                n2[qc[i]] = __shfl_sync(0xffffffffu, nb, 4 * i);
#pragma unroll
                for (int r = 0; r <= NR; ++r)
                {
                  const float2 p = x[pc[i]][r], q0 = x[qc[i]][r];
                  // the second column by the conjugate phase, which makes the product real
                  const float2 q = make_float2(fmaf(pr, q0.x, pm * q0.y), fmaf(pr, q0.y, -pm * q0.x));
                  x[pc[i]][r] = make_float2(fmaf(ci, p.x, -si * q.x), fmaf(ci, p.y, -si * q.y));
                  x[qc[i]][r] = make_float2(fmaf(si, p.x, ci * q.x), fmaf(si, p.y, ci * q.y));
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
              float2 *to = (c < 4 ? left + c * 32 * NR : right + (c - 4) * 32 * NR) + lane;
#pragma unroll
              for (int r = 0; r < NR; ++r) to[r * 32] = x[c][r];
              if (lane < 8) jm[lane * 8 + c] = x[c][NR];
            }
            __syncwarp();
            float2 *vl = at_home(v, bl) + lane, *vr = at_home(v, br) + lane;
#pragma unroll
            for (int r = 0; r < NR; ++r)
            {
              float2 out[8] = {};
#pragma unroll
              for (int i = 0; i < 8; ++i)
              {
                const float2 in = (i < 4 ? vl + i * 32 * NR : vr + (i - 4) * 32 * NR)[r * 32];
#pragma unroll
                for (int j = 0; j < 8; ++j) out[j] = cmul_add(in, jm[i * 8 + j], out[j]);
              }
#pragma unroll
              for (int i = 0; i < 8; ++i) (i < 4 ? vl + i * 32 * NR : vr + (i - 4) * 32 * NR)[r * 32] = out[i];
            }
            __syncwarp();
          }
          sync();
        }
        const int more = static_cast<int>(threadIdx.x) < ranks ? *cluster.map_shared_rank(flags + (sweep & 1), threadIdx.x) : 0;
        if (!__syncthreads_or(more)) return sweep + 1;
      }
      return -1;
    }

    // out(i, j) = sum_x a(x, i) b(x, j) over a 16 x 16 tile, x < depth (svd.cu small_product)
    template <typename T, typename FA, typename FB, typename Out>
    __device__ void product(int depth, FA fa, bool a_x_fast, FB fb, bool b_x_fast, void *stage, Out out)
    {
      T *sa = static_cast<T *>(stage), *sb = sa + kDepth * kPitch;
      const int t = threadIdx.x, i = t & 15, j = (t >> 4) & 15, half = t >> 8;
      const int xa = a_x_fast ? t & 31 : t >> 4, ia = a_x_fast ? t >> 5 : t & 15;
      const int xb = b_x_fast ? t & 31 : t >> 4, jb = b_x_fast ? t >> 5 : t & 15;
      T acc{}, na{}, nb{};
      if (xa < depth) na = fa(xa, ia);
      if (xb < depth) nb = fb(xb, jb);
      for (int x0 = 0; x0 < depth; x0 += kDepth)
      {
        sa[xa * kPitch + ia] = na;
        sb[xb * kPitch + jb] = nb;
        __syncthreads();
        const int x1 = x0 + kDepth;
        if (x1 < depth)
        {
          na = x1 + xa < depth ? fa(x1 + xa, ia) : T{};
          nb = x1 + xb < depth ? fb(x1 + xb, jb) : T{};
        }
#pragma unroll
        for (int x = 0; x < kDepth / 2; ++x)
          acc = cmul_add(sa[(half * 16 + x) * kPitch + i], sb[(half * 16 + x) * kPitch + j], acc);
        __syncthreads();
      }
      if (half == 1) sa[j * kPitch + i] = acc;
      __syncthreads();
      if (half == 0)
      {
        const T o = sa[j * kPitch + i];
        acc.x += o.x;
        acc.y += o.y;
        out(i, j, acc);
      }
      __syncthreads();
    }

    // 3. Jacobi on X = R^H and the factors
    __global__ void __launch_bounds__(kThreads, 1)
      complex_jacobi_kernel(const Entry *__restrict__ table, double2 *__restrict__ u, double *__restrict__ s, double2 *__restrict__ vh,
                            double2 *__restrict__ workspace, int32_t *__restrict__ info)
    {
      extern __shared__ __align__(16) unsigned char dynamic[];
      __shared__ double lambda[kMaxCols];
      __shared__ int rank_of[kMaxCols];
      __shared__ int flags[3];
      __shared__ double big;
      dependent_entry();
      const cg::cluster_group cluster = cg::this_cluster();
      const int ranks = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
      const int block = blockIdx.x / ranks;
      const Entry e = table[block];
      const bool wide = e.cols > e.rows;
      const int len = static_cast<int>(wide ? e.cols : e.rows), k = static_cast<int>(wide ? e.rows : e.cols);
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
      const Places l = layout_of(len, k);
      double2 *ws = workspace + e.ws_off;
      const double2 *q = ws + l.q, *r = ws + l.r;
      double2 *v_cur = ws + l.v0, *v_next = ws + l.v1, *wg = ws + l.w, *g = ws + l.g, *h = ws + l.h;
      float2 *em = reinterpret_cast<float2 *>(ws + l.e);
      const int32_t *order = reinterpret_cast<const int32_t *>(ws + l.order);
      void *stage = dynamic + kDynamic - kStageBytes;
      // X(row, col) = conj(R(col, row)), lower triangular
      double scale = 1.0;  // a power of two: no product under- or overflows
      const auto entry = [&](int row, int col) {
        if (col > row) return make_double2(0.0, 0.0);
        const double2 x = load2(r + static_cast<int64_t>(col) * k + row);
        return make_double2(x.x * scale, -x.y * scale);
      };
      const int tiles = (k + kTile - 1) / kTile;

      // FP32 sweeps
      const int sweepers = k <= kOneSweeper ? 1 : ranks;
      const int rows32 = (k + 31) / 32, ld = 32 * rows32, column_blocks = (k + 7) / 8 * 2, mine = (column_blocks + sweepers - 1) / sweepers;
      float2 *w32 = reinterpret_cast<float2 *>(dynamic), *v32 = w32 + mine * 4 * ld, *jbuf = v32 + mine * 4 * ld;
      if (threadIdx.x == 0) big = 0.0;
      __syncthreads();
      double most = 0.0;
      for (int i = threadIdx.x; i < k * k; i += blockDim.x)
      {
        const double2 x = load2(r + i);
        most = fmax(most, fmax(fabs(x.x), fabs(x.y)));
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) most = fmax(most, __shfl_xor_sync(0xffffffffu, most, o));
      if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<unsigned long long *>(&big), static_cast<unsigned long long>(__double_as_longlong(most)));
      __syncthreads();
      int shift = 0;
      if (big > 0.0 && big < 1.7976931348623157e308) frexp(big, &shift);
      shift = max(-800, min(1000, shift));
      scale = ldexp(1.0, -shift);  // to about one for the FP32 sweeps, then to 2^kBlockExp
      const auto column_of = [&](int i) { return ((i / ld / 4) * sweepers + rank) * 4 + i / ld % 4; };
      int taken = 0;
      if (rank < sweepers)
      {
        for (int i = threadIdx.x; i < mine * 4 * ld; i += blockDim.x)
        {
          const int row = i % ld, col = column_of(i);
          float2 x = make_float2(0.0f, 0.0f);
          if (row < k && col < k) x = to_float(entry(row, col));
          w32[i] = x;
          v32[i] = make_float2(row == col && col < k ? 1.0f : 0.0f, 0.0f);
        }
        switch (rows32)
        {
        case 1: taken = sweeps<1>(cluster, sweepers, w32, v32, k, 1e-5f, jbuf, flags); break;
        case 2: taken = sweeps<2>(cluster, sweepers, w32, v32, k, 1e-5f, jbuf, flags); break;
        case 3: taken = sweeps<3>(cluster, sweepers, w32, v32, k, 1e-5f, jbuf, flags); break;
        case 4: taken = sweeps<4>(cluster, sweepers, w32, v32, k, 1e-5f, jbuf, flags); break;
        default: taken = sweeps<5>(cluster, sweepers, w32, v32, k, 1e-5f, jbuf, flags); break;
        }
        for (int i = threadIdx.x; i < mine * 4 * ld; i += blockDim.x)
        {
          const int row = i % ld, col = column_of(i);
          if (row < k && col < k) v_cur[static_cast<int64_t>(col) * k + row] = make_double2(v32[i].x, v32[i].y);
        }
        if (threadIdx.x == 0) flags[2] = taken;
      }
      cluster.sync();
      taken = cluster.map_shared_rank(flags, 0)[2];
      cluster.sync();
      shift -= kBlockExp;
      scale = ldexp(1.0, -shift);

      // the refinement (svd.cu): E_rc = t e^(i phase) - h_rc / 2 with the phase of the pair's product.  Where W's
      // columns are not orthogonal to round-off after it (rank-deficient blocks), FP64 sweeps follow; V alone
      // is refined (`plain`) until it is orthonormal for them.
      const double tol = 2.220446049250313e-16 * sqrt(static_cast<double>(k));
      bool refined = false, sweep = false, plain = false, last = false;
      for (int it = 0; it < 12 && taken > 0; ++it)
      {
        const double2 *vc = v_cur;
        for (int tile = rank; tile < tiles * tiles; tile += ranks)
        {
          const int tr = tiles - 1 - tile / tiles, tc = tile % tiles;
          product<double2>(
            min(k, (tr + 1) * kTile), [&](int x, int i) { const int row = tr * kTile + i; return row < k ? entry(row, x) : make_double2(0.0, 0.0); }, true,
            [&](int x, int j) { return tc * kTile + j < k ? load2(vc + static_cast<int64_t>(tc * kTile + j) * k + x) : make_double2(0.0, 0.0); }, true, stage,
            [&](int i, int j, double2 sum) {
              const int row = tr * kTile + i, c = tc * kTile + j;
              if (row < k && c < k) wg[static_cast<int64_t>(c) * k + row] = sum;
            });
        }
        cluster.sync();
        int turn = 0;
        if (last)
        {
          refined = true;
          break;
        }
        for (int which = 0; which < 2; ++which)
          for (int tr = 0; tr < tiles; ++tr)
            for (int tc = tr; tc < tiles; ++tc, ++turn)
            {
              if (turn % ranks != rank) continue;
              const double2 *m = which == 0 ? wg : vc;
              double2 *to = which == 0 ? g : h;
              product<double2>(
                k, [&](int x, int i) { return tr * kTile + i < k ? conj2(load2(m + static_cast<int64_t>(tr * kTile + i) * k + x)) : make_double2(0.0, 0.0); }, true,
                [&](int x, int j) { return tc * kTile + j < k ? load2(m + static_cast<int64_t>(tc * kTile + j) * k + x) : make_double2(0.0, 0.0); }, true, stage,
                [&](int i, int j, double2 sum) {
                  const int row = tr * kTile + i, c = tc * kTile + j;
                  if (row <= c && c < k) to[static_cast<int64_t>(c) * k + row] = sum;
                });
            }
        cluster.sync();
        for (int j = threadIdx.x; j < k; j += blockDim.x) lambda[j] = load2(g + static_cast<int64_t>(j) * k + j).x;
        __syncthreads();
        int status = 0;  // above four times tol: 1 a cosine, 2 V^H V - I; 8: either above tol; 4: an angle that is not small
        for (int i = rank * blockDim.x + threadIdx.x; i < k * k; i += ranks * blockDim.x)
        {
          const int c = i / k, row = i - c * k;
          if (row > c) continue;
          const double2 hv = load2(h + i);
          const double off = fmax(fabs(row == c ? 1.0 - hv.x : hv.x), fabs(hv.y));
          if (!(off <= tol)) status |= off <= 4.0 * tol ? 8 : 10;
          if (row == c)
          {
            em[i] = make_float2(static_cast<float>(0.5 * (1.0 - hv.x)), 0.0f);
            continue;
          }
          const double2 gv = load2(g + i);
          const double lr = lambda[row], lc = lambda[c];
          const double limit = tol * tol * lr * lc, square = fma(gv.x, gv.x, gv.y * gv.y);
          const bool open = !(square <= 16.0 * limit);
          if (!(square <= limit)) status |= open ? 9 : 8;
          double2 tangent = make_double2(0.0, 0.0);
          const double2 st = make_double2(fma(-0.5 * hv.x, lr + lc, gv.x), fma(-0.5 * hv.y, lr + lc, gv.y));
          const double size = sqrt(fma(st.x, st.x, st.y * st.y));
          if (!plain && size > 0.0)
          {
            int ex;
            frexp(fmax(lr, lc), &ex);
            float cf, sf;
            const float gf = static_cast<float>(ldexp(size, -ex));
            if (gf > 0.0f)
            {
              angle(static_cast<float>(ldexp(lc - lr, -ex)), gf, cf, sf);
              const float t = sf / cf;
              // (at round-off the angle of a pair of equal values is noise)
              if (open && fabsf(t) > 0.1f) status |= 4;
              if (fabsf(t) <= (open ? 0.1f : 1e-8f)) tangent = make_double2(t * (st.x / size), t * (st.y / size));
            }
          }
          em[static_cast<int64_t>(c) * k + row] = make_float2(static_cast<float>(fma(-0.5, hv.x, tangent.x)), static_cast<float>(fma(-0.5, hv.y, tangent.y)));
          // the lower element: minus the conjugate of the angle's part, the conjugate of h's
          em[static_cast<int64_t>(row) * k + c] = make_float2(static_cast<float>(fma(-0.5, hv.x, -tangent.x)), static_cast<float>(fma(0.5, hv.y, tangent.y)));
        }
        int all = 0;
#pragma unroll
        for (int bit = 1; bit < 16; bit <<= 1) all |= __syncthreads_or(status & bit) ? bit : 0;
        status = all;
        if (threadIdx.x == 0) flags[2] = status;
        cluster.sync();
        status = 0;
        for (int o = 0; o < ranks; ++o) status |= cluster.map_shared_rank(flags, o)[2];
        if ((it >= 1 && (status & 4)) || it >= 5) plain = true;
        refined = !(status & 8);
        taken = it + 1;
        if (refined) break;
        last = !(status & 3) && it < 11;
        if (plain && !last && !(status & 2))
        {
          sweep = true;
          break;
        }
        for (int tile = rank; tile < tiles * tiles; tile += ranks)
        {
          const int tr = tile / tiles, tc = tile % tiles;
          product<float2>(
            k, [&](int x, int i) { return tr * kTile + i < k ? to_float(load2(vc + static_cast<int64_t>(x) * k + tr * kTile + i)) : make_float2(0.0f, 0.0f); }, false,
            [&](int x, int j) { return tc * kTile + j < k ? load2(em + static_cast<int64_t>(tc * kTile + j) * k + x) : make_float2(0.0f, 0.0f); }, true, stage,
            [&](int i, int j, float2 sum) {
              const int row = tr * kTile + i, c = tc * kTile + j;
              if (row < k && c < k)
              {
                const double2 old = load2(vc + static_cast<int64_t>(c) * k + row);
                v_next[static_cast<int64_t>(c) * k + row] = make_double2(old.x + static_cast<double>(sum.x), old.y + static_cast<double>(sum.y));
              }
            });
        }
        cluster.sync();
        double2 *t = v_cur;
        v_cur = v_next;
        v_next = t;
      }
      cluster.sync();

      // FP64 sweeps on W and V where the refinement leaves pairs open (columns at the block's round-off:
      // rank-deficient blocks), four pairs a warp
      if (sweep)
      {
        const int eighth = lane >> 3, part = lane & 7, players = k + (k & 1);
        int left = kMaxSweeps;
        for (bool more = true; more && left > 0; --left)
        {
          bool open = false;
          for (int round = 0; round + 1 < players; ++round)
          {
            for (int first = (rank * warps + warp) * 4; first < players / 2; first += ranks * warps * 4)
            {
              const bool live = first + eighth < players / 2;
              int cp = 0, cq = k;
              if (live) circle_pair(round, first + eighth, players, cp, cq);
              const bool pair = live && cq < k;
              double2 *wp = wg + static_cast<int64_t>(cp) * k, *wq = wg + static_cast<int64_t>(pair ? cq : cp) * k;
              double alpha = 0.0, beta = 0.0, re = 0.0, im = 0.0;
              for (int i = part; i < k; i += 8)
              {
                const double2 x = load2(wp + i), y = load2(wq + i);
                alpha = fma(x.x, x.x, fma(x.y, x.y, alpha));
                beta = fma(y.x, y.x, fma(y.y, y.y, beta));
                re = fma(x.x, y.x, fma(x.y, y.y, re));
                im = fma(x.x, y.y, fma(-x.y, y.x, im));
              }
#pragma unroll
              for (int o = 4; o > 0; o >>= 1)
              {
                alpha += __shfl_xor_sync(0xffffffffu, alpha, o);
                beta += __shfl_xor_sync(0xffffffffu, beta, o);
                re += __shfl_xor_sync(0xffffffffu, re, o);
                im += __shfl_xor_sync(0xffffffffu, im, o);
              }
              const double size = sqrt(fma(re, re, im * im)), norms = sqrt(alpha) * sqrt(beta);
              if (!pair || !(size > tol * norms)) continue;
              open = open || size > 4.0 * tol * norms;
              const double zeta = (beta - alpha) / (2.0 * size);
              const double t = fabs(zeta) > 1e150 ? 0.5 / zeta : copysign(1.0 / (fabs(zeta) + sqrt(fma(zeta, zeta, 1.0))), zeta);
              const double c = 1.0 / sqrt(fma(t, t, 1.0)), sn = c * t, fr = re / size, fi = im / size;
              const auto turn = [&](double2 *pp, double2 *pq) {
                for (int i = part; i < k; i += 8)
                {
                  const double2 x = load2(pp + i), y0 = load2(pq + i);
                  const double2 y = make_double2(fma(fr, y0.x, fi * y0.y), fma(fr, y0.y, -fi * y0.x));
                  pp[i] = make_double2(fma(c, x.x, -sn * y.x), fma(c, x.y, -sn * y.y));
                  pq[i] = make_double2(fma(sn, x.x, c * y.x), fma(sn, x.y, c * y.y));
                }
              };
              turn(wp, wq);
              turn(v_cur + static_cast<int64_t>(cp) * k, v_cur + static_cast<int64_t>(cq) * k);
            }
            cluster.sync();
          }
          open = __syncthreads_or(open);
          if (threadIdx.x == 0) flags[2] = open;
          cluster.sync();
          more = false;
          for (int o = 0; o < ranks; ++o) more = more || cluster.map_shared_rank(flags, o)[2];
          cluster.sync();
        }
        refined = left > 0;
        taken = kMaxSweeps - left;
      }
      // the values and their order, then the factors: U_x = W / sigma and L = Q V
      bool zero = false;
      for (int j = warp; j < k; j += warps)
      {
        double sum = 0.0;
        for (int i = lane; i < k; i += 32)
        {
          const double2 x = load2(wg + static_cast<int64_t>(j) * k + i);
          sum = fma(x.x, x.x, fma(x.y, x.y, sum));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) lambda[j] = sqrt(sum);
        if (sum == 0.0) zero = true;  // no direction, and none needed where the value is not kept
        else if (!(sum >= kLeastSquare && sum < INFINITY)) refined = false;
      }
      refined = __syncthreads_and(refined);
      zero = __syncthreads_or(zero);
      for (int j = threadIdx.x; j < k; j += blockDim.x)
      {
        int above = 0;
        const double sj = lambda[j];
        for (int i = 0; i < k; ++i) above += (lambda[i] > sj || (lambda[i] == sj && i < j)) ? 1 : 0;
        rank_of[j] = above;
        if (rank == 0) s[e.s_off + above] = sj * ldexp(1.0, shift);
      }
      __syncthreads();
      for (int i = rank * blockDim.x + threadIdx.x; i < k * k; i += ranks * blockDim.x)
      {
        const int j = i / k, row = i - j * k, to = order[row];
        const double2 x = load2(wg + i);
        const double sj = lambda[j];
        const double2 ux = sj > 0.0 ? make_double2(x.x / sj, x.y / sj) : make_double2(0.0, 0.0);
        if (wide) u[e.u_off + static_cast<int64_t>(to) * k + rank_of[j]] = ux;
        else vh[e.vh_off + static_cast<int64_t>(rank_of[j]) * k + to] = conj2(ux);
      }
      const int high = (len + kTile - 1) / kTile;
      const double2 *vc = v_cur;
      for (int tile = rank; tile < high * tiles; tile += ranks)
      {
        const int tr = tile / tiles, tc = tile % tiles;
        product<double2>(
          k, [&](int x, int i) { return tr * kTile + i < len ? load2(q + static_cast<int64_t>(tr * kTile + i) * k + x) : make_double2(0.0, 0.0); }, true,
          [&](int x, int j) { return tc * kTile + j < k ? load2(vc + static_cast<int64_t>(tc * kTile + j) * k + x) : make_double2(0.0, 0.0); }, true, stage,
          [&](int i, int j, double2 sum) {
            const int row = tr * kTile + i, c = tc * kTile + j;
            if (row >= len || c >= k) return;
            if (wide) vh[e.vh_off + static_cast<int64_t>(rank_of[c]) * len + row] = conj2(sum);
            else u[e.u_off + static_cast<int64_t>(row) * k + rank_of[c]] = sum;
          });
      }
      if (threadIdx.x == 0 && rank == 0) info[block] = !refined ? -1 : zero ? -2 : taken;
      // no CTA leaves while another may still read its shared memory
      cluster.sync();
    }

    // svd.cu KeepEntry / keep_kernel with complex factors (the values stay real until they are written)
    struct Kept
    {
      int64_t u_off, s_off, vh_off, first_off, second_off, values_off;
      int32_t rows, cols, k, kept, first_ld, column, row, absorb;
    };
    __global__ void complex_keep_kernel(const Kept *__restrict__ table, const double2 *__restrict__ u, const double *__restrict__ s,
                                        const double2 *__restrict__ vh, double2 *__restrict__ first, double2 *__restrict__ second,
                                        double2 *__restrict__ values)
    {
      const Kept e = table[blockIdx.x];
      const double *sv = s + e.s_off;
      if (blockIdx.y == 0 && threadIdx.x == 0)  // the pads after blocks of odd size
      {
        const int64_t one = static_cast<int64_t>(e.rows) * e.first_ld, two = static_cast<int64_t>(e.first_ld) * e.cols;
        if (e.column == 0 && (one & 1)) first[e.first_off + one] = make_double2(0.0, 0.0);
        if (e.row == 0 && (two & 1)) second[e.second_off + two] = make_double2(0.0, 0.0);
      }
      const int32_t at = static_cast<int32_t>(blockIdx.y * blockDim.x + threadIdx.x), step = static_cast<int32_t>(gridDim.y * blockDim.x);
      const auto by = [](double2 x, double f) { return make_double2(x.x * f, x.y * f); };
      for (int32_t i = at; i < e.rows * e.kept; i += step)
      {
        const int32_t r = i / e.kept, j = i - r * e.kept;
        double2 x = u[e.u_off + static_cast<int64_t>(r) * e.k + j];
        if (e.absorb == 1) x = by(x, sv[j]);
        else if (e.absorb == 3) x = by(x, sqrt(sv[j]));
        first[e.first_off + static_cast<int64_t>(r) * e.first_ld + e.column + j] = x;
      }
      for (int32_t i = at; i < e.kept * e.cols; i += step)
      {
        const int32_t j = i / e.cols, c = i - j * e.cols;
        double2 x = vh[e.vh_off + static_cast<int64_t>(j) * e.cols + c];
        if (e.absorb == 2) x = by(x, sv[j]);
        else if (e.absorb == 3) x = by(x, sqrt(sv[j]));
        second[e.second_off + (e.row + j) * static_cast<int64_t>(e.cols) + c] = x;
      }
      for (int32_t j = at; j < e.kept; j += step) values[e.values_off + j] = make_double2(sv[j], 0.0);
    }

    int64_t dynamic_bytes(int64_t k, int64_t ranks)
    {
      const int64_t sweepers = k <= kOneSweeper ? 1 : ranks, ld = (k + 31) / 32 * 32, mine = ((k + 7) / 8 * 2 + sweepers - 1) / sweepers;
      return (2 * mine * 4 * ld + 64 * (kThreads / 32)) * 8;
    }
  } // namespace

  bool complex_svd_takes(int64_t rows, int64_t cols) { return std::min(rows, cols) <= kMaxCols && std::max(rows, cols) < (1 << 24); }

  int64_t complex_svd_workspace(int64_t rows, int64_t cols)
  {
    const int64_t len = std::max(rows, cols), k = std::min(rows, cols);
    return layout_of(len, k).total;
  }

  cudaError_t complex_svd_keep(int32_t count, const void *table, const void *u, const double *s, const void *vh, void *first,
                               void *second, void *values, cudaStream_t stream)
  {
    if (count <= 0) return cudaSuccess;
    complex_keep_kernel<<<dim3(static_cast<unsigned>(count), 8), 256, 0, stream>>>(
      static_cast<const Kept *>(table), static_cast<const double2 *>(u), s, static_cast<const double2 *>(vh),
      static_cast<double2 *>(first), static_cast<double2 *>(second), static_cast<double2 *>(values));
    return cudaGetLastError();
  }

  // The table of the blocks' QR factorisations (qr.cu): matrix, Q, R and workspace places, then len, columns and
  // the strides.
  void complex_svd_qr_entry(int64_t rows, int64_t cols, int64_t ws_off, int64_t *entry)
  {
    const int64_t len = std::max(rows, cols), k = std::min(rows, cols);
    const Places l = layout_of(len, k);
    const auto pack = [](int64_t a, int64_t b) { return a | b << 32; };
    entry[0] = ws_off + l.b;
    entry[1] = ws_off + l.q;
    entry[2] = ws_off + l.r;
    entry[3] = ws_off + l.qr;
    entry[4] = pack(len, k);
    entry[5] = pack(k, 1);
    entry[6] = pack(k, 1);
    entry[7] = pack(k, 1);
  }

  cudaError_t complex_svd_blocks(int32_t count, int64_t largest, int32_t qr_ranks, const void *table, const void *qr_table, const void *a,
                                 void *u, double *s, void *vh, void *workspace, int32_t *info, cudaStream_t stream)
  {
    if (count <= 0) return cudaSuccess;
    static std::once_flag once;
    static cudaError_t configured = cudaSuccess;
    static int most = 1;
    std::call_once(once, [] {
      configured = cudaFuncSetAttribute(complex_jacobi_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kDynamic));
      if (configured == cudaSuccess)
        configured = cudaFuncSetAttribute(complex_jacobi_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      for (int size = 2; size <= 16 && configured == cudaSuccess; size *= 2)
      {
        cudaLaunchConfig_t config = {};
        cudaLaunchAttribute attribute[1];
        attribute[0].id = cudaLaunchAttributeClusterDimension;
        attribute[0].val.clusterDim.x = static_cast<unsigned>(size);
        attribute[0].val.clusterDim.y = attribute[0].val.clusterDim.z = 1;
        config.gridDim = dim3(static_cast<unsigned>(size));
        config.blockDim = dim3(kThreads);
        config.dynamicSmemBytes = kDynamic;
        config.attrs = attribute;
        config.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, complex_jacobi_kernel, &config) != cudaSuccess || clusters < 1)
        {
          cudaGetLastError();
          break;
        }
        most = size;
      }
    });
    if (configured != cudaSuccess) return configured;
    int ranks = std::min(most, largest >= 96 ? 16 : largest >= 12 ? 8 : 1);  // one 16 x 16 tile or less needs no cluster
    while (ranks < most && dynamic_bytes(largest, ranks) > kDynamic) ranks *= 2;
    if (dynamic_bytes(largest, ranks) > kDynamic) return cudaErrorInvalidValue;
    const auto *entries = static_cast<const Entry *>(table);
    auto *ws = static_cast<double2 *>(workspace);
    cudaError_t e = launch_dependent(sort_kernel, static_cast<unsigned>(count), 256, 0, stream, entries, static_cast<const double2 *>(a), ws);
    if (e != cudaSuccess) return e;
    if ((e = qr_blocks(count, qr_ranks, qr_table, ws, ws, ws, ws, true, stream)) != cudaSuccess) return e;
    cudaLaunchConfig_t config = {};
    cudaLaunchAttribute attribute[2];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = static_cast<unsigned>(ranks);
    attribute[0].val.clusterDim.y = attribute[0].val.clusterDim.z = 1;
    attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[1].val.programmaticStreamSerializationAllowed = 1;
    config.gridDim = dim3(static_cast<unsigned>(count) * static_cast<unsigned>(ranks));
    config.blockDim = dim3(kThreads);
    config.dynamicSmemBytes = kDynamic;
    config.stream = stream;
    config.attrs = attribute;
    config.numAttrs = 2;
    return cudaLaunchKernelEx(&config, complex_jacobi_kernel, entries, static_cast<double2 *>(u), s, static_cast<double2 *>(vh), ws, info);
  }
} // namespace ttg

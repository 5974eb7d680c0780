// Thin QR factorisations of the blocks of a tensor in one launch, for moving the orthogonality centre of
// a matrix product state (tentorch/linalg/graded/svd.cpp:203-257, which calls at::linalg_qr once per
// block): Householder reflections in the working precision, with LAPACK's signs (R_jj = beta of dlarfg /
// zlarfg), float64 and complex128.
//
// A thread-block cluster per block, its columns dealt to the ranks in turn and held in shared memory.  A
// step is one cluster barrier: the rank that owns column j has made its reflector and pushed it into
// every rank's shared memory; each rank applies it to its columns right of j, and the warp that
// holds column j + 1 does that column first and makes the next reflector at once.  The chain of a dot
// product, an update, a norm and the scalars bounds a step, and FP64 issue (a warp instruction takes 64
// clocks on a quarter of an SM here): column j + 1 has warp 0 and its quarter to itself, the other columns
// go four to a warp, eight lanes each, on the other quarters, so that four dot products share their
// three shuffled additions.  Q is formed from the unit vectors by the reflectors, the last first, each
// rank its columns.  A block is scaled by a power of two first, so that no square overflows, and a column
// whose squares underflow all the same by one of its own (reflector.cuh).
//
// The site of bond 256 (18 blocks, the largest 92 x 46): 238 us for the whole call, 4661 us with one cuSOLVER
// factorisation per block.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <mutex>

#include "executor.h"
#include "launch.h"
#include "reflector.cuh"

namespace ttg
{
  namespace
  {
    namespace cg = cooperative_groups;

    constexpr int kQrThreads = 512;
    constexpr int64_t kQrSmem = 220 * 1024;
    // Blocks are scaled down no further than to 2^400: the squares do not overflow, and columns far below the
    // largest entry stay in the normal range.
    constexpr int kQrLargest = 400;
    constexpr int kQrBatch = 16;  // reflectors staged at a time while Q is formed

    // Entry (i, j) of the len x columns matrix, entry (i, c) of Q and entry (c, j) of R in their arenas, and
    // the block's part of the workspace, in elements.
    struct QrEntry
    {
      int64_t a, q, r, ws;
      int32_t len, columns;
      int32_t a_row, a_col, q_row, q_col, r_row, r_col;
    };

    // elements of shared memory a rank needs: its columns and two reflectors, or its columns of Q and a
    // batch of reflectors with their scalars
    int64_t qr_elements(int64_t len, int64_t columns, int64_t ranks)
    {
      return ((columns + ranks - 1) / ranks + kQrBatch) * len + kQrBatch;
    }

    __device__ __forceinline__ double zero_of(double) { return 0.0; }
    __device__ __forceinline__ double2 zero_of(double2) { return make_double2(0.0, 0.0); }
    __device__ __forceinline__ double one_of(double) { return 1.0; }
    __device__ __forceinline__ double2 one_of(double2) { return make_double2(1.0, 0.0); }
    // conj(a) b + c
    __device__ __forceinline__ double dot_add(double a, double b, double c) { return fma(a, b, c); }
    __device__ __forceinline__ double2 dot_add(double2 a, double2 b, double2 c)
    {
      return make_double2(fma(a.x, b.x, fma(a.y, b.y, c.x)), fma(a.x, b.y, fma(-a.y, b.x, c.y)));
    }
    // c - w a
    __device__ __forceinline__ double minus(double c, double w, double a) { return fma(-w, a, c); }
    __device__ __forceinline__ double2 minus(double2 c, double2 w, double2 a)
    {
      return make_double2(fma(-w.x, a.x, fma(w.y, a.y, c.x)), fma(-w.x, a.y, fma(-w.y, a.x, c.y)));
    }
    __device__ __forceinline__ double times(double a, double b) { return a * b; }
    __device__ __forceinline__ double2 times(double2 a, double2 b)
    {
      return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
    }
    __device__ __forceinline__ double conj_of(double a) { return a; }
    __device__ __forceinline__ double2 conj_of(double2 a) { return make_double2(a.x, -a.y); }
    __device__ __forceinline__ double plus(double a, double b) { return a + b; }
    __device__ __forceinline__ double2 plus(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
    __device__ __forceinline__ bool is_zero(double a) { return a == 0.0; }
    __device__ __forceinline__ bool is_zero(double2 a) { return a.x == 0.0 && a.y == 0.0; }
    __device__ __forceinline__ double load_l2(const double *p) { return __ldcg(p); }
    __device__ __forceinline__ double2 load_l2(const double2 *p) { return __ldcg(p); }

    template <typename T>
    __global__ void __launch_bounds__(kQrThreads, 1)
      qr_kernel(const QrEntry *__restrict__ table, const T *__restrict__ a, T *__restrict__ q, T *__restrict__ r, T *__restrict__ workspace)
    {
      extern __shared__ __align__(16) unsigned char dynamic[];
      __shared__ T taus[2];
      __shared__ double big, bigs[kQrThreads / 32];
      const cg::cluster_group cluster = cg::this_cluster();
      const int ranks = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
      dependent_entry();
      const QrEntry e = table[blockIdx.x / ranks];
      const int len = e.len, columns = e.columns, k = min(len, columns);
      const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
      const int mine = (columns + ranks - 1) / ranks;
      T *own = reinterpret_cast<T *>(dynamic), *vst = own + static_cast<int64_t>(mine) * len;
      T *qf = workspace + e.ws, *qtau = qf + static_cast<int64_t>(k) * len;  // the reflectors and their scalars
      const auto colp = [&](int c) -> T * { return own + static_cast<int64_t>(c / ranks) * len; };

      // this rank's columns, and the power of two that brings the block's largest entry to at most 2^kQrLargest, a
      // block below one up to it
      double most = 0.0;
      for (int c = rank; c < columns; c += ranks)
        for (int i = threadIdx.x; i < len; i += blockDim.x)
        {
          const T x = a[e.a + static_cast<int64_t>(i) * e.a_row + static_cast<int64_t>(c) * e.a_col];
          colp(c)[i] = x;
          most = fmax(most, largest(x));
        }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) most = fmax(most, __shfl_xor_sync(0xffffffffu, most, o));
      if (lane == 0) bigs[warp] = most;
      __syncthreads();
      if (threadIdx.x == 0)
      {
        for (int w = 1; w < warps; ++w) most = fmax(most, bigs[w]);
        big = most;
      }
      cluster.sync();
      for (int o = 0; o < ranks; ++o) most = fmax(o == 0 ? 0.0 : most, *cluster.map_shared_rank(&big, o));
      int shift = 0;
      if (most > 0.0 && most < 1.7976931348623157e308) frexp(most, &shift);
      if (shift > 0) shift = max(shift - kQrLargest, 0);
      const double down = ldexp(1.0, -shift / 2), down2 = ldexp(1.0, -(shift - shift / 2));  // each in range
      for (int64_t i = threadIdx.x; i < static_cast<int64_t>(mine) * len; i += blockDim.x) own[i] = scaled_by(scaled_by(own[i], down), down2);
      cluster.sync();  // every rank has read the others' maxima

      // column j's reflector by one warp, xn the squared norm below its diagonal
      const auto reflect = [&](int j, double xn) {
        T *col = colp(j);
        T beta, tau, scale;
        column_reflector(col, j, len, xn, beta, tau, scale);
        __syncwarp();
        T *slot = vst + static_cast<int64_t>(j & 1) * len;
        for (int i = j + 1 + lane; !is_zero(tau) && i < len; i += 32)
        {
          const T x = times(col[i], scale);
          qf[static_cast<int64_t>(j) * len + i] = x;
          for (int o = 0; o < ranks; ++o) cluster.map_shared_rank(slot, o)[i] = x;
        }
        if (lane == 0)
        {
          col[j] = beta;
          qtau[j] = tau;
          for (int o = 0; o < ranks; ++o) cluster.map_shared_rank(taus, o)[j & 1] = tau;
        }
      };
      if (rank == 0 && warp == 0 && k > 0)
      {
        const T *col = colp(0);
        double xn = 0.0;
        for (int i = 1 + lane; i < len; i += 32) xn = square(col[i], xn);
        reflect(0, lanes_sum<32>(xn));
      }
      for (int j = 0; j < k; ++j)
      {
        cluster.sync();
        const T *v = vst + static_cast<int64_t>(j & 1) * len;
        const T tau = conj_of(taus[j & 1]);  // H^H is applied
        const int first = (j + ranks - rank) / ranks;  // the first local column right of j
        const bool next = (j + 1) % ranks == rank;     // it is column j + 1
        if (warp == 0)
        {
          if (next && j + 1 < columns)
          {
            T *fc = colp(j + 1);
            double xn = 0.0;
            if (!is_zero(tau))
            {
              T dot = zero_of(tau);
              for (int i = j + 1 + lane; i < len; i += 32) dot = dot_add(v[i], fc[i], dot);
              dot = lanes_sum<32>(dot);
              const T w = times(tau, plus(fc[j], dot));
              for (int i = j + 1 + lane; i < len; i += 32)
              {
                const T x = minus(fc[i], w, v[i]);
                fc[i] = x;
                if (i > j + 1) xn = square(x, xn);
              }
              __syncwarp();
              if (lane == 0) fc[j] = minus(fc[j], w, one_of(w));
            }
            else
              for (int i = j + 2 + lane; i < len; i += 32) xn = square(fc[i], xn);
            __syncwarp();
            if (j + 1 < k) reflect(j + 1, lanes_sum<32>(xn));
          }
        }
        else if ((warp & 3) != 0 && !is_zero(tau))
        {
          const int slot = (warp >> 2) * 3 + (warp & 3) - 1, lanes = lane & 7;
          for (int l0 = first + (next ? 1 : 0) + slot * 4; l0 * ranks + rank < columns; l0 += (warps >> 2) * 12)
          {
            const int c = (l0 + (lane >> 3)) * ranks + rank;
            const bool live = c < columns;
            T *fc = colp(live ? c : l0 * ranks + rank), dot = zero_of(tau);
            for (int i = j + 1 + lanes; i < len; i += 8) dot = dot_add(v[i], fc[i], dot);
            dot = lanes_sum<8>(dot);
            const T head = fc[j], w = times(tau, plus(head, dot));
            __syncwarp();
            if (!live) continue;
            for (int i = j + 1 + lanes; i < len; i += 8) fc[i] = minus(fc[i], w, v[i]);
            if (lanes == 0) fc[j] = minus(head, w, one_of(w));
          }
        }
      }
      cluster.sync();

      // R: this rank's columns down to the diagonal, zeros below, at the block's scale
      const double up = ldexp(1.0, shift / 2), up2 = ldexp(1.0, shift - shift / 2);
      for (int64_t i = threadIdx.x; i < static_cast<int64_t>(mine) * k; i += blockDim.x)
      {
        const int l = static_cast<int>(i / k), c = l * ranks + rank, row = static_cast<int>(i - static_cast<int64_t>(l) * k);
        if (c >= columns) continue;
        const T x = row <= c ? scaled_by(scaled_by(own[static_cast<int64_t>(l) * len + row], up), up2) : zero_of(own[0]);
        r[e.r + static_cast<int64_t>(row) * e.r_row + static_cast<int64_t>(c) * e.r_col] = x;
      }
      __syncthreads();
      // Q: unit vector c through the reflectors c down to 0
      const int cols_q = (k + ranks - 1) / ranks;
      T *stage = own + static_cast<int64_t>(cols_q) * len, *stau = stage + static_cast<int64_t>(kQrBatch) * len;
      for (int64_t i = threadIdx.x; i < static_cast<int64_t>(cols_q) * len; i += blockDim.x)
      {
        const int l = static_cast<int>(i / len), c = l * ranks + rank;
        own[i] = static_cast<int>(i - static_cast<int64_t>(l) * len) == c ? one_of(own[0]) : zero_of(own[0]);
      }
      for (int top = k - 1; top >= 0; top -= kQrBatch)
      {
        const int low = max(top - kQrBatch + 1, 0);
        __syncthreads();
        for (int64_t i = threadIdx.x; i < static_cast<int64_t>(top - low + 1) * len; i += blockDim.x)
        {
          const int t = top - static_cast<int>(i / len), row = static_cast<int>(i % len);
          if (row > t) stage[i] = load_l2(qf + static_cast<int64_t>(t) * len + row);
        }
        if (threadIdx.x < top - low + 1) stau[threadIdx.x] = load_l2(qtau + top - threadIdx.x);
        __syncthreads();
        const int lanes = lane & 7;
        for (int l0 = warp * 4; l0 * ranks + rank < k; l0 += warps * 4)
        {
          const int c = (l0 + (lane >> 3)) * ranks + rank;
          const bool live = c < k;
          T *bc = colp(live ? c : l0 * ranks + rank);
          for (int t = top; t >= low; --t)
          {
            const T tau = stau[top - t];
            if (is_zero(tau)) continue;
            const T *vt = stage + static_cast<int64_t>(top - t) * len;
            T dot = zero_of(tau);
            for (int i = t + 1 + lanes; i < len; i += 8) dot = dot_add(vt[i], bc[i], dot);
            dot = lanes_sum<8>(dot);
            const T head = bc[t], w = times(tau, plus(head, dot));
            __syncwarp();
            if (live && t <= c)
            {
              for (int i = t + 1 + lanes; i < len; i += 8) bc[i] = minus(bc[i], w, vt[i]);
              if (lanes == 0) bc[t] = minus(head, w, one_of(w));
            }
            __syncwarp();
          }
        }
      }
      __syncthreads();
      for (int64_t i = threadIdx.x; i < static_cast<int64_t>(cols_q) * len; i += blockDim.x)
      {
        const int l = static_cast<int>(i / len), c = l * ranks + rank, row = static_cast<int>(i - static_cast<int64_t>(l) * len);
        if (c < k) q[e.q + static_cast<int64_t>(row) * e.q_row + static_cast<int64_t>(c) * e.q_col] = own[i];
      }
      // no CTA leaves while another may still write its shared memory
      cluster.sync();
    }

    // The cluster for a launch: the fewest ranks that hold every block's columns, at least 8 from 16
    // columns on (one CTA below that) and 16 from 96, as far as the GPU can hold such clusters.  (Columns, of wide
    // blocks too: 5 x 3000 takes 103 us with 16 CTAs, 885 with one.)
    template <typename T>
    int qr_ranks(int32_t count, const int64_t *shapes)
    {
      static std::once_flag once;
      static int most = 1;
      std::call_once(once, [] {
        if (cudaFuncSetAttribute(qr_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kQrSmem)) != cudaSuccess ||
            cudaFuncSetAttribute(qr_kernel<T>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
        {
          cudaGetLastError();
          return;
        }
        for (int size = 2; size <= 16; size *= 2)
        {
          cudaLaunchConfig_t config = {};
          cudaLaunchAttribute attribute[1];
          attribute[0].id = cudaLaunchAttributeClusterDimension;
          attribute[0].val.clusterDim.x = static_cast<unsigned>(size);
          attribute[0].val.clusterDim.y = attribute[0].val.clusterDim.z = 1;
          config.gridDim = dim3(static_cast<unsigned>(size));
          config.blockDim = dim3(kQrThreads);
          config.dynamicSmemBytes = kQrSmem;
          config.attrs = attribute;
          config.numAttrs = 1;
          int clusters = 0;
          if (cudaOccupancyMaxActiveClusters(&clusters, qr_kernel<T>, &config) != cudaSuccess || clusters < 1)
          {
            cudaGetLastError();
            break;
          }
          most = size;
        }
      });
      int64_t widest = 0;
      for (int32_t i = 0; i < count; ++i) widest = std::max(widest, shapes[2 * i + 1]);
      const auto fits = [&](int ranks) {
        for (int32_t i = 0; i < count; ++i)
          if (qr_elements(shapes[2 * i], shapes[2 * i + 1], ranks) * static_cast<int64_t>(sizeof(T)) > kQrSmem) return false;
        return true;
      };
      int ranks = std::min(most, widest >= 96 ? 16 : widest >= 16 ? 8 : 1);
      while (ranks < most && !fits(ranks)) ranks *= 2;
      return fits(ranks) ? ranks : 0;
    }
  } // namespace

  int32_t qr_cluster(int32_t count, const int64_t *shapes, bool complex)
  {
    return complex ? qr_ranks<double2>(count, shapes) : qr_ranks<double>(count, shapes);
  }

  // Whether the blocks together take less time here than one after another in cuSOLVER (us, from blocks of 2 x 1 to
  // 1300 x 80 and 5 x 20000 measured one at a time; both within some 15%).  Here a reflector costs its column's chain,
  // by the length that is left, and the passes of 48 columns over a rank; the blocks run side by side.  One block,
  // here and there: 92 x 46 228 and 816, 300 x 150 1277 and 1986, 450 x 200 2288 and 2629, 600 x 300 4193 and 4095,
  // 1000 x 100 2507 and 1464, 20 x 5000 303 and 365, 5 x 20000 524 and 294; complex 300 x 150 2871 and 3187,
  // 400 x 200 4929 and 4463.
  bool qr_pays(int32_t count, const int64_t *shapes, int32_t ranks, bool complex)
  {
    double longest = 0.0, sum = 0.0, others = 85.0;
    for (int32_t i = 0; i < count; ++i)
    {
      const double len = static_cast<double>(shapes[2 * i]), columns = static_cast<double>(shapes[2 * i + 1]), k = std::min(len, columns);
      const double left = len - k / 2, passes = (columns - k / 2) / (48.0 * ranks), share = k / ranks;
      const double t = complex ? k * (0.065 * left + 4.0 * passes + 0.2 * share + 1.5)
                               : k * (0.0255 * left + 2.1 * passes + 0.12 * share + ranks / 32.0);
      longest = std::max(longest, t);
      sum += t;
      others += complex ? 85.0 + k * (17.5 + 0.018 * k + 0.0045 * (columns - k)) : std::min(215.0, 60.0 + 8.0 * k) + k * (8.3 + 0.014 * k);
    }
    return 30.0 + std::max(longest, sum * ranks / device_sms()) < others;
  }

  int64_t qr_workspace(int64_t len, int64_t columns) { return std::min(len, columns) * (len + 1); }

  cudaError_t qr_blocks(int32_t count, int32_t ranks, const void *table, const void *a, void *q, void *r, void *workspace, bool complex,
                        cudaStream_t stream)
  {
    if (count <= 0) return cudaSuccess;
    cudaLaunchConfig_t config = {};
    cudaLaunchAttribute attribute[2];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = static_cast<unsigned>(ranks);
    attribute[0].val.clusterDim.y = attribute[0].val.clusterDim.z = 1;
    attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[1].val.programmaticStreamSerializationAllowed = 1;
    config.gridDim = dim3(static_cast<unsigned>(count) * static_cast<unsigned>(ranks));
    config.blockDim = dim3(kQrThreads);
    config.dynamicSmemBytes = kQrSmem;
    config.stream = stream;
    config.attrs = attribute;
    config.numAttrs = 2;
    const auto *entries = static_cast<const QrEntry *>(table);
    return complex ? cudaLaunchKernelEx(&config, qr_kernel<double2>, entries, static_cast<const double2 *>(a), static_cast<double2 *>(q),
                                        static_cast<double2 *>(r), static_cast<double2 *>(workspace))
                   : cudaLaunchKernelEx(&config, qr_kernel<double>, entries, static_cast<const double *>(a), static_cast<double *>(q),
                                        static_cast<double *>(r), static_cast<double *>(workspace));
  }
} // namespace ttg

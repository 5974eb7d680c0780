// Split-precision block products on the 5th-generation tensor cores (tcgen05).  The numerical scheme
// is the one of gemm.h (Ozaki's error-free splitting: every row of A and column of B cut into S exact
// 7-bit bf16 slices by the slicing pass); this is where the slice products run.
//
//   - A CTA (one per SM) owns 128 x N output tiles, N = 64 or 32, over a range of K.  Warps have
//     roles: one thread copies, one issues the products, eight warps read the sums back.
//   - The slicing pass leaves every slice of a tile over 32 of K as one contiguous piece in the
//     core-matrix layout the products read (8 rows x 16 bytes, K-major, no swizzle; SplitPair), so a
//     stage is 2 S bulk copies (cp.async.bulk) that signal the stage's mbarrier, in a ring of as
//     many stages as fit in shared memory.
//   - The sums of level l = t + u sit in tensor memory at columns l N .. l N + N - 1, and the slices of
//     B follow one another in a stage, so that slice t of A times ALL the slices u < S - t of B is one
//     product of N (S - t) columns landing in levels t .. S - 1: eight tcgen05.mma of up to 256 columns
//     a 16 of K (S = 6) instead of 21 of 64, each reading A from shared memory once.  With 64 columns
//     a product is bound by shared memory (6 KB in 32 clocks), with 256 by the tensor cores.
//   - Every 512 of K (gemm.h kExactChunk) the level sums, exact integers, are read back and folded:
//     the four leading levels as an int64 sum_l lev_l 2^(7 (3 - l)), the rest through one fp32 sum.
//   - FP64 runs at 2 multiply-adds a clock and SM here, 64 times slower than integers: an FP64
//     combination per entry would take longer than the products of a tile of K below 1000.  A tile's
//     value is therefore kept as a fixed-point int64 (head 2^7 + tail with up to 8 more bits) and
//     becomes a double by shifting, with one rounding; the partial tiles of a K that several CTAs
//     share add as integers, exactly, in any order.  Blocks of several pairs (their scales differ),
//     S above 6 and K beyond 2^16 combine in FP64.
// Measured on the SU(2) recoupling of bond 8 x 9 spins (85.9 GFLOP, S = 6: 1.80 PFLOP of slice products)
// 1.16 ms, 1.55 PFLOP/s, 0.78 of the measured bf16 peak; as 21 products of 64 columns staged by cp.async
// from slices a row apart it took 5.99 ms.  The matvec of bond 1001 (both products and their
// slicing) takes 142 us, 425 on mma.sync.
// The roles pass stages, level sums and free tensor memory through mbarriers.  Every wait gives up
// after two seconds or once another has.  The entries whose sums did not come then become NaN: a warp that
// gave up goes on through its CTA's items without waiting, so that every barrier is met and every ticket
// taken (a lost part says so in its ticket, and the whole tile becomes NaN), and the ticket region is left zero.
// On every path out the copies and products in flight are waited for (again with a limit) and the tensor
// memory is freed.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <vector>

#include "executor.h"
#include "gemm.h"
#include "gemm_device.cuh"
#include "launch.h"

namespace ttg
{
  namespace
  {
    constexpr int kTcM = kSliceTileA, kTcK = 32;  // rows of a tile, K per stage
    constexpr int kTcChunkSteps = kExactChunk / kTcK;  // stages between readings of the level sums
    // core-matrix layout of one slice in a stage: 16 bytes per (row, 8 of K); the 4 groups of 8 of K
    // of a row group follow one another (LBO), row groups after them (SBO)
    constexpr int kTcLbo = 128, kTcSbo = kSliceGroup * 2;
    constexpr int kTcSmem = 216 * 1024;
    constexpr int kTcFixedSlices = 6;  // the most slices whose sums the fixed-point values hold
    constexpr int32_t kTcFixedK = 1 << 16;
    constexpr unsigned long long kTcWaitNs = 2000000000ull;

    // 32 columns: sixteen warps read the sums back, eight columns a thread, so that the latency of a small
    // tile's end is short.  64 columns: eight, 32 columns a thread, in two warpgroups of 216 registers;
    // launched with 168 a thread (3 x 128 x 168 of the SM's 65536), the third warpgroup (the copying
    // and the issuing warp) keeps 56: 2 x 216 + 56 = 488 of the 504 they came with.
    template <int S, int N>
    struct TcShape
    {
      static constexpr int slice_a = kTcM * kTcK * 2, slice_b = N * kTcK * 2;  // bytes
      static constexpr int stage = S * (slice_a + slice_b);
      static constexpr int stages = kTcSmem / stage < 6 ? kTcSmem / stage : 6;
      // more than half of the SM's, so that a second CTA never shares it (each holds all 512 columns of
      // its tensor memory)
      static constexpr int bytes = stages * stage > 120 * 1024 ? stages * stage : 120 * 1024;
      static constexpr int warps = N == 32 ? 16 : 8;      // that read the sums back
      static constexpr int cols = N / (warps / 4);        // columns of a tile a thread reads back
      static constexpr int threads = (warps + 4) * 32;
    };

    struct TcArgs
    {
      const uint16_t *sa, *sb;  // slices of A rows and of B columns (SplitPair's layout)
      const int16_t *exps_a, *exps_b;
      double *c;
      const int32_t *relabel;   // per entry of C its place after the leg move that follows, or null
      const DevSplitPair *spairs;
      const TcItem *items;
      const GemmReduce *reduces;
      int32_t longest;
      double *partial;
      int *tickets;
    };
    constexpr int kTcLost = 1 << 16;  // in a ticket: a part of the tile was lost (a tile has fewer parts, at most one a CTA and one)

    __device__ __forceinline__ uint32_t smem_addr(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

    __device__ __forceinline__ uint64_t tc_desc(uint32_t addr)
    {
      // start address, leading (K) and stride (row group) byte offsets in 16-byte units, version 1,
      // base offset 0, no swizzle
      return static_cast<uint64_t>((addr >> 4) & 0x3FFF) | (static_cast<uint64_t>((kTcLbo >> 4) & 0x3FFF) << 16) |
             (static_cast<uint64_t>((kTcSbo >> 4) & 0x3FFF) << 32) | (static_cast<uint64_t>(1) << 46);
    }

    // kind::f16 instruction descriptor: D fp32, A and B bf16, both K-major, N >> 3 at bit 17, M >> 4
    // at bit 24
    __host__ __device__ constexpr uint32_t tc_instr(int n)
    {
      return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(kTcM >> 4) << 24);
    }

    __device__ __forceinline__ void tc_mma(uint32_t tmem, uint64_t a, uint64_t b, uint32_t instr, uint32_t accumulate)
    {
      asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                   "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
                   "l"(a), "l"(b), "r"(instr), "r"(accumulate)
                   : "memory");
    }
    __device__ __forceinline__ void tc_commit(uint64_t *bar)
    {
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
    }
    __device__ __forceinline__ void bar_init(uint64_t *bar, int count)
    {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
    }
    __device__ __forceinline__ void bar_arrive(uint64_t *bar)
    {
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
    }
    __device__ __forceinline__ void bar_expect(uint64_t *bar, uint32_t bytes)
    {
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
    }
    // bytes (a multiple of 16) of global memory into shared memory, counted on `bar` as they land
    __device__ __forceinline__ void bulk_copy(uint32_t dst, const void *src, uint32_t bytes, uint64_t *bar)
    {
      asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
                   "r"(bytes), "r"(smem_addr(bar))
                   : "memory");
    }

    __device__ __forceinline__ unsigned long long tc_now()
    {
      unsigned long long t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      return t;
    }

    // whether the phase with parity `parity` of the mbarrier at `at` is over, looked at for a while by the hardware
    __device__ __forceinline__ bool tc_try(uint32_t at, uint32_t parity)
    {
      uint32_t done;
      asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                   : "=r"(done)
                   : "r"(at), "r"(parity)
                   : "memory");
      return done != 0;
    }

    // Wait for the phase of `bar` with parity `parity`; false when two seconds passed first, or when
    // another wait of the CTA has given up (`failed`, null to wait regardless).
    __device__ __forceinline__ bool tc_wait(uint64_t *bar, uint32_t parity, volatile int *failed)
    {
      const uint32_t at = smem_addr(bar);
      unsigned long long start = 0;
      while (true)
      {
        if (tc_try(at, parity)) return true;
        const unsigned long long now = tc_now();
        if (start == 0) start = now;
        if ((failed && *failed) || now - start > kTcWaitNs)
        {
          if (failed) *failed = 1;
          return false;
        }
      }
    }

    // The same for a whole warp, whose lanes go on together either way (a vote in the loop costs nothing against its
    // branch; one after it 0.5% of a long product).
    __device__ __forceinline__ bool tc_wait_warp(uint64_t *bar, uint32_t parity, volatile int *failed)
    {
      const uint32_t at = smem_addr(bar);
      unsigned long long start = 0;
      while (true)
      {
        if (__all_sync(0xffffffffu, tc_try(at, parity))) return true;
        const unsigned long long now = tc_now();
        if (start == 0) start = now;
        if (__any_sync(0xffffffffu, *failed || now - start > kTcWaitNs))
        {
          *failed = 1;
          return false;
        }
      }
    }

    // 8 columns of one lane of tensor memory
    __device__ __forceinline__ void tc_load8(uint32_t addr, uint32_t *r)
    {
      asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                   : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                   : "r"(addr));
    }

    // The bits a fixed-point value of a pair keeps below the unit of level 4: 8, fewer from K = 4096 on
    // (a value is at most 2^(42 + bits) K).
    __device__ __forceinline__ int fixed_bits(int k) { return k <= 4096 ? 8 : max(0, 8 - (32 - __clz((k - 1) >> 12))); }

    // v 2^e as a double, rounded once (to nearest, ties to even), when it is in the normal range;
    // `outside` collects whether it was not (fixed_slow then gives it).
    __device__ __forceinline__ double fixed_to_double(long long v, int e, bool &outside)
    {
      const unsigned long long sign = static_cast<unsigned long long>(v) & 0x8000000000000000ull;
      const unsigned long long a = static_cast<unsigned long long>(sign ? -v : v);
      const int lz = min(__clzll(static_cast<long long>(a)), 63), field = 1086 - lz + e;
      const unsigned long long m = a << lz, rest = m & 0x7ffull;
      unsigned long long q = m >> 11;
      q += (rest > 0x400ull || (rest == 0x400ull && (q & 1ull))) ? 1ull : 0ull;
      outside |= v != 0 && (field <= 0 || field >= 2046);
      // q has its leading one at bit 52: added to the exponent field one lower, a carry moves it up
      const unsigned long long bits = ((static_cast<unsigned long long>(field - 1) << 52) + q) | sign;
      return __longlong_as_double(static_cast<long long>(v == 0 ? 0ull : bits));
    }
    __device__ __noinline__ double fixed_slow(long long v, int e) { return ldexp(static_cast<double>(v), e); }

    // The 8 x 8 transpose within each group of eight lanes: lane 8 g + i holds entries 0 .. 7 of row i
    // of its group and takes entry i of rows 0 .. 7, so that a store of eight lanes is 64 contiguous
    // bytes instead of eight places a row apart.
    __device__ __forceinline__ void transpose8(long long *v, int lane)
    {
#pragma unroll
      for (int m = 1; m < 8; m <<= 1)
#pragma unroll
        for (int j = 0; j < 8; ++j)
        {
          if (j & m) continue;
          const bool high = lane & m;
          const long long got = __shfl_xor_sync(0xffffffffu, high ? v[j] : v[j | m], m);
          if (high) v[j] = got;
          else v[j | m] = got;
        }
    }

    // The steps of an item, pair by pair: calls f(pair, lo, hi) for the range of the pair's steps that
    // lies in the item; f returns false to stop.
    struct TcPair
    {
      int64_t sa, sb;
      int32_t ksteps, ea, eb;
    };
    template <typename F>
    __device__ __forceinline__ bool tc_segments(const TcArgs &a, const TcItem &it, F f)
    {
      if (it.pair_count == 0) return true;
      int lo = it.s0, hi = min(it.s1, it.ksteps), base = it.ksteps;
      if (lo < hi && !f(TcPair{it.sa, it.sb, it.ksteps, it.ea, it.eb}, lo, hi)) return false;
      for (int p = 1; p < it.pair_count; ++p)
      {
        const DevSplitPair sp = a.spairs[it.pair_begin + p];
        lo = max(it.s0 - base, 0);
        hi = min(it.s1 - base, sp.ksteps);
        base += sp.ksteps;
        if (lo < hi && !f(TcPair{sp.sa, sp.sb, sp.ksteps, sp.ea, sp.eb}, lo, hi)) return false;
      }
      return true;
    }

    template <int S, int N>
    __global__ void __launch_bounds__(TcShape<S, N>::threads, 1) gemm_split_tc_kernel(const __grid_constant__ TcArgs a)
    {
      using Shape = TcShape<S, N>;
      constexpr int kStages = Shape::stages, kCols = Shape::cols, kWarps = Shape::warps;
      extern __shared__ __align__(1024) unsigned char smem[];
      // a stage holds its copies' bytes; a stage's products are done; the level sums are complete, and
      // their tensor memory free again; every product issued is done
      __shared__ __align__(8) uint64_t full[kStages], empty[kStages], sums_full, sums_free, drained;
      __shared__ uint32_t tmem_base;
      __shared__ int failed_flag, last_flag;
      volatile int *failed = &failed_flag;
      const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
      if (warp == 0)
      {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_addr(&tmem_base)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
      }
      if (tid == 32)
      {
        for (int s = 0; s < kStages; ++s)
        {
          bar_init(&full[s], 1);
          bar_init(&empty[s], 1);
        }
        bar_init(&sums_full, 1);
        bar_init(&sums_free, kWarps);
        bar_init(&drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        failed_flag = 0;
      }
      // this CTA's list; the first item is read, as all above is done, while the kernel before still runs
      const TcItem *list = a.items + static_cast<int64_t>(blockIdx.x) * a.longest;
      TcItem it = list[0];
      __syncthreads();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t tmem = tmem_base;
      const auto next = [&](int &at) {
        if (++at < a.longest) it = list[at];
        else it.m = 0;
      };
      // the results of the kernel before are read, and memory that it may still read written, from here on
      asm volatile("griddepcontrol.wait;\n" ::: "memory");

      if (warp >= kWarps)
      {
        if constexpr (N == 64) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp == kWarps && lane == 0)
        {
          // the slices were written through the generic proxy
          asm volatile("fence.proxy.async;" ::: "memory");
          int stage = 0;
          uint32_t phase = 0;
          int64_t issued = 0;
          bool ok = true;
          for (int at = 0; it.m > 0 && ok; next(at))
          {
            const int groups_a = min(kTcM / 8, (it.m - it.m0 + 7) / 8), groups_b = min(N / 8, (it.n - it.n0 + 7) / 8);
            const uint32_t bytes_a = groups_a * kSliceGroup * 2, bytes_b = groups_b * kSliceGroup * 2;
            ok = tc_segments(a, it, [&](const TcPair &sp, int lo, int hi) {
              for (int step = lo; step < hi; ++step)
              {
                if (!tc_wait(&empty[stage], phase ^ 1u, failed)) return false;
                int32_t stride_a, stride_b;
                const uint16_t *ga = a.sa + slice_place(sp.sa, it.m, sp.ksteps, kSliceTileA, it.m0, step, stride_a);
                const uint16_t *gb = a.sb + slice_place(sp.sb, it.n, sp.ksteps, kSliceTileB, it.n0, step, stride_b);
                const uint32_t to = smem_addr(smem) + stage * Shape::stage;
                bar_expect(&full[stage], S * (bytes_a + bytes_b));
#pragma unroll
                for (int t = 0; t < S; ++t)
                {
                  bulk_copy(to + t * Shape::slice_a, ga + t * stride_a, bytes_a, &full[stage]);
                  bulk_copy(to + S * Shape::slice_a + t * Shape::slice_b, gb + t * stride_b, bytes_b, &full[stage]);
                }
                ++issued;
                if (++stage == kStages)
                {
                  stage = 0;
                  phase ^= 1u;
                }
              }
              return true;
            });
          }
          // no copy may still write this CTA's shared memory when it leaves
          if (!ok)
            for (int64_t i = max(static_cast<int64_t>(0), issued - kStages); i < issued; ++i)
              tc_wait(&full[i % kStages], static_cast<uint32_t>(i / kStages) & 1u, nullptr);
        }
        else if (warp == kWarps + 1 && lane == 0)
        {
          int stage = 0;
          uint32_t phase = 0, sums = 0;
          bool ok = true;
          for (int at = 0; it.m > 0 && ok; next(at))
            ok = tc_segments(a, it, [&](const TcPair &, int lo, int hi) {
              for (int step = lo; step < hi; ++step)
              {
                const bool chunk_first = (step - lo) % kTcChunkSteps == 0;
                if (chunk_first && !tc_wait(&sums_free, sums ^ 1u, failed)) return false;
                if (!tc_wait(&full[stage], phase, failed)) return false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a_base = smem_addr(smem) + stage * Shape::stage, b_base = a_base + S * Shape::slice_a;
#pragma unroll
                for (int kk = 0; kk < kTcK / 16; ++kk)
#pragma unroll
                  for (int t = 0; t < S; ++t)
#pragma unroll
                    for (int c = 0; c < N * (S - t); c += 256)
                    {
                      constexpr int most = 256;
                      const int n = N * (S - t) - c < most ? N * (S - t) - c : most;
                      // slice t = 0 reaches every level: its first product starts the chunk's sums
                      const uint32_t accumulate = (chunk_first && kk == 0 && t == 0) ? 0u : 1u;
                      tc_mma(tmem + static_cast<uint32_t>(t * N + c), tc_desc(a_base + t * Shape::slice_a + kk * 2 * kTcLbo),
                             tc_desc(b_base + (c / 8) * kTcSbo + kk * 2 * kTcLbo), tc_instr(n), accumulate);
                    }
                tc_commit(&empty[stage]);
                if (step + 1 == hi || (step + 1 - lo) % kTcChunkSteps == 0)
                {
                  tc_commit(&sums_full);
                  sums ^= 1u;
                }
                if (++stage == kStages)
                {
                  stage = 0;
                  phase ^= 1u;
                }
              }
              return true;
            });
          // no product may still run when the tensor memory is freed
          if (!ok)
          {
            tc_commit(&drained);
            tc_wait(&drained, 0, nullptr);
          }
        }
      }
      else
      {
        if constexpr (N == 64) asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
        // tensor-memory lanes 32 quarter .. + 31 (the quarter a warp may access), columns kCols part ..
        const int quarter = warp & 3, part = warp >> 2, col0 = kCols * part;
        const uint32_t lane_addr = tmem + (static_cast<uint32_t>(32 * quarter) << 16) + static_cast<uint32_t>(col0);
        const auto epilogue_sync = [] { asm volatile("bar.sync 1, %0;\n" ::"n"(kWarps * 32) : "memory"); };
        uint32_t sums = 0;
        bool ok = true;
        for (int at_item = 0; it.m > 0 && ok; next(at_item))
        {
          const int row = it.m0 + 32 * quarter + lane;
          // where the thread stores: rows top .. top + 7 of one column of each run of eight
          const int top = it.m0 + 32 * quarter + (lane & 24), side = it.n0 + col0 + (lane & 7);
          const auto place_of = [&](int c, int j) -> int64_t {
            return top + j < it.m && side + c < it.n ? it.c + static_cast<int64_t>(top + j) * it.n + side + c : -1;
          };
          // the exponents of the row and of the columns (unconditional reads, so that all are in flight
          // together); a tile's of 32 columns, and the places its entries go to, before the sums are there
          const auto exponents = [&](int32_t ea, int32_t eb, int &re, int (&ce)[kCols]) {
            re = a.exps_a[ea + min(row, it.m - 1)];
#pragma unroll
            for (int j = 0; j < kCols; ++j) ce[j] = a.exps_b[eb + min(it.n0 + col0 + j, it.n - 1)];
          };
          // the tile's values: with one pair its level sums, fixed-point integers or doubles, whose scales are
          // taken last; with several, scaled doubles
          const bool single = it.pair_count == 1, fixed = S <= kTcFixedSlices && single && it.k <= kTcFixedK;
          const int bits = fixed_bits(it.k);
          int row_exp = 0, col_exp[kCols];
          int32_t place[8];
          if constexpr (N == 32)
          {
            if (single) exponents(it.ea, it.eb, row_exp, col_exp);
            if (a.relabel)
            {
#pragma unroll
              for (int j = 0; j < 8; ++j)
              {
                const int64_t at = place_of(0, j);
                place[j] = at >= 0 ? a.relabel[at] : -1;
              }
            }
          }
          long long value[kCols];
#pragma unroll
          for (int j = 0; j < kCols; ++j) value[j] = 0;  // also 0.0
          bool some = false;
          ok = ok && tc_segments(a, it, [&](const TcPair &sp, int lo, int hi) {
            long long head[kCols];
            float tail[kCols];
#pragma unroll
            for (int j = 0; j < kCols; ++j)
            {
              head[j] = 0;
              tail[j] = 0.0f;
            }
            for (int step = lo; step < hi; step += kTcChunkSteps)
            {
              if (!tc_wait_warp(&sums_full, sums, failed)) return false;
              sums ^= 1u;
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
              for (int c = 0; c < kCols; c += 8)
#pragma unroll
                for (int l0 = 0; l0 < S; l0 += 3)
                {
                  // three levels of eight columns in flight at a time
                  constexpr int kAhead = 3;
                  uint32_t lev[kAhead][8];
#pragma unroll
                  for (int l = 0; l < kAhead && l0 + l < S; ++l) tc_load8(lane_addr + static_cast<uint32_t>((l0 + l) * N + c), lev[l]);
                  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                  for (int l = 0; l < kAhead && l0 + l < S; ++l)
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                    {
                      const float x = __uint_as_float(lev[l][j]);
                      if (l0 + l < 4)
                        head[c + j] += static_cast<long long>(__float2int_rn(x)) * (1ll << (7 * (3 - l0 - l)));
                      else
                        tail[c + j] = fmaf(x, 1.0f / static_cast<float>(1 << (7 * (l0 + l - 4))), tail[c + j]);
                    }
                }
              asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
              __syncwarp();
              if (lane == 0) bar_arrive(&sums_free);
            }
            if (fixed)
            {
              // the tail in two 32-bit conversions (below 7.1 2^12 K <= 2^31), the fraction exact
#pragma unroll
              for (int j = 0; j < kCols; ++j)
              {
                const float whole = rintf(tail[j]);
                const int low = __float2int_rn((tail[j] - whole) * static_cast<float>(1 << bits));
                value[j] = (head[j] << (7 + bits)) + static_cast<long long>(__float2int_rn(whole)) * (1ll << bits) + low;
              }
            }
            else
            {
              // one FP64 step per entry, and the scales of a pair among several
              int re = 0, ce[kCols] = {};
              if (!single) exponents(sp.ea, sp.eb, re, ce);
#pragma unroll
              for (int j = 0; j < kCols; ++j)
              {
                double x = level_sum(head[j], tail[j]);
                if (!single) x = scaled(x, re + ce[j]);
                if (some) x += __longlong_as_double(value[j]);
                value[j] = __double_as_longlong(x);
              }
            }
            some = true;
            return true;
          });
          bool lost = !ok;
          if (it.slot >= 0)
          {
            // a partial tile, columns of 128 rows so that a warp writes 256 contiguous bytes; the CTA
            // that holds the tile's last ticket sums them in slot order
            long long *out = reinterpret_cast<long long *>(a.partial) + static_cast<int64_t>(it.slot) * kTcM * N + col0 * kTcM +
                             32 * quarter + lane;
#pragma unroll
            for (int j = 0; j < kCols; ++j) __stcg(out + j * kTcM, value[j]);
            const GemmReduce r = a.reduces[it.reduce];
            __threadfence();
            epilogue_sync();
            if (tid == 0)
            {
              const int mine = *failed ? 1 + kTcLost : 1, sum = atomicAdd(a.tickets + it.reduce, mine) + mine;
              last_flag = sum % kTcLost != r.nslots ? 0 : sum < kTcLost ? 1 : 2;
              // every other part of the tile has its ticket: left zero for the next launch
              if (last_flag) a.tickets[it.reduce] = 0;
            }
            epilogue_sync();
            const int last = last_flag;
            epilogue_sync();
            if (last == 0) continue;
            lost = last == 2;
            __threadfence();
            const long long *from = reinterpret_cast<const long long *>(a.partial) + static_cast<int64_t>(r.slot0) * kTcM * N +
                                    col0 * kTcM + 32 * quarter + lane;
#pragma unroll
            for (int c = 0; c < kCols; c += 8)
            {
              // three parts' reads in flight at a time
              constexpr int kAhead = 3;
#pragma unroll
              for (int j = 0; j < 8; ++j) value[c + j] = 0;
              for (int s0 = 0; s0 < r.nslots; s0 += kAhead)
              {
                long long x[kAhead][8];
#pragma unroll
                for (int s = 0; s < kAhead; ++s)
#pragma unroll
                  for (int j = 0; j < 8; ++j)
                    x[s][j] = s0 + s < r.nslots ? __ldcg(from + static_cast<int64_t>(s0 + s) * kTcM * N + (c + j) * kTcM) : 0;
#pragma unroll
                for (int s = 0; s < kAhead; ++s)
#pragma unroll
                  for (int j = 0; j < 8; ++j)
                    value[c + j] = fixed ? value[c + j] + x[s][j]
                                         : __double_as_longlong(__longlong_as_double(value[c + j]) + __longlong_as_double(x[s][j]));
              }
            }
          }
          if (lost)
          {
#pragma unroll 1
            for (int j = 0; j < kCols; ++j)
            {
              int64_t at = it.c + static_cast<int64_t>(row) * it.n + it.n0 + col0 + j;
              if (row >= it.m || it.n0 + col0 + j >= it.n) continue;
              if (a.relabel && (at = a.relabel[at]) < 0) continue;
              a.c[at] = __longlong_as_double(0x7ff8000000000000ll);
            }
            continue;
          }
          if constexpr (N != 32)
            if (single) exponents(it.ea, it.eb, row_exp, col_exp);
          if (single && !fixed)
          {
#pragma unroll
            for (int j = 0; j < kCols; ++j)
              value[j] = __double_as_longlong(scaled(__longlong_as_double(value[j]), row_exp + col_exp[j]));
          }
          if (fixed)
          {
            row_exp -= 42 + bits;
            bool outside = false;
            long long number[kCols];
#pragma unroll
            for (int j = 0; j < kCols; ++j)
              number[j] = __double_as_longlong(fixed_to_double(value[j], row_exp + col_exp[j], outside));
            if (outside)
            {
#pragma unroll 1
              for (int j = 0; j < kCols; ++j)
              {
                long long v = 0;
                int ex = 0;
#pragma unroll
                for (int i = 0; i < kCols; ++i)
                  if (i == j)
                  {
                    v = value[i];
                    ex = row_exp + col_exp[i];
                  }
                const long long slow = __double_as_longlong(fixed_slow(v, ex));
#pragma unroll
                for (int i = 0; i < kCols; ++i)
                  if (i == j) number[i] = slow;
              }
            }
#pragma unroll
            for (int j = 0; j < kCols; ++j) value[j] = number[j];
          }
#pragma unroll
          for (int c = 0; c < kCols; c += 8)
          {
            transpose8(value + c, lane);
            if (a.relabel)
            {
              // straight to its place after the leg move that follows
              if constexpr (N != 32)
              {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                {
                  const int64_t at = place_of(c, j);
                  place[j] = at >= 0 ? a.relabel[at] : -1;
                }
              }
#pragma unroll
              for (int j = 0; j < 8; ++j)
                if (place[j] >= 0) a.c[place[j]] = __longlong_as_double(value[c + j]);
            }
            else
            {
#pragma unroll
              for (int j = 0; j < 8; ++j)
              {
                const int64_t at = place_of(c, j);
                if (at >= 0) a.c[at] = __longlong_as_double(value[c + j]);
              }
            }
          }
          // the alignment pad after an odd-sized block reads as zero in arena-wide sums
          const int64_t entries = static_cast<int64_t>(it.m) * it.n;
          if (!a.relabel && tid == 0 && it.m0 + kTcM >= it.m && it.n0 + N >= it.n && (entries & 1)) a.c[it.c + entries] = 0.0;
        }
      }
      __syncthreads();
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      dependent_release();
      if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
    }
  } // namespace

  // ------------------------------------------------------------------------------------------
  // host
  // ------------------------------------------------------------------------------------------

  // Tiles of 64 columns, of 32 when 64 would leave SMs without a tile (half the time to the end of a
  // small product); a tile whose K is more than an
  // SM's share of the work is cut along K into equal parts of at least sixteen steps, so that the parts
  // fill the SMs once.  A part costs its pipeline's fill, a partial tile of 32 or 64 KB and the ticket
  // (6 us of a 12 us product): the matvec of bond 400 takes 63.5, 49.6, 47.6 and 49.2 us with at
  // least 4, 6, 8 and 16 steps a part, that of bond 512 69.5, 69.2, 69.2 and 64.0, of bond 200 29.4,
  // 30.6, 30.7 and 28.1.
  TcSchedule schedule_tc(const Program &p, const Op &op, const std::vector<SplitPair> *pairs)
  {
    TcSchedule s;
    const auto steps_of = [&p](const GemmBlock &blk) {
      int64_t steps = 0;
      for (int32_t q = 0; q < blk.pair_count; ++q)
        steps += (p.gemm_pairs[static_cast<size_t>(blk.pair_begin + q)].k + kTcK - 1) / kTcK;
      return steps;
    };
    int64_t tiles[2] = {}, total[2] = {};
    for (int64_t b = op.begin; b < op.begin + op.count; ++b)
    {
      const GemmBlock &blk = p.gemm_blocks[static_cast<size_t>(b)];
      const int64_t steps = steps_of(blk), high = (blk.m + kTcM - 1) / kTcM;
      for (int w = 0; w < 2; ++w)
      {
        const int64_t n = high * ((blk.n + (32 << w) - 1) / (32 << w));
        tiles[w] += n;
        total[w] += n * steps;
      }
    }
    const int w = tiles[1] <= p.ctas ? 0 : 1;
    s.n = 32 << w;
    int64_t share = std::max<int64_t>(16, (total[w] + p.ctas - 1) / p.ctas);
    // a ticket per cut tile
    if (tiles[w] > kTicketInts) share = INT32_MAX;
    struct Sized
    {
      TcItem item;
      int64_t work;
    };
    std::vector<Sized> all;
    for (int64_t b = op.begin; b < op.begin + op.count; ++b)
    {
      const GemmBlock &blk = p.gemm_blocks[static_cast<size_t>(b)];
      const int64_t steps = steps_of(blk), parts = std::max<int64_t>(1, (steps + share - 1) / share);
      const int64_t per = (steps + parts - 1) / parts;
      TcItem it{blk.c, 0, 0, blk.m, blk.n, 0, 0, 0, static_cast<int32_t>(steps), -1, -1, blk.pair_begin, blk.pair_count, 0, 0, 0, 0};
      if (pairs && blk.pair_count > 0)
      {
        const SplitPair &sp = (*pairs)[static_cast<size_t>(blk.pair_begin)];
        it.sa = sp.sa;
        it.sb = sp.sb;
        it.k = p.gemm_pairs[static_cast<size_t>(blk.pair_begin)].k;
        it.ksteps = sp.ksteps;
        it.ea = sp.ea;
        it.eb = sp.eb;
      }
      for (it.m0 = 0; it.m0 < blk.m; it.m0 += kTcM)
        for (it.n0 = 0; it.n0 < blk.n; it.n0 += s.n)
        {
          if (parts == 1)
          {
            if (pairs) all.push_back({it, steps + 4});
            continue;
          }
          const int32_t slot0 = static_cast<int32_t>(s.slots);
          TcItem cut = it;
          cut.reduce = static_cast<int32_t>(s.reduces.size());
          for (int64_t s0 = 0; s0 < steps; s0 += per)
          {
            cut.s0 = static_cast<int32_t>(s0);
            cut.s1 = static_cast<int32_t>(std::min(steps, s0 + per));
            cut.slot = static_cast<int32_t>(s.slots++);
            if (pairs) all.push_back({cut, per + 5});
          }
          s.reduces.push_back({static_cast<int32_t>(b), it.m0, it.n0, slot0, static_cast<int32_t>(s.slots) - slot0, 0});
        }
    }
    if (!pairs) return s;
    // the largest first, each to the least loaded SM
    std::stable_sort(all.begin(), all.end(), [](const Sized &x, const Sized &y) { return x.work > y.work; });
    s.ctas = static_cast<int32_t>(std::min<size_t>(static_cast<size_t>(p.ctas), all.size()));
    std::vector<std::vector<int32_t>> lists(static_cast<size_t>(s.ctas));
    std::vector<std::pair<int64_t, int>> heap;
    for (int c = 0; c < s.ctas; ++c) heap.push_back({0, c});
    const auto later = [](const std::pair<int64_t, int> &x, const std::pair<int64_t, int> &y) { return x > y; };
    std::make_heap(heap.begin(), heap.end(), later);
    for (size_t i = 0; i < all.size(); ++i)
    {
      std::pop_heap(heap.begin(), heap.end(), later);
      auto &least = heap.back();
      lists[static_cast<size_t>(least.second)].push_back(static_cast<int32_t>(i));
      least.first += all[i].work;
      std::push_heap(heap.begin(), heap.end(), later);
    }
    for (const auto &list : lists) s.longest = std::max(s.longest, static_cast<int32_t>(list.size()));
    s.items.assign(static_cast<size_t>(s.ctas) * static_cast<size_t>(s.longest), TcItem{});
    for (size_t c = 0; c < lists.size(); ++c)
      for (size_t i = 0; i < lists[c].size(); ++i)
        s.items[c * static_cast<size_t>(s.longest) + i] = all[static_cast<size_t>(lists[c][i])].item;
    return s;
  }

  bool split_tc_large(const Program &p, const Op &op, int32_t slices)
  {
    if (slices < 1) return false;
    // enough whole tiles to give every SM several, and most of the work in them
    double work = 0, tiled = 0;
    int64_t tiles = 0;
    for (int64_t b = op.begin; b < op.begin + op.count; ++b)
    {
      const GemmBlock &blk = p.gemm_blocks[static_cast<size_t>(b)];
      int64_t k = 0;
      for (int32_t q = 0; q < blk.pair_count; ++q) k += p.gemm_pairs[static_cast<size_t>(blk.pair_begin + q)].k;
      const double w = static_cast<double>(blk.m) * blk.n * k;
      work += w;
      tiles += static_cast<int64_t>((blk.m + kTcM - 1) / kTcM) * ((blk.n + 63) / 64);
      if (blk.m >= kTcM / 2 && blk.n >= 32) tiled += w;
    }
    return tiles >= 4 * static_cast<int64_t>(p.ctas) && tiled >= 0.9 * work;
  }

  cudaError_t launch_split_tc(const DeviceTables &t, size_t op_index, int32_t slices,
                              const uint16_t *sa, const uint16_t *sb, const int16_t *exps_a, const int16_t *exps_b,
                              const void *spairs, double *C, double *partial, int *tickets, const int32_t *relabel,
                              cudaStream_t stream)
  {
    const DeviceTables::TcTables &tc = t.tc[op_index];
    const TcArgs args{sa, sb, exps_a, exps_b, C, relabel,
                      static_cast<const DevSplitPair *>(spairs), static_cast<const TcItem *>(tc.items), tc.reduces, tc.longest,
                      partial, tickets};
    cudaError_t e = cudaSuccess;
    switch (slices * 128 + tc.n)
    {
#define TTG_TC(S, N)                                                                                                       \
  case S * 128 + N:                                                                                                        \
  {                                                                                                                        \
    static std::once_flag once;                                                                                            \
    std::call_once(once, [&] {                                                                                             \
      e = cudaFuncSetAttribute(gemm_split_tc_kernel<S, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, TcShape<S, N>::bytes); \
    });                                                                                                                    \
    if (e != cudaSuccess) return e;                                                                                        \
    e = launch_dependent(gemm_split_tc_kernel<S, N>, tc.n_ctas, TcShape<S, N>::threads, TcShape<S, N>::bytes, stream, args);          \
    break;                                                                                                                 \
  }
#define TTG_TC2(S) TTG_TC(S, 32) TTG_TC(S, 64)
      TTG_TC2(1) TTG_TC2(2) TTG_TC2(3) TTG_TC2(4) TTG_TC2(5) TTG_TC2(6) TTG_TC2(7) TTG_TC2(8)
#undef TTG_TC2
#undef TTG_TC
    default: return cudaErrorInvalidValue;
    }
    return e;
  }

} // namespace ttg

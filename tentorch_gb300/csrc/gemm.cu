// Grouped block-pair GEMM for sm_103a: balanced work schedules, the persistent FP64 / complex128
// kernels, the slicing pass of split precision, and its mma.sync kernel, the form beside the tcgen05 one
// (split_tc.cu) for blocks whose tiles there would be padding, and one that the autotuner may pick.  See gemm.h for the numerical scheme.
//
// Both GEMM kernels are persistent: one CTA per SM, held there by its shared-memory request, split
// into independent workers of 128 threads that claim work items from a list sorted largest first
// through an atomic counter.  A tile whose K was cut into several items is reduced by the worker that finishes
// its last item (an atomic ticket per tile): the partials are summed in slot order, so the result
// is deterministic, and no thread ever waits on another CTA.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <numeric>
#include <cmath>
#include <map>
#include <mutex>

#include "executor.h"
#include "gemm.h"
#include "gemm_device.cuh"
#include "launch.h"

namespace ttg
{
  // ------------------------------------------------------------------------------------------
  // schedules (host)
  // ------------------------------------------------------------------------------------------

  namespace
  {
    double op_work(const Program &p, const Op &op)
    {
      double total = 0;
      for (int64_t b = op.begin; b < op.begin + op.count; ++b)
      {
        const GemmBlock &blk = p.gemm_blocks[static_cast<size_t>(b)];
        for (int32_t k = 0; k < blk.pair_count; ++k)
          total += static_cast<double>(blk.m) * blk.n * p.gemm_pairs[static_cast<size_t>(blk.pair_begin + k)].k;
      }
      return total;
    }

    int64_t up256(int64_t bytes) { return (bytes + 255) / 256 * 256; }
  } // namespace

  GemmSchedule schedule_gemm(const Program &p, const Op &op, int bm, int bn, bool full, bool lanes, bool whole)
  {
    GemmSchedule s;
    // The workers of one SM share its FP64 pipe, so what has to balance is the work per SM: items
    // of a few per SM (a matvec's stage has only ~10^5 multiply-adds per SM), each a tile over a
    // K range of at least 16, dealt to the SMs largest first, each to the least loaded (LPT).
    // Cost of an item: the 16 x 8 DMMA fragments it computes (fragments wholly outside the block are
    // skipped) times its K range, plus per staged K step (its copies and barriers) and per item
    // (claim, write or partial tile) a quarter of a full tile over 16 of K.
    // On FMA lanes (complex128): its live entries' multiply-adds, and per staged step of 16 and per item
    // the time of 1024 (a quarter of a 16 x 16 tile over 16).
    const auto cost = [bm, bn, lanes](double rows, double cols, double k)
    {
      if (lanes) return std::ceil(rows * cols / 32.0) * 32.0 * k + 1024.0 * (std::ceil(k / 16.0) + 1.0);
      const double frag = std::ceil(rows / 16.0) * 16.0 * std::ceil(cols / 8.0) * 8.0;
      return frag * k + 0.25 * bm * bn * 16.0 * (std::ceil(k / kDmmaStepK) + 1.0);
    };
    double total = 0;
    for (int64_t b = op.begin; b < op.begin + op.count; ++b)
    {
      const GemmBlock &blk = p.gemm_blocks[static_cast<size_t>(b)];
      int64_t ktotal = 0;
      for (int32_t k = 0; k < blk.pair_count; ++k) ktotal += p.gemm_pairs[static_cast<size_t>(blk.pair_begin + k)].k;
      for (int32_t m0 = 0; m0 < blk.m; m0 += bm)
        for (int32_t n0 = 0; n0 < blk.n; n0 += bn)
          total += cost(std::min(bm, blk.m - m0), std::min(bn, blk.n - n0), static_cast<double>(ktotal));
    }
    const double target = std::max(total / (p.ctas * 6.0), cost(bm, bn, 16.0));
    struct Sized
    {
      GemmItem item;
      double work;
    };
    std::vector<Sized> items;
    int64_t n_items = 0;
    for (int64_t b = op.begin; b < op.begin + op.count; ++b)
    {
      const GemmBlock &blk = p.gemm_blocks[static_cast<size_t>(b)];
      int64_t ktotal = 0;
      for (int32_t k = 0; k < blk.pair_count; ++k) ktotal += p.gemm_pairs[static_cast<size_t>(blk.pair_begin + k)].k;
      for (int32_t m0 = 0; m0 < blk.m; m0 += bm)
        for (int32_t n0 = 0; n0 < blk.n; n0 += bn)
        {
          const double rows = std::min(bm, blk.m - m0), cols = std::min(bn, blk.n - n0);
          const double work = cost(rows, cols, static_cast<double>(ktotal));
          int64_t chunks = whole ? 1 : std::max<int64_t>(1, static_cast<int64_t>(std::ceil(work / target)));
          int64_t kc = (ktotal + chunks - 1) / std::max<int64_t>(chunks, 1);
          kc = std::max<int64_t>(16, (kc + 15) / 16 * 16);
          chunks = ktotal > 0 ? (ktotal + kc - 1) / kc : 1;
          const int32_t bi = static_cast<int32_t>(b);
          n_items += chunks;
          if (chunks == 1)
          {
            if (full) items.push_back({{bi, m0, n0, 0, static_cast<int32_t>(ktotal), -1, -1, 0}, work});
            continue;
          }
          const int32_t slot0 = static_cast<int32_t>(s.slots), reduce = static_cast<int32_t>(s.reduces.size());
          for (int64_t c = 0; c < chunks; ++c)
          {
            const int64_t k0 = c * kc, k1 = std::min(ktotal, (c + 1) * kc);
            if (full)
              items.push_back({{bi, m0, n0, static_cast<int32_t>(k0), static_cast<int32_t>(k1), static_cast<int32_t>(s.slots),
                                reduce, 0},
                               cost(rows, cols, static_cast<double>(k1 - k0))});
            ++s.slots;
          }
          s.reduces.push_back({bi, m0, n0, slot0, static_cast<int32_t>(chunks), 0});
        }
    }
    s.n_items = n_items;
    if (!full) return s;
    // largest first, equal work in the order made
    std::vector<int32_t> order(items.size());
    std::iota(order.begin(), order.end(), 0);
    std::sort(order.begin(), order.end(), [&items](int32_t a, int32_t b)
              { return items[static_cast<size_t>(a)].work > items[static_cast<size_t>(b)].work ||
                       (items[static_cast<size_t>(a)].work == items[static_cast<size_t>(b)].work && a < b); });
    // LPT: each item to the CTA with the least work so far (ties to the lower index)
    const int ctas = static_cast<int>(std::min<size_t>(static_cast<size_t>(p.ctas), std::max<size_t>(items.size(), 1)));
    std::vector<std::pair<double, int>> heap;
    heap.reserve(static_cast<size_t>(ctas));
    for (int c = 0; c < ctas; ++c) heap.push_back({0.0, c});
    const auto later = [](const std::pair<double, int> &a, const std::pair<double, int> &b)
    { return a.first > b.first || (a.first == b.first && a.second > b.second); };
    std::make_heap(heap.begin(), heap.end(), later);
    std::vector<int32_t> cta_of(items.size());
    s.cta_begin.assign(static_cast<size_t>(ctas) + 1, 0);
    for (const int32_t i : order)
    {
      std::pop_heap(heap.begin(), heap.end(), later);
      auto &least = heap.back();
      cta_of[static_cast<size_t>(i)] = least.second;
      ++s.cta_begin[static_cast<size_t>(least.second) + 1];
      least.first += items[static_cast<size_t>(i)].work;
      std::push_heap(heap.begin(), heap.end(), later);
    }
    // the lists back to back, each in the order its items were dealt
    for (int c = 0; c < ctas; ++c) s.cta_begin[static_cast<size_t>(c) + 1] += s.cta_begin[static_cast<size_t>(c)];
    std::vector<int32_t> fill(s.cta_begin.begin(), s.cta_begin.end() - 1);
    s.items.resize(items.size());
    for (const int32_t i : order)
      s.items[static_cast<size_t>(fill[static_cast<size_t>(cta_of[static_cast<size_t>(i)])]++)] = items[static_cast<size_t>(i)].item;
    return s;
  }

  void gemm_operands(const Program &p, const Op &op, std::vector<OperandBlock> &left, std::vector<OperandBlock> &right)
  {
    std::map<int64_t, int> seen_a, seen_b;
    left.clear();
    right.clear();
    for (int64_t b = op.begin; b < op.begin + op.count; ++b)
    {
      const GemmBlock &blk = p.gemm_blocks[static_cast<size_t>(b)];
      for (int32_t k = 0; k < blk.pair_count; ++k)
      {
        const GemmPair &pr = p.gemm_pairs[static_cast<size_t>(blk.pair_begin + k)];
        if (seen_a.emplace(pr.a, 0).second) left.push_back({pr.a, blk.m, pr.k});
        if (seen_b.emplace(pr.b, 0).second) right.push_back({pr.b, pr.k, blk.n});
      }
    }
  }

  SplitSchedule schedule_split(const Program &p, const Op &op, bool full)
  {
    SplitSchedule s;
    if (full) s.pairs.assign(p.gemm_pairs.size(), SplitPair{0, 0, 0, 0, 0, 0});
    // slices: every distinct left block's rows, every distinct right block's columns, in the layout of
    // SplitPair; exponents: one per row of A, one per column of B
    std::map<int64_t, std::pair<int64_t, int32_t>> a_at, b_at;  // arena offset -> (slice offset, exponent base)
    const auto pad32 = [](int64_t k) { return (k + kSplitStepK - 1) / kSplitStepK * kSplitStepK; };
    std::vector<SplitGroup> b_groups;
    const auto cut = [full](std::vector<SplitGroup> &out, int64_t src, int64_t base, int32_t lines, int32_t len, int32_t line_step,
                            int32_t entry_step, int32_t tile, int32_t exp)
    {
      const int32_t ksteps = (len + kSplitStepK - 1) / kSplitStepK;
      for (int32_t l = 0; full && l < lines; l += 8)
      {
        SplitGroup g{src + static_cast<int64_t>(l) * line_step, 0, len, line_step, entry_step, std::min(8, lines - l), exp + l, 0, 0, 0};
        g.dst = slice_place(base, lines, ksteps, tile, l, 0, g.slice_stride);
        g.step_stride = kMaxSlices * g.slice_stride;
        out.push_back(g);
      }
      return static_cast<int64_t>((lines + 7) / 8) * ksteps * kMaxSlices * kSliceGroup;
    };
    for (int64_t bi = op.begin; bi < op.begin + op.count; ++bi)
    {
      const GemmBlock &blk = p.gemm_blocks[static_cast<size_t>(bi)];
      for (int32_t k = 0; k < blk.pair_count; ++k)
      {
        const size_t pi = static_cast<size_t>(blk.pair_begin + k);
        const GemmPair &pr = p.gemm_pairs[pi];
        s.longest_line = std::max<int64_t>(s.longest_line, pr.k);
        auto fa = a_at.find(pr.a);
        if (fa == a_at.end())
        {
          fa = a_at.emplace(pr.a, std::make_pair(s.slice_a, static_cast<int32_t>(s.exps_a))).first;
          s.slice_a += cut(s.groups, pr.a, s.slice_a, blk.m, pr.k, pr.k, 1, kSliceTileA, static_cast<int32_t>(s.exps_a));
          s.exps_a += blk.m;
        }
        auto fb = b_at.find(pr.b);
        if (fb == b_at.end())
        {
          fb = b_at.emplace(pr.b, std::make_pair(s.slice_b, static_cast<int32_t>(s.exps_b))).first;
          s.slice_b += cut(b_groups, pr.b, s.slice_b, blk.n, pr.k, 1, blk.n, kSliceTileB, static_cast<int32_t>(s.exps_b));
          s.exps_b += blk.n;
        }
        if (full)
          s.pairs[pi] = SplitPair{fa->second.first, fb->second.first, static_cast<int32_t>(pad32(pr.k) / kSplitStepK),
                                  fa->second.second, fb->second.second, 0};
      }
    }
    s.exps = s.exps_a + s.exps_b;
    s.groups_a = static_cast<int64_t>(s.groups.size());
    s.groups.insert(s.groups.end(), b_groups.begin(), b_groups.end());
    // items: one pair's K range each (a multiple of 32), about two per worker, never below a tile
    // over 256 of K (one exact level chunk: smaller items cost more in folds and partial tiles than
    // they gain in spread; at bond 512 the split matvec took 147 us with 128 and 123 us with 256)
    const double target =
      std::max(op_work(p, op) / (p.ctas * kSplitWorkers * 2.0), static_cast<double>(kSplitTileM) * kSplitTileN * kSplitChunk);
    struct Sized
    {
      SplitItem item;
      double work;
    };
    std::vector<Sized> items, tile;
    for (int64_t bi = op.begin; bi < op.begin + op.count; ++bi)
    {
      const GemmBlock &blk = p.gemm_blocks[static_cast<size_t>(bi)];
      for (int32_t m0 = 0; m0 < blk.m; m0 += kSplitTileM)
        for (int32_t n0 = 0; n0 < blk.n; n0 += kSplitTileN)
        {
          const double rows = std::min(kSplitTileM, blk.m - m0), cols = std::min(kSplitTileN, blk.n - n0);
          // a warp's 16 x 16 quarter outside the block skips its products
          const double quarters = std::ceil(rows / 16.0) * std::ceil(cols / 16.0);
          const auto cost = [quarters](double k)
          { return quarters * 256.0 * (std::ceil(k / kSplitStepK) * kSplitStepK + 2.0 * kSplitStepK * (std::ceil(k / kSplitChunk) + 1.0)); };
          tile.clear();
          for (int32_t k = 0; k < blk.pair_count; ++k)
          {
            const int32_t pi = blk.pair_begin + k;
            const int64_t K = p.gemm_pairs[static_cast<size_t>(pi)].k;
            const double work = rows * cols * static_cast<double>(K);
            int64_t chunks = std::max<int64_t>(1, static_cast<int64_t>(std::ceil(work / target)));
            const int64_t kc = pad32((K + chunks - 1) / chunks);
            chunks = (K + kc - 1) / kc;
            for (int64_t c = 0; c < chunks; ++c)
            {
              const int64_t k0 = c * kc, k1 = std::min<int64_t>(K, (c + 1) * kc);
              tile.push_back({{static_cast<int32_t>(bi), m0, n0, pi, static_cast<int32_t>(k0), static_cast<int32_t>(k1), 0, -1},
                              cost(static_cast<double>(k1 - k0))});
            }
          }
          if (tile.size() == 1)
          {
            tile[0].item.slot = -1;
            if (full) items.push_back(tile[0]);
          }
          else if (tile.empty())
          {
            if (full) items.push_back({{static_cast<int32_t>(bi), m0, n0, -1, 0, 0, -1, -1}, cost(0.0)});  // no pair: zeros
          }
          else
          {
            const int32_t slot0 = static_cast<int32_t>(s.slots), reduce = static_cast<int32_t>(s.reduces.size());
            for (Sized &t : tile)
            {
              t.item.slot = static_cast<int32_t>(s.slots++);
              t.item.reduce = reduce;
              if (full) items.push_back(t);
            }
            s.reduces.push_back({static_cast<int32_t>(bi), m0, n0, slot0, static_cast<int32_t>(tile.size()), 0});
          }
        }
    }
    if (!full) return s;
    std::stable_sort(items.begin(), items.end(), [](const Sized &a, const Sized &b) { return a.work > b.work; });
    // dealt to the SMs like the FP64 items (largest first onto the least loaded)
    const int ctas = static_cast<int>(std::min<size_t>(static_cast<size_t>(p.ctas), std::max<size_t>(items.size(), 1)));
    std::vector<std::vector<SplitItem>> lists(static_cast<size_t>(ctas));
    std::vector<std::pair<double, int>> heap;
    for (int c = 0; c < ctas; ++c) heap.push_back({0.0, c});
    const auto later = [](const std::pair<double, int> &a, const std::pair<double, int> &b)
    { return a.first > b.first || (a.first == b.first && a.second > b.second); };
    std::make_heap(heap.begin(), heap.end(), later);
    for (const Sized &it : items)
    {
      std::pop_heap(heap.begin(), heap.end(), later);
      auto &least = heap.back();
      lists[static_cast<size_t>(least.second)].push_back(it.item);
      least.first += it.work;
      std::push_heap(heap.begin(), heap.end(), later);
    }
    s.cta_begin.push_back(0);
    for (const auto &list : lists)
    {
      s.items.insert(s.items.end(), list.begin(), list.end());
      s.cta_begin.push_back(static_cast<int32_t>(s.items.size()));
    }
    return s;
  }

  namespace
  {
    // bytes of the partial tiles of either form of the split products
    int64_t split_partial_bytes(const SplitSchedule &s, const TcSchedule &tc)
    {
      return up256(std::max<int64_t>(s.slots * kSplitTileM * kSplitTileN * 8, tc.slots * kSliceTileA * tc.n * 8));
    }
    // bytes of split scratch: slices of A and of B (bf16), exponents (int16), partial tiles, tickets
    int64_t split_bytes(const SplitSchedule &s, const TcSchedule &tc)
    {
      return up256(2 * s.slice_a) + up256(2 * s.slice_b) + up256(2 * s.exps) + split_partial_bytes(s, tc) +
             up256(4 * (static_cast<int64_t>(s.reduces.size()) + 1));
    }
    // The complex128 tile of an op: 32 x 32 where such tiles are many beside their K.  A tile has its first copies, its
    // sums' meeting and its claim for itself, which with a short K is most of its time; with a long K and few tiles an
    // SM's share is too coarse.  Measured (us, 16 x 16 and 32 x 32): 4000 x 4000 x 4 879 and 498, x 16 2117 and 1668, x 128
    // 13391 and 13084; 1000 x 1000 x 16 135 and 121, x 32 241 and 233, x 64 443 and 454; 30000 x 8 x 3 32 and 20;
    // 300 x 300 x 16 19 and 24; the environment of bond 256/17 144, 144 and 135 by this line.
    int lanes_tile(const Program &p, const Op &op)
    {
      int64_t tiles = 0, longest = 0;
      for (int64_t b = op.begin; b < op.begin + op.count; ++b)
      {
        const GemmBlock &blk = p.gemm_blocks[static_cast<size_t>(b)];
        int64_t k = 0;
        for (int32_t q = 0; q < blk.pair_count; ++q) k += p.gemm_pairs[static_cast<size_t>(blk.pair_begin + q)].k;
        longest = std::max(longest, k);
        tiles += static_cast<int64_t>((blk.m + 2 * kLanesTile - 1) / (2 * kLanesTile)) * ((blk.n + 2 * kLanesTile - 1) / (2 * kLanesTile));
      }
      return tiles >= p.ctas * std::max<int64_t>(10, longest) / 5 ? 2 * kLanesTile : kLanesTile;
    }
    // bytes of FP64 scratch: partial tiles (`entry` bytes an entry), tickets
    int64_t f64_bytes(const GemmSchedule &s, int tile, int entry)
    {
      return up256(s.slots * tile * tile * entry) + up256(4 * (static_cast<int64_t>(s.reduces.size()) + 1));
    }
  } // namespace

  int device_sms()
  {
    static std::atomic<int> cached[64] = {};
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64)
    {
      cudaGetLastError();
      return 152;
    }
    int n = cached[device].load(std::memory_order_relaxed);
    if (n > 0) return n;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || n <= 0)
    {
      cudaGetLastError();
      return 152;
    }
    cached[device].store(n, std::memory_order_relaxed);
    return n;
  }

  int64_t plan_gemms(Program &p)
  {
    p.ctas = device_sms();
    auto plans = std::make_shared<GemmPlans>();
    plans->f64.resize(p.ops.size());
    plans->split.resize(p.ops.size());
    plans->cache_a.assign(p.ops.size(), -1);
    plans->cache_b.assign(p.ops.size(), -1);
    int64_t need = 0;
    for (size_t i = 0; i < p.ops.size(); ++i)
    {
      const Op &op = p.ops[i];
      if (op.kind != OpKind::gemm) continue;
      plans->f64[i] = schedule_gemm(p, op, kF64TileM, kF64TileN, false);
      // the split schedule itself is built on the first split launch (most plans never run one);
      // here only its scratch
      need = std::max(need, (f64_bytes(plans->f64[i], kF64TileM, 8) + 7) / 8);
      // complex arenas count elements of 16 bytes
      const int lanes = lanes_tile(p, op);
      need = std::max(need, (f64_bytes(schedule_gemm(p, op, lanes, lanes, false, true), lanes, 16) + 15) / 16);
      // a chain's one launch holds the partial tiles of both its products at once
      if (static_cast<int32_t>(i) == p.chain_second)
      {
        // its items are cut for the FMA kernel (chain.cu)
        p.chain_slots = chain_partial_slots(p);
        need = std::max(need, (up256(p.chain_slots * kF64TileM * kF64TileN * 8) + 7) / 8);
      }
      const SplitSchedule sizes = schedule_split(p, op, false);
      need = std::max(need, (split_bytes(sizes, schedule_tc(p, op)) + 7) / 8);
      // the slices of a prepared operand's value go into its arena
      for (int side = 0; side < 2; ++side)
      {
        const int32_t buffer = side == 0 ? op.src : op.src2;
        if (buffer < 0) continue;
        const int32_t operand = p.buffers[static_cast<size_t>(buffer)].prepared_of;
        if (operand < 0) continue;
        if (plans->prepared_bytes.empty())
        {
          plans->prepared_bytes.assign(static_cast<size_t>(p.n_inputs), 0);
          for (int32_t j = 0; j < p.n_inputs; ++j)
            if (p.prepared[static_cast<size_t>(j)] >= 0)
              plans->prepared_bytes[static_cast<size_t>(j)] = up256(p.buffers[static_cast<size_t>(p.prepared[static_cast<size_t>(j)])].size * 8);
        }
        SliceCache c;
        c.op = static_cast<int32_t>(i);
        c.side = side;
        c.operand = operand;
        c.offset = plans->prepared_bytes[static_cast<size_t>(operand)];
        const int64_t slice = side == 0 ? sizes.slice_a : sizes.slice_b, exps = side == 0 ? sizes.exps_a : sizes.exps_b;
        c.exps_offset = c.offset + up256(2 * slice);
        c.bytes = up256(2 * slice) + up256(2 * exps);
        plans->prepared_bytes[static_cast<size_t>(operand)] += c.bytes;
        (side == 0 ? plans->cache_a : plans->cache_b)[i] = static_cast<int32_t>(plans->caches.size());
        plans->caches.push_back(c);
      }
    }
    p.gemm_plans = std::move(plans);
    return need;
  }

  // ------------------------------------------------------------------------------------------
  // device
  // ------------------------------------------------------------------------------------------

  namespace
  {
    // After a worker has written a partial tile: take the tile's ticket; the worker holding the last
    // ticket sums every partial of the tile in slot order into C.  The fences order the partial
    // writes before the ticket and the ticket before the reads (reads bypass L1).
    // `scale` gives an entry of the tile from its sum.
    struct Unscaled
    {
      template <typename T>
      __device__ T operator()(T v, const DevBlock &, int, int) const { return v; }
    };
    template <typename T, int BM, int BN, typename Scale = Unscaled>
    __device__ void finish_partial(int worker, int lt, int *flag, int *tickets, const GemmReduce *reduces, int reduce,
                                   const DevBlock *blocks, const T *partial, T *C, const int32_t *relabel = nullptr,
                                   Scale scale = Scale())
    {
      __threadfence();
      worker_sync(worker);
      const GemmReduce r = reduces[reduce];
      if (lt == 0) *flag = atomicAdd(tickets + reduce, 1) == r.nslots - 1;
      worker_sync(worker);
      const bool last = *flag;
      worker_sync(worker);
      if (!last) return;
      // every other partial of the tile has taken its ticket: leave the counter zero for the next launch
      if (lt == 0) tickets[reduce] = 0;
      __threadfence();
      const DevBlock blk = blocks[r.block];
      // every entry of the tile sums its slots in slot order; the loads of four slots for all of the
      // thread's entries are issued together, so a deep split costs a few L2 round trips, not one
      // per slot
      constexpr int PER = BM * BN / kWorkerThreads;
      T sum[PER];
#pragma unroll
      for (int k = 0; k < PER; ++k) sum[k] = zero_t<T>();
      const T *base = partial + static_cast<int64_t>(r.slot0) * BM * BN + lt;
      int s = 0;
      for (; s + 4 <= r.nslots; s += 4)
      {
        T v[4][PER];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int k = 0; k < PER; ++k) v[u][k] = __ldcg(base + static_cast<int64_t>(s + u) * BM * BN + k * kWorkerThreads);
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int k = 0; k < PER; ++k) sum[k] = add_t(sum[k], v[u][k]);
      }
      for (; s < r.nslots; ++s)
#pragma unroll
        for (int k = 0; k < PER; ++k) sum[k] = add_t(sum[k], __ldcg(base + static_cast<int64_t>(s) * BM * BN + k * kWorkerThreads));
#pragma unroll
      for (int k = 0; k < PER; ++k)
      {
        const int e = lt + k * kWorkerThreads;
        const int gm = r.m0 + e / BN, gn = r.n0 + e % BN;
        if (gm >= blk.m || gn >= blk.n) continue;
        const int64_t at = blk.c + static_cast<int64_t>(gm) * blk.n + gn;
        const T value = scale(sum[k], blk, gm, gn);
        if (!relabel)
          C[at] = value;
        else if (relabel[at] >= 0)
          C[relabel[at]] = value;  // straight to its place after the leg move that follows
      }
      const int64_t entries = static_cast<int64_t>(blk.m) * blk.n;
      if (!relabel && lt == 0 && r.m0 + BM >= blk.m && r.n0 + BN >= blk.n && (entries & 1)) C[blk.c + entries] = zero_t<T>();
    }

    // ---------------------------------------------------------------------------------------
    // FP64 / complex128
    // ---------------------------------------------------------------------------------------

    // Persistent: kF64Workers workers of 128 threads, each computing 16 x 16 (lanes_tile: or 32 x 32) tiles over a K range on FP64
    // FMA lanes.  A complex multiply-add is four FP64 ones and a warp's FP64 instruction takes 64 clocks
    // on a quarter of an SM, so what counts is that no lane works on padding and none waits for copies:
    //   - a tile's live entries times R phases of K (R a power of two, as many as fill the worker's 1024
    //     slots, at most the 16 K of a step) are dealt to the threads, eight independent chains each at most,
    //     and the phases of an entry summed at the end (a 10 x 10 block as 32 x 32 padded entries spent ten
    //     times its multiply-adds); 32 x 32 tiles over 32 of K hold an SM for 32 us, and few do not balance
    //     (the Fibonacci recoupling of 16 multiplets, all full tiles, takes 3.97 ms with them and 3.85 with
    //     16 x 16);
    //   - K advances through two shared stages, the next one's cp.async in flight during a step.
    // The three products of an environment update at bond 203 (13 charges) take 19, 42 and 26 us; with
    // padded 32 x 32 tiles and one synchronous stage 70, 94 and 66.
    constexpr int kLanesK = 16, kLanesPer = 8;
    constexpr int kLanesSlots = kLanesPer * kWorkerThreads;
    constexpr int lanes_bytes(int tile) { return kF64Workers * (2 * 2 * kLanesK * (tile + 1) + kLanesSlots) * 16; }

    __device__ __forceinline__ void copy16(double2 *dst, const double2 *src, bool in)
    {
      const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
      asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(in ? 16 : 0) : "memory");
    }

    template <int Tile>
    __global__ void __launch_bounds__(kF64Workers * kWorkerThreads, 1)
      gemm_c128_kernel(const double2 *__restrict__ A, const double2 *__restrict__ B, double2 *__restrict__ C,
                       const DevBlock *__restrict__ blocks, const DevPair *__restrict__ pairs,
                       const GemmItem *__restrict__ items, const int32_t *__restrict__ cta_begin, const GemmReduce *__restrict__ reduces,
                       int64_t n_reduces, double2 *__restrict__ partial, int *__restrict__ tickets)
    {
      dependent_entry();
      constexpr int BM = Tile, BN = Tile, BK = kLanesK, P = Tile + 1;
      extern __shared__ __align__(16) unsigned char smem_raw[];
      const int worker = threadIdx.x / kWorkerThreads, lt = threadIdx.x % kWorkerThreads;
      double2 *stage_base = reinterpret_cast<double2 *>(smem_raw) + static_cast<int64_t>(worker) * (2 * 2 * BK * P + kLanesSlots);
      double2 *slots = stage_base + 2 * 2 * BK * P;
      __shared__ int flags[kF64Workers];
      // this CTA's list of items (dealt by the host, largest first, to balance the SMs); its
      // workers take them in order through a shared counter
      __shared__ int next[kF64Workers];
      __shared__ int taken;
      if (threadIdx.x == 0) taken = 0;
      __syncthreads();
      const int64_t list_begin = cta_begin[blockIdx.x], list_end = cta_begin[blockIdx.x + 1];
      for (int64_t idx = list_begin + local_claim(worker, lt, next + worker, &taken); idx < list_end;
           idx = list_begin + local_claim(worker, lt, next + worker, &taken))
      {
        const GemmItem it = items[idx];
        const DevBlock blk = blocks[it.block];
        const int rows = min(BM, blk.m - it.m0), cols = min(BN, blk.n - it.n0), live = rows * cols;
        int shift = 0;
        while ((1 << shift) < BK && (live << (shift + 1)) <= kLanesSlots) ++shift;
        const int phases = 1 << shift, count = live << shift;
        const int mine = count > lt ? (count - lt + kWorkerThreads - 1) / kWorkerThreads : 0;
        // slot v: entry v >> shift, phase v & (phases - 1)
        int pa[kLanesPer], pb[kLanesPer];
        double2 acc[kLanesPer];
#pragma unroll
        for (int i = 0; i < kLanesPer; ++i)
        {
          const int v = min(lt + i * kWorkerThreads, count - 1), e = v >> shift, row = e / cols, k = v & (phases - 1);
          pa[i] = k * P + row;
          pb[i] = BK * P + k * P + (e - row * cols);
          acc[i] = make_double2(0.0, 0.0);
        }
        const auto load = [&](int stage, const double2 *a, const double2 *b, int K, int k0, int hi)
        {
          double2 *as = stage_base + stage * 2 * BK * P, *bs = as + BK * P;
          for (int i = lt; i < rows * BK; i += kWorkerThreads)
          {
            const int row = i / BK, kk = i % BK;
            const bool in = k0 + kk < hi;
            copy16(as + kk * P + row, in ? a + static_cast<int64_t>(it.m0 + row) * K + k0 + kk : a, in);
          }
          for (int i = lt; i < BK * cols; i += kWorkerThreads)
          {
            const int kk = i / cols, c = i - kk * cols;
            const bool in = k0 + kk < hi;
            copy16(bs + kk * P + c, in ? b + static_cast<int64_t>(k0 + kk) * blk.n + it.n0 + c : b, in);
          }
          copy_commit();
        };
        int32_t kbase = 0;
        for (int32_t pi = 0; pi < blk.pair_count; ++pi)
        {
          const DevPair pr = pairs[blk.pair_begin + pi];
          const int K = pr.k;
          const int lo = max(it.k0 - kbase, 0), hi = min(it.k1 - kbase, K);
          kbase += K;
          if (lo >= hi) continue;
          load(0, A + pr.a, B + pr.b, K, lo, hi);
          int stage = 0;
          for (int k0 = lo; k0 < hi; k0 += BK, stage ^= 1)
          {
            if (k0 + BK < hi)
              load(stage ^ 1, A + pr.a, B + pr.b, K, k0 + BK, hi);
            else
              copy_commit();  // an empty group keeps the count of the wait below
            copy_wait_one();
            worker_sync(worker);
            const double2 *base = stage_base + stage * 2 * BK * P;
            const int steps = min(BK, hi - k0);  // entries of the stage past `hi` are zeros
            for (int kk = 0; kk < steps; kk += phases)
#pragma unroll
              for (int i = 0; i < kLanesPer; ++i)
                if (i < mine) acc[i] = cfma(base[kk * P + pa[i]], base[kk * P + pb[i]], acc[i]);
            worker_sync(worker);
          }
        }
        // the phases of each entry, summed in order
        if (shift != 0)
        {
#pragma unroll
          for (int i = 0; i < kLanesPer; ++i)
            if (i < mine) slots[lt + i * kWorkerThreads] = acc[i];
          worker_sync(worker);
#pragma unroll
          for (int i = 0; i < kLanesPer; ++i)
          {
            const int e = lt + i * kWorkerThreads;
            double2 sum = make_double2(0.0, 0.0);
            if (e < live)
              for (int f = 0; f < phases; ++f) sum = add_t(sum, slots[(e << shift) + f]);
            acc[i] = sum;
          }
        }
#pragma unroll
        for (int i = 0; i < kLanesPer; ++i)
        {
          const int e = lt + i * kWorkerThreads;
          if (e >= live) continue;
          const int row = e / cols, c = e - row * cols;
          if (it.slot >= 0) partial[static_cast<int64_t>(it.slot) * BM * BN + row * BN + c] = acc[i];
          else C[blk.c + static_cast<int64_t>(it.m0 + row) * blk.n + it.n0 + c] = acc[i];
        }
        if (it.slot >= 0)
        {
          finish_partial<double2, BM, BN>(worker, lt, flags + worker, tickets, reduces, it.reduce, blocks, partial, C);
          continue;
        }
        // the alignment pad after an odd-sized block reads as zero in arena-wide sums
        const int64_t entries = static_cast<int64_t>(blk.m) * blk.n;
        if (lt == 0 && it.m0 + BM >= blk.m && it.n0 + BN >= blk.n && (entries & 1)) C[blk.c + entries] = make_double2(0.0, 0.0);
      }
    }

    // The float64 products on the FP64 matrix instruction (mma m16n8k8 f64): each of
    // a worker's 4 warps owns a 16 x 16 quarter of the 32 x 32 tile as two m16n8 accumulators; per
    // 8 of K staged in shared memory a warp issues 2 DMMA.
    __global__ void __launch_bounds__(kF64Workers * kWorkerThreads, 1)
      gemm_dmma_kernel(const double *__restrict__ A, const double *__restrict__ B, double *__restrict__ C,
                       const DevBlock *__restrict__ blocks, const DevPair *__restrict__ pairs,
                       const GemmItem *__restrict__ items, const int32_t *__restrict__ cta_begin, const GemmReduce *__restrict__ reduces,
                       int64_t n_reduces, double *__restrict__ partial, int *__restrict__ tickets)
    {
      dependent_entry();
      constexpr int BM = kF64TileM, BN = kF64TileN, BK = kDmmaStepK;
      extern __shared__ __align__(16) unsigned char smem_raw[];
      const int worker = threadIdx.x / kWorkerThreads, lt = threadIdx.x % kWorkerThreads;
      // rows of 36 doubles: a warp's fragment loads (k = lane % 4 (+ 4), row = lane / 4 (+ 8)) then
      // fall on distinct bank pairs within each half warp.  Two stages of A (k-major) and B per worker.
      constexpr int P = 36;
      double *stage_base = reinterpret_cast<double *>(smem_raw) + static_cast<size_t>(worker) * 2 * 2 * BK * P;
      __shared__ int flags[kF64Workers];
      const int warp = lt >> 5, lane = lt & 31;
      const int wm = warp >> 1, wn = warp & 1;
      const int fr = lane >> 2, fk = lane & 3;  // fragment row (or column) and k of this lane
      // this CTA's list of items (dealt by the host, largest first, to balance the SMs); its
      // workers take them in order through a shared counter
      __shared__ int next[kF64Workers];
      __shared__ int taken;
      if (threadIdx.x == 0) taken = 0;
      __syncthreads();
      const int64_t list_begin = cta_begin[blockIdx.x], list_end = cta_begin[blockIdx.x + 1];
      for (int64_t idx = list_begin + local_claim(worker, lt, next + worker, &taken); idx < list_end;
           idx = list_begin + local_claim(worker, lt, next + worker, &taken))
      {
        const GemmItem it = items[idx];
        const DevBlock blk = blocks[it.block];
        double acc[2][4] = {};
        const bool live_i = it.m0 + wm * 16 < blk.m;
        const bool live_j[2] = {it.n0 + wn * 16 < blk.n, it.n0 + wn * 16 + 8 < blk.n};
        int32_t kbase = 0;
        for (int32_t pi = 0; pi < blk.pair_count; ++pi)
        {
          const DevPair pr = pairs[blk.pair_begin + pi];
          const int K = pr.k;
          const int lo = max(it.k0 - kbase, 0), hi = min(it.k1 - kbase, K);
          kbase += K;
          if (lo >= hi) continue;
          const double *a = A + pr.a;
          const double *b = B + pr.b;
          // K in steps of BK through two shared stages: the copies of step s + 1 (cp.async, entries
          // outside the block or past hi filled with zeros) are in flight while step s computes
          const auto load = [&](int stage, int k0)
          {
            double *as = stage_base + stage * 2 * BK * P, *bs = as + BK * P;
            for (int i = lt; i < BM * BK; i += kWorkerThreads)
            {
              const int r = i / BK, kk = i % BK;
              const int gm = it.m0 + r, gk = k0 + kk;
              const bool in = gm < blk.m && gk < hi;
              copy8(as + kk * P + r, in ? a + static_cast<int64_t>(gm) * K + gk : a, in);
            }
            for (int i = lt; i < BK * BN; i += kWorkerThreads)
            {
              const int kk = i / BN, cc = i % BN;
              const int gk = k0 + kk, gn = it.n0 + cc;
              const bool in = gk < hi && gn < blk.n;
              copy8(bs + kk * P + cc, in ? b + static_cast<int64_t>(gk) * blk.n + gn : b, in);
            }
            copy_commit();
          };
          load(0, lo);
          int stage = 0;
          for (int k0 = lo; k0 < hi; k0 += BK, stage ^= 1)
          {
            if (k0 + BK < hi)
              load(stage ^ 1, k0 + BK);
            else
              copy_commit();  // an empty group keeps the count of the wait below
            copy_wait_one();
            worker_sync(worker);
            const double(*as)[P] = reinterpret_cast<const double(*)[P]>(stage_base + stage * 2 * BK * P);
            const double(*bs)[P] = reinterpret_cast<const double(*)[P]>(stage_base + stage * 2 * BK * P + BK * P);
            const int steps = min(BK, hi - k0);
            // a 16 x 8 fragment wholly outside the block costs the FP64 pipe as much as a full one:
            // skip it (warp-uniform); a full step runs unrolled with no bound, so the fragment loads
            // of the next k are issued ahead of the products of this one.  Entries of the stage past
            // `hi` are zeros, so a last step rounded up to 8 adds nothing.
            const auto step_k = [&](int kb)
            {
              double af[4], bf[2][2];
#pragma unroll
              for (int h = 0; h < 4; ++h) af[h] = as[kb + fk + (h >> 1) * 4][wm * 16 + (h & 1) * 8 + fr];
#pragma unroll
              for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) bf[j][h] = bs[kb + fk + h * 4][wn * 16 + j * 8 + fr];
#pragma unroll
              for (int j = 0; j < 2; ++j)
                if (live_j[j]) dmma16(acc[j], af, bf[j]);
            };
            if (live_i && live_j[0])  // the warp's 16 x 16 quarter touches the block
            {
              if (steps == BK)
              {
#pragma unroll
                for (int kb = 0; kb < BK; kb += 8) step_k(kb);
              }
              else
                for (int kb = 0; kb < steps; kb += 8) step_k(kb);
            }
            worker_sync(worker);
          }
        }
        if (it.slot >= 0)
        {
          double *out = partial + static_cast<int64_t>(it.slot) * BM * BN;
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int h = 0; h < 4; ++h) out[(wm * 16 + (h >> 1) * 8 + fr) * BN + wn * 16 + j * 8 + fk * 2 + (h & 1)] = acc[j][h];
          finish_partial<double, BM, BN>(worker, lt, flags + worker, tickets, reduces, it.reduce, blocks, partial, C);
          continue;
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int h = 0; h < 4; ++h)
          {
            const int gm = it.m0 + wm * 16 + (h >> 1) * 8 + fr, gn = it.n0 + wn * 16 + j * 8 + fk * 2 + (h & 1);
            if (gm < blk.m && gn < blk.n) C[blk.c + static_cast<int64_t>(gm) * blk.n + gn] = acc[j][h];
          }
        const int64_t entries = static_cast<int64_t>(blk.m) * blk.n;
        if (lt == 0 && it.m0 + BM >= blk.m && it.n0 + BN >= blk.n && (entries & 1)) C[blk.c + entries] = 0.0;
      }
    }

    // ---------------------------------------------------------------------------------------
    // split precision
    // ---------------------------------------------------------------------------------------

    // One CTA per group of eight lines (rows of A, columns of B): the power of two 2^e that bounds each
    // line, then each entry as the integer round(x 2^(56-e)) cut into `slices` balanced 7-bit digits
    // (|q_1| <= 128, |q_t| <= 64 after it), exact in bf16, into the layout of SplitPair, zeros past the
    // line's end.  A thread takes eight consecutive entries of one line, so that it writes 16 bytes a
    // slice, a warp 512 contiguous ones; consecutive threads are consecutive lines, so that the columns
    // of B, neighbours in memory, are read in runs of 64 bytes.  The first kHeld runs of a thread stay in
    // registers between the maximum and the cut (lines of up to 512 with 256 threads); the rest are read
    // again.  Bound by the bytes it reads and writes.
    constexpr int kHeld = 2;

    __global__ void __launch_bounds__(256)
      split_groups_kernel(const double *__restrict__ a, const double *__restrict__ b, uint16_t *__restrict__ slices_a,
                          uint16_t *__restrict__ slices_b, int16_t *__restrict__ exps_a, int16_t *__restrict__ exps_b,
                          const SplitGroup *__restrict__ groups, int64_t groups_a, int64_t group_begin, int slices_n)
    {
      __shared__ unsigned long long most[8][8];
      // the table is read while the kernel before still runs
      const int64_t at = group_begin + blockIdx.x;
      const SplitGroup g = groups[at];
      dependent_entry();
      dependent_release();  // to the product, which sets up its barriers and tensor memory meanwhile
      const bool left = at < groups_a;
      const int line = threadIdx.x & 7, first = threadIdx.x >> 3, runs = blockDim.x >> 3;
      const bool live = line < g.lines;
      const double *src = (left ? a : b) + g.src + static_cast<int64_t>(line) * g.line_step;
      uint16_t *dst = (left ? slices_a : slices_b) + g.dst + line * 8;
      const int total = (g.len + kSplitStepK - 1) / kSplitStepK * (kSplitStepK / 8);  // runs of a line, padding among them
      const auto read = [&](int run, double (&x)[8])
      {
#pragma unroll
        for (int j = 0; j < 8; ++j)
        {
          const int k = run * 8 + j;
          x[j] = live && k < g.len ? src[static_cast<int64_t>(k) * g.entry_step] : 0.0;
        }
      };
      unsigned long long big = 0;
      const auto larger = [&](const double (&x)[8])
      {
#pragma unroll
        for (int j = 0; j < 8; ++j)
        {
          // the largest |entry| by its bits (positive doubles order as integers)
          const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(x[j])) & 0x7fffffffffffffffull;
          big = bits > big ? bits : big;
        }
      };
      // (zeros, and no reads, past the line's end: every read of the thread is in flight together)
      double held[kHeld][8];
#pragma unroll
      for (int h = 0; h < kHeld; ++h) read(first + h * runs, held[h]);
#pragma unroll
      for (int h = 0; h < kHeld; ++h) larger(held[h]);
      for (int run = first + kHeld * runs; run < total; run += runs)
      {
        double x[8];
        read(run, x);
        larger(x);
      }
#pragma unroll
      for (int off = 8; off < 32; off <<= 1)
      {
        const unsigned long long o = __shfl_xor_sync(0xffffffffu, big, off);
        big = o > big ? o : big;
      }
      if ((threadIdx.x & 31) < 8) most[threadIdx.x >> 5][line] = big;
      __syncthreads();
      for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) big = most[w][line] > big ? most[w][line] : big;
      // its frexp exponent e: every |entry| < 2^e
      const int e = frexp_exponent(big);
      if (live && first == 0) (left ? exps_a : exps_b)[g.exp + line] = static_cast<int16_t>(e);
      const auto cut = [&](int run, const double (&x)[8])
      {
        // The first t + 1 digits are the integer rounded to nearest, halves up, at that place, so that any
        // number of slices is as near to the entry as it can be (fields of seven bits of the integer plus
        // half a unit of each digit, -64 to 63, are off by up to 0.504 of the last kept one); digit t is what
        // that prefix adds to the one before, of which 32 bits suffice.
        long long r[8];
        uint32_t prefix[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
        {
          r[j] = scaled_integer(x[j], 56 - e);
          prefix[j] = 0;
        }
        if (56 - e > kSubnormalScale)  // a line below the normal range
        {
#pragma unroll
          for (int j = 0; j < 8; ++j) r[j] *= 1ll << (56 - e - kSubnormalScale);
        }
        uint16_t *out = dst + static_cast<int64_t>(run >> 2) * g.step_stride + (run & 3) * 64;
#pragma unroll
        for (int t = 0; t < kMaxSlices; ++t)
        {
          if (t >= slices_n) break;
          uint32_t word[4];
#pragma unroll
          for (int j = 0; j < 8; ++j)
          {
            const int place = 49 - 7 * t;
            const uint32_t now = static_cast<uint32_t>((r[j] + ((1ll << place) >> 1)) >> place);
            const int q = static_cast<int>(now - (prefix[j] << 7));
            prefix[j] = now;
            // |q| <= 128: the fp32 of 12582912 + q holds q in its last bits, and q is exact in bf16
            const uint32_t f = __float_as_uint(__int_as_float(0x4b400000 + q) - 12582912.0f) >> 16;
            word[j >> 1] = j & 1 ? word[j >> 1] | f << 16 : f;
          }
          *reinterpret_cast<uint4 *>(out + static_cast<int64_t>(t) * g.slice_stride) = make_uint4(word[0], word[1], word[2], word[3]);
        }
      };
      if (!live) return;
#pragma unroll
      for (int h = 0; h < kHeld; ++h)
        if (first + h * runs < total) cut(first + h * runs, held[h]);
      for (int run = first + kHeld * runs; run < total; run += runs)
      {
        double x[8];
        read(run, x);
        cut(run, x);
      }
    }

    template <int S>
    __host__ __device__ constexpr int split_worker_bytes() { return 2 * S * (kSplitTileM + kSplitTileN) * kRow * 2; }

    // Persistent: kSplitWorkers workers of 128 threads (4 warps of 16 x 16), each computing 32 x 32
    // tiles of one pair over a K range.  All S slices of a 32-wide K step are staged in the worker's
    // shared memory with 16-byte cp.async, double buffered; every A and B slice fragment of a k16
    // step is loaded once with ldmatrix and reused for the S(S+1)/2 products.  Level sums stay exact
    // in fp32 for 256 of K and are then folded into FP64 with the pair's row and column scales: the
    // four leading levels exactly, the rest (weights <= 2^-42 of the first) through one fp32 sum.
    template <int S>
    __global__ void __launch_bounds__(kSplitWorkers * kWorkerThreads, 1)
      gemm_split_kernel(const uint16_t *__restrict__ sa_all, const uint16_t *__restrict__ sb_all,
                        const int16_t *__restrict__ exps_a, const int16_t *__restrict__ exps_b, double *__restrict__ C,
                        const DevBlock *__restrict__ blocks, const DevSplitPair *__restrict__ spairs,
                        const SplitItem *__restrict__ items, const int32_t *__restrict__ cta_begin, const GemmReduce *__restrict__ reduces,
                        int64_t n_reduces, double *__restrict__ partial, int *__restrict__ tickets,
                        const int32_t *__restrict__ relabel)
    {
      dependent_entry();
      extern __shared__ __align__(16) unsigned char smem_raw[];
      const int worker = threadIdx.x / kWorkerThreads, lt = threadIdx.x % kWorkerThreads;
      uint16_t *sA = reinterpret_cast<uint16_t *>(smem_raw + worker * split_worker_bytes<S>());  // [2][S][32][kRow]
      uint16_t *sB = sA + 2 * S * kSplitTileM * kRow;                                           // [2][S][32][kRow]
      __shared__ int flags[kSplitWorkers];
      const int warp = lt >> 5, lane = lt & 31;
      const int g = lane >> 2, tig = lane & 3;
      const int wm = warp >> 1, wn = warp & 1;
      __shared__ int next[kSplitWorkers];
      __shared__ int taken;
      if (threadIdx.x == 0) taken = 0;
      __syncthreads();
      const int64_t list_begin = cta_begin[blockIdx.x], list_end = cta_begin[blockIdx.x + 1];
      for (int64_t idx = list_begin + local_claim(worker, lt, next + worker, &taken); idx < list_end;
           idx = list_begin + local_claim(worker, lt, next + worker, &taken))
      {
        const SplitItem it = items[idx];
        const DevBlock blk = blocks[it.block];
        double acc[2][4] = {};
        const int r0 = it.m0 + wm * 16 + g, c0 = it.n0 + wn * 16 + tig * 2;
        // the warp's 16 x 16 quarter of the tile touches the block (warp-uniform)
        const bool live = it.m0 + wm * 16 < blk.m && it.n0 + wn * 16 < blk.n;
        if (it.pair >= 0 && it.k1 > it.k0)
        {
          const DevSplitPair sp = spairs[it.pair];
          const int rows = min(kSplitTileM, blk.m - it.m0), cols = min(kSplitTileN, blk.n - it.n0);
          const auto load = [&](int stage, int k) {
            int32_t stride_a, stride_b;
            const uint16_t *ga = sa_all + slice_place(sp.sa, blk.m, sp.ksteps, kSliceTileA, it.m0, k / kSplitStepK, stride_a);
            const uint16_t *gb = sb_all + slice_place(sp.sb, blk.n, sp.ksteps, kSliceTileB, it.n0, k / kSplitStepK, stride_b);
            const auto piece = [](int r, int q) { return (r >> 3) * kSliceGroup + q * 64 + (r & 7) * 8; };
            for (int c = lt; c < S * kSplitTileM * 4; c += kWorkerThreads)
            {
              const int t = c / (kSplitTileM * 4), r = (c / 4) % kSplitTileM, q = c % 4;
              const bool ok = r < rows;
              cp_async16(sA + ((stage * S + t) * kSplitTileM + r) * kRow + q * 8, ga + (ok ? t * stride_a + piece(r, q) : 0),
                         ok ? 16 : 0);
            }
            for (int c = lt; c < S * kSplitTileN * 4; c += kWorkerThreads)
            {
              const int u = c / (kSplitTileN * 4), r = (c / 4) % kSplitTileN, q = c % 4;
              const bool ok = r < cols;
              cp_async16(sB + ((stage * S + u) * kSplitTileN + r) * kRow + q * 8, gb + (ok ? u * stride_b + piece(r, q) : 0),
                         ok ? 16 : 0);
            }
            cp_async_commit();
          };
          const int steps = (it.k1 - it.k0 + kSplitStepK - 1) / kSplitStepK;
          long long acc_int[2][4] = {};
          float acc_tail[2][4] = {};
          float lev[S][2][4];
#pragma unroll
          for (int l = 0; l < S; ++l)
#pragma unroll
            for (int ns = 0; ns < 2; ++ns)
#pragma unroll
              for (int q = 0; q < 4; ++q) lev[l][ns][q] = 0.0f;
          const int er0 = r0 < blk.m ? exps_a[sp.ea + r0] : 0, er1 = r0 + 8 < blk.m ? exps_a[sp.ea + r0 + 8] : 0;
          int ec[2][2];
#pragma unroll
          for (int ns = 0; ns < 2; ++ns)
#pragma unroll
            for (int h = 0; h < 2; ++h) ec[ns][h] = c0 + ns * 8 + h < blk.n ? exps_b[sp.eb + c0 + ns * 8 + h] : 0;
          load(0, it.k0);
          for (int step = 0; step < steps; ++step)
          {
            const int stage = step & 1;
            if (step + 1 < steps)
            {
              load(stage ^ 1, it.k0 + (step + 1) * kSplitStepK);
              cp_async_wait<1>();
            }
            else
              cp_async_wait<0>();
            worker_sync(worker);
#pragma unroll
            for (int kk = 0; kk < kSplitStepK; kk += 16)
            {
              if (!live) break;
              uint32_t af[S][4], bf[S][4];
#pragma unroll
              for (int t = 0; t < S; ++t)
              {
                ldmatrix_x4(af[t], sA + ((stage * S + t) * kSplitTileM + wm * 16 + (lane & 15)) * kRow + kk + (lane >> 4) * 8);
                ldmatrix_x4(bf[t], sB + ((stage * S + t) * kSplitTileN + wn * 16 + (lane & 7) + ((lane >> 4) << 3)) * kRow +
                                     kk + ((lane >> 3) & 1) * 8);
              }
#pragma unroll
              for (int t = 0; t < S; ++t)
#pragma unroll
                for (int u = 0; u + t < S; ++u)
                {
                  mma_bf16(lev[t + u][0], af[t], bf[u][0], bf[u][1]);
                  mma_bf16(lev[t + u][1], af[t], bf[u][2], bf[u][3]);
                }
            }
            worker_sync(worker);
            if ((step + 1) % (kSplitChunk / kSplitStepK) == 0 || step + 1 == steps)
            {
              // the four leading levels are exact integers (below 2^24 over a chunk of <= 256 of K):
              // combined exactly in int64 as sum_l lev_l 2^(7 (3 - l)); the rest in fp32
#pragma unroll
              for (int ns = 0; ns < 2; ++ns)
#pragma unroll
                for (int q = 0; q < 4; ++q)
                {
                  float tail = 0.0f;
#pragma unroll
                  for (int l = S - 1; l >= 4; --l) tail = fmaf(lev[l][ns][q], ldexpf(1.0f, -7 * (l - 4)), tail);
                  long long head = 0;
#pragma unroll
                  for (int l = 0; l < 4; ++l)
                    head = head * 128 + (l < S ? static_cast<long long>(__float2int_rn(lev[l][ns][q])) : 0ll);
                  acc_int[ns][q] += head;
                  acc_tail[ns][q] += tail;
#pragma unroll
                  for (int l = 0; l < S; ++l) lev[l][ns][q] = 0.0f;
                }
            }
          }
          // one FP64 step per entry, and the row and column scales unless several items share the K of
          // the block's only pair
          const bool last = it.slot < 0 || blk.pair_count != 1;
#pragma unroll
          for (int ns = 0; ns < 2; ++ns)
#pragma unroll
            for (int q = 0; q < 4; ++q)
            {
              const double x = level_sum(acc_int[ns][q], acc_tail[ns][q]);
              acc[ns][q] = last ? scaled(x, (q < 2 ? er0 : er1) + ec[ns][q & 1]) : x;
            }
        }
        if (it.slot >= 0)
        {
          double *out = partial + static_cast<int64_t>(it.slot) * kSplitTileM * kSplitTileN;
#pragma unroll
          for (int ns = 0; ns < 2; ++ns)
#pragma unroll
            for (int q = 0; q < 4; ++q)
              out[(wm * 16 + g + (q >= 2 ? 8 : 0)) * kSplitTileN + wn * 16 + ns * 8 + tig * 2 + (q & 1)] = acc[ns][q];
          finish_partial<double, kSplitTileM, kSplitTileN>(
            worker, lt, flags + worker, tickets, reduces, it.reduce, blocks, partial, C, relabel,
            [&](double v, const DevBlock &b, int gm, int gn) {
              if (b.pair_count != 1) return v;
              const DevSplitPair sp = spairs[b.pair_begin];
              return scaled(v, exps_a[sp.ea + gm] + exps_b[sp.eb + gn]);
            });
          continue;
        }
#pragma unroll
        for (int ns = 0; ns < 2; ++ns)
#pragma unroll
          for (int q = 0; q < 4; ++q)
          {
            const int gm = r0 + (q >= 2 ? 8 : 0), gn = c0 + ns * 8 + (q & 1);
            if (gm >= blk.m || gn >= blk.n) continue;
            const int64_t at = blk.c + static_cast<int64_t>(gm) * blk.n + gn;
            if (!relabel)
              C[at] = acc[ns][q];
            else if (relabel[at] >= 0)
              C[relabel[at]] = acc[ns][q];  // straight to its place after the leg move that follows
          }
        const int64_t entries = static_cast<int64_t>(blk.m) * blk.n;
        if (!relabel && lt == 0 && it.m0 + kSplitTileM >= blk.m && it.n0 + kSplitTileN >= blk.n && (entries & 1))
          C[blk.c + entries] = 0.0;
      }
    }


    // Shared memory that holds one CTA per SM: at least 120 KiB, so a second never fits beside it.
    constexpr int kPinBytes = 120 * 1024;

    template <typename K>
    cudaError_t configure(K kernel, int bytes, std::once_flag &once)
    {
      cudaError_t e = cudaSuccess;
      std::call_once(once, [&] { e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); });
      return e;
    }

    template <int S>
    cudaError_t launch_split_s(const uint16_t *sa, const uint16_t *sb, const int16_t *exps_a, const int16_t *exps_b, double *C, const DevBlock *blocks, const DevSplitPair *spairs,
                               const SplitItem *items, const int32_t *cta_begin, int32_t n_ctas, int64_t longest,
                               const GemmReduce *reduces, int64_t n_reduces, double *partial, int *tickets,
                               const int32_t *relabel, cudaStream_t stream)
    {
      const int bytes = std::max(kSplitWorkers * split_worker_bytes<S>(), kPinBytes);
      static std::once_flag once;
      cudaError_t e = configure(gemm_split_kernel<S>, bytes, once);
      if (e != cudaSuccess) return e;
      // one CTA per list the schedule dealt, as many workers as its longest list needs
      const int workers = static_cast<int>(std::clamp<int64_t>(longest, 1, kSplitWorkers));
      return launch_dependent(gemm_split_kernel<S>, n_ctas, workers * kWorkerThreads, bytes, stream, sa, sb, exps_a, exps_b,
                              C, blocks, spairs, items, cta_begin, reduces, n_reduces, partial, tickets,
                              relabel);
    }
  } // namespace

  // ------------------------------------------------------------------------------------------
  // launchers
  // ------------------------------------------------------------------------------------------

  namespace
  {
    // The FP64 tables of a GEMM op, built on its first FP64 launch.
    cudaError_t ensure_f64(const Program &p, DeviceTables &t, size_t op_index, bool complex)
    {
      std::lock_guard<std::mutex> lock(t.mutex);
      DeviceTables::GemmTables &dst = (complex ? t.gemm_complex : t.gemm)[op_index];
      if (dst.ready) return cudaSuccess;
      const int tile = complex ? lanes_tile(p, p.ops[op_index]) : kF64TileM;
      dst.tile = tile;
      const GemmSchedule s = schedule_gemm(p, p.ops[op_index], tile, tile, true, complex);

      dst.n_items = static_cast<int64_t>(s.items.size());
      dst.n_reduces = static_cast<int64_t>(s.reduces.size());
      dst.slots = s.slots;
      dst.n_ctas = static_cast<int32_t>(s.cta_begin.size()) - 1;
      dst.longest = 0;
      for (size_t c = 0; c + 1 < s.cta_begin.size(); ++c)
        dst.longest = std::max<int64_t>(dst.longest, s.cta_begin[c + 1] - s.cta_begin[c]);
      TableStaging staging;
      staging.add(s.items, reinterpret_cast<void **>(&dst.items));
      staging.add(s.reduces, reinterpret_cast<void **>(&dst.reduces));
      staging.add(s.cta_begin, reinterpret_cast<void **>(&dst.cta_begin));
      const cudaError_t e = staging.commit(&dst.base);
      if (e != cudaSuccess) return e;
      dst.ready = true;
      return cudaSuccess;
    }
  } // namespace

  cudaError_t launch_gemm_f64(const Program &p, DeviceTables &t, size_t op_index, const void *A, const void *B, void *C,
                              bool complex, void *scratch, int *ticket_region, cudaStream_t stream)
  {
    if (const cudaError_t built = ensure_f64(p, t, op_index, complex); built != cudaSuccess) return built;
    const auto &sched = (complex ? t.gemm_complex : t.gemm)[op_index];
    if (sched.n_items == 0) return cudaSuccess;
    const auto *blocks = reinterpret_cast<const DevBlock *>(t.blocks);
    const auto *pairs = reinterpret_cast<const DevPair *>(t.pairs);
    char *base = static_cast<char *>(scratch);
    void *partial = base;
    // the workspace's ticket region (zero, and left zero by the kernel) when it holds them all,
    // else tickets of our own in the scratch, cleared first
    int *tickets = ticket_region;
    cudaError_t e = cudaSuccess;
    if (sched.n_reduces > kTicketInts)
    {
      tickets = reinterpret_cast<int *>(base + up256(sched.slots * sched.tile * sched.tile * (complex ? 16 : 8)));
      if ((e = cudaMemsetAsync(tickets, 0, static_cast<size_t>(sched.n_reduces) * 4, stream)) != cudaSuccess) return e;
    }
    // one CTA per list the schedule dealt, as many workers as its longest list needs (at most four)
    const int grid = sched.n_ctas;
    const int workers = static_cast<int>(std::clamp<int64_t>(sched.longest, 1, kF64Workers));
    if (complex)
    {
      const bool large = sched.tile != kLanesTile;
      const auto kernel = large ? gemm_c128_kernel<2 * kLanesTile> : gemm_c128_kernel<kLanesTile>;
      const int bytes = std::max<int>(lanes_bytes(sched.tile), kPinBytes);
      static std::once_flag once[2];
      if ((e = configure(kernel, bytes, once[large])) != cudaSuccess) return e;
      e = launch_dependent(kernel, grid, workers * kWorkerThreads, bytes, stream,
                           static_cast<const double2 *>(A), static_cast<const double2 *>(B), static_cast<double2 *>(C), blocks,
                           pairs, static_cast<const GemmItem *>(sched.items), static_cast<const int32_t *>(sched.cta_begin),
                           static_cast<const GemmReduce *>(sched.reduces), sched.n_reduces, static_cast<double2 *>(partial),
                           tickets);
    }
    else
    {
      const int bytes = std::max<int>(kF64Workers * 2 * 2 * kDmmaStepK * 36 * 8, kPinBytes);
      static std::once_flag once;
      if ((e = configure(gemm_dmma_kernel, bytes, once)) != cudaSuccess) return e;
      e = launch_dependent(gemm_dmma_kernel, grid, workers * kWorkerThreads, bytes, stream, static_cast<const double *>(A),
                           static_cast<const double *>(B), static_cast<double *>(C), blocks, pairs,
                           static_cast<const GemmItem *>(sched.items), static_cast<const int32_t *>(sched.cta_begin),
                           static_cast<const GemmReduce *>(sched.reduces), sched.n_reduces, static_cast<double *>(partial),
                           tickets);
    }
    return e;
  }

  namespace
  {
    // The split tables of a GEMM op, built on its first split use.
    cudaError_t ensure_split(const Program &p, const Op &op, DeviceTables &t, size_t op_index)
    {
      std::lock_guard<std::mutex> lock(t.mutex);
      DeviceTables::SplitTables &dst = t.split[op_index];
      if (dst.ready) return cudaSuccess;
      const SplitSchedule s = schedule_split(p, op, true);
      dst.n_items = static_cast<int64_t>(s.items.size());
      dst.n_reduces = static_cast<int64_t>(s.reduces.size());
      dst.n_groups_a = s.groups_a;
      dst.n_groups_b = static_cast<int64_t>(s.groups.size()) - s.groups_a;
      dst.longest_line = s.longest_line;
      dst.partial_bytes = split_partial_bytes(s, schedule_tc(p, op));
      dst.slice_a = s.slice_a;
      dst.slice_b = s.slice_b;
      dst.exps_a = s.exps_a;
      dst.exps = s.exps;
      dst.slots = s.slots;
      dst.n_ctas = static_cast<int32_t>(s.cta_begin.size()) - 1;
      dst.longest = 0;
      for (size_t c = 0; c + 1 < s.cta_begin.size(); ++c)
        dst.longest = std::max<int64_t>(dst.longest, s.cta_begin[c + 1] - s.cta_begin[c]);
      TableStaging staging;
      staging.add(s.cta_begin, reinterpret_cast<void **>(&dst.cta_begin));
      staging.add(s.items, &dst.items);
      staging.add(s.reduces, reinterpret_cast<void **>(&dst.reduces));
      staging.add(s.pairs, &dst.pairs);
      staging.add(s.groups, &dst.groups);
      DeviceTables::TcTables &tc = t.tc[op_index];
      const TcSchedule ts = schedule_tc(p, op, &s.pairs);
      staging.add(ts.items, &tc.items);
      staging.add(ts.reduces, reinterpret_cast<void **>(&tc.reduces));
      tc.n_ctas = ts.ctas;
      tc.longest = ts.longest;
      tc.n = ts.n;
      // Products of one step of K whose tiles do not go by it but by their end: a 128 x 64 tile takes an SM about
      // 10.5 us (22 with the FP64 sums of seven and eight slices), a 32 x 32 one on mma.sync 3.65 (3.1), so blocks of
      // few rows and many columns, a tile mostly padding, run there: 8 x 30000 x 3 with six slices 36 us, 51 on
      // tcgen05 (eight: 38 and 86); 30000 x 8 x 3 44 and 32, 4000 x 4000 x 16 375 and 141 (eight: 313 and 295).
      // Up to a tile an SM both are latency.
      int64_t tiles = 0, small = 0;
      for (int64_t b = op.begin; b < op.begin + op.count; ++b)
      {
        const GemmBlock &blk = p.gemm_blocks[static_cast<size_t>(b)];
        tiles += static_cast<int64_t>((blk.m + kSliceTileA - 1) / kSliceTileA) * ((blk.n + ts.n - 1) / ts.n);
        small += static_cast<int64_t>((blk.m + kSplitTileM - 1) / kSplitTileM) * ((blk.n + kSplitTileN - 1) / kSplitTileN);
      }
      if (s.longest_line <= kSplitStepK && tiles > p.ctas)
      {
        tc.padding[0] = 3.65 * small < 10.5 * tiles;
        tc.padding[1] = 3.1 * small < 22.0 * tiles;
      }
      const cudaError_t e = staging.commit(&dst.base);
      if (e != cudaSuccess) return e;
      dst.ready = true;
      return cudaSuccess;
    }

    cudaError_t launch_groups(const DeviceTables::SplitTables &sched, const double *A, const double *B, uint16_t *sa,
                              uint16_t *sb, int16_t *exps_a, int16_t *exps_b, int64_t begin, int64_t end, int slices,
                              cudaStream_t stream)
    {
      if (begin >= end) return cudaSuccess;
      // threads for a whole line of 8 x 8 entries a thread, four warps at least
      const int threads = sched.longest_line > 128 ? 256 : 128;
      return launch_dependent(split_groups_kernel, static_cast<unsigned>(end - begin), threads, 0, stream, A, B, sa, sb, exps_a,
                              exps_b, static_cast<const SplitGroup *>(sched.groups), sched.n_groups_a, begin, slices);
    }
  } // namespace

  cudaError_t fill_slice_caches(const Program &p, DeviceTables &t, int32_t operand, const void *arena, cudaStream_t stream)
  {
    if (!p.gemm_plans) return cudaSuccess;
    for (const SliceCache &c : p.gemm_plans->caches)
    {
      if (c.operand != operand) continue;
      const Op &op = p.ops[static_cast<size_t>(c.op)];
      cudaError_t e = ensure_split(p, op, t, static_cast<size_t>(c.op));
      if (e != cudaSuccess) return e;
      const auto &sched = t.split[static_cast<size_t>(c.op)];
      if (sched.n_items == 0) continue;
      char *base = static_cast<char *>(const_cast<void *>(arena));
      auto *slices = reinterpret_cast<uint16_t *>(base + c.offset);
      auto *exps = reinterpret_cast<int16_t *>(base + c.exps_offset);
      const auto *value = static_cast<const double *>(arena);
      e = c.side == 0 ? launch_groups(sched, value, nullptr, slices, nullptr, exps, nullptr, 0, sched.n_groups_a, kMaxSlices, stream)
                      : launch_groups(sched, nullptr, value, nullptr, slices, nullptr, exps, sched.n_groups_a,
                                      sched.n_groups_a + sched.n_groups_b, kMaxSlices, stream);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }

  cudaError_t launch_gemm_split(const Program &p, const Op &op, DeviceTables &t, size_t op_index, const double *A,
                                const double *B, double *C, int32_t slices, void *scratch, int *ticket_region,
                                const void *const *prepared, cudaStream_t stream, const int32_t *relabel, bool tensor_cores)
  {
    cudaError_t e = ensure_split(p, op, t, op_index);
    if (e != cudaSuccess) return e;
    const auto &sched = t.split[op_index];
    if (sched.n_items == 0) return cudaSuccess;
    char *base = static_cast<char *>(scratch);
    auto *sa = reinterpret_cast<uint16_t *>(base);
    base += up256(2 * sched.slice_a);
    auto *sb = reinterpret_cast<uint16_t *>(base);
    base += up256(2 * sched.slice_b);
    auto *exps_a = reinterpret_cast<int16_t *>(base);
    auto *exps_b = exps_a + sched.exps_a;
    base += up256(2 * sched.exps);
    auto *partial = reinterpret_cast<double *>(base);
    base += sched.partial_bytes;
    // a side whose operand's prepared arena the caller holds was cut when the arena was prepared
    int64_t begin = 0, end = sched.n_groups_a + sched.n_groups_b;
    if (p.gemm_plans && prepared)
    {
      const int32_t ca = p.gemm_plans->cache_a[op_index], cb = p.gemm_plans->cache_b[op_index];
      if (ca >= 0 && prepared[p.gemm_plans->caches[static_cast<size_t>(ca)].operand])
      {
        const SliceCache &c = p.gemm_plans->caches[static_cast<size_t>(ca)];
        char *arena = static_cast<char *>(const_cast<void *>(prepared[c.operand]));
        sa = reinterpret_cast<uint16_t *>(arena + c.offset);
        exps_a = reinterpret_cast<int16_t *>(arena + c.exps_offset);
        begin = sched.n_groups_a;
      }
      if (cb >= 0 && prepared[p.gemm_plans->caches[static_cast<size_t>(cb)].operand])
      {
        const SliceCache &c = p.gemm_plans->caches[static_cast<size_t>(cb)];
        char *arena = static_cast<char *>(const_cast<void *>(prepared[c.operand]));
        sb = reinterpret_cast<uint16_t *>(arena + c.offset);
        exps_b = reinterpret_cast<int16_t *>(arena + c.exps_offset);
        end = sched.n_groups_a;
      }
    }
    if ((e = launch_groups(sched, A, B, sa, sb, exps_a, exps_b, begin, end, slices, stream)) != cudaSuccess) return e;
    static const bool tc_enabled = []
    {
      const char *v = std::getenv("TENTORCH_GB300_TCGEN05");
      return !(v && v[0] == '0');
    }();
    if (tc_enabled && tensor_cores && !t.tc[op_index].padding[slices > 6])
      return launch_split_tc(t, op_index, slices, sa, sb, exps_a, exps_b, sched.pairs, C, partial, ticket_region, relabel,
                             stream);
    int *tickets = ticket_region;
    if (sched.n_reduces > kTicketInts)
    {
      tickets = reinterpret_cast<int *>(base);
      if ((e = cudaMemsetAsync(tickets, 0, static_cast<size_t>(sched.n_reduces) * 4, stream)) != cudaSuccess) return e;
    }
    const auto *blocks = reinterpret_cast<const DevBlock *>(t.blocks);
    const auto *spairs = reinterpret_cast<const DevSplitPair *>(sched.pairs);
    const auto *items = reinterpret_cast<const SplitItem *>(sched.items);
    switch (slices)
    {
#define TTG_SPLIT(S)                                                                                                    \
  case S:                                                                                                               \
    e = launch_split_s<S>(sa, sb, exps_a, exps_b, C, blocks, spairs, items,                                             \
                          sched.cta_begin, sched.n_ctas, sched.longest, sched.reduces, sched.n_reduces, partial, tickets,  \
                          relabel, stream);                                                                             \
    break;
      TTG_SPLIT(1) TTG_SPLIT(2) TTG_SPLIT(3) TTG_SPLIT(4) TTG_SPLIT(5) TTG_SPLIT(6) TTG_SPLIT(7) TTG_SPLIT(8)
#undef TTG_SPLIT
    default: return cudaErrorInvalidValue;
    }
    return e;
  }

  // The device copies of every GEMM op's schedules and slicing lines, staged into the program's
  // one table allocation.
  void stage_gemm(const Program &p, DeviceTables &t, TableStaging &staging)
  {
    t.gemm.assign(p.ops.size(), {});
    t.gemm_complex.assign(p.ops.size(), {});
    t.split.assign(p.ops.size(), {});
    t.tc.assign(p.ops.size(), {});
    if (!p.gemm_plans) return;
    for (size_t i = 0; i < p.ops.size(); ++i)
    {
      if (p.ops[i].kind != OpKind::gemm) continue;
      // the FP64 tables are built on the op's first FP64 launch (ensure_f64)
    }
  }

} // namespace ttg

// Grouped block-pair GEMM schedules and launchers.
//
// A GEMM op of a program computes every output block C_b = sum over its pairs A_p B_p.  Its output
// tiles are cut into work items of roughly equal multiply-add count, each covering a contiguous
// range of the tile's K (concatenated over the tile's pairs), so one long block product is spread
// over many SMs.  An item that covers its whole tile writes C; otherwise it writes a partial tile
// to scratch and a reduction sums the partials of the tile in a fixed order (deterministic, no
// atomics).
//
// Split precision (gemm.cu): every row of A and column of B is scaled by a power of two so that
// its entries lie in [-1, 1], then cut into `s` slices of 7 bits held exactly as bf16 integers
// (|q_1| <= 128, |q_t| <= 64).  The products of slices are sums of integers that fp32 accumulates
// exactly over a K-chunk (kExactChunk), so the only rounding is the final FP64 combination and the
// truncation after s slices (about 2^-7s of the row and column maxima): Ozaki's error-free
// splitting (K. Ozaki, T. Ogita, S. Oishi, S. M. Rump, Numer. Algorithms 59 (2012)) on bf16
// tensor cores with fp32 accumulation.
#pragma once

#include <cstdint>
#include <vector>

#include "program.h"

namespace ttg
{
  struct GemmItem
  {
    int32_t block, m0, n0, k0, k1, slot;  // slot -1: the item covers its tile and writes C
    int32_t reduce, pad;                   // the tile's GemmReduce when slot >= 0
  };
  struct GemmReduce
  {
    int32_t block, m0, n0, slot0, nslots, pad;
  };
  struct GemmSchedule
  {
    std::vector<GemmItem> items;     // grouped by the CTA that runs them
    std::vector<GemmReduce> reduces;
    std::vector<int32_t> cta_begin;  // CTA b runs items [cta_begin[b], cta_begin[b + 1])
    int64_t slots = 0;               // partial tiles of bm x bn doubles
    int64_t n_items = 0;             // items (also when only the sizes were computed)
  };
  // The SMs of the current device (cached per device), or 152, a GB300's count, when no device is
  // visible (plans compiled on a host without a GPU).  A plan's persistent GEMM launches spread
  // their items over this many CTAs, one per SM (Program::ctas, fixed when the plan is compiled).
  int device_sms();

  // Split precision works pair by pair: an item is one pair's K range (a multiple of 32 long, but
  // for the pair's last one), so a tile with several pairs or chunks always goes through partials.
  struct SplitItem
  {
    int32_t block, m0, n0, pair, k0, k1, slot, reduce;
  };
  // Where a pair's slices and exponents sit in scratch.  The rows of A and the columns of B ("lines")
  // are cut into kMaxSlices slices and kept in the order the tensor cores read them: lines in tiles of
  // kSliceTileA (A) or kSliceTileB (B), K in steps of 32; per tile and step the slices one after
  // another, each as groups of 8 lines x 32 of K (512 bytes: four runs of 8 lines x 16 bytes, the
  // core matrices of tcgen05's K-major layout without swizzle).  A tile over one step is then one
  // contiguous piece a slice, which a bulk copy brings into shared memory as the products read it;
  // the last tile of a block keeps only the groups it has (slice_place below).
  struct SplitPair
  {
    int64_t sa, sb;  // elements: the first tile of the A lines, of the B lines
    int32_t ksteps, ea, eb, pad;
  };
  // Up to eight lines to slice together.
  struct SplitGroup
  {
    int64_t src, dst;                   // the first line's first entry; its place in the first step's first slice
    int32_t len, line_step, entry_step; // entries a line, source elements between lines and between entries
    int32_t lines, exp;                 // lines in the group, the first one's exponent
    int32_t slice_stride, step_stride, pad;  // elements between slices, between steps of K
  };
  struct SplitSchedule
  {
    std::vector<SplitItem> items;
    std::vector<GemmReduce> reduces;
    std::vector<SplitPair> pairs;    // one per GemmPair of the program (only this op's are filled)
    std::vector<SplitGroup> groups;  // rows of A then columns of B
    int64_t groups_a = 0;
    int64_t slice_a = 0, slice_b = 0;  // elements of all slices of A (B)
    int64_t exps_a = 0, exps_b = 0;    // int16 exponents of the rows of A, of the columns of B
    int64_t exps = 0;                  // both
    int64_t slots = 0;
    int64_t longest_line = 0;          // the longest K
    std::vector<int32_t> cta_begin;    // CTA b runs items [cta_begin[b], cta_begin[b + 1])
  };
  // The split-precision schedule of a GEMM op; with full = false only its sizes (slices, exponents,
  // partial slots, reductions), for sizing the scratch without building its tables.
  SplitSchedule schedule_split(const Program &p, const Op &op, bool full = true);

  // Tile sizes of the two kernels.
  constexpr int kF64TileM = 32, kF64TileN = 32;
  constexpr int kLanesTile = 16;  // rows and columns of a complex128 tile (or twice these: gemm.cu lanes_tile)
  constexpr int kDmmaStepK = 32;  // K staged per step (two stages in flight) in the DMMA kernel
  constexpr int kSplitTileM = 32, kSplitTileN = 32, kSplitStepK = 32;
  // Persistent launches: one CTA per SM (held there by its shared memory), several workers of 128
  // threads per CTA taking items round robin.
  constexpr int kF64Workers = 4, kSplitWorkers = 2, kWorkerThreads = 128;
  constexpr int kMaxSlices = 8;
  // K over which the sums of slice products stay integers of at most 2^24, which fp32 adds exactly:
  // level l sums 2^12 (l + 3) a K at most (2^14 for l = 0), so 512 holds through level 5.  Levels 6
  // and 7 weigh 2^-14 and less of level 4, whose rounding theirs stays below.
  constexpr int kExactChunk = 512;
  constexpr int kSplitChunk = 256;  // the K after which the mma.sync kernel folds its level sums
  constexpr int kSliceTileA = 128, kSliceTileB = 64;  // lines of a tile of slices
  constexpr int kSliceGroup = 8 * 32;                 // elements of eight lines over 32 of K

  // The element of the first slice of line `line` (a multiple of 8) at a step of K, for `lines` lines
  // starting at `base` in tiles of `tile`; the elements between slices there in `slice_stride`.
#ifdef __CUDACC__
  __host__ __device__
#endif
  inline int64_t slice_place(int64_t base, int32_t lines, int32_t ksteps, int32_t tile, int32_t line, int32_t step,
                             int32_t &slice_stride)
  {
    const int32_t t = line / tile, full = tile / 8, left = (lines - t * tile + 7) / 8;
    const int32_t groups = left < full ? left : full;
    slice_stride = groups * kSliceGroup;
    return base + (static_cast<int64_t>(t) * ksteps * full + static_cast<int64_t>(step) * groups) * kMaxSlices * kSliceGroup +
           static_cast<int64_t>((line - t * tile) / 8) * kSliceGroup;
  }

  // The work of split products on the tensor cores (split_tc.cu): an item is a 128 x n output tile
  // over steps [s0, s1) of 32 of K (its block's pairs one after another, each in whole steps).  It
  // carries its block and first pair, so that a CTA has all it needs of most tiles after one read.
  struct TcItem
  {
    int64_t c, sa, sb;                 // the block's place in C, the first pair's slices (SplitPair)
    int32_t m, n, m0, n0;              // the block, the tile's corner; m 0 ends a CTA's list
    int32_t s0, s1, slot, reduce;
    int32_t pair_begin, pair_count;
    int32_t k, ksteps, ea, eb;         // the first pair
  };
  struct TcSchedule
  {
    std::vector<TcItem> items;  // `longest` places a CTA, its list and then items of m 0
    std::vector<GemmReduce> reduces;
    int32_t ctas = 0, longest = 0;
    int32_t n = 64;     // columns of a tile
    int64_t slots = 0;  // partial tiles of 128 x n doubles
  };
  // With `pairs` (the op's, from schedule_split) the whole schedule, else its sizes.
  TcSchedule schedule_tc(const Program &p, const Op &op, const std::vector<SplitPair> *pairs = nullptr);

  // The FP64 schedule of a GEMM op; with full = false only its sizes (items, partial slots,
  // reductions), for sizing the scratch: the items are dealt on the op's first FP64 launch.
  // `lanes`: costed for the FMA-lane kernel (complex128) rather than DMMA fragments; `whole`: no tile is
  // cut along K.
  GemmSchedule schedule_gemm(const Program &p, const Op &op, int bm, int bn, bool full = true, bool lanes = false, bool whole = false);
  // The partial tiles (32 x 32 doubles each) the one launch of a program's product chain may hold
  // (chain.cu; 0 without a chain).
  int64_t chain_partial_slots(const Program &p);
  // The key of a plan's block-size histogram (autotune.cpp).
  uint64_t tune_key(const Program &p);

  // Scratch doubles a program's GEMM ops need at most (FP64 partials, or slices + exponents +
  // partials for split precision), laid out per op from offset 0.
  // Per op of a program (empty for the ops that are not GEMMs): the FP64 and the split schedules.
  // The slices of a GEMM operand that is an operand's prepared value (fixed while the arena is
  // unchanged: the head and tail of a Lanczos window) are cut once, when the arena is prepared,
  // into the arena after the prepared value: kMaxSlices slices (any fewer are a prefix of them)
  // and the exponents, in the order of SplitPair.
  struct SliceCache
  {
    int32_t op;       // the GEMM op
    int32_t side;     // 0: its A (rows), 1: its B (columns)
    int32_t operand;  // whose prepared arena holds it
    int64_t offset;   // bytes into that arena: the slices, then the exponents at exps_offset
    int64_t exps_offset;
    int64_t bytes;
  };
  struct GemmPlans
  {
    std::vector<GemmSchedule> f64;
    std::vector<SplitSchedule> split;
    std::vector<SliceCache> caches;
    std::vector<int32_t> cache_a, cache_b;  // per op: its A's (B's) cache, -1 for none
    std::vector<int64_t> prepared_bytes;    // per operand: bytes of its prepared arena with caches
  };
  // Schedule every GEMM op of the program into p.gemm_plans and return the scratch elements the
  // launches need (partial tiles, tickets, slices).
  int64_t plan_gemms(Program &p);

  // Find a product -> leg move -> product chain among the program's ops (Program::chain_*), from
  // the ops alone; whether the move is a one-to-one relabelling is checked on its first launch.
  void detect_chain(Program &p);
  // One FP64 work item of a chain: stage 0 items belong to the first product (their results go to
  // the moved layout), stage 1 items to the second (they start once every stage 0 tile is done).
  struct ChainItem
  {
    int32_t stage, block, m0, n0, k0, k1, slot, reduce, window, pad;  // window: the program of a batched launch
  };
  struct ChainReduce
  {
    int32_t stage, block, m0, n0, slot0, nslots, pad0, pad1;
  };
  // Programs a batched chain launch takes at most (tt_plan_execute_batch).
  constexpr int kChainBatch = 64;

  // The distinct left blocks (offset, rows, cols) and right blocks of one GEMM op.
  struct OperandBlock
  {
    int64_t offset;
    int32_t rows, cols;
  };
  void gemm_operands(const Program &p, const Op &op, std::vector<OperandBlock> &left, std::vector<OperandBlock> &right);

} // namespace ttg

// How pt_gemm splits a product over blocks, and what a block takes of its SM.  Host arithmetic alone: a plain C++ compiler takes this file.
#pragma once
#include <algorithm>
#include <cstdint>

namespace pt {
namespace tc {

constexpr int BM = 128;            // weight rows per CTA
constexpr int BKB = 128;           // bytes of k per stage and operand row (one 128-byte swizzle atom)
constexpr int MAX_CLUSTER = 8;     // k-slices of a tile (one cluster)
constexpr int A_TILE = BM * BKB;   // 16 KB: 128 rows x 128 bytes of k, 128-byte swizzle
constexpr int RAW_TILE = BM * 32;  // 4 KB: 128 rows x 64 k of packed nibbles
constexpr int RAW_STEP = 2 * RAW_TILE;   // a step of the INT4 kernel: 128 k

// A block waits without a limit in two places: for tensor memory that another block of its SM holds, and, if its tile has k-slices, for the
// other blocks of its cluster.  Launches of several streams share the SMs, so that these two waits must not close a circle whatever
// products meet: a block that holds columns and waits for its cluster, whose other block waits for columns of the same kind elsewhere.
// It cannot if at most two blocks of these kernels fit an SM and two that may be in clusters always find their columns.  So every block
// takes at least SHARED_SMEM, which leaves no room for a third, and one that takes all 512 columns and may be in a cluster takes ALONE_SMEM, beside
// which none fits.  (Blocks without a cluster wait for nobody while they hold columns.)
constexpr uint32_t SM_SMEM = 228 * 1024, BLOCK_RESERVE = 1024;      // shared memory of an SM, and what the system takes of it for each block
constexpr uint32_t SHARED_SMEM = 89 * 1024, ALONE_SMEM = 138 * 1024, PAIR_SMEM = 120 * 1024;
constexpr int SM_COLUMNS = 512;
static_assert(3 * (SHARED_SMEM + BLOCK_RESERVE) > SM_SMEM, "three blocks on an SM");
static_assert(ALONE_SMEM + SHARED_SMEM + 2 * BLOCK_RESERVE > SM_SMEM, "a block beside one that takes all columns");
static_assert(2 * PAIR_SMEM + 2 * BLOCK_RESERVE > SM_SMEM, "two blocks of two accumulators of 256 columns");

struct GemmAsk {
  bool int4, bf16, fp16;
  int m, n_out, k_in;
  int ksplit;              // 0: chosen here
  int group_rows;          // grouped weights (BF16): rows of a tile; 0: not grouped
  int sms;
};
struct GemmPlan {
  bool fits;
  int mb, n_tiles, m_tiles;        // activation rows of a tile (a multiple of 16, at most 256), tiles
  int n_kb, ksplit, kb_per_split;  // k blocks (of 128 bytes of operand row; INT4: of 128 k), k-slices, k blocks of a slice
  int na;                          // weight tiles of a block
  int int4_groups;                 // groups of transform warps
  int stages, raw_stages, threads;
  int tmem_columns;
  bool x_warps;                    // warps fetch the activations, not TMA
  bool sent, few;                  // the slices send their sums to the block that writes them, otherwise it fetches them; that, or a whole tile of so few rows
  uint32_t sum_offset;             // where the slices' sums arrive behind the operands (0: in their place)
  uint32_t stage_bytes, smem;
};

constexpr int gemm_ceil(int a, int b) { return (a + b - 1) / b; }

// Tiles of the INT4 kernel.  A CTA spends on a step (128 k) the longer of transform and single-thread roles (about 350 cycles) and MMAs (4 mb
// cycles), then its epilogue, and the CTAs run in rounds over the SMs: of all row counts per tile (steps of 16) and k-slices the pair with
// the least time by this count is taken.
struct Int4Plan { int mb, ksplit; };
static inline Int4Plan plan_int4(int m, int n_tiles, int n_steps, int ksplit_req, int sms) {
  Int4Plan best{16, 1};
  double least = 1e30;
  for (int mb = 16; mb <= 256; mb += 16) {
    const int m_tiles = gemm_ceil(m, mb);
    if (mb > 16 && m_tiles == gemm_ceil(m, mb - 16)) continue;    // fewer rows per tile do as well
    for (int ks = 1; ks <= MAX_CLUSTER; ++ks) {
      if (ksplit_req > 0 ? ks != std::min(std::min(ksplit_req, MAX_CLUSTER), n_steps) : ks > 1 && n_steps / ks < 4) continue;
      const long long ctas = (long long)n_tiles * m_tiles * ks, rounds = (ctas + sms - 1) / sms;
      const double t = (double)rounds * (gemm_ceil(n_steps, ks) * (double)std::max(350, 4 * mb) + 1500 + 8 * mb) + (ks > 1 ? 2500 + 6 * mb : 0);
      if (t < least) { least = t; best = {mb, ks}; }
    }
  }
  return best;
}

// How many k-slices, of at most `most`, save more than their sums cost: 0.2 us for a k block that a CTA does not have to take (more above 128
// rows, where the MMAs are the longer part) against half a microsecond and (8 + 44 / slices) ns per row of the tile for the meetings of the
// cluster.  Fitted on B200 to 768 x 384 .. 8192 and 4096 x 384 .. 8192 in FP8 at 8 .. 512 rows, us whole and in 2 and 4 slices: 768 x 768 at 16 rows 4.3, 4.7, 4.3;
// at 256 rows 7.8, 14.9, 12.2; 768 x 4096 at 16 rows 9.8, 7.6, 5.6; at 256 rows 15.3, 18.8, 12.7 (8 slices 11.1).
// (Sums that are sent, see below, make slices of few rows cheaper, and the line still holds: 768 x 768 at 16 rows whole, 2 and 4 slices 3.2, 3.5, 3.4; 768 x 4096 at
// 16 rows 8.6, 6.4, 4.4, 8 slices 3.8.)
// A BF16 tile whose rows are no multiple of 32 leaves element by element when it is whole: a microsecond more.
static inline int slices_that_pay(int most, int n_kb, int mb, bool slow_whole) {
  const double block = 200.0 + (mb > 128 ? 1.1 * (mb - 128) : 0.0);
  int best = 1;
  double most_saved = slow_whole ? -1000.0 : 0.0;
  for (int s = 2; s <= most; ++s) {
    const double saved = block * (n_kb - gemm_ceil(n_kb, s)) - 500.0 - mb * (8.0 + 44.0 / s);
    if (saved > most_saved) { most_saved = saved; best = s; }
  }
  return best;
}

// Which slices' sums are sent to the block that writes them, and which are fetched by it (gemm_tc.cu).  Sent sums save two meetings of the cluster, but the four warps of a
// block that sum them take group after group of four rows: worth it up to 32 rows and where a block has at most two groups, with a short k one (three if they leave as fp16).  us sent / fetched / before
// there was sending, BF16: 2048 x 2048 at 24 rows in 8 slices 4.5 / 5.2 / 5.2, 1600 x 1600 in 7 4.4 / 5.4 / 5.2, 8192 x 1024 in 4 6.2 / 6.7 / 6.4; but 2304 x 768 in 4 4.6 / 4.1 / 4.1,
// 2048 x 512 in 2 5.0 / 4.5 / 4.3; at 64 rows 10304 x 2048 in 3 13.6 / 11.9 / 12.0, 2048 x 2048 in 8 7.1 / 7.0 / 6.8.  FP8 12288 x 4096 at 9 rows in 2 10.5 / 11.1 / 11.1.
// INT4, whose eight or sixteen warps sum, up to 64 rows (on average over 11 sizes 24 to 48 rows 4 % less than fetched; 64 rows level).
constexpr int SENT_ROWS = 32, SENT_ROWS_INT4 = 64;
// Shared memory for the sums of the slices that are sent: a block's share of the groups of four rows, from every slice.  Behind the operands where that takes at most
// SUM_SMEM, so that a block can send before the one that sums has finished its products.
constexpr uint32_t SUM_SMEM = 32 * 1024;
static inline uint32_t sum_bytes(int mb, int ksplit) { return ksplit > 1 ? (uint32_t)gemm_ceil(mb / 4, ksplit) * ksplit * BM * 16 : 0; }

static inline GemmPlan plan_gemm(const GemmAsk &a) {
  GemmPlan p{};
  const bool wide = a.bf16 || a.fp16;
  p.mb = std::min(256, gemm_ceil(a.m, 16) * 16);
  p.n_tiles = gemm_ceil(a.n_out, BM);
  // 16-bit weights: fewer activation rows per tile before k-slices (whose sums cost two meetings of a cluster) when there are not enough tiles
  if (a.group_rows) p.mb = a.group_rows;
  else if (wide)
    while (p.mb > 64 && p.n_tiles * gemm_ceil(a.m, p.mb) * 4 < a.sms * 3) p.mb = gemm_ceil(p.mb, 32) * 16;
  p.m_tiles = gemm_ceil(a.m, p.mb);
  p.n_kb = wide ? a.k_in / 64 : a.k_in / 128;
  // k-slices: fill the GPU when there are few tiles, with at least PT_TC_MIN_KB k-blocks per CTA.  Not to the brim: the slices of a tile
  // start together in one cluster, and 36 clusters of eight did not fit 148 SMs of two CTAs each at once (4608 x 4096 at 8 rows: 14.7 us
  // with 8 slices, 11.1 with 7; 12288 x 4096: 26 us with 3 slices, 20 with 2).
#ifndef PT_TC_MIN_KB
#define PT_TC_MIN_KB 3
#endif
  int ksplit = a.ksplit;
  if (a.int4) {
    const Int4Plan plan = plan_int4(a.m, p.n_tiles, p.n_kb, a.ksplit, a.sms);
    p.mb = plan.mb;
    ksplit = plan.ksplit;
  } else if (ksplit <= 0) {
    ksplit = std::max(1, (p.mb <= 64 ? 2 : 1) * a.sms * 7 / 8 / (p.n_tiles * p.m_tiles));   // two CTAs fit an SM up to 64 activation rows
    // (with several blocks of activation rows a slice's sums cost more than its share of a short k saves: 128 x 2048 at 512 .. 8192
    // rows takes 19 - 21 us whole and 27 - 41 us in slices)
    ksplit = std::max(1, std::min(ksplit, p.n_kb / (wide && p.m_tiles > 1 ? 32 : PT_TC_MIN_KB)));
    if (!(wide && p.m_tiles > 1)) ksplit = slices_that_pay(std::min(ksplit, MAX_CLUSTER), p.n_kb, p.mb, a.bf16 && a.m % 32 != 0);
  }
  ksplit = std::min(ksplit, MAX_CLUSTER);
  p.m_tiles = gemm_ceil(a.m, p.mb);
  ksplit = std::max(1, std::min(ksplit, p.n_kb));
  p.kb_per_split = gemm_ceil(p.n_kb, ksplit);
  p.ksplit = gemm_ceil(p.n_kb, p.kb_per_split);

  // BF16 without k-slices: two weight tiles per CTA when half as many CTAs still fill the GPU
#ifndef PT_TC_PAIR
#define PT_TC_PAIR 1
#endif
  p.na = PT_TC_PAIR && a.bf16 && p.ksplit == 1 && p.mb >= 128 && p.n_tiles >= 2 && (long long)gemm_ceil(p.n_tiles, 2) * p.m_tiles >= a.sms ? 2 : 1;
  const int most_sent = a.int4 ? SENT_ROWS_INT4 : SENT_ROWS;
  p.sent = p.ksplit > 1 && p.mb <= most_sent && (a.int4 || gemm_ceil(p.mb / 4, p.ksplit) <= (p.n_kb < 16 ? 1 : a.bf16 ? 2 : 3));
  p.few = p.sent || (p.ksplit == 1 && p.mb <= most_sent);
  // (Sums that are fetched take 512 bytes per row of the ring.)
  const uint32_t b_bytes = (uint32_t)p.mb * BKB, sums = p.sent ? sum_bytes(p.mb, p.ksplit) : p.ksplit > 1 ? p.mb * BM * 4 : 0;
  uint32_t behind = p.sent && sums <= SUM_SMEM ? sums : 0;
  if (a.int4) {
    const bool two = p.mb <= 128 && p.n_tiles * p.m_tiles * p.ksplit > a.sms;     // two CTAs per SM (each has half the tensor memory)
    p.int4_groups = !two && p.mb <= 128 ? 4 : 2;                                  // above 128 rows a step's MMAs take longer than half a transform
    p.threads = (3 + 4 * p.int4_groups) * 32;
    // slots: 64 tensor-memory columns beside the accumulator and 256 bytes of shared memory per row each
    p.stages = two ? (p.mb <= 64 ? 3 : 2) : (p.mb <= 128 ? 4 : p.mb <= 208 ? 3 : 2);
    p.stage_bytes = 2 * b_bytes;
    const uint32_t slots = p.stages * p.stage_bytes, room = (two ? (behind ? 110 : 104) : 217) * 1024u;
    if (room < slots + behind + (p.stages + p.int4_groups) * RAW_STEP) behind = 0;
    p.raw_stages = (int)std::min<uint32_t>(12, (room - slots - behind) / RAW_STEP);
    p.sum_offset = behind ? slots + p.raw_stages * RAW_STEP : 0;
    p.smem = slots + p.raw_stages * RAW_STEP + behind + 1024;
    p.fits = p.stages >= p.int4_groups && p.raw_stages >= p.stages + p.int4_groups && sums <= p.smem - 1024;
    p.tmem_columns = ((p.mb + 31) & ~31) + 64 * p.stages <= 256 ? 256 : 512;
    if (p.tmem_columns == SM_COLUMNS) p.smem = std::max(p.smem, ALONE_SMEM);
  } else {
    p.threads = 64 + 128 * p.na;   // warp 0: producer, warp 1: MMA + tensor-memory allocation, then four epilogue warps per accumulator
    p.stage_bytes = p.na * A_TILE + ((b_bytes + 1023u) & ~1023u);
    // Up to 64 activation rows a stage is small, and what limits the kernel is the one thread per CTA that issues the MMAs (about
    // 75 cycles per tcgen05.mma whatever its N): two CTAs per SM (half the shared memory each) issue side by side.  Measured on
    // B200, FP8 65024 x 4096 at 8 / 32 rows: 63 / 66 us with one CTA per SM, 45 / 47 us with two.
#ifndef PT_TC_BUDGET_SMALL_KB
#define PT_TC_BUDGET_SMALL_KB 100
#endif
    // 16-bit weights also with large tiles when there are more of them than SMs: the epilogue of one CTA then hides behind the products of
    // the other (two accumulators of 256 columns fill the tensor memory).
    const bool small = p.mb <= 64 || (wide && !(p.ksplit > 1 && p.mb > 128) && p.na * p.mb <= 256 && (long long)p.n_tiles * p.m_tiles * p.ksplit > a.sms);
    p.stages = (int)std::min<uint32_t>(8, ((small ? PT_TC_BUDGET_SMALL_KB : 200) * 1024u + std::min(behind, (small ? 110 - PT_TC_BUDGET_SMALL_KB : 16) * 1024u) - behind) / p.stage_bytes);
    p.sum_offset = behind ? p.stages * p.stage_bytes : 0;
    p.smem = p.stages * p.stage_bytes + behind + 1024;
    // (A whole tile of a short k gains nothing from warps that fetch: FP8 768 x 768 at 16 rows 3.4 us so, 3.2 by TMA.)
    p.x_warps = (p.ksplit > 1 || p.n_kb >= 16) && p.na == 1 && p.mb <= 32 && p.stages >= 4;
    p.fits = p.stages >= 2 && sums <= p.smem - 1024;
    int columns = 32;
    while (columns < p.mb) columns <<= 1;
    p.tmem_columns = p.na * columns;
    if (p.tmem_columns == SM_COLUMNS) p.smem = std::max(p.smem, PAIR_SMEM);       // (no k-slices, so no cluster)
  }
  p.smem = std::max(p.smem, SHARED_SMEM);
  return p;
}

}  // namespace tc
}  // namespace pt

// How a small product of few activation rows is split over blocks (gemm_few.cu).  Host arithmetic alone: a plain C++ compiler takes this file.
#pragma once
#include <algorithm>
#include <cstdint>

namespace pt {
namespace few {

constexpr int ROWS = 8;                            // activation rows, at most
constexpr int UNIT = 16;                           // weight rows of a warp
constexpr int MAX_WARPS = 12;                      // multiplying warps of a block
constexpr int MAX_STAGES = 12;
constexpr int MAX_CLUSTER = 8;
constexpr uint32_t UNIT_BYTES = 2048, ROW_BYTES = 128;      // of a k block (64 k): of a unit's weights, of an activation row
constexpr uint32_t ITEM = ROWS * 20 * 4;           // sums of a unit and eight activation rows: rows of 16 floats, padded to 20
constexpr uint32_t BUDGET = 104 * 1024;            // shared memory of a block: two fit an SM, so that the next launch's can fetch weights while this one ends

struct Plan {
  int units, warps_k, slices;      // units of a block; its warps that share a unit's k; blocks of a cluster that share it
  int kb_per_slice, stages, blocks;
  uint32_t stage_bytes, sum_offset, smem;
};
constexpr int ceil_to(int a, int b) { return (a + b - 1) / b; }

// Which products may come here: up to eight rows, of matrices up to 8 MB or of a short k, where a block's tile is over before it has begun.
static inline bool small(int m, int n_out, int k_in) { return m <= ROWS && (k_in <= 1024 || (long long)n_out * k_in <= 1 << 22); }

// ... and which of them are faster here than in tensor memory (gemm_few.cu has the times of small ones).  Not large ones whose tiles of 128 weight rows fill the last round
// there (two a SM) to four fifths: 32003 x 512 at 1 row 6.2 us there and 6.8 here, 65536 x 768 17.1 and 18.4; where they leave more of it empty it is the other
// way: 50257 x 768 15.8 and 12.9, 20000 x 1024 9.3 and 8.1, 16384 x 1024 7.2 and 6.8.  Nor large ones of k up to 256, of which one or two stages are all: 16384 x 256 3.1
// there, 3.4 here; unless the tiles are more than a round (50257 x 256 7.4, 5.8).
static inline bool pays(int n_out, int k_in, int sms) {
  const int tiles = ceil_to(n_out, 128), rounds = ceil_to(tiles, 2 * sms);
  const bool filled = tiles * 5 >= rounds * 2 * sms * 4;
  return k_in <= 256 ? n_out <= 8192 || (rounds > 1 && !filled) : (long long)n_out * k_in <= 1 << 22 || !filled;
}

static inline Plan split(int n_units, int n_kb, int units, int warps_k, int slices) {
  Plan p{units, warps_k, slices, 0, 0, 0, 0, 0, 0};
  p.kb_per_slice = ceil_to(n_kb, slices);
  p.slices = ceil_to(n_kb, p.kb_per_slice);
  p.blocks = ceil_to(n_units, units) * p.slices;
  p.stage_bytes = warps_k * (units * UNIT_BYTES + ROWS * ROW_BYTES);
  const uint32_t sums = (uint32_t)ceil_to(units, p.slices) * p.slices * warps_k * ITEM;
  p.stages = std::min({MAX_STAGES, (int)((BUDGET - 1024 - sums) / p.stage_bytes), std::max(2, ceil_to(p.kb_per_slice, warps_k))});
  p.sum_offset = p.stages * p.stage_bytes;
  p.smem = p.sum_offset + sums + 1024;
  return p;
}

// The split with the least time by a linear model of what a block does (us: k blocks of a warp, a cluster's meeting, activations and weights to fetch, parts
// of a sum, warps), fitted on B200 to 24 sizes of 640 x 2048 .. 2048 x 2048 and 8000 x 512 at 1 and 8 rows, some 100 splits of each: what it takes is
// on average 4 % above the best.  (Up to 1024 k clusters give 0.1 us at most: none.)  More blocks than SMs only if they are small, so that they share the SMs.
// Matrices of more than twice the size that it was fitted to take rounds of two blocks an SM: us at 8 rows by the model / so, fp16, 12288 x 1024 8.0 / 6.6, 16384 x 768 6.5 / 5.7, 20000 x 1024
// 9.5 / 8.2, 50257 x 768 14.1 / 13.3, 128256 x 1024 48.6 / 43.4.
static inline Plan make_plan(int m, int n_out, int k_in, int sms) {
  const int n_units = ceil_to(n_out, UNIT), n_kb = k_in / 64;
  if ((long long)n_out * k_in > 1 << 23) {     // (k up to 1024) what counts is that the blocks fill every round of two an SM evenly
    const int rounds = ceil_to(n_units, 2 * sms * MAX_WARPS), units = ceil_to(n_units, 2 * sms * rounds);
    return split(n_units, n_kb, units, std::min(n_kb, units <= 2 ? 3 : units <= 5 ? 2 : 1), 1);
  }
  Plan best = split(n_units, n_kb, MAX_WARPS, 1, 1);       // (many rounds of blocks)
  double least = 1e30;
  for (int units = 1; units <= MAX_WARPS; ++units)
    for (int warps = 1; units * warps <= MAX_WARPS && warps <= n_kb; ++warps)
      for (int slices = 1; slices <= (n_kb > 16 ? MAX_CLUSTER : 1); ++slices) {
        const Plan p = split(n_units, n_kb, units, warps, slices);
        if (p.slices != slices || p.stages < 2 || p.blocks > 2 * sms || (p.blocks > sms && units * warps > 6)) continue;
        const int rounds = ceil_to(p.blocks, sms), steps = ceil_to(p.kb_per_slice, warps), parts = slices * warps;
        const double weights = (double)rounds * p.kb_per_slice * units * UNIT_BYTES, rows = (double)rounds * p.kb_per_slice * m * ROW_BYTES;
        const double stream = std::max((double)n_out * k_in * 2 / (sms * 23.0), weights / 50.0);       // cycles
        const double us = 0.177 * steps + (slices > 1 ? 0.353 : 0.0) + 0.304e-4 * rows + 0.053e-5 * weights + 3.822e-4 * stream + (rounds > 1 ? 0.138 : 0.0) + 0.0181 * parts +
                          0.0588 * units * warps - (warps > 1 && slices == 1 ? 0.105 : 0.0) + 0.0353 * ceil_to(units, slices) * parts / (units * warps) + 0.002 * slices;
        if (us < least) { least = us; best = p; }
      }
  return best;
}

// The same for a size that this thread has met lately: the search takes the host 4.5 us where clusters are an option (0.4 up to 1024 k), as long as half a
// call that is not captured in a graph; a size that is kept takes 10 ns.  (A place in the table and the three behind it are a size's.)
static inline const Plan &kept_plan(int m, int n_out, int k_in, int sms) {
  struct Kept { int m, n_out, k_in, sms; Plan plan; };       // (m = 0: nothing yet)
  constexpr unsigned PLACES = 128, WAYS = 4;
  static thread_local Kept kept[PLACES];
  static thread_local unsigned turn = 0;
  const unsigned first = ((unsigned)n_out * 2654435769u ^ (unsigned)k_in * 2246822519u ^ (unsigned)m * 3266489917u) >> 25;
  for (unsigned i = 0; i < WAYS; ++i) {
    const Kept &e = kept[(first + i) % PLACES];
    if (e.m == m && e.n_out == n_out && e.k_in == k_in && e.sms == sms) return e.plan;
  }
  Kept &e = kept[(first + turn++ % WAYS) % PLACES];
  e = {m, n_out, k_in, sms, make_plan(m, n_out, k_in, sms)};
  return e.plan;
}

}  // namespace few
}  // namespace pt

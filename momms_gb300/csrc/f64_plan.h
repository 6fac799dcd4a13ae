// How a plain f64 problem is cut into work units, and what its split needs of
// scratch. Host code without CUDA, so that tests check the plans of every shape
// against the scratch that holds their partial tiles on the CPU.
#pragma once
#include <stdint.h>

#include <algorithm>

namespace momms {

// What a split plan of the model may use, the same for every caller: partial
// tiles within 160 of 128 x 128 doubles (counted on the 128 grid, which a tile
// of 32, 16 or 8 divides), and the 1280 counters that two splits of so many
// 32 x 32 tiles take.
constexpr int64_t kSplitTileCap = 160, kSplitCounterCap = 1280;
inline bool f64_split_fits(int64_t m, int64_t n, int splits) {
  return ((m + 127) / 128) * ((n + 127) / 128) * splits <= kSplitTileCap;
}

// Square output tiles of ts = 32, 16 or 8, k in `splits` ranges of kb_split
// k-blocks of 16. Depends only on the shape, the tuning table and the SM count.
struct F64Plan {
  int ts, tiles_m, tiles_n, splits;
  int64_t kb_split;
  int run;  // k-blocks whose products a warp sums in one chain (f64_run)
  int64_t tiles() const { return (int64_t)tiles_m * tiles_n; }
  int64_t units() const { return tiles() * splits; }
  // doubles of a split's partial tiles, one of ts x ts per unit
  int64_t partial_elems() const { return splits > 1 ? units() * ts * ts : 0; }
  double unit_cost;  // FP64-pipe clocks of one SM per unit
};

inline int clamp_splits(int s, int64_t kblocks) {
  return std::max(1, (int)std::min<int64_t>(s, std::max<int64_t>(1, kblocks)));
}

// A warp sums its products of `run` k-blocks in one chain (16 products an entry
// and k-block, or 4 where the tile's four warps share each k-block: steps of 16
// and 8), the runs in turn, then the warps, then the splits. For products of
// either sign the mean square error of such a sum is proportional to
//   chain + runs + splits (+ 5 for the four warps),
// each of runs and splits counted where there is more than one. The run is the
// longest chain, at most 256 products, whose error is no larger than that of
// the same product cut on the 128 x 128 grid, k split while tiles leave SMs idle
// and each range keeps two k-blocks: every run costs one addition per entry,
// 0.5 % of the time at 256 products and 3 % at 32. (256 throughout had 2.2 times
// the error of that grid's split at 384 x 384 x 512, 1.8 times at 384 x 384 x 1024.)
// A tuned split count is what that grid would use as well: 256 products.
inline int f64_run(const F64Plan& p, int64_t m, int64_t n, int64_t k, int sm_count, bool tuned) {
  const int per = p.ts > 16 ? 16 : 4;  // products of an entry per k-block and warp
  if (tuned) return 256 / per;
  auto div_up = [](int64_t a, int64_t b) { return (a + b - 1) / b; };
  const int64_t kblocks = div_up(k, 16), tiles = div_up(m, 128) * div_up(n, 128);
  const int64_t ranges = tiles < sm_count
                             ? std::max<int64_t>(1, std::min<int64_t>({sm_count / tiles, kblocks / 2, 32}))
                             : 1;
  const int64_t kb_range = div_up(kblocks, ranges), used = div_up(kblocks, kb_range);
  const int64_t most = std::min(k, 16 * kb_range) + (used > 1 ? used : 0);
  int best = 1;
  int64_t best_error = INT64_MAX;
  for (int run = 256 / per; run >= 1; --run) {
    const int64_t runs = div_up(std::min(p.kb_split, kblocks), run);
    const int64_t error = std::min<int64_t>(run, std::min(p.kb_split, kblocks)) * per + (runs > 1 ? runs : 0) +
                          (p.splits > 1 ? p.splits : 0) + (per == 4 ? 5 : 0);
    if (error <= most) return run;
    if (error < best_error) {
      best_error = error;
      best = run;
    }
  }
  return best;
}

// The f64 plan minimises the FP64 pipe's time on the busiest SM plus what a
// split costs at its end. One SM takes 128 clocks per 8 x 8 x 4 DMMA whatever
// the tile, so the sum per SM (units dealt round-robin, the SM's four CTAs
// sharing the pipe) is what balance can change: tiles of 32 where they are
// many, of 16 (8, for a few dozen rows and columns) or k splits where a last
// wave would be thin or SMs would idle. Splitting adds one FP64 addition per output and split, and
// a partial write, a fence, an atomic and the last arriver's reads in series
// (about 3 us). `tuned`: the tuning table's split count, kept as it is, or 0.
inline F64Plan f64_model(int64_t m, int64_t n, int64_t k, int sm_count, int tuned) {
  constexpr double kBlockStep = 128.0, kUnitFill = 300.0, kSplitTail = 6000.0, kSplitTailEach = 200.0;
  auto div_up = [](int64_t a, int64_t b) { return (a + b - 1) / b; };
  const int64_t kblocks = div_up(k, 16), ksteps = div_up(k, 4);
  F64Plan best{};
  double best_t = -1.0;
  for (int ts = 32; ts >= 8; ts /= 2) {
    F64Plan p{};
    p.ts = ts;
    p.tiles_m = (int)div_up(m, ts);
    p.tiles_n = (int)div_up(n, ts);
    const int64_t tiles = p.tiles();
    const double blocks = (double)std::min<int64_t>(div_up(m, 8), ts / 8) * std::min<int64_t>(div_up(n, 8), ts / 8);
    const int most = !tuned && tiles > kSplitCounterCap ? 1 : (int)std::min<int64_t>(32, kblocks);
    // a tuned split count is kept as it is: smaller tiles only where its
    // counters still fit
    if (tuned && ts < 32 && clamp_splits(tuned, kblocks) > 1 && tiles > kSplitCounterCap) break;
    int prev = 0;
    for (int want = 1; want <= most; ++want) {
      if (tuned) want = clamp_splits(tuned, kblocks);
      p.kb_split = div_up(kblocks, want);
      p.splits = (int)div_up(kblocks, p.kb_split);
      if (!tuned && p.splits > 1 && !f64_split_fits(m, n, p.splits)) break;
      if (p.splits != prev) {
        prev = p.splits;
        const double steps = (double)std::min<int64_t>(4 * p.kb_split, ksteps);
        // warps with one block of their own keep the pipe at 0.7 of its rate
        const double rate = ts == 8 || (ts == 32 && m <= 16 && n <= 16) ? 0.7 : 1.0;
        // per output: alpha and beta (or nothing), and the four warps' sum
        p.unit_cost = blocks * (kBlockStep / rate * steps + (p.splits == 1 ? 64.0 : 0.0) + (ts < 32 ? 96.0 : 0.0)) + kUnitFill;
        double t = (double)div_up(p.units(), sm_count) * p.unit_cost;
        if (p.splits > 1)
          t += kSplitTail + kSplitTailEach * p.splits +
               (double)div_up(tiles, sm_count) * blocks * 32.0 * (p.splits + 1);
        if (best_t < 0.0 || t < best_t) {
          best_t = t;
          best = p;
        }
      }
      if (tuned) break;
    }
  }
  best.run = f64_run(best, m, n, k, sm_count, tuned != 0);
  return best;
}

}  // namespace momms

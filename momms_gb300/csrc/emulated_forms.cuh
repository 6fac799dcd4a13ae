// The two forms of an emulated product (digit pairs, or residues modulo coprime
// numbers), which of them a product takes, and what each needs of scratch. Host
// code only, so that tests compare the byte counts on the CPU.
#pragma once
#include <math.h>

#include <algorithm>
#include <vector>

#include "crt_elem.cuh"
#include "internal.h"
#include "ozaki_elem.cuh"
#include "slicegemm.cuh"

namespace momms {
namespace forms {

using elem::kDigitBits;
// k per launch (kOzakiMaxK): the largest product of two digits is 2^16, so a
// single pair's int32 sum stays below 2^31 for up to 511 k-blocks of 64
constexpr int64_t kMaxK = kOzakiMaxK;
static_assert((kMaxK / 64) * 64 * (1ll << (2 * kDigitBits)) < (1ll << 31), "int32 digit sums must stay exact");
// an int32 group sum's bound (sums of the pairs' worst cases)
constexpr double kGroupLimit = 2147483647.0;
// one TMEM chunk's bound: integers up to 2^24 are exact in FP32
constexpr double kChunkBound = 16777216.0;
// the residue form runs from this k (crt_applies)
constexpr int64_t kCrtMinK = 128;

// The slice-product schedule for ns slices over k: diagonals d = t + u from
// the smallest weight (d = ns+1) to the largest (d = 2), each diagonal's pairs
// (t, d-t) in t order, cut into accumulation groups whose worst-case int32
// sums (k * 2^bits_t * 2^bits_u over the group's pairs; the top digit has
// `bits` bits, the centred ones bits-1) stay within kGroupLimit. A group's
// A TMEM chunk keeps its sum within kChunkBound: a k-block of pair (t, u)
// adds at most 64 * 2^bits_t * 2^bits_u, so a pair's weight is that product
// in units of 2^10 and a chunk's capacity kChunkBound / 64 / 2^10 (a lone
// pair: 4, 8 or 16 k-blocks of 64 for 8-bit digits; at small k one chunk
// spans several pairs of a group).
constexpr int kChunkUnitLog2 = 10;
constexpr int kChunkCap = (int)(kChunkBound / 64.0) >> kChunkUnitLog2;
struct Schedule {
  int np = 0, ng = 0;
  uint8_t pair_a[sp::MAX_PAIRS], pair_b[sp::MAX_PAIRS];
  int group_begin[sp::MAX_GROUPS + 1];
  int pair_w[sp::MAX_PAIRS];
  uint8_t level[sp::MAX_GROUPS];  // d - 2
};

inline bool ozaki_schedule(int ns, int64_t k, Schedule* sc) {
  const int bits = kDigitBits;
  const int64_t kblocks = ceil_div(std::min<int64_t>(std::max<int64_t>(k, 1), kMaxK), 64);
  const double kspan = (double)kblocks * 64.0;
  auto prod = [&](int t, int u) { return 1 << ((t == 1 ? bits : bits - 1) + (u == 1 ? bits : bits - 1)); };
  sc->np = sc->ng = 0;
  for (int d = ns + 1; d >= 2; --d) {
    double gsum = 0.0;
    bool open = false;
    for (int t = 1; t <= ns; ++t) {
      const int u = d - t;
      if (u < 1 || u > ns) continue;
      const int pb = prod(t, u);
      if (open && gsum + kspan * pb > kGroupLimit) open = false;  // this pair starts the next group
      if (!open) {
        if (sc->ng >= sp::MAX_GROUPS) return false;
        sc->group_begin[sc->ng] = sc->np;
        sc->level[sc->ng] = (uint8_t)(d - 2);
        ++sc->ng;
        gsum = 0.0;
        open = true;
      }
      if (sc->np >= sp::MAX_PAIRS) return false;
      sc->pair_a[sc->np] = (uint8_t)(t - 1);
      sc->pair_b[sc->np] = (uint8_t)(u - 1);
      sc->pair_w[sc->np] = std::max(1, pb >> kChunkUnitLog2);
      ++sc->np;
      gsum += kspan * pb;
    }
  }
  sc->group_begin[sc->ng] = sc->np;
  return true;
}

// Moduli that hold an ns-slice product whose sums of scaled magnitudes
// (sum_p |a_ip b_pj| 2^-e_i 2^-f_j, at most k) stay within `sum`: P > 2 |R|,
// |R| <= sum 2^(16 ns), with 2 % to spare for the quotient's rounding
// (crt::kFracBits). More moduli than R needs do not change the result.
inline int crt_moduli(int ns, double sum) {
  const double need = 16.0 * ns + log2(std::max(sum, (double)kCrtMinK)) + 1.0 + 0.03;
  double have = 0.0;
  int n = 0;
  while (n < crt::kMaxModuli && have < need) have += log2((double)crt::kModuli[n++]);
  return n;
}
// Whether an ns-slice product runs by residues: where the model below says it
// is the faster form. From the sizes alone (those of the whole product, where
// it is streamed in blocks), so that a product gives the same bits alone, in a
// batch, streamed and from packed operands. The rates are measured ones:
//  * slice products: 0.26 us per 256 x 256 x 64 step of a CTA pair, 76 pairs,
//    a group's steps in series (7 pairs of digits, or one modulus, each over
//    all of k: what decides for few tiles), and per group and entry what of
//    the epilogue they do not hide: 0.53 ps (digits: 4 bytes of plane), 0.2 ps;
//  * recombination 7.4 ps per entry (7 digit groups), 10.4 ps (16 moduli);
//  * operand planes 2 bytes per slice or modulus, 8 read, at 6 TB/s;
//  * packed operands have their digits, and no residues: 2 bytes read per
//    slice and written per modulus, at 9 TB/s (much of it stays in L2).
// The residue form has to be faster either way, by 3 us where operands are not
// packed: 3776 x 247 x 2224 from packs, 8 slices, 115 us by digits and 156 by
// residues, 1000 x 1000 x 1000, 7 slices, 62 and 56.
// Both forms, 7 slices, ms per call: 8192 x 8192 x 128 1.33 (digits) and 1.40,
// x 256 1.61 and 1.56, x 1024 3.17 and 2.48, x 8192 20.9 and 13.1; 65536 x 256 x
// 256 0.64 and 0.75; the slice kernel alone at 512^3 0.030 and 0.014.
inline bool crt_applies(int ns, int64_t m, int64_t n, int64_t k) {
  if (ns < 5 || k < kCrtMinK) return false;
  const int N = crt_moduli(ns, k);
  Schedule sc;
  if (!ozaki_schedule(ns, k, &sc)) return true;
  constexpr double kPairs = 76.0, kStep = 0.26e6, kMargin = 3e6;  // ps
  const double mn = (double)m * n, ops = (double)(m + n) * k;
  const double tiles = (double)(ceil_div(m, 256) * ceil_div(n, 256)), steps = (double)ceil_div(k, 64) * kStep;
  auto products = [&](double pairs, double longest) { return steps * std::max(pairs * tiles / kPairs, longest); };
  const double digits = products(sc.np, ns) + mn * (0.53 * sc.ng + 2.7 + 0.67 * sc.ng);
  const double residues = products(N, 1.0) + mn * (0.2 * N + 0.65 * N);
  return residues + ops * (8 + 2 * N) / 6.0 + kMargin < digits + ops * (8 + 2 * ns) / 6.0 &&
         residues + ops * (2 * ns + 2 * N) / 9.0 < digits;
}

// What an emulated product's scratch consists of.
struct Sizes {
  double ops;  // elements of one plane of both operands
  double own;  // the same of the operands that are not packed
  double c;    // entries of C, padded to whole tiles
};
inline Sizes sizes_of(int64_t m, int64_t n, int64_t k, bool tight) {
  const double ops = (double)(m + n) * (double)plane_row(std::min(k, kMaxK), 8, tight);
  return Sizes{ops, ops, (double)round_up(m, sp::BM) * (double)round_up(n, sp::BN)};
}
// Operand planes and group planes: the digit form's (packed operands bring
// their digits), or the residue form's with `per` of its N moduli per pass.
inline double digit_scratch(int ns, int64_t k, const Sizes& z) {
  Schedule sc;
  const double ng = ozaki_schedule(ns, k, &sc) ? sc.ng : sp::MAX_GROUPS;
  return 2.0 * ns * z.own + 4.0 * ng * z.c;
}
inline double crt_scratch(int per, int N, const Sizes& z) { return 2.0 * per * z.ops + N * z.c; }
// The residue form keeps to `limit` bytes, the digit form's scratch or more, by
// walking the moduli in several passes, each with its own operand planes: at
// 8192^3 two passes of 8 moduli instead of 4.6 GB of planes, for one more read
// of the operands (0.2 of 13 ms). Where a call is small a second pass shows:
// 2600 x 2600 x 2600 786 us in two, 754 in one, 4096 x 1024 x 4096 728 and 678.
inline int crt_per_pass(int N, const Sizes& z, double limit) {
  int per = N;
  while (per > 1 && crt_scratch(per, N, z) > limit) --per;
  const int passes = (int)ceil_div(N, per);
  return (int)ceil_div(N, passes);
}
// What a call may take where the device has room for it, `digits` the digit
// form's scratch: kFreeScratch, or the digits that packed operands bring on top (in passes within the
// digit form's own scratch, 8192 x 8192 x 8192 from packs re-reads the digits
// nine times). A call under stream capture has its scratch allocated when its
// graph is launched, where no second choice is left: kCapturedScratch, enough
// for one pass of the small calls to which a pass matters. `tight`: no more
// than the digit form's.
constexpr double kCapturedScratch = 512.0 * (1 << 20);
inline double scratch_limit(int ns, const Sizes& z, double digits, bool tight, bool captured) {
  if (tight) return digits;
  if (captured) return std::max(digits, kCapturedScratch);
  return std::max(digits + 2.0 * ns * (z.ops - z.own), (double)kFreeScratch);
}
// The most an ns-slice product takes, whatever its operands (an automatic count
// may need fewer moduli than k asks for, and then more of them fit a pass).
inline double emulated_scratch(int ns, int64_t m, int64_t n, int64_t k, bool tight) {
  const Sizes z = sizes_of(m, n, k, tight);
  const double d = digit_scratch(ns, k, z);
  const int64_t kk = std::min(k, kMaxK);
  if (!crt_applies(ns, m, n, kk) || tight) return d;
  const int N = crt_moduli(ns, (double)kk);
  return std::max(d, std::min(crt_scratch(N, N, z), scratch_limit(ns, z, d, false, false)));
}

// A plan holds the scratch of the problems it runs in one slice launch for as
// long as it lives, residues in one pass. Which of its problems do: those that
// add least beyond the digit form, while the sum stays within `limit` (a plan of
// eight 4096 x 1024 x 4096 products would hold 5.9 GB for 3.3 by digits). The
// others, the largest, run on their own, each in scratch that the next reuses.
inline double batch_extra(int ns, int64_t m, int64_t n, int64_t k) {
  if (!crt_applies(ns, m, n, k)) return 0.0;
  const Sizes z = sizes_of(m, n, k, false);
  const int N = crt_moduli(ns, k);
  return std::max(0.0, crt_scratch(N, N, z) - digit_scratch(ns, k, z));
}
inline std::vector<char> batch_members(const std::vector<double>& extra, double limit) {
  std::vector<size_t> order(extra.size());
  for (size_t i = 0; i < order.size(); ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](size_t x, size_t y) { return extra[x] < extra[y]; });
  std::vector<char> in(extra.size(), 0);
  double sum = 0.0;
  for (size_t i : order) in[i] = (sum += extra[i]) <= limit;
  return in;
}

}  // namespace forms
}  // namespace momms

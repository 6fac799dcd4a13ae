// The plain f64 plans (momms_gb300/csrc/f64_plan.h) of every kind of shape
// against what holds their split's partial tiles and counters. Prints "OK" or
// the first plans that do not fit. With the argument "rms": one line per shape,
// "m n k ratio", of the rms error of dot products summed in the plan's order
// over that of the 128 x 128 grid's order (chains of 16 k products of each range
// of k, ranges in turn), both with FP32 sums against FP64 ones.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "f64_plan.h"

using momms::F64Plan;

static int failures = 0;

static void check(int64_t m, int64_t n, int64_t k, int sms, int tuned) {
  const F64Plan p = momms::f64_model(m, n, k, sms, tuned);
  const int64_t kblocks = (k + 15) / 16;
  bool ok = (p.ts == 32 || p.ts == 16 || p.ts == 8) && (int64_t)p.tiles_m * p.ts >= m && (int64_t)p.tiles_n * p.ts >= n &&
            p.splits >= 1 && p.splits <= 32 && p.kb_split * p.splits >= kblocks && p.kb_split * (p.splits - 1) < kblocks;
  // a thread's partials lie in its unit's ts x ts doubles (dmma_core.cuh, finish_unit)
  const int threads = p.ts > 8 ? 128 : 32, outputs = p.ts == 32 ? 8 : 2;
  ok = ok && threads * outputs == p.ts * p.ts;
  // the scratch of calls that cannot allocate: 160 tiles of 128 x 128 doubles and 1280 counters
  const bool split = p.splits > 1;
  // (with a launch's unit counters, also within the 21 MB that admission and streaming charge for it)
  const bool room = !split || (p.partial_elems() <= 160 * 128 * 128 && p.tiles() <= 1280 &&
                               p.partial_elems() * 8 + p.tiles() * 4 + 16 <= 21 * 1024 * 1024);
  if (!tuned) ok = ok && room;  // a tuned plan may ask for more, and is refused there
  else if (split && momms::f64_split_fits(m, n, p.splits)) ok = ok && room;
  if (!ok && failures++ < 10)
    printf("%lld x %lld x %lld, %d SMs, tuned %d: step %d, splits %d, %lld tiles, %lld partial doubles\n", (long long)m,
           (long long)n, (long long)k, sms, tuned, p.ts, p.splits, (long long)p.tiles(), (long long)p.partial_elems());
}

static unsigned long long seed = 1;
static double rnd() {
  seed = seed * 6364136223846793005ull + 1442695040888963407ull;
  return (double)(seed >> 11) / 9007199254740992.0;
}

// a . b as a unit's warps, its runs and its splits sum it (dmma_core.cuh)
static float dot(const std::vector<float>& a, const std::vector<float>& b, int64_t k, int ts, int splits, int64_t kb_split,
                 int64_t run) {
  const int64_t kblocks = (k + 15) / 16;
  const int warps = ts > 16 ? 1 : 4, per = 16 / warps;
  float sum = 0.0f;
  for (int s = 0; s < splits; ++s) {
    float part = 0.0f;
    for (int w = 0; w < warps; ++w) {
      float total = 0.0f;
      for (int64_t kb = s * kb_split, end = std::min(kblocks, kb + kb_split); kb < end; kb += run) {
        float chain = 0.0f;
        for (int64_t q = kb; q < std::min(end, kb + run); ++q)
          for (int64_t i = 16 * q + per * w; i < std::min(k, 16 * q + per * (w + 1)); ++i) chain = std::fma(a[i], b[i], chain);
        total = kb == s * kb_split ? chain : total + chain;
      }
      part = w == 0 ? total : part + total;
    }
    sum = s == 0 ? part : sum + part;
  }
  return sum;
}

static void rms(int64_t m, int64_t n, int64_t k, bool positive) {
  const F64Plan p = momms::f64_model(m, n, k, 152, 0);
  const int64_t kblocks = (k + 15) / 16, tiles = ((m + 127) / 128) * ((n + 127) / 128);
  const int64_t want = tiles < 152 ? std::max<int64_t>(1, std::min<int64_t>({152 / tiles, kblocks / 2, 32})) : 1;
  const int64_t range = (kblocks + want - 1) / want, ranges = (kblocks + range - 1) / range;
  std::vector<float> a(k), b(k);
  double plan = 0.0, grid = 0.0;
  for (int i = 0; i < 20000; ++i) {
    double exact = 0.0;
    for (int64_t q = 0; q < k; ++q) {
      a[q] = (float)(positive ? rnd() : 2 * rnd() - 1), b[q] = (float)(positive ? rnd() : 2 * rnd() - 1);
      exact += (double)a[q] * b[q];
    }
    const double x = dot(a, b, k, p.ts, p.splits, p.kb_split, p.run) - exact;
    const double y = dot(a, b, k, 32, (int)ranges, range, kblocks) - exact;
    plan += x * x, grid += y * y;
  }
  printf("%lld %lld %lld %.4f\n", (long long)m, (long long)n, (long long)k, std::sqrt(plan / grid));
}

int main(int argc, char**) {
  if (argc > 1) {
    const int64_t shapes[][3] = {{384, 384, 512}, {384, 384, 1024}, {128, 1500, 500}, {768, 768, 512}, {512, 512, 512},
                                 {256, 256, 256}, {600, 500, 700},  {44, 746, 1024},  {64, 64, 2000},  {93, 110, 77},
                                 {1024, 1024, 1024}, {200, 200, 200}};
    for (auto& s : shapes)
      for (bool positive : {false, true}) rms(s[0], s[1], s[2], positive);
    return 0;
  }
  static_assert(momms::kSplitTileCap == 160 && momms::kSplitCounterCap == 1280, "the scratch of the no-alloc entry point");
  const int sm_counts[] = {152, 132, 148, 160, 1};
  const int64_t known[][3] = {{512, 512, 1024}, {512, 512, 8192}, {384, 384, 2048}, {256, 256, 4096}, {112, 736, 512},
                              {256, 768, 16384}, {747, 287, 16741}, {8, 8, 100000}, {20, 12, 5000}, {1024, 1024, 4096}};
  for (int sms : sm_counts)
    for (auto& s : known)
      for (int tuned : {0, 1, 2, 7, 32}) check(s[0], s[1], s[2], sms, tuned);
  auto size = [&](double most) { return (int64_t)std::exp(rnd() * std::log(most)); };
  for (int i = 0; i < 200000; ++i)
    check(size(6000.0), size(6000.0), size(300000.0), sm_counts[i % 5], i % 3 ? 0 : 1 + (int)(rnd() * 32));
  for (int64_t x = 1; x <= 1300; x += 3)
    for (int64_t k : {16, 100, 1024, 9000}) check(x, x + x % 5, k, 152, 0);
  if (failures) return printf("%d plans\n", failures), 1;
  puts("OK");
  return 0;
}

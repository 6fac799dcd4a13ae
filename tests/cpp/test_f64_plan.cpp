// The plain f64 plans (momms_gb300/csrc/f64_plan.h) of every kind of shape
// against what holds their split's partial tiles and counters. Prints "OK" or
// the first plans that do not fit.
#include <cmath>
#include <cstdio>
#include <cstdlib>

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
  const bool room = !split || (p.partial_elems() <= 160 * 128 * 128 && p.tiles() <= 1280);
  if (!tuned) ok = ok && room;  // a tuned plan may ask for more, and is refused there
  else if (split && momms::f64_split_fits(m, n, p.splits)) ok = ok && room;
  if (!ok && failures++ < 10)
    printf("%lld x %lld x %lld, %d SMs, tuned %d: step %d, splits %d, %lld tiles, %lld partial doubles\n", (long long)m,
           (long long)n, (long long)k, sms, tuned, p.ts, p.splits, (long long)p.tiles(), (long long)p.partial_elems());
}

int main() {
  static_assert(momms::kSplitTileCap == 160 && momms::kSplitCounterCap == 1280, "the scratch of the no-alloc entry point");
  const int sm_counts[] = {152, 132, 148, 160, 1};
  const int64_t known[][3] = {{512, 512, 1024}, {512, 512, 8192}, {384, 384, 2048}, {256, 256, 4096}, {112, 736, 512},
                              {256, 768, 16384}, {747, 287, 16741}, {8, 8, 100000}, {20, 12, 5000}, {1024, 1024, 4096}};
  for (int sms : sm_counts)
    for (auto& s : known)
      for (int tuned : {0, 1, 2, 7, 32}) check(s[0], s[1], s[2], sms, tuned);
  unsigned long long seed = 1;
  auto rnd = [&]() {
    seed = seed * 6364136223846793005ull + 1442695040888963407ull;
    return (double)(seed >> 11) / 9007199254740992.0;
  };
  auto size = [&](double most) { return (int64_t)std::exp(rnd() * std::log(most)); };
  for (int i = 0; i < 200000; ++i)
    check(size(6000.0), size(6000.0), size(300000.0), sm_counts[i % 5], i % 3 ? 0 : 1 + (int)(rnd() * 32));
  for (int64_t x = 1; x <= 1300; x += 3)
    for (int64_t k : {16, 100, 1024, 9000}) check(x, x + x % 5, k, 152, 0);
  if (failures) return printf("%d plans\n", failures), 1;
  puts("OK");
  return 0;
}

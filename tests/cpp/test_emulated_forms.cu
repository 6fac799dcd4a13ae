// Host-side check of the emulated product's scratch (momms_gb300/csrc/
// emulated_forms.cuh): the residue form's least passes stay within what the
// digit form would take for the same call, packed operands' digits not counted.
// Runs on the CPU: no kernel is instantiated or launched.
#include <cmath>
#include <cstdio>

#include "emulated_forms.cuh"

using namespace momms;
using namespace momms::forms;

static int failures = 0;
static void expect(bool ok, const char* what, int ns, int64_t m, int64_t n, int64_t k) {
  if (!ok && failures++ < 10) printf("%s: %d slices, %lld x %lld x %lld\n", what, ns, (long long)m, (long long)n, (long long)k);
}

static void check(int ns, int64_t m, int64_t n, int64_t k) {
  if (!crt_applies(ns, m, n, k)) return;
  const int N = crt_moduli(ns, (double)k);
  for (bool tight : {false, true})
    for (int packs = 0; packs < 4; ++packs) {  // bit 0: A packed, bit 1: B
      Sizes z = sizes_of(m, n, k, tight);
      const double row = (double)plane_row(k, 8, tight);
      z.own = ((packs & 1 ? 0.0 : (double)m) + (packs & 2 ? 0.0 : (double)n)) * row;
      const double digits = digit_scratch(ns, k, z);
      const double limit = scratch_limit(ns, z, digits, tight, false);
      const int least = crt_per_pass(N, z, digits), most = crt_per_pass(N, z, limit);
      expect(least >= 1 && least <= most && most <= N, "passes", ns, m, n, k);
      // one modulus per pass is the least there is: from packs it can be more than their digit form takes
      expect(crt_scratch(least, N, z) <= digits || (packs && least == 1), "least passes", ns, m, n, k);
      if (!packs) expect(crt_scratch(least, N, z) <= digits, "within the digit form", ns, m, n, k);
      expect(crt_scratch(most, N, z) <= limit || most == 1, "free scratch", ns, m, n, k);
      if (tight) expect(most == least, "tight", ns, m, n, k);
      // under capture: at most the digit form's or 512 MB
      const int captured = crt_per_pass(N, z, scratch_limit(ns, z, digits, tight, true));
      expect(crt_scratch(captured, N, z) <= std::max(digits, 512.0 * (1 << 20)) || (packs && captured == 1), "captured", ns, m, n, k);
      // what admission and streaming charge for it, whatever number of moduli the data need
      for (int moduli = crt_moduli(ns, 1.0); moduli <= N; ++moduli) {
        const int per = crt_per_pass(moduli, z, limit);
        expect(crt_scratch(per, moduli, z) <= emulated_scratch(ns, m, n, k, tight), "charge", ns, m, n, k);
      }
    }
}

int main() {
  unsigned long long seed = 7;
  auto rnd = [&]() {
    seed = seed * 6364136223846793005ull + 1442695040888963407ull;
    return (double)(seed >> 11) / 9007199254740992.0;
  };
  auto size = [&](double low, double high) { return (int64_t)std::exp(std::log(low) + rnd() * std::log(high / low)); };
  const int64_t known[][3] = {{8192, 8192, 8192}, {4096, 1024, 4096}, {2600, 2600, 2600}, {512, 512, 8192}, {1000, 1000, 1000}};
  for (auto& s : known)
    for (int ns = 5; ns <= 15; ++ns) check(ns, s[0], s[1], s[2]);
  // 8192 x 8192 x 8192 from packs of 7 digits: the digit form's 1.9 GB of group sums, not its 3.8 GB with planes
  Sizes z = sizes_of(8192, 8192, 8192, false);
  z.own = 0.0;
  expect(crt_scratch(crt_per_pass(17, z, digit_scratch(7, 8192, z)), 17, z) <= 1.9e9, "packs", 7, 8192, 8192, 8192);
  for (int i = 0; i < 20000; ++i) check(5 + i % 11, size(32, 20000), size(32, 20000), size(128, 32704));
  // plans: what their problems hold together beyond the digit form
  for (int trial = 0; trial < 300; ++trial) {
    std::vector<double> extra;
    double together = 0.0;
    const int count = 1 + (int)(rnd() * 60);
    for (int i = 0; i < count; ++i) extra.push_back(batch_extra(5 + (int)(rnd() * 6), size(64, 5000), size(64, 5000), size(64, 5000)));
    const std::vector<char> in = batch_members(extra, (double)kFreeScratch);
    double left = 0.0;
    for (int i = 0; i < count; ++i) (in[i] ? together : left) += extra[i];
    expect(together <= (double)kFreeScratch, "plan", 0, count, 0, 0);
    expect(together + left > (double)kFreeScratch || left == 0.0, "all of a small plan", 0, count, 0, 0);
  }
  expect(batch_extra(7, 4096, 1024, 4096) * 8 > (double)kFreeScratch, "known plan", 7, 4096, 1024, 4096);
  if (failures) return printf("%d failures\n", failures), 1;
  puts("OK");
  return 0;
}

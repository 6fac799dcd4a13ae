// Host harness for momms_gb300/csrc/crt_elem.cuh: reads cases from stdin.
//   0 ns e bits            residues of the double's scaled integer, every modulus
//   1 ns n scale b0..bn-1  bits of the double that the first n residues' bytes stand for
#include <stdio.h>

#include "crt_elem.cuh"

using namespace momms;

static constexpr crt::ModulusTable kTable = crt::make_moduli();

template <int NS>
static void residues(double v, int e) {
  float f[crt::limbs_of(NS)];
  crt::limbs<NS>(v, e, f);
  for (int l = 0; l < crt::kMaxModuli; ++l) printf("%d ", (int)crt::residue_of_limbs<crt::limbs_of(NS)>(f, kTable.m[l]));
  printf("\n");
}

template <int NW>
static double value(int n, const unsigned* r, int scale) {
  crt::Weights w;
  crt::make_weights(n, &w);
  crt::Sums<NW> s;
  s.start(w);
  for (int l = 0; l < n; ++l) s.add(r[l], w.w[l], w.frac[l]);
  uint32_t R[NW];
  s.finish(w, R);
  return words_to_double<NW>(R, scale);
}

int main() {
  int kind, ns;
  while (scanf("%d %d", &kind, &ns) == 2) {
    if (kind == 0) {
      int e;
      unsigned long long b;
      if (scanf("%d %llu", &e, &b) != 2) return 1;
      double v;
      memcpy(&v, &b, 8);
      switch (ns) {
#define X(N) case N: residues<N>(v, e); break;
        X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15)
#undef X
      }
    } else {
      int n, scale;
      unsigned r[crt::kMaxModuli];
      if (scanf("%d %d", &n, &scale) != 2) return 1;
      for (int l = 0; l < n; ++l)
        if (scanf("%u", &r[l]) != 1) return 1;
      double v = 0.0;
      switch (crt::words_of(ns)) {
        case 5: v = value<5>(n, r, scale); break;
        case 6: v = value<6>(n, r, scale); break;
        case 7: v = value<7>(n, r, scale); break;
        case 8: v = value<8>(n, r, scale); break;
        default: v = value<4>(n, r, scale);
      }
      unsigned long long b;
      memcpy(&b, &v, 8);
      printf("%llu\n", b);
    }
  }
  return 0;
}

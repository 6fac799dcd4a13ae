// Residue arithmetic of the emulated FP64 product (Ozaki scheme II: Ozaki,
// Uchino, Imamura 2025, "Ozaki Scheme II: A GEMM-oriented emulation of
// floating-point matrix multiplication using an integer modular technique").
//
// The rows of A and columns of B are scaled to integers X of 8s bits as in
// the digit scheme (ozaki_elem.cuh), but the integer product R = sum_p X_a X_b
// is formed modulo pairwise coprime p_l <= 256 instead of digit pair by digit
// pair: the residues of X are symmetric (|r| <= 128, exact in fp16), each
// modulus is one fp16 product, and R comes back from its residues by the
// Chinese remainder theorem, exactly, once the moduli's product P passes
// 2 |R|. 7 slices of 8 bits need 28 digit products and keep R's leading
// part; 16 moduli hold all of R (17 from k = 5300).
//
// Host-callable, so that tests compare every function with integer arithmetic.
#pragma once
#include <stdint.h>

#include "exact_round.cuh"
#include "ozaki_elem.cuh"

namespace momms {
namespace crt {

constexpr int kMaxModuli = 36;
constexpr int kModuli[kMaxModuli] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217,
                                     211, 199, 197, 193, 191, 181, 179, 173, 167, 163, 157, 151,
                                     149, 139, 137, 131, 127, 113, 109, 107, 103, 101, 97,  89};
constexpr bool pairwise_coprime() {
  for (int i = 0; i < kMaxModuli; ++i)
    for (int j = 0; j < i; ++j) {
      int a = kModuli[i], b = kModuli[j];
      while (b) {
        const int t = a % b;
        a = b;
        b = t;
      }
      if (a != 1) return false;
    }
  return true;
}
static_assert(pairwise_coprime(), "the moduli must be pairwise coprime");

// An integer X of 8s bits is reduced from limbs of 14 bits: t = sum_i limb_i *
// (2^(14 i) mod p), the powers symmetric, is below 2^24 in magnitude for every
// s and p here, so t is exact in FP32 and so is its remainder.
constexpr int kLimbBits = 14, kMaxLimbs = 9, kMaxDigits = 15;
constexpr int limbs_of(int ns) { return (8 * ns + kLimbBits - 1) / kLimbBits; }
constexpr int pow2_mod(int e, int p) {  // symmetric 2^e mod p
  int r = 1;
  for (int i = 0; i < e; ++i) r = 2 * r % p;
  return 2 * r > p ? r - p : r;
}
struct Modulus {
  float p, inv;
  float limb[kMaxLimbs];    // 2^(14 i) mod p
  float digit[kMaxDigits];  // 2^(8 i) mod p
};
struct ModulusTable {
  Modulus m[kMaxModuli];
};
constexpr ModulusTable make_moduli() {
  ModulusTable t{};
  for (int l = 0; l < kMaxModuli; ++l) {
    t.m[l].p = (float)kModuli[l];
    t.m[l].inv = (float)(1.0 / kModuli[l]);
    for (int i = 0; i < kMaxLimbs; ++i) t.m[l].limb[i] = (float)pow2_mod(kLimbBits * i, kModuli[l]);
    for (int i = 0; i < kMaxDigits; ++i) t.m[l].digit[i] = (float)pow2_mod(8 * i, kModuli[l]);
  }
  return t;
}

__host__ __device__ __forceinline__ float fma_f(float a, float b, float c) {
#ifdef __CUDA_ARCH__
  return __fmaf_rn(a, b, c);
#else
  return __builtin_fmaf(a, b, c);
#endif
}

// The limbs of v's scaled integer, with v's sign.
template <int NS>
__host__ __device__ __forceinline__ void limbs(double v, int e, float (&f)[limbs_of(NS)]) {
  constexpr int L = limbs_of(NS);
  using U = typename elem::Word<NS>::type;
  U X = elem::scaled_integer<NS, U>(v, e);
  const uint32_t sign = elem::is_negative(v) ? 0x80000000u : 0u;
MOMMS_UNROLL
  for (int i = 0; i < L; ++i) {
    // below 2^23: under the exponent of 2^23 the bits are 2^23 + limb
    const uint32_t u = (uint32_t)X & (i < L - 1 ? (1u << kLimbBits) - 1 : 0x7fffu);
    uint32_t b = 0x4B000000u | u;
    float x;
    memcpy(&x, &b, 4);
    x -= 8388608.0f;
    memcpy(&b, &x, 4);
    b ^= sign;
    memcpy(&f[i], &b, 4);
    X >>= kLimbBits;
  }
}

// Symmetric remainder of an integer |t| <= 2^24 (|r| <= 128 for every modulus:
// t/p is rounded from a value off by less than 2^-7.7, at most p/2 + 1/2 + ...
// stays below 129).
__host__ __device__ __forceinline__ float remainder_of(float t, float p, float inv) {
  const float q = fma_f(t, inv, 12582912.0f) - 12582912.0f;  // nearest integer to t/p (1.5 * 2^23)
  return fma_f(-q, p, t);
}

// Digits (|d| <= 128) taken in pairs d + 256 d' (|.| <= 32896) for the residue of
// a number of ns digits: as many as keep the sum of pairs and digits times
// 2^(8 i) mod p (at most 127 in magnitude; modulo 256 zero from i = 1 on) within
// 2^24: four pairs above the first reach 16.74 of 16.78 million, five would not,
// and nor would four and three or more single digits.
constexpr int pairs_of_digits(int ns) { return ns <= 10 ? ns / 2 : 4; }

template <int L>
__host__ __device__ __forceinline__ float residue_of_limbs(const float (&f)[L], const Modulus& m) {
  float t = f[0];
MOMMS_UNROLL
  for (int i = 1; i < L; ++i) t = fma_f(f[i], m.limb[i], t);
  return remainder_of(t, m.p, m.inv);
}

// A product's residue as it is stored: (r + 128) mod 256 of the symmetric
// residue r, one byte (r = 128, possible for 256 alone, wraps to -128).
//
// Reconstruction of R from the first n moduli, modulo 2^(32 words): R =
// sum_l r_l w_l - Q P with w_l = (P / p_l) ((P / p_l)^-1 mod p_l) and Q the
// integer nearest to sum_l r_l w_l / P. The byte's bias and an offset that
// keeps Q positive are in the sums' starting values; Q's fractions carry
// kFracBits bits, an error of at most 36 * 128 / 2^19 < 0.009, which the
// moduli leave room for (crt_moduli).
constexpr int kMaxWords = 8, kFracBits = 18, kQOffset = 8192;
struct Weights {
  uint32_t frac[kMaxModuli];          // w_l / P
  uint32_t w[kMaxModuli][kMaxWords];
  uint32_t negp[kMaxWords];           // -P
  uint32_t start[kMaxWords];          // kQOffset P - 128 sum_l w_l
  uint32_t qstart;                    // kQOffset + 1/2 - 128 sum_l w_l / P
};
inline void make_weights(int n, Weights* out) {
  constexpr int NB = kMaxWords + 2;  // P has at most 36 * 8 bits
  uint32_t P[NB] = {1}, S[NB] = {0};
  auto mul = [&](uint32_t (&x)[NB], uint32_t f) {
    uint64_t c = 0;
    for (int i = 0; i < NB; ++i) {
      c += (uint64_t)x[i] * f;
      x[i] = (uint32_t)c;
      c >>= 32;
    }
  };
  auto add = [&](uint32_t (&x)[NB], const uint32_t (&y)[NB], bool negate) {
    uint64_t c = negate ? 1 : 0;
    for (int i = 0; i < NB; ++i) {
      c += (uint64_t)x[i] + (negate ? (uint32_t)~y[i] : y[i]);
      x[i] = (uint32_t)c;
      c >>= 32;
    }
  };
  for (int l = 0; l < n; ++l) mul(P, (uint32_t)kModuli[l]);
  uint32_t q0 = ((uint32_t)kQOffset << kFracBits) + (1u << (kFracBits - 1));
  for (int l = 0; l < n; ++l) {
    const uint32_t p = (uint32_t)kModuli[l];
    uint32_t q[NB];
    uint64_t r = 0;
    for (int i = NB - 1; i >= 0; --i) {
      r = (r << 32) | P[i];
      q[i] = (uint32_t)(r / p);
      r %= p;
    }
    uint32_t qm = 0;  // (P / p) mod p
    for (int i = NB - 1; i >= 0; --i) qm = (uint32_t)((((uint64_t)qm << 32) | q[i]) % p);
    uint32_t inv = 1;
    while (qm * inv % p != 1) ++inv;
    mul(q, inv);
    for (int i = 0; i < kMaxWords; ++i) out->w[l][i] = q[i];
    out->frac[l] = ((inv << kFracBits) + p / 2) / p;
    q0 -= 128 * out->frac[l];
    add(S, q, false);
  }
  out->qstart = q0;
  uint32_t neg[NB] = {0}, start[NB];
  add(neg, P, true);
  for (int i = 0; i < NB; ++i) start[i] = P[i];
  mul(start, (uint32_t)kQOffset);
  mul(S, 128);
  add(start, S, true);
  for (int i = 0; i < kMaxWords; ++i) {
    out->negp[i] = neg[i];
    out->start[i] = start[i];
  }
}

// Words of R: |R| <= k 2^(16 s) < 2^(16 s + 15) for k <= 32704; at least the
// four that words_to_double takes.
constexpr int words_of(int ns) { return ns <= 7 ? 4 : (16 * ns + 16 + 31) / 32; }

// The sums of one entry. The top word needs only its low 32 bits.
template <int NW>
struct Sums {
  unsigned long long a[NW - 1];
  uint32_t top, q;
  __host__ __device__ __forceinline__ void start(const Weights& wt) {
    MOMMS_UNROLL
    for (int i = 0; i < NW - 1; ++i) a[i] = wt.start[i];
    top = wt.start[NW - 1];
    q = wt.qstart;
  }
  __host__ __device__ __forceinline__ void add(uint32_t byte, const uint32_t* w, uint32_t frac) {
    MOMMS_UNROLL
    for (int i = 0; i < NW - 1; ++i) a[i] += (unsigned long long)byte * w[i];
    top += byte * w[NW - 1];
    q += byte * frac;
  }
  // R, two's complement, least word first
  __host__ __device__ __forceinline__ void finish(const Weights& wt, uint32_t (&out)[NW]) const {
    const uint32_t Q = q >> kFracBits;
    unsigned long long c = 0;
    MOMMS_UNROLL
    for (int i = 0; i < NW - 1; ++i) {
      c += a[i] + (unsigned long long)Q * wt.negp[i];
      out[i] = (uint32_t)c;
      c >>= 32;
    }
    out[NW - 1] = (uint32_t)c + top + Q * wt.negp[NW - 1];
  }
};

}  // namespace crt
}  // namespace momms

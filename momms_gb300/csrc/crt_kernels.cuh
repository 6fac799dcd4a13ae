// Device passes of the residue form of the emulated product (crt_elem.cuh):
// operand -> residue planes, and residues of the products -> C.
#pragma once
#include <cuda_fp16.h>

#include "crt_elem.cuh"
#include "planes.cuh"
#include "slicegemm.cuh"

namespace momms {
namespace crt {

static __constant__ ModulusTable c_moduli = make_moduli();

__device__ __forceinline__ uint32_t half2_bits(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// remainder_of of two integers.
__device__ __forceinline__ float2 remainder_of2(float2 t, const Modulus& md) {
  const float2 big = make_float2(12582912.0f, 12582912.0f), nbig = make_float2(-12582912.0f, -12582912.0f);
  const float2 nq = add2(fma2(t, make_float2(-md.inv, -md.inv), big), nbig);
  return fma2(nq, make_float2(md.p, md.p), t);
}

// Residue planes l0..l1-1 of operand views under their row exponents, in the
// run layout of planes.cuh: plane l holds every element's residue modulo
// kModuli[l] as fp16. A thread takes the limbs of its run's 8 elements once
// and walks the moduli with them in registers, one 16-byte store per plane; at
// 8192^2 it writes at 5.6 TB/s.
template <int NS, typename RowExp>
struct ResidueBody {
  using Tin = double;
  static constexpr int RUN = 8, kContigLg = planes::kRowsContigLgPlanes, L = limbs_of(NS);
  template <bool R_CONTIG>
  static int rows(int lg) { return planes::run_rows(lg); }
  template <bool R_CONTIG>
  static int64_t cols(int lg, int iters) { return ((int64_t)RUN << lg) * iters; }
  RowExp re[2];
  __half* out[2];
  int64_t ldp, plane_elems[2];
  int l0, l1;

  template <bool R_CONTIG>
  __device__ __forceinline__ void run(const planes::View<double>& v, int z, const planes::BlockPlace& at) const {
    const planes::Chunk<R_CONTIG> c(v.lg);
    const int64_t pe = plane_elems[z];
    for (int64_t r = (int64_t)at.y * c.rows + c.rl; r < v.R; r += (int64_t)at.ny * c.rows) {
      const int e = re[z].row(r);
      if (at.x == 0 && c.ru == 0) re[z].first(r, e);
      const double* xr = v.x + r * v.sr;
      __half* outr = out[z] + r * ldp;
#pragma unroll 1
      for (int it = 0; it < v.iters; ++it) {
        const int64_t p = planes::run_col(at.x, c, it, RUN, v.iters);
        if (p >= v.K) break;
        float f[RUN][L];
        {
          double x[RUN];
          planes::load_run<R_CONTIG, RUN>(xr, v.sp, p, v.K, v.vec, x);
#pragma unroll
          for (int i = 0; i < RUN; ++i) limbs<NS>(x[i], e, f[i]);
        }
        __half* dst = outr + p;
#pragma unroll 2
        for (int l = l0; l < l1; ++l, dst += pe) {
          const Modulus& md = c_moduli.m[l];
          uint32_t w[RUN / 2];
#pragma unroll
          for (int q = 0; q < RUN / 2; ++q) {
            // residue_of_limbs of the pair, in packed operations
            float2 t = make_float2(f[2 * q][0], f[2 * q + 1][0]);
#pragma unroll
            for (int i = 1; i < L; ++i)
              t = fma2(make_float2(f[2 * q][i], f[2 * q + 1][i]), make_float2(md.limb[i], md.limb[i]), t);
            t = remainder_of2(t, md);
            w[q] = half2_bits(t.x, t.y);
          }
          *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
    }
  }
};

// The same planes from one or two operands' digit planes ([NS][elems], the top
// digit first; packed operands), one per grid row: the residue of
// sum_t digit_t 2^(8 t), exact in FP32. Both in one launch, and digits taken in
// pairs (the FMAs per modulus bound it): 200 x 200 x 200 from packs 31 -> 21 us,
// the pass itself at 1000 x 1000 x 1000 24 -> 19 us.
struct PackedDigits {
  const __half* digits[2];
  int64_t elems[2];
  __half* out[2];
};
template <int NS>
__global__ void __launch_bounds__(256)
    residues_of_digits_kernel(const __grid_constant__ PackedDigits P, int l0, int l1) {
  dependency_wait();
  dependents_may_start();
  const __half* __restrict__ digits = P.digits[blockIdx.y];
  __half* __restrict__ out = P.out[blockIdx.y];
  const int64_t elems = P.elems[blockIdx.y];
  // D pairs of digits (16 bits and a sign), then the digits above them
  constexpr int D = pairs_of_digits(NS), T = NS - D;
  for (int64_t v = (int64_t)blockIdx.x * 256 + threadIdx.x; v * 8 < elems; v += (int64_t)gridDim.x * 256) {
    float2 f[T][4];
#pragma unroll
    for (int t = 0; t < T; ++t) {
      // the pair's low digit and its high one, or one digit above the pairs
      const int low = t < D ? NS - 1 - 2 * t : NS - 1 - D - t;
      const uint4 u = __ldg(reinterpret_cast<const uint4*>(digits + low * elems) + v);
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) f[t][q] = __half22float2(*reinterpret_cast<const __half2*>(&w[q]));
      if (t < D) {
        const uint4 h = __ldg(reinterpret_cast<const uint4*>(digits + (low - 1) * elems) + v);
        const uint32_t x[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
        for (int q = 0; q < 4; ++q)
          f[t][q] = fma2(__half22float2(*reinterpret_cast<const __half2*>(&x[q])), make_float2(256.0f, 256.0f), f[t][q]);
      }
    }
    __half* dst = out + v * 8;
#pragma unroll 2
    for (int l = l0; l < l1; ++l, dst += elems) {
      const Modulus& md = c_moduli.m[l];
      uint32_t o[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float2 t = f[0][q];
#pragma unroll
        for (int i = 1; i < T; ++i) {
          const float c = md.digit[i < D ? 2 * i : D + i];
          t = fma2(f[i][q], make_float2(c, c), t);
        }
        t = remainder_of2(t, md);
        o[q] = half2_bits(t.x, t.y);
      }
      *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

template <int NS>
void launch_residues_of_digits(const PackedDigits& p, int count, int l0, int l1, int sm_count, cudaStream_t s) {
  const int64_t most = count > 1 ? (p.elems[0] > p.elems[1] ? p.elems[0] : p.elems[1]) : p.elems[0];
  const int64_t blocks = std::min<int64_t>(ceil_div_dev(most / 8, 256), (int64_t)sm_count * 8);
  launch_dependent(residues_of_digits_kernel<NS>, dim3((unsigned)blocks, (unsigned)count), 256, 0, s, p, l0, l1);
}

struct CombineParams {
  const uint8_t* res;  // residue planes of the products (sp::Params, residue form)
  int64_t plane;       // bytes per plane
  int64_t mpad;
  int moduli;
  int scale_off;  // -16 s
  int alpha_sign, beta_zero;  // alpha_sign: 1 or -1 when alpha is that, else 0
  int64_t m;
  int64_t j0, j1;  // columns of C this launch finishes (j0 a multiple of 4)
  const int* row_exp;
  const int* col_exp;
  double alpha, beta;
  double* c;
  int64_t rsc, csc;
  Weights wt;
};

// A thread finishes four columns of one row: one 32-bit load per modulus, R of
// each entry by the remainder theorem (NW words), one rounding, C's update.
// Per entry and modulus that is NW - 1 wide and two plain multiply-adds with
// constant-bank operands, which is why the modulus count N is a template
// argument (a runtime count, its weights fetched by indexed constant loads:
// 342 instructions per entry and 1.32 ms at 8192^2 with 16 moduli).
template <int NW, int N>
__global__ void __launch_bounds__(256, NW == 4 ? 4 : (NW <= 6 ? 3 : 2)) combine_kernel(const __grid_constant__ CombineParams p) {
  dependency_wait();
  const int64_t row = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (row >= p.m) return;
  const int er = p.row_exp[row];
  // a block's place in the planes is uniform; only the row within its two tiles varies
  const uint32_t roff = (threadIdx.x / sp::BM) * (sp::BM * sp::BN) + 4 * (threadIdx.x % sp::BM);
  const uint8_t* base = p.res + (int64_t)blockIdx.x * (2 * sp::BM * sp::BN);
  double* crow = p.c + row * p.rsc;
  // a sign flipped as an FP64 negation would be an FP64 addition
  const long long flip = p.alpha_sign < 0 ? (long long)(1ull << 63) : 0;
  for (int64_t j = p.j0 + 4 * (int64_t)blockIdx.y; j < p.j1; j += 4 * (int64_t)gridDim.y) {
    const uint8_t* src = base + (j / sp::BN) * (p.mpad * sp::BN) + (j % sp::BN) * sp::BM;
    const int live = (int)min((int64_t)4, p.j1 - j);
    uint32_t w[N];
#pragma unroll
    for (int l = 0; l < N; ++l) w[l] = __ldcs(reinterpret_cast<const unsigned*>(src + l * p.plane + roff));
    double* cp = crow + j * p.csc;
    double c_old[4] = {0.0, 0.0, 0.0, 0.0};
    if (!p.beta_zero) {
      const double* q = cp;
#pragma unroll
      for (int i = 0; i < 4; ++i, q += p.csc)
        if (i < live) c_old[i] = *q;
    }
    Sums<NW> sum[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) sum[q].start(p.wt);
    // moduli outermost: a modulus' weights are fetched once for the four entries
#pragma unroll
    for (int l = 0; l < N; ++l)
#pragma unroll
      for (int q = 0; q < 4; ++q) sum[q].add(__byte_perm(w[l], 0, 0x4440 + q), p.wt.w[l], p.wt.frac[l]);
#pragma unroll
    for (int q = 0; q < 4; ++q, cp += p.csc) {
      if (q >= live) break;
      const int ec = p.col_exp[j + q];
      double v;
      if (er == INT32_MAX || ec == INT32_MAX) {
        v = __longlong_as_double(0x7ff8000000000000ll);
      } else {
        uint32_t R[NW];
        sum[q].finish(p.wt, R);
        v = words_to_double<NW>(R, er + ec + p.scale_off);
      }
      // FP64 operations cost 0.12 ms each at 8192^2: alpha = 1 and -1 take none.
      // (asm volatile: the compiler would multiply and select.)
      v = __longlong_as_double(__double_as_longlong(v) ^ flip);
      if (p.alpha_sign == 0) asm volatile("mul.rn.f64 %0, %0, %1;" : "+d"(v) : "d"(p.alpha));
      if (!p.beta_zero) asm volatile("fma.rn.f64 %0, %1, %2, %0;" : "+d"(v) : "d"(p.beta), "d"(c_old[q]));
      *cp = v;
    }
  }
}

}  // namespace crt
}  // namespace momms

// The slice-pair GEMM engine on tcgen05: C-tile accumulation of sums of
// products of operand "planes" (precision slices of A and B) through TMEM.
//
//   for each output tile (persistent, one CTA per SM, 128 x 256 tiles):
//     for each group g (processed in order):
//       S_g = sum over pairs (a, b) in g of  A_plane[a] * B_plane[b]^T
//       accumulated in TMEM in chunks (runs of (pair, k-block) steps within a
//       bound, Params::pair_w); each finished chunk is handed to the
//       epilogue (ping-pong TMEM buffers)
//
// Planes are K-major in HBM ([plane][row][k], k contiguous) and are loaded by
// TMA as 128-byte-wide k-blocks with the 128B swizzle that the tcgen05 shared
// memory descriptors expect. Warp roles: warp 0 issues TMA, warp 1 (one
// thread) issues tcgen05.mma and commits, warps 2..9 drain TMEM.
//
// Three epilogues:
//   EPI_F32   : one group; finished chunks are summed in FP32 registers
//               (round to nearest) and C = alpha*sum + beta*C is written at
//               the end of the tile. Used by the split-TF32 f32 path (pairs
//               lo*hi, hi*lo, hi*hi).
//   EPI_OZAKI : integer-valued slices; every chunk is exact in FP32 (the
//               host sizes chunks so that sums of absolute products stay
//               within 2^24) and is converted and added into int32
//               accumulators; at the end of each group the
//               exact sums are written to that group's int32 plane (the FP64
//               recombination runs afterwards in its own kernel, so no FP64
//               work sits in this pipeline).
//   EPI_BOUND : one group of one pair, bf16 magnitude planes |a| 2^-e_i and
//               |b| 2^-f_j rounded toward zero: the FP32 sum is a lower bound
//               L_ij of (|A||B|)_ij 2^-(e_i+f_j) (after a factor for the
//               accumulation's rounding). Nothing is stored per entry: each
//               tile reduces the worst-case error ratios
//                 q1 = (sum_p |a_ip| 2^-e_i + sum_p |b_pj| 2^-f_j) / L_ij,
//                 q2 = k / L_ij
//               (upward-rounded) to two maxima posted with atomicMax, and
//               counts the entries with L_ij = 0; from these the host picks a
//               slice count that holds for every entry. With count_only the
//               planes are 0/1 indicators of nonzero elements and only the
//               entries with a nonzero sum are counted.
#pragma once
#include <stdlib.h>

#include <algorithm>
#include <atomic>
#include <type_traits>
#include <vector>

#include "tc_common.cuh"

namespace momms {
namespace sp {

// A stage holds one k-block of each operand: 128 bytes of k per row (64 fp16
// or 32 fp32 elements) in the 128-byte swizzle. (64-byte k-blocks with the
// 64-byte swizzle fit nine stages instead of four but measured 25 % slower:
// twice the TMA row requests per byte.)
constexpr int BM = 128, BN = 256, STAGES = 4;
constexpr int ROW_BYTES = 128;
constexpr int KSTEPS = ROW_BYTES / 32;  // MMAs per stage (each consumes 32 bytes of k)
constexpr int A_TILE = BM * ROW_BYTES;
constexpr int B_TILE = BN * ROW_BYTES;
constexpr int STAGE_BYTES = A_TILE + B_TILE;  // 48 KB
constexpr int EPI_WARPS = 8;                     // 2 per TMEM lane quarter
constexpr int EPI_COLS = BN / (EPI_WARPS / 4);   // columns drained per thread
constexpr int THREADS = (2 + EPI_WARPS) * 32;
constexpr int TMEM_COLS = 512;  // two 128 x 256 f32 accumulators
constexpr int SMEM_BYTES = 1024 + STAGES * STAGE_BYTES + 256;
constexpr int MAX_GROUPS = 160, MAX_PAIRS = 160, MAX_MODULI = 36;

enum { EPI_F32 = 0, EPI_OZAKI = 1, EPI_BOUND = 2 };

struct Params {
  int64_t m, n;
  int kblocks;  // k-blocks per plane
  int kelems;   // elements per k-block (64 for f16, 32 for tf32: 128 bytes)
  int tiles_m, tiles_n;
  int ngroups;
  int gchunk;  // groups per work unit: a tile's groups may run as separate units (0 = all)
  int group_begin[MAX_GROUPS + 1];
  // TMEM accumulation chunks: a chunk is a run of consecutive (pair, k-block)
  // steps of one group whose weights pair_w sum to at most chunk_cap; with
  // merge_pairs a chunk continues from one pair into the next (the Ozaki
  // path, whose chunk sums are exact, so chunking never changes a result),
  // otherwise every pair starts a new chunk. group_chunks[g]: chunks of
  // group g (plan_chunks).
  int pair_w[MAX_PAIRS];
  int chunk_cap, merge_pairs;
  int group_chunks[MAX_GROUPS];
  uint8_t pair_a[MAX_PAIRS], pair_b[MAX_PAIRS];
  // EPI_F32
  float alpha_f, beta_f;
  float* c32;
  // EPI_OZAKI: exact group sums, one int32 plane per group, tile-blocked:
  // element (row, col) at (col / BN) * (tiles_m * BM * BN) + (row / BM) * BM * BN
  // + (col % BN) * BM + row % BM, so that each CTA tile is written as one
  // contiguous block
  // Residue form (residue != 0): group g is one modulus, its sum is reduced
  // to a symmetric residue r and its plane holds bytes (r + 128) mod 256: four
  // columns of a row per 32-bit word, word (col / 4, row) of a tile at
  // (col % BN / 4) * BM + row % BM (the tile's 32 KB block in the same place)
  int* sbuf;
  int64_t plane;  // bytes between group planes in the residue form, else ints
  int64_t rsc, csc;
  int residue;
  struct Modulus {
    float p, inv;
  } mod[MAX_MODULI];
  // EPI_BOUND: row sums of the scaled magnitudes of A (m) and B's columns
  // (n) in units of 2^-40, each term rounded up; k; the maxima (bit patterns of
  // non-negative floats)
  const unsigned long long* msum_a;
  const unsigned long long* msum_b;
  float kf;
  unsigned* bound_out;                // [0], [1]: the maxima; [4], [5]: the largest row sum of A's and B's magnitudes
  unsigned long long* bound_count;  // entries counted
  int count_only;
  int64_t unit_begin;  // grouped launches: this problem's first work unit
  unsigned* status;
};

// A grouped launch of the CTA-pair kernel: many problems, each with its own
// Params (schedule, sizes, output) and tensor maps, in device memory. Work
// unit u belongs to the last problem whose unit_begin <= u.
struct GroupTable {
  const Params* probs;      // sorted by unit_begin
  const CUtensorMap* maps;  // [2 * nprobs]: each problem's A map and B half-tile map (64-byte aligned)
  int nprobs;
  int64_t units;
};

__device__ __forceinline__ bool aborted(volatile int* flag) { return *flag != 0; }

// Output tile of work item t: groups of 16 m-tiles swept n-tile by n-tile,
// so that the ~152 tiles in flight at once share 16 A row panels and about
// 10 B column panels of each slice plane in L2 (a plain column-major sweep
// would touch a whole 128 MB plane per pair at m = 8192).
template <int G>
__device__ __forceinline__ void tile_coords(int64_t t, int tiles_m, int tiles_n, int& tm, int& tn) {
  const int64_t per_group = (int64_t)G * tiles_n;
  const int64_t g = t / per_group, r = t % per_group;
  const int first = (int)(g * G);
  const int gm = min(G, tiles_m - first);
  tm = first + (int)(r % gm);
  tn = (int)(r / gm);
}

// Accumulators of drained chunks: Ozaki sums are int32 (each chunk value is
// an integer of magnitude <= 2^24, exact in FP32, converted exactly);
// split-TF32 sums are FP32.
template <int EPI>
using EpiAcc = typename std::conditional<EPI == EPI_OZAKI, int, float>::type;

// Drains one TMEM chunk (this thread's row, NC columns from taddr) into S.
// The loads run one 16-column batch ahead of the adds: a batch's wait comes
// after the previous batch's adds.
template <int EPI, int NC>
__device__ __forceinline__ void drain_chunk(uint32_t taddr, EpiAcc<EPI> (&S)[NC]) {
  uint32_t ra[16], rb[16];
  tc::ld16(taddr, ra);
#pragma unroll
  for (int pc = 0; pc < NC / 16; ++pc) {
    uint32_t(&cur)[16] = (pc & 1) ? rb : ra;
    uint32_t(&nxt)[16] = (pc & 1) ? ra : rb;
    tc::ld_wait(cur);
    if (pc + 1 < NC / 16) tc::ld16(taddr + (pc + 1) * 16, nxt);
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      if (EPI == EPI_OZAKI) S[pc * 16 + j] += __float2int_rz(__uint_as_float(cur[j]));
      else S[pc * 16 + j] += __uint_as_float(cur[j]);
    }
  }
}

// EPI_BOUND: this thread's row against its NC columns, reduced over the warp
// and posted to the maxima. Every lane calls it (rows past m contribute 0).
// `sb`: shared memory for this warp's NC column sums.
//
// The maxima are of quotients by S, upward but for the reciprocal: q1's are
// products with the hardware's approximate one (at most one unit in the last
// place off, 2^-23), six instructions per entry with the sum's own. The host
// raises them by that and scales S down to its lower bound in FP64
// (bound_quotients). In all they are above the entries' own by at most 2^-21, as
// four upward-rounded FP32 operations would leave them. (Those, formed where they
// could raise the maximum, and column sums by shuffle took 25 of the 30 us of a
// 512 x 512 x 512 bound, 0.23 ms at 8192 x 8192 x 64; a second look at the
// entries near the maximum, for the exact one, cost 1-4 us of 14.)
//
// The sums of magnitudes are read before the tile's product is there
// (bound_sums), and the posted maxima all at once: each is a trip to L2 or
// beyond that nothing else would hide. With the columns past n set apart and a
// reciprocal without denormals (20 instructions per entry before): 512 x 512 x
// 512 16.4 -> 14.2 us, 8192 x 8192 x 256 100 -> 67.
struct BoundSums {
  float sa = 0.0f, mb = 0.0f;  // this row's sum; the largest column sum this lane read
};
template <int NC>
__device__ __forceinline__ BoundSums bound_sums(const Params& p, int64_t row, int64_t col0, float* sb) {
  BoundSums b;
  if (p.count_only) return b;
  const int lane = threadIdx.x & 31, nvalid = (int)min((int64_t)NC, max((int64_t)0, p.n - col0));
  unsigned long long w[NC / 32], a = 0;
#pragma unroll
  for (int q = 0; q < NC / 32; ++q) w[q] = 32 * q + lane < nvalid ? p.msum_b[col0 + 32 * q + lane] : 0;
  if (row < p.m) a = p.msum_a[row];
#pragma unroll
  for (int q = 0; q < NC / 32; ++q) {
    const float v = __fmul_ru(__ull2float_ru(w[q]), 0x1p-40f);
    sb[32 * q + lane] = v;
    b.mb = fmaxf(b.mb, v);
  }
  b.sa = __fmul_ru(__ull2float_ru(a), 0x1p-40f);
  __syncwarp();
  return b;
}
template <int NC>
__device__ __forceinline__ void bound_tile(const Params& p, int64_t row, int64_t col0, float (&S)[NC],
                                           const BoundSums& sums, float* sb) {
  const int lane = threadIdx.x & 31;
  float m1 = 0.0f, m2 = 0.0f, ma = sums.sa, mb = sums.mb;
  unsigned cnt = 0;
  // columns of this tile inside C (the same for the whole warp)
  const int nvalid = (int)min((int64_t)NC, max((int64_t)0, p.n - col0));
  const bool rv = row < p.m;
  if (p.count_only) {
    if (rv) {
#pragma unroll
      for (int j = 0; j < NC; ++j) cnt += (j < nvalid && S[j] > 0.0f) ? 1u : 0u;
    }
  } else {
    if (rv) {
      const float sa = sums.sa;
      float smin = INFINITY;
      // columns past n count as covered
      if (nvalid < NC) {
#pragma unroll
        for (int j = 0; j < NC; ++j) S[j] = j < nvalid ? S[j] : INFINITY;
      }
#pragma unroll
      for (int j = 0; j < NC; j += 4) {
        const float4 b4 = *reinterpret_cast<const float4*>(sb + j);
        const float b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float s = S[j + q];
          float r;  // a sum that flushes to zero takes the row through the other loop
          asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(s));
          m1 = fmaxf(m1, __fmul_ru(__fadd_ru(sa, b[q]), r));
          smin = fminf(smin, s);
        }
      }
      // S = 0: no p with both a_ip and b_pj nonzero (the entry has no error), or
      // every term below FP32's range: counted, the host tells the two apart.
      // Such rows (and any whose smallest sum an approximate reciprocal would
      // take past FP32's range) go through their entries again.
      if (smin < 0x1p-100f) {
        m1 = 0.0f;
        smin = INFINITY;
#pragma unroll 1
        for (int j = 0; j < nvalid; ++j) {
          float s = 0.0f;
#pragma unroll
          for (int q = 0; q < NC; ++q) s = q == j ? S[q] : s;
          if (s > 0.0f) {
            m1 = fmaxf(m1, __fdiv_ru(__fadd_ru(sa, sb[j]), s));
            smin = fminf(smin, s);
          } else {
            ++cnt;
          }
        }
      }
      if (smin < INFINITY) m2 = __fdiv_ru(p.kf, smin);
    }
    __syncwarp();  // before the next tile's column sums
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    m1 = fmaxf(m1, __shfl_xor_sync(0xffffffffu, m1, o));
    m2 = fmaxf(m2, __shfl_xor_sync(0xffffffffu, m2, o));
    ma = fmaxf(ma, __shfl_xor_sync(0xffffffffu, ma, o));
    mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, o));
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  }
  if (lane == 0) {
    // Non-negative floats order like their bit patterns. Every warp of every
    // tile reports here: the maxima only grow, so a warp below the value
    // already posted skips its atomic (same-address atomics serialise in L2;
    // at 8192 x 8192 x 64 they cost most of the kernel).
    if (!p.count_only) {
      const volatile unsigned* cur = p.bound_out;
      const unsigned c0 = cur[0], c1 = cur[1], c4 = cur[4], c5 = cur[5];
      if (__float_as_uint(m1) > c0) atomicMax(&p.bound_out[0], __float_as_uint(m1));
      if (__float_as_uint(m2) > c1) atomicMax(&p.bound_out[1], __float_as_uint(m2));
      if (__float_as_uint(ma) > c4) atomicMax(&p.bound_out[4], __float_as_uint(ma));
      if (__float_as_uint(mb) > c5) atomicMax(&p.bound_out[5], __float_as_uint(mb));
    }
    if (cnt) atomicAdd(p.bound_count, (unsigned long long)cnt);
  }
}

// Split-TF32 epilogue: asks L2 for the C lines this thread's warp will
// read at the end of the tile (beta != 0), issued when the tile starts, so
// that the epilogue's loads of C hit L2 instead of HBM. Column-major C: a
// warp's 32 rows of one column are one 128-byte line, so lane L takes the
// columns L, L + 32, ... of the thread's EPI_COLS; other layouts are left to
// the loads themselves.
template <int NC>
__device__ __forceinline__ void prefetch_c_rows(const Params& p, int64_t row_of_lane0, int64_t col0, int lane) {
  if (p.beta_f == 0.0f || p.rsc != 1 || row_of_lane0 >= p.m) return;
  const float* base = p.c32 + row_of_lane0;
#pragma unroll
  for (int j = lane; j < NC; j += 32) {
    const int64_t col = col0 + j;
    if (col < p.n) asm volatile("prefetch.global.L2 [%0];" ::"l"(base + col * p.csc));
  }
}

// Symmetric residues of exact integers |v| <= 2^24: at most p/2 and a
// rounding of the quotient beyond (|r| <= 128). Two at a time: the FP32
// operations are packed pairs. nq: the nearest integers to -v/p.
struct ResidueOf {
  float2 ninv, p;
  __device__ __forceinline__ explicit ResidueOf(const Params::Modulus& m)
      : ninv(make_float2(-m.inv, -m.inv)), p(make_float2(m.p, m.p)) {}
  __device__ __forceinline__ float2 operator()(float2 v) const {
    const float2 big = make_float2(12582912.0f, 12582912.0f), nbig = make_float2(-12582912.0f, -12582912.0f);
    const float2 nq = add2(fma2(v, ninv, big), nbig);
    return fma2(nq, p, v);
  }
};

// Walks one TMEM chunk (this thread's row, NC columns from taddr) 16 columns
// at a time, the next batch's load in flight: fn(first column, 16 values).
template <int NC, typename F>
__device__ __forceinline__ void for_batches(uint32_t taddr, F&& fn) {
  uint32_t ra[16], rb[16];
  tc::ld16(taddr, ra);
#pragma unroll
  for (int pc = 0; pc < NC / 16; ++pc) {
    uint32_t(&cur)[16] = (pc & 1) ? rb : ra;
    uint32_t(&nxt)[16] = (pc & 1) ? ra : rb;
    tc::ld_wait(cur);
    if (pc + 1 < NC / 16) tc::ld16(taddr + (pc + 1) * 16, nxt);
    fn(pc * 16, cur);
  }
}

// The bytes of four symmetric residues, one word. Under the exponent of 2^23
// a float's low byte is (r + 128) mod 256; modulo 255 a residue of 128 would
// not survive that (modulo 256 it does), so it becomes -127 first.
template <bool P255>
__device__ __forceinline__ uint32_t residue_bytes(float2 a, float2 b) {
  if (P255) {
    a.x = a.x > 127.0f ? -127.0f : a.x;
    a.y = a.y > 127.0f ? -127.0f : a.y;
    b.x = b.x > 127.0f ? -127.0f : b.x;
    b.y = b.y > 127.0f ? -127.0f : b.y;
  }
  const float2 k = make_float2(8388736.0f, 8388736.0f);
  a = add2(a, k);
  b = add2(b, k);
  return __byte_perm(__byte_perm(__float_as_uint(a.x), __float_as_uint(a.y), 0x0040),
                     __byte_perm(__float_as_uint(b.x), __float_as_uint(b.y), 0x0040), 0x5410);
}

// One residue group of one tile: its chunks' residues to the plane's words
// `out` of this thread's row (see Params::sbuf), `live` columns of it. Each
// chunk's values are reduced in FP32 (three packed operations of the wide FMA
// pipe per pair; the conversion to int32 of the digit form runs at an eighth
// of that pipe's rate).
template <int NC, bool P255, typename Wait, typename Release>
__device__ __forceinline__ bool residue_group(const Params::Modulus& m, int chunks, uint32_t* out, int live, Wait&& wait,
                                              Release&& release) {
  const ResidueOf res(m);
  auto pair = [](const uint32_t(&v)[16], int j) { return make_float2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])); };
  if (chunks == 1) {
    // straight from TMEM to bytes
    const uint32_t taddr = wait();
    if (taddr == ~0u) return false;
    for_batches<NC>(taddr, [&](int j0, const uint32_t(&v)[16]) {
#pragma unroll
      for (int j = 0; j < 16; j += 4) {
        const uint32_t w = residue_bytes<P255>(res(pair(v, j)), res(pair(v, j + 2)));
        if (j0 + j < live) out[((j0 + j) / 4) * BM] = w;
      }
    });
    release();
    return true;
  }
  // several chunks: the residues, plus 128, are summed as pairs of 16-bit
  // fields (at most 32 chunks of at most 256), half the registers of FP32 sums
  uint32_t S[NC / 2];
#pragma unroll
  for (int j = 0; j < NC / 2; ++j) S[j] = 0;
  for (int c = 0; c < chunks; ++c) {
    const uint32_t taddr = wait();
    if (taddr == ~0u) return false;
    for_batches<NC>(taddr, [&](int j0, const uint32_t(&v)[16]) {
#pragma unroll
      for (int j = 0; j < 16; j += 2) {
        const float2 r = add2(res(pair(v, j)), make_float2(8388736.0f, 8388736.0f));
        S[(j0 + j) / 2] += __byte_perm(__float_as_uint(r.x), __float_as_uint(r.y), 0x5410);
      }
    });
    release();
  }
  const float nbias = -(8388608.0f + 128.0f * (float)chunks);
  auto sum = [&](int i) {
    return add2(make_float2(__uint_as_float(0x4B000000u | (S[i] & 0xffffu)), __uint_as_float(0x4B000000u | (S[i] >> 16))),
                make_float2(nbias, nbias));
  };
#pragma unroll
  for (int j = 0; j < NC; j += 4) {
    const uint32_t w = residue_bytes<P255>(res(sum(j / 2)), res(sum(j / 2 + 1)));
    if (j < live) out[(j / 4) * BM] = w;
  }
  return true;
}

// EPI_OZAKI: publishes a group's exact int32 sums of this thread's row.
template <int NC>
__device__ __forceinline__ void publish_sums(int* out, int live, const int (&S)[NC]) {
#pragma unroll
  for (int j = 0; j < NC; ++j)
    if (j < live) out[j * BM] = S[j];
}

// The epilogue of EPI_OZAKI's groups [g0, g1) of one tile: wait() returns
// the TMEM address of the next finished chunk or ~0 on a timeout, release()
// hands its buffer back. Returns false on a timeout.
template <int NC, typename Wait, typename Release>
__device__ __forceinline__ bool ozaki_groups(const Params& p, int g0, int g1, int64_t row, int64_t col0, int tm, int tn,
                                             int col_in_tile, int r_local, Wait&& wait, Release&& release) {
  const int live = row < p.m ? (int)max((int64_t)0, min((int64_t)NC, p.n - col0)) : 0;
  const size_t tile = (size_t)tn * ((size_t)p.tiles_m * BM * BN) + (size_t)tm * (BM * BN);
  for (int g = g0; g < g1; ++g) {
    const int chunks = p.group_chunks[g];
    if (p.residue) {
      uint32_t* out = reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(p.sbuf) + (size_t)g * p.plane + tile) +
                      (size_t)(col_in_tile / 4) * BM + r_local;
      const bool ok = p.mod[g].p == 255.0f ? residue_group<NC, true>(p.mod[g], chunks, out, live, wait, release)
                                           : residue_group<NC, false>(p.mod[g], chunks, out, live, wait, release);
      if (!ok) return false;
    } else {
      int S[NC];
#pragma unroll
      for (int j = 0; j < NC; ++j) S[j] = 0;
      for (int c = 0; c < chunks; ++c) {
        const uint32_t taddr = wait();
        if (taddr == ~0u) return false;
        drain_chunk<EPI_OZAKI, NC>(taddr, S);
        release();
      }
      // tile-blocked plane: this CTA's 128 x 256 tile is one contiguous block,
      // column after column of 128 rows (see the host's plane layout)
      publish_sums<NC>(p.sbuf + (size_t)g * p.plane + tile + (size_t)col_in_tile * BM + r_local, live, S);
    }
  }
  return true;
}

// The epilogue of EPI_F32 and EPI_BOUND for one tile (groups [g0, g1)), as ozaki_groups.
template <int EPI, int NC, typename Wait, typename Release>
__device__ __forceinline__ bool float_groups(const Params& p, int g0, int g1, int64_t row, int64_t col0, Wait&& wait,
                                             Release&& release, float* sb) {
  // per-thread FP32 sums of finished chunks, rounded to nearest, which keeps
  // the tensor core's internal accumulation to one chunk at a time
  float S[NC];
  BoundSums sums;
  if constexpr (EPI == EPI_BOUND) sums = bound_sums<NC>(p, row, col0, sb);
#pragma unroll
  for (int j = 0; j < NC; ++j) S[j] = 0.0f;
  for (int g = g0; g < g1; ++g) {
    for (int c = 0; c < p.group_chunks[g]; ++c) {
      const uint32_t taddr = wait();
      if (taddr == ~0u) return false;
      drain_chunk<EPI_F32, NC>(taddr, S);
      release();
    }
  }
  if constexpr (EPI == EPI_BOUND) bound_tile<NC>(p, row, col0, S, sums, sb);
  if (EPI == EPI_F32 && row < p.m) {
    // C is read 8 columns at a time, every load of a group issued before
    // the first use (one memory round trip per group, not per element)
    float* crow = p.c32 + row * p.rsc;
#pragma unroll
    for (int j0 = 0; j0 < NC; j0 += 8) {
      float c0[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int64_t col = col0 + j0 + j;
        c0[j] = (p.beta_f != 0.0f && col < p.n) ? crow[col * p.csc] : 0.0f;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int64_t col = col0 + j0 + j;
        if (col < p.n) {
          const float v = (float)S[j0 + j] * p.alpha_f;
          crow[col * p.csc] = (p.beta_f == 0.0f) ? v : fmaf(p.beta_f, c0[j], v);
        }
      }
    }
  }
  return true;
}

// C's columns [c0, c1) of a tile from the sums of the cluster's CTAs (each
// BM x BN by columns at `part` of its shared memory), added in rank order.
// A warp takes one column at a time, a lane four of its rows.
__device__ __forceinline__ void reduce_columns(const Params& p, const float* part, int64_t row0, int64_t col0, int c0,
                                               int c1, int ranks, int warp, int lane) {
  const int64_t row = row0 + lane * 4;
  const int rows = (int)min((int64_t)4, p.m - row);
  for (int c = c0 + warp; c < c1; c += THREADS / 32) {
    if (col0 + c >= p.n) break;
    float* cp = p.c32 + row * p.rsc + (col0 + c) * p.csc;
    float old[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (p.beta_f != 0.0f) {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (q < rows) old[q] = cp[q * p.rsc];
    }
    const float* src = part + c * BM + lane * 4;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
    for (int r = 0; r < ranks; ++r) {
      const float4 w = ld_cluster_f4(mapa_shared(src, (uint32_t)r));
      v.x += w.x, v.y += w.y, v.z += w.z, v.w += w.w;
    }
    const float out[4] = {v.x * p.alpha_f, v.y * p.alpha_f, v.z * p.alpha_f, v.w * p.alpha_f};
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (q < rows) cp[q * p.rsc] = p.beta_f == 0.0f ? out[q] : fmaf(p.beta_f, old[q], out[q]);
  }
}

// Split (EPI_F32, few tiles): a cluster of CTAs per tile, each with a range of
// the k-blocks of every pair. Each CTA leaves its sums in shared memory, and
// reduces a range of the tile's columns over the cluster, in rank order. One
// CTA's chain of MMAs bounds such a product (0.33 us per k-block of a pair):
// split-TF32 1024 x 1024 x 1024 52 -> 29 us as 4 CTAs per tile. The exchange
// through the cluster's shared memory needs no scratch and no second kernel.
template <int KIND, int EPI, bool SPLIT = false>
__global__ void __launch_bounds__(THREADS, 1)
    slice_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const __grid_constant__ Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;  // [2]
  uint64_t* tempty = tfull + 2;      // [2]
  uint64_t* drain = tempty + 2;      // used only when aborting
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // work units: output tiles (times group chunks), one CTA each
  const int64_t unit0 = SPLIT ? (int64_t)cluster_id_x() : (int64_t)blockIdx.x;
  const int64_t unit_step = SPLIT ? (int64_t)cluster_count_x() : (int64_t)gridDim.x;
  const int rank = SPLIT ? (int)cluster_ctarank() : 0, ranks = SPLIT ? (int)cluster_nctarank() : 1;
  const int kb0 = p.kblocks * rank / ranks, kb1 = p.kblocks * (rank + 1) / ranks;
  const int units_m = p.tiles_m;
  // work unit t: tile (pair) t % tile_units, groups [g_begin(t), g_end(t)) -
  // group-major, so that units in flight read the same digit planes
  const int64_t tile_units = (int64_t)units_m * p.tiles_n;
  const int gchunk = p.gchunk > 0 ? p.gchunk : p.ngroups;
  const int64_t units = tile_units * ceil_div_dev(p.ngroups, gchunk);
  auto g_begin = [&](int64_t t) { return (int)(t / tile_units) * gchunk; };
  auto g_end = [&](int64_t t) { return min(p.ngroups, g_begin(t) + gchunk); };
  // round r hands units [r*step, (r+1)*step) to the CTAs (clusters), in
  // reverse order on odd rounds: units are ordered by falling cost (largest
  // groups first), so this snake order evens out the per-CTA totals
  auto unit_at = [&](int64_t r) {
    return r * unit_step + ((r & 1) ? (unit_step - 1 - unit0) : unit0);
  };
  auto coords = [&](int64_t t, int& tm, int& tn) { tile_coords<16>(t, units_m, p.tiles_n, tm, tn); };

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], EPI_WARPS);
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(tmem_slot, TMEM_COLS);
    tc::tmem_relinquish();
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem_base = *tmem_slot;
  dependency_wait_few();

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      prefetch_tensormap(&tmA);
      prefetch_tensormap(&tmB);
      int stage = 0;
      uint32_t ph = 0;
      uint32_t armed = 0;  // bit s: stage s has been armed at least once
      uint32_t last_ph = 0;  // bit s: parity of the phase last armed on stage s
      for (int64_t r = 0; r * unit_step < units && !aborted(abort_flag); ++r) {
        const int64_t t = unit_at(r);
        if (t >= units) continue;
        int tm, tn;
        coords(t % tile_units, tm, tn);
        for (int g = g_begin(t); g < g_end(t); ++g) {
          for (int pi = p.group_begin[g]; pi < p.group_begin[g + 1]; ++pi) {
            for (int kb = kb0; kb < kb1; ++kb) {
              if (!mbar_wait_bounded(&empty[stage], ph ^ 1)) {
                report_status(p.status, DEV_TIMEOUT_EMPTY);
                *abort_flag = 1;
                // let every copy already issued land before the CTA exits
                for (int s = 0; s < STAGES; ++s)
                  if ((armed >> s) & 1u) mbar_wait_bounded(&full[s], (last_ph >> s) & 1u);
                goto producer_done;
              }
              armed |= 1u << stage;
              last_ph = (last_ph & ~(1u << stage)) | (ph << stage);
              mbar_arrive_expect_tx(&full[stage], STAGE_BYTES);
              uint8_t* sa = smem + stage * STAGE_BYTES;
              tma_load_3d(sa, &tmA, &full[stage], kb * p.kelems, tm * BM, p.pair_a[pi]);
              tma_load_3d(sa + A_TILE, &tmB, &full[stage], kb * p.kelems, tn * BN, p.pair_b[pi]);
              if (++stage == STAGES) {
                stage = 0;
                ph ^= 1;
              }
            }
          }
        }
      }
    producer_done:;
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    if (lane == 0) {
      const uint32_t idv = tc::idesc(tc::kind_fmt(KIND), BM, BN);
      int stage = 0;
      uint32_t ph = 0;
      int buf = 0;
      uint32_t acc_ph[2] = {0, 0};
      for (int64_t r = 0; r * unit_step < units && !aborted(abort_flag); ++r) {
        const int64_t t = unit_at(r);
        if (t >= units) continue;
        for (int g = g_begin(t); g < g_end(t); ++g) {
          int load = 0;
          bool open = false;
          uint32_t d_tmem = 0;
          for (int pp = p.group_begin[g]; pp < p.group_begin[g + 1]; ++pp) {
            const int w = p.pair_w[pp];
            if (open && !p.merge_pairs) {
              tc::commit(&tfull[buf]);
              acc_ph[buf] ^= 1;
              buf ^= 1;
              open = false;
            }
            for (int st = kb0; st < kb1;) {
              if (open && load + w > p.chunk_cap) {
                tc::commit(&tfull[buf]);
                acc_ph[buf] ^= 1;
                buf ^= 1;
                open = false;
              }
              bool fresh = false;
              if (!open) {
                if (!mbar_wait_bounded(&tempty[buf], acc_ph[buf] ^ 1)) {
                  report_status(p.status, DEV_TIMEOUT_TMEM);
                  *abort_flag = 1;
                  goto mma_done;
                }
                tc::fence_after();
                d_tmem = tmem_base + (uint32_t)(buf * BN);
                load = 0;
                open = fresh = true;
              }
              // the k-blocks of this pair that still fit in the open chunk
              const int s0 = st, s1 = min(kb1, st + (p.chunk_cap - load) / w);
              for (; st < s1; ++st) {
                if (!mbar_wait_bounded(&full[stage], ph)) {
                  report_status(p.status, DEV_TIMEOUT_FULL);
                  *abort_flag = 1;
                  goto mma_done;
                }
                tc::fence_after();
                const uint32_t a_addr = smem_u32(smem + stage * STAGE_BYTES);
                const uint32_t b_addr = a_addr + A_TILE;
#pragma unroll
                for (int kk = 0; kk < KSTEPS; ++kk)
                  tc::mma<KIND>(d_tmem, tc::sdesc_k128(a_addr + kk * 32), tc::sdesc_k128(b_addr + kk * 32), idv,
                                (fresh && st == s0 && kk == 0) ? 0u : 1u);
                tc::commit(&empty[stage]);
                if (++stage == STAGES) {
                  stage = 0;
                  ph ^= 1;
                }
              }
              load += (s1 - s0) * w;
            }
          }
          if (open) {
            tc::commit(&tfull[buf]);
            acc_ph[buf] ^= 1;
            buf ^= 1;
          }
        }
      }
    mma_done:
      if (aborted(abort_flag)) {
        // wait (bounded) until every MMA issued so far has completed, so that
        // TMEM is not released under a running MMA
        tc::commit(drain);
        mbar_wait_bounded(drain, 0);
      }
    }
  } else {
    // ------------------------------ epilogue ------------------------------
    const int q = warp & 3;              // TMEM lane quarter this warp may access
    const int h = (warp - 2) >> 2;       // column group: cols h*EPI_COLS .. +EPI_COLS-1
    __shared__ float4 s_sums[EPI == EPI_BOUND ? EPI_WARPS * EPI_COLS / 4 : 1];
    float* sb = reinterpret_cast<float*>(s_sums) + (EPI == EPI_BOUND ? (warp - 2) * EPI_COLS : 0);
    const int r_local = q * 32 + lane;
    int buf = 0;
    uint32_t acc_ph[2] = {0, 0};
    for (int64_t r = 0; r * unit_step < units && !aborted(abort_flag); ++r) {
      const int64_t t = unit_at(r);
      if (t >= units) continue;
      int tm, tn;
      coords(t % tile_units, tm, tn);
      const int64_t row = (int64_t)tm * BM + r_local;
      const int64_t col0 = (int64_t)tn * BN + h * EPI_COLS;
      if (EPI == EPI_F32 && !SPLIT) prefetch_c_rows<EPI_COLS>(p, (int64_t)tm * BM + q * 32, col0, lane);
      // the next finished chunk's TMEM address (~0: timed out), and its release
      auto wait = [&]() -> uint32_t {
        if (!mbar_wait_bounded(&tfull[buf], acc_ph[buf])) {
          report_status(p.status, DEV_TIMEOUT_MMA);
          *abort_flag = 1;
          return ~0u;
        }
        tc::fence_after();
        return tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN + h * EPI_COLS);
      };
      auto release = [&]() {
        tc::fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty[buf]);
        acc_ph[buf] ^= 1;
        buf ^= 1;
      };
      if constexpr (SPLIT) {
        // one unit per cluster; the stages are free once its chunks are done
        float S[EPI_COLS];
#pragma unroll
        for (int j = 0; j < EPI_COLS; ++j) S[j] = 0.0f;
        const int chunks = p.group_begin[1] * ((kb1 - kb0 + p.chunk_cap - 1) / p.chunk_cap);
        for (int c = 0; c < chunks; ++c) {
          const uint32_t taddr = wait();
          if (taddr == ~0u) goto epi_done;
          drain_chunk<EPI, EPI_COLS>(taddr, S);
          release();
        }
        float* part = reinterpret_cast<float*>(smem) + h * EPI_COLS * BM + r_local;
#pragma unroll
        for (int j = 0; j < EPI_COLS; ++j) part[j * BM] = S[j];
      } else if constexpr (EPI == EPI_OZAKI) {
        if (!ozaki_groups<EPI_COLS>(p, g_begin(t), g_end(t), row, col0, tm, tn, h * EPI_COLS, r_local, wait, release))
          goto epi_done;
      } else {
        if (!float_groups<EPI, EPI_COLS>(p, g_begin(t), g_end(t), row, col0, wait, release, sb)) goto epi_done;
      }
    }
  epi_done:;
  }

  // reconverge each warp (its lane 0 may have run a role loop alone) before
  // the CTA-wide barrier, which requires whole warps
  __syncwarp();
  if constexpr (SPLIT) {
    cluster_sync();  // every CTA's sums are in place
    int tm, tn;
    coords(unit0, tm, tn);
    reduce_columns(p, reinterpret_cast<const float*>(smem), (int64_t)tm * BM, (int64_t)tn * BN, BN * rank / ranks,
                   BN * (rank + 1) / ranks, ranks, warp, lane);
    cluster_sync();  // before any of them is gone
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after();
    tc::tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------
// CTA-pair kernel (cta_group::2). A cluster of two CTAs computes a 256 x 256
// output tile with one MMA stream: each CTA holds 128 rows of A and 128 rows
// (columns of the output) of B per stage, and the even CTA issues
// tcgen05.mma.cta_group::2, which reads both CTAs' shared memory and writes
// 128 output rows into each CTA's TMEM. Against the single-CTA kernel this
// reads two thirds of the shared-memory bytes per FLOP (the B half is read
// once for both SMs) and a stage is 32 KB, so seven stages fit.
//   full[s]   (even CTA)  both CTAs' TMA loads complete here (64 KB)
//   empty[s]  (each CTA)  the even CTA's commit, multicast: stage s is free
//   tfull[b]  (each CTA)  the even CTA's commit, multicast: accumulator b done
//   tempty[b] (even CTA)  all 16 epilogue warps of the pair: b drained
// ---------------------------------------------------------------------------
constexpr int P_STAGE_BYTES = A_TILE + B_TILE / 2;  // 32 KB
// Stages: seven, or six where the epilogue needs shared memory of its own (the
// bound's column sums).
template <int EPI>
constexpr int pair_stages() { return EPI == EPI_BOUND ? 6 : 7; }
template <int EPI>
constexpr int pair_smem() { return 1024 + pair_stages<EPI>() * P_STAGE_BYTES + 256; }

template <int KIND, int EPI, bool GROUPED = false>
__global__ void __launch_bounds__(THREADS, 1)
    slice_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmBh,
                           const __grid_constant__ Params p, const __grid_constant__ GroupTable gt) {
  constexpr int PSTAGES = pair_stages<EPI>();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + PSTAGES * P_STAGE_BYTES);
  uint64_t* empty = full + PSTAGES;
  uint64_t* tfull = empty + PSTAGES;  // [2]
  uint64_t* tempty = tfull + 2;       // [2]
  uint64_t* drain = tempty + 2;       // used only when aborting
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = (rank == 0);
  const int64_t unit0 = (int64_t)cluster_id_x(), unit_step = (int64_t)cluster_count_x();
  // A problem's work units: vertical tile pairs x chunks of its groups,
  // group-major (units in flight read the same digit planes).
  auto tile_units_of = [](const Params& P) { return (int64_t)((P.tiles_m + 1) / 2) * P.tiles_n; };
  auto gchunk_of = [](const Params& P) { return P.gchunk > 0 ? P.gchunk : P.ngroups; };
  const int64_t units = GROUPED ? gt.units : tile_units_of(p) * ceil_div_dev(p.ngroups, gchunk_of(p));
  unsigned* status = GROUPED ? gt.probs[0].status : p.status;
  // round r hands units [r*step, (r+1)*step) to the CTAs (clusters), in
  // reverse order on odd rounds: units are ordered by falling cost (largest
  // groups first), so this snake order evens out the per-CTA totals
  auto unit_at = [&](int64_t r) {
    return r * unit_step + ((r & 1) ? (unit_step - 1 - unit0) : unit0);
  };
  // Calls fn(problem, its A map, its B map, unit within the problem).
  auto with_unit = [&](int64_t u, auto&& fn) -> bool {
    if constexpr (GROUPED) {
      int lo = 0, hi = gt.nprobs - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (gt.probs[mid].unit_begin <= u) lo = mid;
        else hi = mid - 1;
      }
      const Params& P = gt.probs[lo];
      return fn(P, &gt.maps[2 * lo], &gt.maps[2 * lo + 1], u - P.unit_begin);
    } else {
      return fn(p, &tmA, &tmBh, u);
    }
  };
  // tile of unit t of problem P (rank 1 of an odd last pair reads zero rows, writes nothing)
  auto coords = [&](const Params& P, int64_t t, int& tm, int& tn) {
    int um;
    tile_coords<8>(t % tile_units_of(P), (P.tiles_m + 1) / 2, P.tiles_n, um, tn);
    tm = 2 * um + (int)rank;
  };
  auto groups_of = [&](const Params& P, int64_t t, int& g0, int& g1) {
    const int gc = gchunk_of(P);
    g0 = (int)(t / tile_units_of(P)) * gc;
    g1 = min(P.ngroups, g0 + gc);
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < PSTAGES; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull[b], 1);
      mbar_init(&tempty[b], 2 * EPI_WARPS);
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tc::tmem_alloc2(tmem_slot, TMEM_COLS);
    tc::tmem_relinquish2();
  }
  tc::fence_before();
  __syncthreads();
  cluster_sync();  // the pair's barriers exist before any remote arrival
  tc::fence_after();
  const uint32_t tmem_base = *tmem_slot;
  dependency_wait_few();

  if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs) ------------------------------
    if (lane == 0) {
      if (!GROUPED) {
        prefetch_tensormap(&tmA);
        prefetch_tensormap(&tmBh);
      }
      int stage = 0;
      uint32_t ph = 0;
      auto produce = [&](const Params& P, const CUtensorMap* mA, const CUtensorMap* mB, int64_t t) -> bool {
        int tm, tn, g0, g1;
        coords(P, t, tm, tn);
        groups_of(P, t, g0, g1);
        for (int g = g0; g < g1; ++g) {
          for (int pi = P.group_begin[g]; pi < P.group_begin[g + 1]; ++pi) {
            for (int kb = 0; kb < P.kblocks; ++kb) {
              if (!mbar_wait_bounded(&empty[stage], ph ^ 1)) {
                report_status(status, DEV_TIMEOUT_EMPTY);
                *abort_flag = 1;
                return false;
              }
              if (leader) mbar_arrive_expect_tx(&full[stage], 2 * P_STAGE_BYTES);
              uint8_t* sa = smem + stage * P_STAGE_BYTES;
              const uint32_t bar = mapa_shared(&full[stage], 0);
              tma_load_3d_pair(sa, mA, bar, kb * P.kelems, tm * BM, P.pair_a[pi]);
              tma_load_3d_pair(sa + A_TILE, mB, bar, kb * P.kelems, tn * BN + (int)rank * (BN / 2), P.pair_b[pi]);
              if (++stage == PSTAGES) {
                stage = 0;
                ph ^= 1;
              }
            }
          }
        }
        return true;
      };
      bool ok = true;
      for (int64_t r = 0; r * unit_step < units && ok && !aborted(abort_flag); ++r) {
        const int64_t u = unit_at(r);
        if (u >= units) continue;
        ok = with_unit(u, produce);
      }
      if (ok && !aborted(abort_flag)) {
        // every stage released: no commit from the even CTA is still on its
        // way to this CTA's barriers
        for (int i = 0; i < PSTAGES; ++i) {
          if (!mbar_wait_bounded(&empty[stage], ph ^ 1)) {
            report_status(status, DEV_TIMEOUT_EMPTY);
            *abort_flag = 1;
            break;
          }
          if (++stage == PSTAGES) {
            stage = 0;
            ph ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (even CTA) ------------------------------
    if (lane == 0 && leader) {
      const uint32_t idv = tc::idesc(tc::kind_fmt(KIND), 2 * BM, BN);
      int stage = 0;
      uint32_t ph = 0;
      int buf = 0;
      uint32_t acc_ph[2] = {0, 0};
      auto issue = [&](const Params& P, const CUtensorMap*, const CUtensorMap*, int64_t t) -> bool {
        int g0, g1;
        groups_of(P, t, g0, g1);
        for (int g = g0; g < g1; ++g) {
          int load = 0;
          bool open = false;
          uint32_t d_tmem = 0;
          for (int pp = P.group_begin[g]; pp < P.group_begin[g + 1]; ++pp) {
            const int w = P.pair_w[pp];
            if (open && !P.merge_pairs) {
              tc::commit2_mc(&tfull[buf], (uint16_t)0x3);
              acc_ph[buf] ^= 1;
              buf ^= 1;
              open = false;
            }
            for (int st = 0; st < P.kblocks;) {
              if (open && load + w > P.chunk_cap) {
                tc::commit2_mc(&tfull[buf], (uint16_t)0x3);
                acc_ph[buf] ^= 1;
                buf ^= 1;
                open = false;
              }
              bool fresh = false;
              if (!open) {
                if (!mbar_wait_bounded(&tempty[buf], acc_ph[buf] ^ 1)) {
                  report_status(status, DEV_TIMEOUT_TMEM);
                  *abort_flag = 1;
                  return false;
                }
                tc::fence_after();
                d_tmem = tmem_base + (uint32_t)(buf * BN);
                load = 0;
                open = fresh = true;
              }
              // the k-blocks of this pair that still fit in the open chunk
              const int s0 = st, s1 = min(P.kblocks, st + (P.chunk_cap - load) / w);
              for (; st < s1; ++st) {
                if (!mbar_wait_bounded(&full[stage], ph)) {
                  report_status(status, DEV_TIMEOUT_FULL);
                  *abort_flag = 1;
                  return false;
                }
                tc::fence_after();
                const uint32_t a_addr = smem_u32(smem + stage * P_STAGE_BYTES);
                const uint32_t b_addr = a_addr + A_TILE;
#pragma unroll
                for (int kk = 0; kk < KSTEPS; ++kk)
                  tc::mma2<KIND>(d_tmem, tc::sdesc_k128(a_addr + kk * 32), tc::sdesc_k128(b_addr + kk * 32), idv,
                                (fresh && st == s0 && kk == 0) ? 0u : 1u);
                tc::commit2_mc(&empty[stage], (uint16_t)0x3);
                if (++stage == PSTAGES) {
                  stage = 0;
                  ph ^= 1;
                }
              }
              load += (s1 - s0) * w;
            }
          }
          if (open) {
            tc::commit2_mc(&tfull[buf], (uint16_t)0x3);
            acc_ph[buf] ^= 1;
            buf ^= 1;
          }
        }
        return true;
      };
      bool ok = true;
      for (int64_t r = 0; r * unit_step < units && ok && !aborted(abort_flag); ++r) {
        const int64_t u = unit_at(r);
        if (u >= units) continue;
        ok = with_unit(u, issue);
      }
      if (aborted(abort_flag)) {
        tc::commit2_mc(drain, (uint16_t)0x1);
        mbar_wait_bounded(drain, 0);
      }
    }
  } else {
    // ------------------------------ epilogue (both CTAs) ------------------------------
    const int q = warp & 3;
    const int h = (warp - 2) >> 2;
    __shared__ float4 s_sums[EPI == EPI_BOUND ? EPI_WARPS * EPI_COLS / 4 : 1];
    float* sb = reinterpret_cast<float*>(s_sums) + (EPI == EPI_BOUND ? (warp - 2) * EPI_COLS : 0);
    const int r_local = q * 32 + lane;
    const uint32_t tempty_leader[2] = {mapa_shared(&tempty[0], 0), mapa_shared(&tempty[1], 0)};
    int buf = 0;
    uint32_t acc_ph[2] = {0, 0};
    auto drain_unit = [&](const Params& P, const CUtensorMap*, const CUtensorMap*, int64_t t) -> bool {
      int tm, tn, g0, g1;
      coords(P, t, tm, tn);
      groups_of(P, t, g0, g1);
      const int64_t row = (int64_t)tm * BM + r_local;
      const int64_t col0 = (int64_t)tn * BN + h * EPI_COLS;
      if (EPI == EPI_F32) prefetch_c_rows<EPI_COLS>(P, (int64_t)tm * BM + q * 32, col0, lane);
      auto wait = [&]() -> uint32_t {
        if (!mbar_wait_bounded(&tfull[buf], acc_ph[buf])) {
          report_status(status, DEV_TIMEOUT_MMA);
          *abort_flag = 1;
          return ~0u;
        }
        tc::fence_after();
        return tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN + h * EPI_COLS);
      };
      auto release = [&]() {
        tc::fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster_relaxed(tempty_leader[buf]);
        acc_ph[buf] ^= 1;
        buf ^= 1;
      };
      if constexpr (EPI == EPI_OZAKI)
        return ozaki_groups<EPI_COLS>(P, g0, g1, row, col0, tm, tn, h * EPI_COLS, r_local, wait, release);
      else
        return float_groups<EPI, EPI_COLS>(P, g0, g1, row, col0, wait, release, sb);
    };
    bool ok = true;
    for (int64_t r = 0; r * unit_step < units && ok && !aborted(abort_flag); ++r) {
      const int64_t u = unit_at(r);
      if (u >= units) continue;
      ok = with_unit(u, drain_unit);
    }
  }

  __syncwarp();
  tc::fence_before();
  __syncthreads();
  cluster_sync();  // both CTAs are done with each other's barriers and TMEM
  if (warp == 1) {
    tc::fence_after();
    tc::tmem_dealloc2(tmem_base, TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
// Chunk counts of every group (Params::group_chunks) under the chunk rule
// the MMA issuer applies step by step: a chunk takes a pair's k-blocks while
// their weights fit in chunk_cap, continues into the next pair only with
// merge_pairs, and a new chunk holds floor(chunk_cap / w) k-blocks of a pair
// of weight w. Returns false if a weight exceeds the capacity.
inline bool plan_chunks(Params& p) {
  const int cap = p.chunk_cap;
  for (int g = 0; g < p.ngroups; ++g) {
    int n = 0, load = 0;
    bool open = false;
    for (int pp = p.group_begin[g]; pp < p.group_begin[g + 1]; ++pp) {
      const int w = p.pair_w[pp];
      if (w < 1 || w > cap) return false;
      int rem = p.kblocks;
      if (open && p.merge_pairs) {
        const int take = std::min(rem, (cap - load) / w);
        rem -= take;
        load += take * w;
      } else {
        open = false;
      }
      if (rem > 0) {
        const int per = cap / w;
        const int fresh = (rem + per - 1) / per;
        n += fresh;
        load = (rem - (fresh - 1) * per) * w;
        open = true;
      }
    }
    p.group_chunks[g] = n;
  }
  return true;
}

template <int KIND, int EPI>
inline cudaError_t set_slice_attrs() {
  cudaError_t e = cudaFuncSetAttribute(slice_gemm_kernel<KIND, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       SMEM_BYTES);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(slice_gemm_pair_kernel<KIND, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             pair_smem<EPI>());
  if constexpr (EPI == EPI_F32)
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(slice_gemm_kernel<KIND, EPI, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               SMEM_BYTES);
  if (e == cudaSuccess && EPI == EPI_OZAKI)
    e = cudaFuncSetAttribute(slice_gemm_pair_kernel<KIND, EPI, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             pair_smem<EPI>());
  return e;
}

// Kernel variants: 0 = one CTA per tile, 2 = CTA pairs with cta_group::2 MMA
// 3 = a cluster of CTAs per tile, each a range of k
// (1 is not used: it was a cluster kernel sharing B tiles by multicast loads).
enum { SLICE_SINGLE = 0, SLICE_PAIR = 2, SLICE_SPLIT = 3 };

inline cudaLaunchConfig_t cluster_config(int ctas, int smem, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = (size_t)smem;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ctas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cfg;
}

// The variant to use on the current device and how many CTA pairs fit at
// once; queried once per device. MOMMS_SLICE_VARIANT=0 restricts the choice to
// the single-CTA kernel (default and MOMMS_SLICE_VARIANT=2: the pair kernel
// wherever the device can co-schedule pairs).
template <int KIND, int EPI>
inline int slice_variant(int* clusters) {
  static std::atomic<int> cache_v[64], cache_n[64];
  static std::atomic<bool> init[64];
  int dev = 0;
  *clusters = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return SLICE_SINGLE;
  if (!init[dev].load()) {
    const char* env = getenv("MOMMS_SLICE_VARIANT");
    const bool want_pair = !(env && env[0] == '0');
    int v = SLICE_SINGLE, n = 0;
    if (want_pair) {
      cudaLaunchAttribute attr[2];
      cudaLaunchConfig_t cfg = cluster_config(2, pair_smem<EPI>(), attr);
      int c = 0;
      if (cudaOccupancyMaxActiveClusters(&c, (const void*)slice_gemm_pair_kernel<KIND, EPI>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        c = 0;
      }
      if (c > 0) {
        v = SLICE_PAIR;
        n = c;
      }
    }
    cache_v[dev].store(v);
    cache_n[dev].store(n);
    init[dev].store(true);
  }
  *clusters = cache_n[dev].load();
  return cache_v[dev].load();
}

// How many clusters of `ctas` of the split kernel fit the current device at
// once; queried once per device and size (0: none).
template <int KIND>
inline int split_clusters(int ctas) {
  static std::atomic<int> cache[64][4];  // the count + 1
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  std::atomic<int>& c = cache[dev][ctas == 8 ? 3 : ctas / 2];
  int n = c.load();
  if (!n) {
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = cluster_config(ctas, SMEM_BYTES, attr);
    if (cudaOccupancyMaxActiveClusters(&n, (const void*)slice_gemm_kernel<KIND, EPI_F32, true>, &cfg) != cudaSuccess) {
      cudaGetLastError();
      n = 0;
    }
    c.store(++n);
  }
  return n - 1;
}

// The split kernel: clusters of `ctas`, one per tile.
template <int KIND>
inline cudaError_t launch_slice_split(const CUtensorMap& tmA, const CUtensorMap& tmB, const Params& p, int ctas,
                                      cudaStream_t s) {
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = cluster_config(ctas, SMEM_BYTES, attr);
  cfg.gridDim = dim3((unsigned)((int64_t)p.tiles_m * p.tiles_n * ctas));
  cfg.stream = s;
  return cudaLaunchKernelEx(&cfg, slice_gemm_kernel<KIND, EPI_F32, true>, tmA, tmB, p);
}

// Launches the slice kernel. The pair kernel needs at least two m-tiles (its
// units are vertical tile pairs) and takes tmB_half, whose box is BN/2 rows
// (each CTA of a pair stages its half of the B tile); the single-CTA kernel
// takes tmB_full. *variant receives the one run.
template <int KIND, int EPI>
inline cudaError_t launch_slice(const CUtensorMap& tmA, const CUtensorMap& tmB_full, const CUtensorMap& tmB_half,
                                const Params& p, int sm_count, cudaStream_t s, int* variant) {
  int clusters = 0;
  const int v = p.tiles_m >= 2 ? slice_variant<KIND, EPI>(&clusters) : SLICE_SINGLE;
  *variant = v;
  const int64_t tile_units = v == SLICE_PAIR ? (int64_t)((p.tiles_m + 1) / 2) * p.tiles_n
                                             : (int64_t)p.tiles_m * p.tiles_n;
  const int64_t slots = v == SLICE_PAIR ? clusters : sm_count;
  Params q = p;
  if (!plan_chunks(q)) return cudaErrorInvalidValue;
  q.gchunk = p.ngroups;
  // Few tiles: a tile's accumulation groups (each writes its own int32 plane)
  // can run as separate work units. Pick the split whose schedule of units
  // (group-major, handed out in the kernel's snake order; cost = k-blocks of
  // the unit's pairs plus 8 for its pipeline fill) finishes first.
  if (EPI == EPI_OZAKI && p.residue && tile_units < 4 * slots) {
    // groups of equal cost: the makespan is rounds times a unit's
    double best = -1.0;
    for (int gc = p.ngroups; gc >= 1; gc = gc == 1 ? 0 : (gc + 1) / 2) {
      const int64_t units = tile_units * ((p.ngroups + gc - 1) / gc);
      const double makespan = (double)((units + slots - 1) / slots) * (8.0 + (double)gc * (double)p.kblocks);
      if (best < 0.0 || makespan < best * 0.97) {
        best = makespan;
        q.gchunk = gc;
      }
    }
  } else if (EPI == EPI_OZAKI && tile_units < 4 * slots && p.ngroups > 1) {
    double best = -1.0;
    std::vector<double> load((size_t)slots);
    for (int gc = p.ngroups; gc >= 1; gc = gc == 1 ? 0 : (gc + 1) / 2) {
      std::fill(load.begin(), load.end(), 0.0);
      const int chunks = (p.ngroups + gc - 1) / gc;
      int64_t u = 0;
      for (int c = 0; c < chunks; ++c) {
        const int g0 = c * gc, g1 = std::min(p.ngroups, g0 + gc);
        const double cost = 8.0 + (double)(p.group_begin[g1] - p.group_begin[g0]) * (double)p.kblocks;
        for (int64_t tu = 0; tu < tile_units; ++tu, ++u) {
          const int64_t r = u / slots, i = u % slots;
          load[(size_t)((r & 1) ? slots - 1 - i : i)] += cost;  // the kernel's snake order
        }
      }
      const double makespan = *std::max_element(load.begin(), load.end());
      if (best < 0.0 || makespan < best * 0.97) {  // a finer split must gain 3 %
        best = makespan;
        q.gchunk = gc;
      }
    }
  }
  const int64_t units = tile_units * ((p.ngroups + q.gchunk - 1) / q.gchunk);
  if (v == SLICE_PAIR) {
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = cluster_config(2, pair_smem<EPI>(), attr);
    cfg.gridDim = dim3((unsigned)(2 * std::min<int64_t>(units, clusters)));
    cfg.stream = s;
    return cudaLaunchKernelEx(&cfg, slice_gemm_pair_kernel<KIND, EPI>, tmA, tmB_half, q, GroupTable{});
  }
  const int grid = (int)std::min<int64_t>(units, sm_count);
  return launch_dependent(slice_gemm_kernel<KIND, EPI>, dim3((unsigned)grid), THREADS, SMEM_BYTES, s, tmA, tmB_full, q);
}

}  // namespace sp
}  // namespace momms

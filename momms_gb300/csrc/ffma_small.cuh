// The FP32 kernel of small products: 32 x 32 output tiles, 128 threads of 2 x 4
// outputs, k in stages of 32 through a 4-deep cp.async ring.
//
// A 128 x 128 tile of a product with few tiles and a short k runs on a handful
// of SMs and waits out one global-memory round trip per 16 of k: 256 x 300 x 200
// took 28.7 us on 6 CTAs. Here it is 80 CTAs whose first 128 of k are in flight
// before the first FMA. Shared memory feeds a 2 x 4 block at half of the FMA
// rate at best, so larger products keep the large tiles. Every output is the
// same fma chain over k (and the same split order) as in the other tiles, so the
// tile never changes a result.
//
// An operand is staged along its contiguous index, [k][x] or [x][k], by
// 16-byte copies where its rows are aligned and whole, else by 4-byte copies;
// the FMA loop takes four k at a time, one 8- or 16-byte load per k and operand
// on average in either layout (rows of [x][k] are 36 floats apart: the eight
// rows a load touches fall on different banks).
#pragma once
#include "ffma_core.cuh"

namespace momms {
namespace ffma {

struct Small {
  static constexpr int TILE = 32, KB = 32, STAGES = 4, THREADS = 128, CTAS_PER_SM = 4;
  static constexpr int KROW = KB + 4;                 // floats per x row of a k-contiguous stage
  static constexpr int OP = TILE * KROW;              // floats per operand and stage (x-contiguous: KB * TILE)
  static constexpr int SMEM_BYTES = STAGES * 2 * OP * 4;
};

template <int BYTES>
__device__ __forceinline__ void cp_async_f32(float* dst, const float* src, bool valid) {
  if (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid ? 4 : 0) : "memory");
}

// One operand's stage: x from x0 (X in all), k in [k0, k1), k1 the unit's end;
// elements outside are zero.
template <bool XC>
__device__ __forceinline__ void stage_small(float* s, const float* base, int64_t sx, int64_t sk, int64_t x0, int64_t X,
                                            int64_t k0, int64_t k1, bool vec) {
  const int xl = (int)min(X - x0, (int64_t)Small::TILE), kl = (int)min(k1 - k0, (int64_t)Small::KB);
  const float* src = base + x0 * sx + k0 * sk;
  const int t = threadIdx.x;
  if (vec && xl == Small::TILE && kl == Small::KB) {
    // 8 pieces of 4 elements along the contiguous index
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row = (t >> 3) + 16 * i, col = (t & 7) * 4;
      cp_async_f32<16>(s + row * (XC ? Small::TILE : Small::KROW) + col,
                       src + (XC ? row * sk + col : row * sx + col), true);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = (t >> 5) + 4 * i, col = t & 31;  // [k][x] or [x][k]
      const bool ok = XC ? (col < xl && row < kl) : (row < xl && col < kl);
      const float* q = XC ? src + col * sx + row * sk : src + row * sx + col * sk;
      cp_async_f32<4>(s + row * (XC ? Small::TILE : Small::KROW) + col, ok ? q : base, ok);
    }
  }
}

// v[kk][i]: element x + i of the operand at k + kk, for four k.
template <bool XC, int N>
__device__ __forceinline__ void fragment_small(const float* s, int x, int k, float (&v)[4][N]) {
  if (XC) {
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      if (N == 2) {
        const float2 u = *reinterpret_cast<const float2*>(s + (k + kk) * Small::TILE + x);
        v[kk][0] = u.x, v[kk][1] = u.y;
      } else {
        const float4 u = *reinterpret_cast<const float4*>(s + (k + kk) * Small::TILE + x);
        v[kk][0] = u.x, v[kk][1] = u.y, v[kk][N - 2] = u.z, v[kk][N - 1] = u.w;
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float4 u = *reinterpret_cast<const float4*>(s + (x + i) * Small::KROW + k);
      v[0][i] = u.x, v[1][i] = u.y, v[2][i] = u.z, v[3][i] = u.w;
    }
  }
}

// Accumulates k in [k0, k1) of the tile whose first row and column are m0, n0.
template <bool A_XC, bool B_XC>
__device__ __forceinline__ void small_unit(const Operands& o, int64_t m0, int64_t n0, int64_t k0, int64_t k1,
                                           float (&acc)[2][4], float* smem) {
  auto stage = [&](int64_t at, int slot) {
    float* s = smem + slot * 2 * Small::OP;
    if (at < k1) {
      stage_small<A_XC>(s, o.a, o.rsa, o.csa, m0, o.m, at, k1, o.vec);
      stage_small<B_XC>(s + Small::OP, o.b, o.csb, o.rsb, n0, o.n, at, k1, o.vec);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < Small::STAGES - 1; ++i) stage(k0 + i * Small::KB, i);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r0 = (warp & 1) * 16 + (lane & 7) * 2, c0 = (warp >> 1) * 16 + (lane >> 3) * 4;
  int slot = 0;
  for (int64_t at = k0; at < k1; at += Small::KB) {
    asm volatile("cp.async.wait_group %0;" ::"n"(Small::STAGES - 2) : "memory");
    __syncthreads();  // the stage is in for every thread, and the slot refilled next has been read
    stage(at + (Small::STAGES - 1) * Small::KB, (slot + Small::STAGES - 1) % Small::STAGES);
    const float* s = smem + slot * 2 * Small::OP;
#pragma unroll
    for (int k = 0; k < Small::KB; k += 4) {
      float a[4][2], b[4][4];
      fragment_small<A_XC, 2>(s, r0, k, a);
      fragment_small<B_XC, 4>(s + Small::OP, c0, k, b);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[kk][i], b[kk][j], acc[i][j]);
    }
    slot = (slot + 1) % Small::STAGES;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();  // before the next unit's stages
}

// Epilogue, as ffma_finish: partials [splits][32 * 32] per tile, summed by the
// last split in split order.
__device__ __forceinline__ void small_finish(const Epi& e, float (&acc)[2][4], int64_t m0, int64_t n0, int splits, int sp,
                                             float* tile_partials, unsigned* counter, int* s_last) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t row = m0 + (warp & 1) * 16 + (lane & 7) * 2, col = n0 + (warp >> 1) * 16 + (lane >> 3) * 4;
  auto update = [&]() {
    float c0[2][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 2; ++i)
        c0[i][j] = (e.beta != 0.0f && row + i < e.m && col + j < e.n) ? e.c[(row + i) * e.rsc + (col + j) * e.csc] : 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (row + i < e.m && col + j < e.n) {
          const float t = acc[i][j] * e.alpha;
          e.c[(row + i) * e.rsc + (col + j) * e.csc] = (e.beta == 0.0f) ? t : fmaf(e.beta, c0[i][j], t);
        }
  };
  if (splits == 1) {
    update();
    return;
  }
  constexpr int E = Small::TILE * Small::TILE;
  float* part = tile_partials + (size_t)sp * E;
#pragma unroll
  for (int u = 0; u < 8; ++u) part[u * Small::THREADS + tid] = acc[u >> 2][u & 3];
  __threadfence();
  __syncthreads();
  if (tid == 0) *s_last = atomicAdd(counter, 1u) == (unsigned)(splits - 1) ? 1 : 0;
  __syncthreads();
  if (*s_last) {
    __threadfence();
#pragma unroll
    for (int u = 0; u < 8; ++u) acc[u >> 2][u & 3] = __ldcg(tile_partials + u * Small::THREADS + tid);
    for (int q = 1; q < splits; ++q) {
      float w[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) w[u] = __ldcg(tile_partials + (size_t)q * E + u * Small::THREADS + tid);
#pragma unroll
      for (int u = 0; u < 8; ++u) acc[u >> 2][u & 3] += w[u];
    }
    update();
    if (tid == 0) *counter = 0u;
  }
  __syncthreads();
}

}  // namespace ffma
}  // namespace momms

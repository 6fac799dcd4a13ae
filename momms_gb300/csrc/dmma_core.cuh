// Building blocks of the FP64 DMMA GEMM kernels (single-problem and grouped):
// staging of 128B-swizzled A/B tiles, the warp-level DMMA k loop, and the
// epilogue with optional split-k fix-up.
//
// GB300 issues FP64 at about 2 FMAs per SM and clock, so one m8n8k4 DMMA
// occupies an SM for ~128 clocks and operand feeding costs nothing at any tile
// size: a 16 x 16 tile needs 0.5 B per FLOP, 4 GB/s per SM. What small tiles
// buy is balance. The tile is 32 x 32 (four DMMA warps, each 2 x 2 blocks of
// 8 x 8 interleaved over the tile, so that the live blocks of an edge tile
// spread over the warps), one producer warp, k-blocks of 16 in a 5-stage ring
// and four CTAs per SM: a CTA's epilogue and pipeline fill run under the other
// three's DMMAs. A problem may step its tiles by 16 or 8 instead of 32 (`ts`,
// see f64_plan.h): then every warp takes the whole tile for one k step of 4
// of each k-block, and the four partial sums meet in shared memory. (One
// block per warp over all of k ran the FP64 pipe at 0.70 of its rate, 0.72
// TFLOP/s at 1024^3 against 1.09 for four blocks per warp: a warp needs
// several independent DMMAs.)
//
// An operand is staged in the orientation of its contiguous index: x (the
// non-k index) contiguous as 16-wide sub-tiles [BK][16], k contiguous as
// [32][BK], both with the 128-byte swizzle. Operands TMA can address (16-byte
// base and stride) arrive by TMA, any others by 8-byte cp.async from the
// producer warp's lanes straight into the same layout, so no operand is ever
// repacked in memory first.
#pragma once
#include "common.cuh"

namespace momms {
namespace dmma {

constexpr int TILE = 32, BK = 16, STAGES = 5;
constexpr int CONSUMER_WARPS = 4;  // 2 (m) x 2 (n), blocks interleaved
constexpr int THREADS = (CONSUMER_WARPS + 1) * 32;
constexpr int CONSUMERS = CONSUMER_WARPS * 32;
constexpr int CTAS_PER_SM = 4;
constexpr int OP_STAGE = TILE * BK * 8;  // bytes of one operand's k-block
constexpr int SUB = BK * 128;  // one 16-wide sub-tile of an x-contiguous operand
constexpr int RED_BYTES = CONSUMER_WARPS * 16 * 16 * 8;  // the warps' partial sums of a 16-stepped tile
constexpr int SMEM_BYTES = 1024 + STAGES * 2 * OP_STAGE + RED_BYTES + 2 * STAGES * 8 + 16;
constexpr int GROUP_SMEM = (SMEM_BYTES - 1024 + 1023) / 1024 * 1024;  // from one group's shared memory to the next's
constexpr int smem_bytes(int groups) { return SMEM_BYTES + (groups - 1) * GROUP_SMEM; }

// Byte offset of element (r, kk) in a k-contiguous tile: rows of 16 doubles
// (128 bytes), 128B swizzle (16-byte chunk index XOR row mod 8).
__device__ __forceinline__ uint32_t off_kc(int r, int kk) {
  return r * 128 + ((((kk >> 1) ^ (r & 7))) << 4) + ((kk & 1) << 3);
}
// Byte offset of element (x, kk) in an x-contiguous tile stored as 16-wide
// sub-tiles of [BK rows of k][16 doubles of x], each 128B-swizzled.
__device__ __forceinline__ uint32_t off_xc(int x, int kk) {
  return (x >> 4) * SUB + kk * 128 + (((((x & 15) >> 1) ^ (kk & 7))) << 4) + ((x & 1) << 3);
}

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// Among the DMMA warps of one group (dgemm_body).
__device__ __forceinline__ void consumer_sync(int group) {
  asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(CONSUMERS) : "memory");
}

// How the kernels read an operand: xc, the staged layout (x contiguous); tma,
// through the tensor map, else element (x, k) at ptr[x*sx + k*sk].
struct Operand {
  const double* ptr;
  int64_t sx, sk;
  int xc, tma;
};

// Output description for the epilogue.
struct Epi {
  int64_t m, n;
  double alpha, beta;
  double* c;
  int64_t rsc, csc;
};

// 8-byte asynchronous copy global -> shared; zero-fills when !valid.
__device__ __forceinline__ void cp_async8(void* dst, const double* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid ? 8 : 0)
               : "memory");
}

// One operand's k-block by the producer warp's lanes: consecutive lanes take
// consecutive elements of the staged layout's contiguous index (16 of them per
// group of 16 lanes, the two groups two apart along the other index). x0: the
// tile's first x, ext: the x to stage (16 or 32), X and K the matrix extents;
// elements outside are zero.
__device__ __forceinline__ void stage_async(const Operand& o, uint8_t* dst, int64_t x0, int64_t k0, int ext,
                                            int64_t X, int64_t K, int lane) {
  const int fast = lane & 15, slow = lane >> 4;
  const int xl = (int)min(X - x0, (int64_t)ext), kl = (int)min(K - k0, (int64_t)BK);
  const double* base = o.ptr + x0 * o.sx + k0 * o.sk;
  if (o.xc) {
    for (int xb = 0; xb < ext; xb += 16) {
      const int x = xb + fast;
      const double* src = base + x * o.sx + slow * o.sk;
#pragma unroll
      for (int i = 0; i < BK / 2; ++i, src += 2 * o.sk) {
        const int kk = slow + 2 * i;
        const bool ok = x < xl && kk < kl;
        cp_async8(dst + off_xc(x, kk), ok ? src : o.ptr, ok);
      }
    }
  } else {
    const double* src = base + slow * o.sx + fast * o.sk;
#pragma unroll 8
    for (int x = slow; x < ext; x += 2, src += 2 * o.sx) {
      const bool ok = x < xl && fast < kl;
      cp_async8(dst + off_kc(x, fast), ok ? src : o.ptr, ok);
    }
  }
}

// One operand's k-block by TMA (one lane): `ext` of x, which the map's box
// matches (x-contiguous: boxes 16 wide).
__device__ __forceinline__ void stage_tma(const Operand& o, const CUtensorMap* map, uint64_t* bar, uint8_t* dst,
                                          int32_t x0, int32_t k0, int ext) {
  if (o.xc) {
    tma_load_2d(dst, map, bar, x0, k0);
    if (ext > 16) tma_load_2d(dst + SUB, map, bar, x0 + 16, k0);
  } else {
    tma_load_2d(dst, map, bar, k0, x0);
  }
}

// x staged per operand and k-block for tiles stepped by ts.
__host__ __device__ constexpr int stage_extent(int ts) { return ts > 16 ? TILE : 16; }

// Arrivals on a stage's full barrier: every producer lane, once its own copies
// have landed, and lane 0 once more by an ordinary arrival. That one releases
// lane 0's plain stores (the unit's tag): a cp.async arrival is made when the
// copies land and orders no other store of its thread.
constexpr unsigned FULL_ARRIVALS = 33;

// Producer warp: k-blocks [kb0, kb1) of the output tile whose first row and
// column are m0, n0. Every lane arrives on the stage's full barrier once its
// own copies have landed; lane 0 adds the TMA bytes, and releases what it
// stored before (FULL_ARRIVALS). Returns false if a bounded wait expired.
__device__ __forceinline__ bool produce_unit(const CUtensorMap* tmA, const CUtensorMap* tmB, const Operand& a,
                                             const Operand& b, int64_t m, int64_t n, int64_t k, int ts, int64_t m0,
                                             int64_t n0, int64_t kb0, int64_t kb1, uint8_t* sA, uint8_t* sB,
                                             uint64_t* full, uint64_t* empty, int& stage, uint32_t& phase, int lane,
                                             unsigned* status) {
  const int ext = stage_extent(ts);
  const uint32_t tx = (uint32_t)(ext * BK * 8) * ((a.tma ? 1 : 0) + (b.tma ? 1 : 0));
  for (int64_t kb = kb0; kb < kb1; ++kb) {
    const bool free_stage = mbar_wait_bounded(&empty[stage], phase ^ 1);
    if (!__all_sync(0xffffffffu, free_stage)) {
      if (lane == 0) report_status(status, DEV_TIMEOUT_EMPTY);
      return false;
    }
    uint8_t* a_dst = sA + stage * OP_STAGE;
    uint8_t* b_dst = sB + stage * OP_STAGE;
    const int32_t kc = (int32_t)(kb * BK);
    if (lane == 0 && tx) {
      // the stage may have held another problem's cp.async data: order those
      // (released by the wait above) before this TMA's writes
      fence_proxy_async();
      mbar_expect_tx(&full[stage], tx);
      if (a.tma) stage_tma(a, tmA, &full[stage], a_dst, (int32_t)m0, kc, ext);
      if (b.tma) stage_tma(b, tmB, &full[stage], b_dst, (int32_t)n0, kc, ext);
    }
    if (!a.tma) stage_async(a, a_dst, m0, kc, ext, m, k, lane);
    if (!b.tma) stage_async(b, b_dst, n0, kc, ext, n, k, lane);
    if (a.tma && b.tma) mbar_arrive(&full[stage]);
    else mbar_arrive_cp_async(&full[stage]);
    if (lane == 0) mbar_arrive(&full[stage]);
    if (++stage == STAGES) {
      stage = 0;
      phase ^= 1;
    }
  }
  return true;
}

// What a DMMA warp multiplies and what it stores.
//  ts 32: it multiplies its blocks 8 wm + 16 i, 8 wn + 16 j (i, j in {0, 1}) for
//         every k step, and stores them;
//  ts 16: it multiplies blocks 8 i, 8 j of the 16 x 16 tile for k step `warp`
//         of each k-block, and stores block 8 wm, 8 wn of the four warps' sum;
//  ts 8:  the same with the one block 0, 0 (which warp 0 stores).
// Rows and columns stop at row_end, col_end (the tile's end or the matrix's).
struct Place {
  int ra, rb, step;          // tile row / column of block (0, 0) multiplied, distance to the next
  int ks0, ks1;              // k steps of each k-block
  uint32_t live;             // bit 2i + j: block (i, j) holds an element (warp-uniform)
  int64_t row, col;          // of this lane's first stored element; further ones 16 apart
  int64_t row_end, col_end;
};
__device__ __forceinline__ Place place_of(int64_t m0, int64_t n0, int ts, int64_t m, int64_t n, int warp, int lane) {
  const int wm = warp >> 1, wn = warp & 1;
  const bool whole = ts <= 16;
  Place p;
  p.ra = whole ? 0 : 8 * wm;
  p.rb = whole ? 0 : 8 * wn;
  p.step = ts > 16 ? 16 : 8;
  p.ks0 = whole ? warp : 0;
  p.ks1 = whole ? warp + 1 : BK / 4;
  p.row_end = min(m, m0 + ts);
  p.col_end = min(n, n0 + ts);
  p.row = m0 + 8 * wm + (lane >> 2);
  p.col = n0 + 8 * wn + 2 * (lane & 3);
  p.live = 0;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
      if (m0 + p.ra + p.step * i < p.row_end && n0 + p.rb + p.step * j < p.col_end) p.live |= 1u << (2 * i + j);
  return p;
}

// Consumer: accumulate k-blocks [kb0, kb1) of the current unit into acc, each
// run of `run` k-blocks in a chain of its own that is then added to the total
// (F64Plan::run).
// Blocks entirely outside the output and k steps past K are not multiplied
// (both would add zeros). Returns false if a bounded wait expired.
__device__ __forceinline__ bool consume_unit(int a_xc, int b_xc, int64_t k, int64_t kb0, int64_t kb1, const Place& p,
                                             const uint8_t* sA, const uint8_t* sB, uint64_t* full, uint64_t* empty,
                                             int& stage, uint32_t& phase, int lane, int run, double (&acc)[2][2][2],
                                             unsigned* status) {
  double total[2][2][2] = {};
  int left = run;
  bool added = false;
  auto add = [&]() {
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (p.live & (1u << (u >> 1))) total[u >> 2][(u >> 1) & 1][u & 1] += acc[u >> 2][(u >> 1) & 1][u & 1];
  };
  const int ra = p.ra + (lane >> 2), rb = p.rb + (lane >> 2);
  for (int64_t kb = kb0; kb < kb1; ++kb) {
    if (!mbar_wait_bounded(&full[stage], phase)) {
      report_status(status, DEV_TIMEOUT_FULL);
      return false;
    }
    const uint8_t* a = sA + stage * OP_STAGE;
    const uint8_t* b = sB + stage * OP_STAGE;
    const int steps = (int)min((int64_t)p.ks1, (k - kb * BK + 3) / 4);
#pragma unroll 4
    for (int ks = p.ks0; ks < steps; ++ks) {
      const int kk = ks * 4 + (lane & 3);
      double af[2], bf[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = ra + p.step * i;
        af[i] = *reinterpret_cast<const double*>(a + (a_xc ? off_xc(r, kk) : off_kc(r, kk)));
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int r = rb + p.step * j;
        bf[j] = *reinterpret_cast<const double*>(b + (b_xc ? off_xc(r, kk) : off_kc(r, kk)));
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
          if (p.live & (1u << (2 * i + j))) dmma(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[stage]);
    if (++stage == STAGES) {
      stage = 0;
      phase ^= 1;
    }
    if (--left == 0 && kb + 1 < kb1) {
      add();
      added = true;
      left = run;
#pragma unroll
      for (int u = 0; u < 8; ++u) acc[u >> 2][(u >> 1) & 1][u & 1] = 0.0;
    }
  }
  if (added) {
    add();
#pragma unroll
    for (int u = 0; u < 8; ++u) acc[u >> 2][(u >> 1) & 1][u & 1] = total[u >> 2][(u >> 1) & 1][u & 1];
  }
  return true;
}

// ts 16 and 8: the four warps' partial sums of the tile, added in warp order;
// each warp is left with its block in acc[0][0].
__device__ __forceinline__ void reduce_warps(double (&acc)[2][2][2], double* red, int warp, int lane, int group) {
#pragma unroll
  for (int u = 0; u < 8; ++u) red[(warp * 8 + u) * 32 + lane] = acc[u >> 2][(u >> 1) & 1][u & 1];
  consumer_sync(group);
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    double v = red[(2 * warp + q) * 32 + lane];
#pragma unroll
    for (int w = 1; w < CONSUMER_WARPS; ++w) v += red[(w * 8 + 2 * warp + q) * 32 + lane];
    acc[0][0][q] = v;
  }
  consumer_sync(group);  // read before the next unit's sums are written
}

// Epilogue of one unit. With splits == 1 the tile goes straight to C.
// Otherwise this split's partial tile is published in `tile_partials`
// ([splits][ts * ts], thread-interleaved: at steps of 16 a thread owns two
// outputs, at steps of 8 the first warp's threads do), and the last split to arrive on
// `counter` sums all partials in split order 0..splits-1 (a fixed order: the
// result does not depend on which CTA finishes last), writes C and resets
// the counter to zero.
//
// A thread owns eight outputs; their loads (C for beta != 0, the partials two
// splits at a time) are issued before the first value is used.
__device__ __forceinline__ void finish_unit(const Epi& e, const double (&acc)[2][2][2], const Place& p, int ts,
                                            int splits, int sp, double* tile_partials, unsigned* counter, int ctid,
                                            int group, int* s_last) {
  // output u = 4i + 2j + q of this thread
  auto live = [&](int u) { return p.row + 16 * (u >> 2) < p.row_end && p.col + 16 * ((u >> 1) & 1) + (u & 1) < p.col_end; };
  auto cptr = [&](int u) {
    return e.c + (p.row + 16 * (u >> 2)) * e.rsc + (p.col + 16 * ((u >> 1) & 1) + (u & 1)) * e.csc;
  };
  auto update = [&](const double (&v)[8]) {
    double c0[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) c0[u] = (e.beta != 0.0 && live(u)) ? *cptr(u) : 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (live(u)) {
        const double t = v[u] * e.alpha;
        *cptr(u) = (e.beta == 0.0) ? t : fma(e.beta, c0[u], t);
      }
  };
  double v[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) v[u] = acc[u >> 2][(u >> 1) & 1][u & 1];
  if (splits == 1) {
    update(v);
    return;
  }
  // Partials exist only for the tile's entries inside C.
  const int elems = ts * ts, own = ts > 8 ? CONSUMERS : 32;
  double* part = tile_partials + (size_t)sp * elems;
#pragma unroll
  for (int u = 0; u < 8; ++u)
    if (live(u)) part[u * own + ctid] = v[u];
  __threadfence();
  consumer_sync(group);
  if (ctid == 0) {
    unsigned prev = atomicAdd(counter, 1u);
    *s_last = (prev == (unsigned)(splits - 1)) ? 1 : 0;
  }
  consumer_sync(group);
  if (*s_last) {
    __threadfence();
    constexpr int T = 2;  // splits loaded together
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = live(u) ? __ldcg(tile_partials + u * own + ctid) : 0.0;
    for (int t0 = 1; t0 < splits; t0 += T) {
      double w[T][8];
#pragma unroll
      for (int t = 0; t < T; ++t)
#pragma unroll
        for (int u = 0; u < 8; ++u)
          w[t][u] = (t0 + t < splits && live(u))
                        ? __ldcg(tile_partials + (size_t)(t0 + t) * elems + u * own + ctid)
                        : 0.0;
#pragma unroll
      for (int t = 0; t < T; ++t)
        if (t0 + t < splits) {
#pragma unroll
          for (int u = 0; u < 8; ++u) v[u] += w[t][u];
        }
    }
    update(v);
    if (ctid == 0) *counter = 0u;
  }
  consumer_sync(group);
}

// Shared-memory carve-up and barrier initialisation common to the kernels.
struct Smem {
  uint8_t* sA;
  uint8_t* sB;
  double* red;
  uint64_t* full;
  uint64_t* empty;
  int* s_last;
};

__device__ __forceinline__ Smem setup_smem(uint8_t* smem_raw, int group, int tid) {
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023)) +
                  group * GROUP_SMEM;
  Smem s;
  s.sA = smem;
  s.sB = smem + STAGES * OP_STAGE;
  s.red = reinterpret_cast<double*>(s.sB + STAGES * OP_STAGE);
  s.full = reinterpret_cast<uint64_t*>(s.sB + STAGES * OP_STAGE + RED_BYTES);
  s.empty = s.full + STAGES;
  s.s_last = reinterpret_cast<int*>(s.empty + STAGES);
  if (tid == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&s.full[i], FULL_ARRIVALS);
      mbar_init(&s.empty[i], CONSUMER_WARPS);
    }
    fence_barrier_init();
  }
  __syncthreads();
  return s;
}

// One unit of work: an output tile's k range.
struct Unit {
  int64_t tile, kb0, kb1;  // tile: index of its counter and partials within the problem
  int tm, tn, sp;
};

// One problem, as the kernels see it.
struct DProblem {
  int64_t m, n, k;
  Operand a, b;
  Epi e;
  int tiles_m, tiles_n, splits, ts, run;
  int64_t kb_split;
  int64_t unit_begin;  // grouped launches: the problem's first unit
  double* partials;    // splits > 1: [tiles][splits][ts * ts]
  unsigned* counters;  // splits > 1: [tiles], zero on entry and on exit
};

// A persistent CTA over a source of units (Src: total(), and unit(u, fn) which
// calls fn(problem, A map, B map, Unit) with problem a DProblem), or GROUPS of
// such CTAs, each with its own warps, barriers and shared memory, as one: where
// they have to be on one SM.
// With `next` units are handed out dynamically: the producer warp takes the
// next unit from the global counter (numbered costliest first, so this is
// longest-processing-time-first list scheduling by the actual durations; a
// static deal of 4096 equal units over 608 CTAs left one SM in four with 28
// units against 26.9 on average: 1.055 against 1.095 TFLOP/s at 2048^3).
// Without, the CTA takes units blockIdx.x, blockIdx.x + gridDim.x, ...
// Either way the producer tags the first stage it fills for a unit with the
// unit's index, which the DMMA warps read when they reach that stage; -1 ends.
template <int GROUPS = 1, typename Src>
__device__ __forceinline__ void dgemm_body(const Src& src, unsigned long long* next, unsigned* status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ long long s_units[GROUPS][STAGES];
  const int group = GROUPS > 1 ? threadIdx.x / THREADS : 0, tid = threadIdx.x - group * THREADS;
  long long* const s_stage_unit = s_units[group];
  const Smem sm = setup_smem(smem_raw, group, tid);
  const int warp = tid >> 5, lane = tid & 31;
  const long long total = src.total();
  int stage = 0;
  uint32_t phase = 0;
  if (warp == CONSUMER_WARPS) {
    bool ok = true;
    // a tag is written while its stage is free (every DMMA warp read the
    // previous tag before releasing it) and published by lane 0's ordinary
    // arrival on the stage (release) to the warps' wait (acquire)
    auto tag = [&](long long u) {
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(&sm.empty[stage], phase ^ 1));
      if (ok && lane == 0) s_stage_unit[stage] = u;
      if (!ok && lane == 0) report_status(status, DEV_TIMEOUT_EMPTY);
    };
    for (long long u = (long long)blockIdx.x * GROUPS + group;; u += (long long)gridDim.x * GROUPS) {
      if (next) {
        if (lane == 0) u = (long long)atomicAdd(next, 1ull);
        u = __shfl_sync(0xffffffffu, u, 0);
      }
      if (u >= total) break;
      tag(u);
      if (!ok) break;
      src.unit(u, [&](const DProblem& P, const CUtensorMap* ma, const CUtensorMap* mb, const Unit& w) {
        ok = produce_unit(ma, mb, P.a, P.b, P.m, P.n, P.k, P.ts, (int64_t)w.tm * P.ts, (int64_t)w.tn * P.ts, w.kb0,
                          w.kb1, sm.sA, sm.sB, sm.full, sm.empty, stage, phase, lane, status);
      });
      if (!ok) break;
    }
    if (ok) {
      tag(-1);
      if (ok) mbar_arrive(&sm.full[stage]);
      if (ok && lane == 0) mbar_arrive(&sm.full[stage]);
    }
    cp_async_wait_all();
    if (next && lane == 0) {
      // the last group out resets the counters for the next launch
      __threadfence();
      const unsigned long long done = atomicAdd(next + 1, 1ull);
      if (done == (unsigned long long)gridDim.x * GROUPS - 1) {
        next[0] = 0ull;
        next[1] = 0ull;
        __threadfence();
      }
    }
    return;
  }
  for (;;) {
    if (!mbar_wait_bounded(&sm.full[stage], phase)) {
      report_status(status, DEV_TIMEOUT_FULL);
      return;
    }
    const long long u = s_stage_unit[stage];
    if (u < 0) return;
    bool ok = true;
    src.unit(u, [&](const DProblem& P, const CUtensorMap*, const CUtensorMap*, const Unit& w) {
      const Place at = place_of((int64_t)w.tm * P.ts, (int64_t)w.tn * P.ts, P.ts, P.m, P.n, warp, lane);
      double acc[2][2][2] = {};
      ok = consume_unit(P.a.xc, P.b.xc, P.k, w.kb0, w.kb1, at, sm.sA, sm.sB, sm.full, sm.empty, stage, phase, lane,
                        P.run, acc, status);
      if (!ok) return;
      if (P.ts <= 16) reduce_warps(acc, sm.red, warp, lane, group);
      finish_unit(P.e, acc, at, P.ts, P.splits, w.sp,
                  P.splits > 1 ? P.partials + (size_t)w.tile * P.splits * (P.ts * P.ts) : nullptr,
                  P.splits > 1 ? P.counters + w.tile : nullptr, tid, group, sm.s_last);
    });
    if (!ok) return;
  }
}

}  // namespace dmma
}  // namespace momms

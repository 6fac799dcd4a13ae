// f32 GEMM as an error-compensated 3-term split-TF32 product on tcgen05.
//
// Each operand is split once into two TF32 planes, x = hi + lo with
// hi = tf32_rna(x) and lo = tf32_rna(x - hi) (the subtraction is exact), and
// C = beta*C + alpha*(A_lo B_hi + A_hi B_lo + A_hi B_hi) is accumulated in one
// FP32 TMEM accumulator (the dropped A_lo B_lo term is below 2^-22 relative;
// Markidis et al. 2018, Ootomo & Yokota 2022). The small cross terms are
// accumulated first. The result stays inside the f32 componentwise bound
// |dC| <= 2k u_32 (|A||B|) that the plain FFMA path meets.
#include <algorithm>
#include <cstdlib>

#include "internal.h"
#include "planes.cuh"
#include "slicegemm.cuh"

namespace momms {

namespace {
struct Tf32SplitOp {
  static constexpr int PLANES = 2;  // hi, lo
  using Tout = float;
  using Word = uint2;  // one pair's float2 bits
  __device__ __forceinline__ int row(int64_t) const { return 0; }
  __device__ __forceinline__ void first(int64_t, int) const {}
  __device__ __forceinline__ static void split(float v, float* hi_out, float* lo_out) {
    uint32_t hi, lo;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(v));
    const float rest = v - __uint_as_float(hi);
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(rest));
    *hi_out = __uint_as_float(hi);
    *lo_out = __uint_as_float(lo);
  }
  // two neighbouring elements of a row: their hi pair and lo pair
  __device__ __forceinline__ void pack(float v0, float v1, int, uint2 (&out)[2]) const {
    float h0, h1, l0, l1;
    split(v0, &h0, &l0);
    split(v1, &h1, &l1);
    out[0] = make_uint2(__float_as_uint(h0), __float_as_uint(h1));
    out[1] = make_uint2(__float_as_uint(l0), __float_as_uint(l1));
  }
};

int64_t tiles(int64_t rows, int64_t cols) { return ceil_div(rows, sp::BM) * ceil_div(cols, sp::BN); }

// CTAs per tile where the tiles are fewer than the GPU has room for: the split
// of k (1: none) whose waves end first, from 0.33 us per k-block of a pair and
// 5 us per wave, 7 with the reduction. Measured (us, 1 / 2 / 4 / 8 CTAs, the
// pair kernel for 1): 512^3 32 / 26 / 22 / 20; 1024^3 52 / 37 / 29 / 54;
// 1500^3 73 / 54 / 62 / 101; 2048^3 102 / 114 / 127 / 189; 2560^3 212 / 200 /
// 225 / 333; 64 x 64 x 4096 139 / 77 / 47 / 31.
int split_ctas(int64_t m, int64_t n, int kblocks, int sms) {
  const int64_t pairs = ceil_div(m, 2 * sp::BM) * ceil_div(n, sp::BN), units = std::min(tiles(m, n), tiles(n, m));
  if (pairs > sms) return 1;
  double best = 0.92 * (double)ceil_div(pairs, sms / 2) * (3 * 0.33 * kblocks + 5.0);
  int ctas = 1;
  for (int z = 2; z <= 8 && z <= kblocks; z *= 2) {
    const int fit = sp::split_clusters<1>(z);
    if (fit < 1) break;
    const double t = (double)ceil_div(units, fit) * (3 * 0.33 * (double)ceil_div(kblocks, z) + 7.0);
    if (t < best) {
      best = t;
      ctas = z;
    }
  }
  return ctas;
}
}  // namespace

int set_attrs_tf32() {
  cudaError_t e = sp::set_slice_attrs<1, sp::EPI_F32>();
  return e == cudaSuccess ? MOMMS_OK : cuda_fail(e, "cudaFuncSetAttribute(split-TF32)");
}

void tf32_operand_planes(const F32View* v, int count, int64_t K, int64_t kp, cudaStream_t s) {
  planes::Views<float> vs{};
  planes::PlanesBody<float, Tf32SplitOp> body{};
  body.ldp = kp;
  for (int i = 0; i < count; ++i) {
    vs.v[i] = planes::make_view(v[i].x, v[i].sr, v[i].sp, v[i].R, K);
    body.planes[i] = v[i].planes;
    body.plane_elems[i] = v[i].R * kp;
  }
  KernelTimer kt(MOMMS_KERNEL_PREP, s);
  note_launch(planes::launch_to_planes(vs, count, body, s));
}

int launch_sgemm_tf32x3(const DevGemm& g, cudaStream_t s) {
  DeviceState* ds = device_state();
  if (!ds) return MOMMS_ERR_NO_DEVICE;
  // Few tiles: a cluster of CTAs per tile. The same split for every block of a
  // streamed product and for either orientation, so that neither changes a bit.
  const int kblocks = (int)ceil_div(g.k, 32);
  const int ctas = split_ctas(g.whole_m ? g.whole_m : g.m, g.whole_n ? g.whole_n : g.n, kblocks, ds->sm_count);
  // The epilogue's lanes hold consecutive rows of the tile, so C is taken
  // transposed (C^T = B^T A^T) where its columns are the closer ones: 32-lane
  // stores of one line instead of 32 (6000 x 3001 x 4099, C by rows: 627 ->
  // 543 us); a split product takes the orientation of fewer tiles. Every
  // product and the order of the sums stay the same.
  const int64_t fewer = ctas > 1 ? tiles(g.n, g.m) - tiles(g.m, g.n) : 0;
  const bool flip = fewer ? fewer < 0 : std::llabs(g.c.cs) < std::llabs(g.c.rs);
  const int ia = flip ? 1 : 0, ib = 1 - ia;  // the operand (0 = A, 1 = B) that gives the tile's rows, columns
  const int64_t rows = flip ? g.n : g.m, cols = flip ? g.m : g.n;
  // packed operands (momms_pack) bring their planes
  int64_t kp[2];
  size_t plane[2], own = 0;
  for (int i = 0; i < 2; ++i) {
    kp[i] = g.pk[i] ? g.pk[i]->kp : plane_row(g.k, 4, g.tight);
    plane[i] = (size_t)((i ? g.n : g.m) * kp[i]);
    if (!g.pk[i]) own += 2 * plane[i];
  }
  void* buf = nullptr;
  cudaError_t ce = cudaSuccess;
  if (own && (ce = scratch_alloc(&buf, own * sizeof(float), s)) != cudaSuccess)
    return cuda_fail(ce, "split-TF32 planes");
  ScratchGuard free_buf(buf, s);
  float* planes[2];
  for (int i = 0; i < 2; ++i)
    planes[i] = g.pk[i] ? static_cast<float*>(g.pk[i]->planes)
                        : static_cast<float*>(buf) + (i && !g.pk[0] ? 2 * plane[0] : 0);
  const F32View views[2] = {{static_cast<const float*>(g.a.ptr), g.a.rs, g.a.cs, g.m, planes[0]},
                            {static_cast<const float*>(g.b.ptr), g.b.cs, g.b.rs, g.n, planes[1]}};
  if (!g.pk[0] && !g.pk[1] && !g.staging) {
    tf32_operand_planes(views, 2, g.k, kp[0], s);
  } else {
    // each operand's split waits only for that operand
    for (int i = 0; i < 2; ++i) {
      if (g.pk[i]) continue;
      if ((ce = wait_operand(g, i, s)) != cudaSuccess) return cuda_fail(ce, "operand staging");
      tf32_operand_planes(&views[i], 1, g.k, kp[i], s);
    }
  }

  CUtensorMap tmA, tmB, tmB_half;
  auto map = [&](CUtensorMap* m, int i, int64_t R, int box_rows) {
    const uint64_t dims[3] = {(uint64_t)g.k, (uint64_t)R, 2};
    const uint64_t strides[2] = {(uint64_t)kp[i] * 4, (uint64_t)plane[i] * 4};
    const uint32_t box[3] = {32, (uint32_t)box_rows, 1};  // 128-byte k-blocks
    return encode_tiled(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, planes[i], dims, strides, box,
                        CU_TENSOR_MAP_SWIZZLE_128B);
  };
  int rc = map(&tmA, ia, rows, sp::BM);
  if (!rc) rc = map(&tmB, ib, cols, sp::BN);
  if (!rc) rc = map(&tmB_half, ib, cols, sp::BN / 2);  // one CTA's half of the B tile for the pair kernel
  if (rc) return rc;

  sp::Params p;
  memset(&p, 0, sizeof(p));
  p.m = rows;
  p.n = cols;
  p.kelems = 32;
  p.kblocks = kblocks;
  p.tiles_m = (int)ceil_div(rows, sp::BM);
  p.tiles_n = (int)ceil_div(cols, sp::BN);
  p.ngroups = 1;
  p.group_begin[0] = 0;
  p.group_begin[1] = 3;
  // small cross terms first, then hi*hi
  p.pair_a[0] = !flip; p.pair_b[0] = flip;  // A_lo * B_hi
  p.pair_a[1] = flip; p.pair_b[1] = !flip;  // A_hi * B_lo
  p.pair_a[2] = 0; p.pair_b[2] = 0;  // A_hi * B_hi
  // 256 k per tensor-core accumulation (8 k-blocks of one pair), then an RN
  // add in registers; chunks never span pairs
  for (int i = 0; i < 3; ++i) p.pair_w[i] = 1;
  p.chunk_cap = 8;
  p.merge_pairs = 0;
  p.alpha_f = (float)g.alpha;
  p.beta_f = (float)g.beta;
  p.c32 = static_cast<float*>(g.c.ptr);
  p.rsc = flip ? g.c.cs : g.c.rs;
  p.csc = flip ? g.c.rs : g.c.cs;
  p.status = ds->status;

  // the epilogue reads C
  if ((ce = wait_operand(g, 2, s)) != cudaSuccess) return cuda_fail(ce, "operand staging");
  {
    KernelTimer kt(MOMMS_KERNEL_SLICE_TF32, s);
    int variant = sp::SLICE_SPLIT;
    call_info().splits = ctas;
    if (ctas > 1) ce = sp::launch_slice_split<1>(tmA, tmB, p, ctas, s);
    else ce = sp::launch_slice<1, sp::EPI_F32>(tmA, tmB, tmB_half, p, ds->sm_count, s, &variant);
    if (ce != cudaSuccess) return cuda_fail(ce, "split-TF32 slice launch");
    call_info().slice_variant = variant;
  }
  note_launch();
  ce = launch_status();
  if (ce != cudaSuccess) return cuda_fail(ce, "split-TF32 launch");
  return MOMMS_OK;
}

}  // namespace momms

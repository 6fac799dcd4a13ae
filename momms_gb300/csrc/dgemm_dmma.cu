// Plain f64 GEMM on the FP64 tensor-core MMA (DMMA, mma.sync m8n8k4.f64).
//
// Replaces the reference's PackA/PackB copiers (src/composables/pack.rs:51-133)
// with TMA (or cp.async) staging of 128B-swizzled tiles in a 5-stage
// shared-memory ring, its PartM/PartN/ParallelN loops
// (src/composables/part.rs:7-79, src/composables/parallel_range.rs:130-154)
// with a persistent CTA-tile scheduler, its PartK slabs (part.rs:81-120) with
// an in-register k loop plus optional split-k, and the d6x8 microkernel
// (ukernels/bli_gemm_haswell_asm_d6x8.c:666-1200) with warp-level DMMA.
//
// The epilogue keeps the microkernel's order: acc is scaled by alpha and then
// c = fma(beta, c, acc); beta == 0 stores without reading C (d6x8.c:889-1192).
// Unlike the reference, C is rounded once per element, not once per KC=192
// slab; both stay inside |dC| <= 2k u (|A||B|).
//
// Bound by GB300's FP64 rate (about 1.1 TFLOP/s per GPU): see dmma_core.cuh
// for why the tile is 32 x 32 and f64_plan.h for how units are cut.
#include <stdio.h>
#include <string.h>

#include "dmma_core.cuh"
#include "internal.h"

namespace momms {
namespace dmma {

struct Params {
  DProblem prob;
  TileSched sched;  // tiles stepped by prob.ts
  unsigned long long* next;  // unit counter and finished-CTA counter, both zero; null: static deal
  unsigned* status;
};

// The launch's one problem as a source of units.
struct One {
  const Params& p;
  const CUtensorMap *ma, *mb;
  __device__ __forceinline__ long long total() const { return p.sched.units(); }
  template <typename F>
  __device__ __forceinline__ void unit(long long u, F&& fn) const {
    Unit w;
    p.sched.decode(u, w.tm, w.tn, w.sp);
    w.tile = u / p.sched.splits;
    w.kb0 = w.sp * p.prob.kb_split;
    w.kb1 = min(ceil_div_dev(p.prob.k, BK), w.kb0 + p.prob.kb_split);
    fn(p.prob, ma, mb, w);
  }
};

__global__ void __launch_bounds__(THREADS, CTAS_PER_SM)
    dgemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ Params p) {
  dependency_wait_few();
  dgemm_body(One{p, &tmA, &tmB}, p.next, p.status);
}

}  // namespace dmma

// ---------------------------------------------------------------------------
// Host launcher
// ---------------------------------------------------------------------------

// rows x cols operand where `x_is_rows` says whether the non-k index is the
// row index (A: rows = m) or the column index (B: cols = n).
DmmaOrient dmma_orient(const DevMat& v, int64_t rows, int64_t cols, bool x_is_rows) {
  DmmaOrient o;
  o.sx = x_is_rows ? v.rs : v.cs;
  o.sk = x_is_rows ? v.cs : v.rs;
  const int64_t x_ext = x_is_rows ? rows : cols, k_ext = x_is_rows ? cols : rows;
  const bool aligned = (reinterpret_cast<uintptr_t>(v.ptr) & 15) == 0;
  const bool xc = o.sx == 1 && (k_ext == 1 || (o.sk > 0 && o.sk % 2 == 0 && o.sk >= x_ext));
  const bool kc = o.sk == 1 && (x_ext == 1 || (o.sx > 0 && o.sx % 2 == 0 && o.sx >= k_ext));
  o.tma = aligned && (xc || kc);
  // cp.async reads along the smaller stride
  o.xc = o.tma ? xc : (k_ext == 1 || (x_ext > 1 && o.sx <= o.sk));
  return o;
}

int dmma_operand(const DevMat& v, int64_t rows, int64_t cols, bool x_is_rows, int ts, dmma::Operand* op,
                 CUtensorMap* map) {
  const DmmaOrient o = dmma_orient(v, rows, cols, x_is_rows);
  *op = dmma::Operand{static_cast<const double*>(v.ptr), o.sx, o.sk, o.xc ? 1 : 0, o.tma ? 1 : 0};
  if (!o.tma) return MOMMS_OK;
  const int64_t x_ext = x_is_rows ? rows : cols, k_ext = x_is_rows ? cols : rows;
  uint64_t dims[2], strides[1];
  uint32_t box[2];
  if (o.xc) {
    dims[0] = (uint64_t)x_ext, dims[1] = (uint64_t)k_ext;
    strides[0] = (uint64_t)(k_ext == 1 ? round_up(x_ext * 8, 16) : o.sk * 8);
    box[0] = 16, box[1] = dmma::BK;
  } else {
    dims[0] = (uint64_t)k_ext, dims[1] = (uint64_t)x_ext;
    strides[0] = (uint64_t)(x_ext == 1 ? round_up(k_ext * 8, 16) : o.sx * 8);
    box[0] = dmma::BK, box[1] = (uint32_t)dmma::stage_extent(ts);
  }
  return encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, v.ptr, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

int set_attrs_dmma() {
  const cudaError_t e = cudaFuncSetAttribute(dmma::dgemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             dmma::SMEM_BYTES);
  return e == cudaSuccess ? MOMMS_OK : cuda_fail(e, "cudaFuncSetAttribute(dgemm)");
}

int dmma_problem(const DevGemm& g, const F64Plan& plan, dmma::DProblem* P, CUtensorMap* tmA, CUtensorMap* tmB) {
  memset(P, 0, sizeof(*P));
  memset(tmA, 0, sizeof(*tmA));
  memset(tmB, 0, sizeof(*tmB));
  P->m = g.m, P->n = g.n, P->k = g.k;
  P->e = dmma::Epi{g.m, g.n, g.alpha, g.beta, static_cast<double*>(g.c.ptr), g.c.rs, g.c.cs};
  P->tiles_m = plan.tiles_m, P->tiles_n = plan.tiles_n;
  P->splits = plan.splits, P->ts = plan.ts, P->run = plan.run;
  P->kb_split = plan.kb_split;
  // A: rows m, cols k, x = m. B: rows k, cols n, x = n.
  const int rc = dmma_operand(g.a, g.m, g.k, true, plan.ts, &P->a, tmA);
  return rc ? rc : dmma_operand(g.b, g.k, g.n, false, plan.ts, &P->b, tmB);
}

namespace {
int dmma_params(const DevGemm& g, const F64Plan& plan, unsigned* status, dmma::Params* p, CUtensorMap* tmA,
                CUtensorMap* tmB) {
  p->sched = TileSched{plan.tiles_m, plan.tiles_n, plan.splits, 8, plan.kb_split * dmma::BK};
  p->next = nullptr;
  p->status = status;
  return dmma_problem(g, plan, &p->prob, tmA, tmB);
}
}  // namespace

int launch_dgemm_dmma(const DevGemm& g, cudaStream_t s) {
  using namespace dmma;
  DeviceState* ds = device_state();
  if (!ds) return MOMMS_ERR_NO_DEVICE;
  cudaError_t ce;
  if ((ce = wait_operands(g, s)) != cudaSuccess) return cuda_fail(ce, "operand staging");
  const F64Plan plan = f64_plan(g.m, g.n, g.k, ds->sm_count);
  Params p;
  CUtensorMap tmA, tmB;
  const int rc = dmma_params(g, plan, ds->status, &p, &tmA, &tmB);
  if (rc) return rc;
  call_info().splits = plan.splits;
  // split-k partials and counters, and the unit counter of a launch with more
  // units than CTAs
  const int64_t slots = (int64_t)CTAS_PER_SM * ds->sm_count;
  const bool dynamic = plan.units() > slots;
  const size_t part_bytes = (size_t)plan.partial_elems() * sizeof(double);
  const size_t zero_bytes = (dynamic ? 2 * sizeof(unsigned long long) : 0) +
                            (plan.splits > 1 ? (size_t)plan.tiles() * sizeof(unsigned) : 0);
  void* ws = nullptr;
  if (zero_bytes && (ce = scratch_alloc(&ws, part_bytes + zero_bytes, s)) != cudaSuccess)
    return cuda_fail(ce, "split-k workspace");
  ScratchGuard free_ws(ws, s);  // back to the pool in stream order, after the kernel if it was launched
  if (ws) {
    char* zero = static_cast<char*>(ws) + part_bytes;
    if ((ce = cudaMemsetAsync(zero, 0, zero_bytes, s)) != cudaSuccess) return cuda_fail(ce, "memset counters");
    if (dynamic) {
      p.next = reinterpret_cast<unsigned long long*>(zero);
      zero += 2 * sizeof(unsigned long long);
    }
    p.prob.partials = static_cast<double*>(ws);
    p.prob.counters = reinterpret_cast<unsigned*>(zero);
  }
  const int grid = (int)std::min<int64_t>(plan.units(), slots);
  {
    KernelTimer kt(MOMMS_KERNEL_DGEMM_DMMA, s);
    launch_dependent(dgemm_kernel, dim3((unsigned)grid), THREADS, SMEM_BYTES, s, tmA, tmB, p);
  }
  note_launch();
  ce = launch_status();
  return ce == cudaSuccess ? MOMMS_OK : cuda_fail(ce, "dgemm_dmma launch");
}

}  // namespace momms

// ---------------------------------------------------------------------------
// momms_dgemm_noalloc: the f64 GEMM for callers that cannot allocate device
// memory. Same kernel and same tile / split-k plan as momms_dgemm on device
// operands; the split-k scratch comes from a fixed device-global array instead
// of the stream-ordered pool.
// ---------------------------------------------------------------------------
#include <mutex>

namespace momms {
namespace {

constexpr size_t kNoallocPartialTiles = kSplitTileCap;  // 128 x 128 f64 partial tiles
constexpr size_t kNoallocPartialBytes = kNoallocPartialTiles * 128 * 128 * sizeof(double);
constexpr size_t kNoallocCounterSlots = kSplitCounterCap;  // per-output-tile arrival counters
constexpr size_t kNoallocBytes = kNoallocPartialBytes + kNoallocCounterSlots * sizeof(unsigned);
static_assert(kNoallocBytes == MOMMS_NOALLOC_SCRATCH_BYTES + 1024, "scratch layout must match the header's sizes");

// The scratch itself. Every GPU that loads this library holds these bytes
// until the process exits; every call of momms_dgemm_noalloc on a device uses
// the same bytes. In host code this name is only a stand-in for the device
// address: host code passes the address from cudaGetSymbolAddress instead.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoallocBytes];
// The no-alloc calls' status word: a kernel whose bounded wait expires ORs a
// DEV_* bit in here (momms_noalloc_status reads and clears it). Like the
// scratch, one word per device for the life of the process.
static __device__ unsigned g_noalloc_status;

struct NoallocDevice {
  bool ready = false;
  void* scratch = nullptr;   // device address of g_noalloc_scratch on this device
  unsigned* status = nullptr;  // device address of g_noalloc_status on this device
  int sm_count = 0;
};
std::mutex g_noalloc_mu;
NoallocDevice g_noalloc_dev[64];

// One-time set-up per device, run by the first call on that device with the
// device current: looks up the scratch array's device address and the SM
// count, and raises the kernels' shared-memory limit. Allocates nothing.
int noalloc_setup(NoallocDevice*& out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  if (dev < 0 || dev >= 64) return fail(MOMMS_ERR_NO_DEVICE, "device ordinal %d out of range", dev);
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  NoallocDevice& d = g_noalloc_dev[dev];
  if (!d.ready) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(no-alloc scratch)");
    void* st = nullptr;
    e = cudaGetSymbolAddress(&st, g_noalloc_status);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(no-alloc status)");
    int sms = 0;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaDeviceGetAttribute");
    e = cudaFuncSetAttribute(dmma::dgemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dmma::SMEM_BYTES);
    if (e != cudaSuccess) return cuda_fail(e, "cudaFuncSetAttribute");
    d.scratch = p;
    d.status = static_cast<unsigned*>(st);
    d.sm_count = sms;
    d.ready = true;
  }
  out = &d;
  return MOMMS_OK;
}

}  // namespace

// The no-alloc status word of the current device (nullptr with the error
// recorded if the set-up fails); used by the wait-expiry self-test.
unsigned* noalloc_status_word() {
  NoallocDevice* nd = nullptr;
  return noalloc_setup(nd) ? nullptr : nd->status;
}
}  // namespace momms

extern "C" int momms_dgemm_noalloc(int64_t m, int64_t n, int64_t k, const double* alpha, const double* a,
                                   int64_t rs_a, int64_t cs_a, const double* b, int64_t rs_b, int64_t cs_b,
                                   const double* beta, double* c, int64_t rs_c, int64_t cs_c, void* stream) {
  using namespace momms;
  using namespace momms::dmma;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (!alpha || !beta) return fail(MOMMS_ERR_INVALID_ARG, "alpha/beta pointer is null");
  if (m < 0 || n < 0 || k < 0) return fail(MOMMS_ERR_INVALID_ARG, "negative size");
  if (m > INT32_MAX || n > INT32_MAX || k > INT32_MAX) return fail(MOMMS_ERR_INVALID_ARG, "dimension above 2^31-1");
  if (m == 0 || n == 0 || k == 0) return MOMMS_OK;  // as momms_dgemm: k == 0 leaves C as it is
  if (!a || !b || !c) return fail(MOMMS_ERR_INVALID_ARG, "null operand pointer");
  if (rs_a < 0 || cs_a < 0 || rs_b < 0 || cs_b < 0 || rs_c < 0 || cs_c < 0)
    return fail(MOMMS_ERR_INVALID_ARG, "negative stride");
  if (m > 1 && n > 1 && rs_c == cs_c) return fail(MOMMS_ERR_INVALID_ARG, "C has equal strides");
  int cur = -1;
  if (cudaGetDevice(&cur) != cudaSuccess) {
    cudaGetLastError();
    return fail(MOMMS_ERR_NO_DEVICE, "no current CUDA device");
  }
  const void* ptrs[3] = {a, b, c};
  for (const void* p : ptrs) {
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess ||
        !(at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged)) {
      cudaGetLastError();
      return fail(MOMMS_ERR_INVALID_ARG,
                  "momms_dgemm_noalloc takes device operands only (staging host memory would allocate)");
    }
    // the kernels' TMA reads go to this device's memory only
    if (at.type == cudaMemoryTypeDevice && at.device != cur)
      return fail(MOMMS_ERR_INVALID_ARG, "operand is memory of device %d, the current device is %d", at.device,
                  cur);
  }
  NoallocDevice* nd = nullptr;
  int rc = noalloc_setup(nd);
  if (rc) return rc;

  DevGemm g;
  g.dtype = MOMMS_DTYPE_F64;
  g.m = m; g.n = n; g.k = k;
  g.alpha = *alpha; g.beta = *beta;
  g.a = DevMat{const_cast<double*>(a), rs_a, cs_a};
  g.b = DevMat{const_cast<double*>(b), rs_b, cs_b};
  g.c = DevMat{c, rs_c, cs_c};
  if (!dmma_orient(g.a, g.m, g.k, true).tma || !dmma_orient(g.b, g.k, g.n, false).tma)
    return fail(MOMMS_ERR_INVALID_ARG,
                "momms_dgemm_noalloc needs A and B with unit stride along one index, the other stride a multiple of "
                "2 elements and 16-byte aligned bases (other layouts would need a repack copy)");

  // The same plan as momms_dgemm, so both give the same result.
  const F64Plan plan = f64_plan(g.m, g.n, g.k, nd->sm_count);
  const size_t part_bytes = (size_t)plan.partial_elems() * sizeof(double);
  if (plan.splits > 1 && (!f64_split_fits(m, n, plan.splits) || part_bytes > kNoallocPartialBytes ||
                          (size_t)plan.tiles() > kNoallocCounterSlots))
    return fail(MOMMS_ERR_INVALID_ARG,
                "this problem needs %lld split-k partial tiles of 128x128 doubles (%zu bytes, %lld counters); the "
                "no-alloc scratch holds %zu (%zu bytes, %zu counters)",
                (long long)(ceil_div(m, 128) * ceil_div(n, 128) * plan.splits), part_bytes, (long long)plan.tiles(),
                kNoallocPartialTiles, kNoallocPartialBytes, kNoallocCounterSlots);
  Params p;
  CUtensorMap tmA, tmB;
  // waits report in the no-alloc status word, not the library's allocated one
  rc = dmma_params(g, plan, nd->status, &p, &tmA, &tmB);
  if (rc) return rc;
  if (plan.splits > 1) {
    p.prob.partials = static_cast<double*>(nd->scratch);
    p.prob.counters = reinterpret_cast<unsigned*>(static_cast<unsigned char*>(nd->scratch) + kNoallocPartialBytes);
    // counters must start at zero; the array keeps whatever the last call left
    cudaError_t e = cudaMemsetAsync(p.prob.counters, 0, (size_t)plan.tiles() * sizeof(unsigned), s);
    if (e != cudaSuccess) return cuda_fail(e, "clear split-k counters");
  }
  const int grid = (int)std::min<int64_t>(p.sched.units(), (int64_t)CTAS_PER_SM * nd->sm_count);
  dgemm_kernel<<<grid, THREADS, SMEM_BYTES, s>>>(tmA, tmB, p);
  note_launch();
  cudaError_t e = launch_status();
  if (e != cudaSuccess) return cuda_fail(e, "dgemm_noalloc launch");
  return MOMMS_OK;
}

extern "C" int momms_noalloc_status(uint32_t* bits) {
  using namespace momms;
  NoallocDevice* nd = nullptr;
  int rc = noalloc_setup(nd);
  if (rc) return rc;
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return cuda_fail(e, "cudaDeviceSynchronize");
  unsigned w = 0;
  const unsigned zero = 0;
  e = cudaMemcpyFromSymbol(&w, g_noalloc_status, sizeof(unsigned));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_noalloc_status, &zero, sizeof(unsigned));
  if (e != cudaSuccess) return cuda_fail(e, "no-alloc status word");
  if (bits) *bits = w;
  if (w) return fail(MOMMS_ERR_DEVICE_TIMEOUT, "no-alloc status bits 0x%x", w);
  return MOMMS_OK;
}

// Grouped persistent launches: many independent GEMMs in one kernel per
// dtype, and the execution plans (momms_plan_*) that hold their problem
// tables, workspaces and an optional CUDA graph.
//
// Every plain f64 problem contributes tiles x splits work units to one
// persistent DMMA kernel and every plain f32 problem to one persistent FFMA
// kernel. Units are ordered by decreasing cost (longest first) and handed to
// the CTAs through a global atomic counter. Each problem keeps the split
// count a single launch of its shape uses (the tuning table or the model,
// tune.cu: the runtime analogue of the reference's compile-time block
// sizes), and its k-splits are reduced in a fixed order, so a problem's
// result does not depend on the rest of the batch.
#include <string.h>

#include <algorithm>
#include <mutex>
#include <numeric>
#include <vector>

#include "dmma_core.cuh"
#include "ffma_core.cuh"
#include "internal.h"

namespace momms {
namespace grouped {

using dmma::DProblem;

struct SProblem {
  ffma::Operands o;
  ffma::Epi e;
  int tiles_m, tiles_n, splits, pad;
  int64_t kb_split;
  int64_t unit_begin;
  int64_t part_offset;
  int64_t counter_offset;
};

template <typename P>
__device__ __forceinline__ int find_problem(const P* probs, int nprobs, int64_t u) {
  int lo = 0, hi = nprobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (probs[mid].unit_begin <= u) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// A table of problems, ordered by their first unit, as a source of units.
struct Many {
  const CUtensorMap* maps;
  const DProblem* probs;
  int nprobs;
  long long units;
  __device__ __forceinline__ long long total() const { return units; }
  template <typename F>
  __device__ __forceinline__ void unit(long long u, F&& fn) const {
    const int pi = find_problem(probs, nprobs, u);
    const DProblem& P = probs[pi];
    const int64_t local = u - P.unit_begin;
    dmma::Unit w;
    w.sp = (int)(local % P.splits);
    w.tile = local / P.splits;
    w.tm = (int)(w.tile % P.tiles_m);
    w.tn = (int)(w.tile / P.tiles_m);
    w.kb0 = w.sp * P.kb_split;
    w.kb1 = min(ceil_div_dev(P.k, dmma::BK), w.kb0 + P.kb_split);
    fn(P, &maps[2 * pi], &maps[2 * pi + 1], w);
  }
};

// Every plain f64 problem's units, dealt dynamically (dgemm_body); the last
// CTA resets the unit counter, so a captured plan relaunches as is.
// GROUPS = CTAS_PER_SM: an SM's CTAs as one, for launches capped to some of the
// SMs. The CTAs of a grid are spread over all SMs that can take one: four small
// ones for each SM of the cap ran on every SM, and a request whose kernel needs a
// whole SM waited for the large one beside it to end (emulated 512 x 512 x 512
// beside f64 4096 x 4096 x 2048: 52 ms, 0.07 as one CTA on each SM of the cap).
template <int GROUPS>
__global__ void __launch_bounds__(dmma::THREADS * GROUPS, dmma::CTAS_PER_SM / GROUPS)
    dgemm_grouped_kernel(const CUtensorMap* __restrict__ maps, const DProblem* __restrict__ probs, int nprobs,
                         int64_t total_units, unsigned long long* next_unit, unsigned* status) {
  dmma::dgemm_body<GROUPS>(Many{maps, probs, nprobs, total_units}, next_unit, status);
}

template <int TM, typename Off>
__global__ void __launch_bounds__(ffma::Tile<TM>::THREADS, ffma::Tile<TM>::CTAS_PER_SM)
    sgemm_grouped_kernel(const SProblem* __restrict__ probs, int nprobs, int64_t total_units,
                         unsigned long long* next_unit, float* partials, unsigned* counters) {
  using namespace ffma;
  extern __shared__ float4 ffma_smem[];
  __shared__ int s_last;
  __shared__ long long s_unit;
  for (;;) {
    if (threadIdx.x == 0) s_unit = (long long)atomicAdd(next_unit, 1ull);
    __syncthreads();
    const int64_t u = s_unit;
    __syncthreads();
    if (u >= total_units) break;
    const int pi = find_problem(probs, nprobs, u);
    const SProblem& P = probs[pi];
    const int64_t local = u - P.unit_begin;
    const int sp = (int)(local % P.splits);
    const int64_t tile = local / P.splits;
    const int tm = (int)(tile % P.tiles_m), tn = (int)(tile / P.tiles_m);
    const int64_t kblocks = ceil_div_dev(P.o.k, BK);
    const int64_t kb0 = sp * P.kb_split, kb1 = min(kblocks, kb0 + P.kb_split);
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
    prefetch_c_tile<TM>(P.e, tm, tn);
    ffma_unit_any<TM, Off>(P.o, tm, tn, kb0, kb1, acc, reinterpret_cast<float*>(ffma_smem));
    ffma_finish<TM>(P.e, acc, tm, tn, P.splits, sp,
                    P.splits > 1 ? partials + P.part_offset + (size_t)tile * P.splits * TM * TM : nullptr,
                    P.splits > 1 ? counters + P.counter_offset + tile : nullptr, &s_last);
  }
  // the last CTA out resets the unit counter for the next launch of the plan
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned long long done = atomicAdd(next_unit + 1, 1ull);
    if (done == (unsigned long long)gridDim.x - 1) {
      next_unit[0] = 0ull;
      next_unit[1] = 0ull;
      __threadfence();
    }
  }
}

}  // namespace grouped

// ---------------------------------------------------------------------------
// Plans
// ---------------------------------------------------------------------------

struct PlanProblem {
  momms_gemm_desc d;
  int slices;  // Ozaki: frozen slice count
  bool tight;  // DevGemm::tight
  DevGemm gemm() const {
    DevGemm g = devgemm_of(d);
    g.tight = tight;
    return g;
  }
};

struct Plan {
  int device = -1;
  // stream-ordered mode (used by the server): allocations, uploads and frees
  // are enqueued on `stream` instead of synchronising the device
  bool async = false;
  cudaStream_t stream = nullptr;
  std::vector<char> host_tables;  // upload sources, alive until destroy
  // f64 plain group
  int nd = 0;
  int64_t d_units = 0;
  grouped::DProblem* d_probs = nullptr;  // device
  CUtensorMap* d_maps = nullptr;         // device
  double* d_partials = nullptr;
  unsigned* d_counters = nullptr;
  unsigned long long* d_next = nullptr;  // unit counter + finished-CTA counter
  // f32 plain groups, one per FFMA tile (0: 128 x 128, 1: 64 x 64), each
  // one persistent launch
  struct SGroup {
    int ns = 0;
    int64_t units = 0;
    grouped::SProblem* probs = nullptr;
    float* partials = nullptr;
    unsigned* counters = nullptr;
    unsigned long long* next = nullptr;
    bool wide = false;  // some f32 operand needs 64-bit element offsets
  } sg[2];
  // problems run by their own launch sequence (Ozaki, split-TF32)
  std::vector<PlanProblem> other;
  // two or more emulated problems with fixed slice counts: one slice launch
  OzakiBatch* ozb = nullptr;
  // captured graph
  cudaGraphExec_t graph = nullptr;
  std::vector<void*> allocs;
};

namespace {

int plan_alloc(Plan* p, void** out, size_t bytes) {
  if (bytes == 0) {
    *out = nullptr;
    return MOMMS_OK;
  }
  cudaError_t e = p->async ? scratch_alloc(out, bytes, p->stream) : device_malloc(out, bytes);
  if (e != cudaSuccess) return cuda_fail(e, "plan allocation");
  p->allocs.push_back(*out);
  return MOMMS_OK;
}

void plan_free(Plan* p) {
  if (p->graph) cudaGraphExecDestroy(p->graph);
  ozaki_batch_destroy(p->ozb);
  for (void* a : p->allocs) {
    if (p->async) cudaFreeAsync(a, p->stream);
    else cudaFree(a);
  }
  delete p;
}

bool on_device(const void* ptr) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, ptr) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged;
}

}  // namespace

int set_attrs_grouped() {
  cudaError_t e = cudaFuncSetAttribute(grouped::dgemm_grouped_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       dmma::smem_bytes(1));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(grouped::dgemm_grouped_kernel<dmma::CTAS_PER_SM>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, dmma::smem_bytes(dmma::CTAS_PER_SM));
  return e == cudaSuccess ? MOMMS_OK : cuda_fail(e, "cudaFuncSetAttribute(grouped)");
}

// Copies host bytes to the device: synchronously, or stream-ordered from a
// copy kept in the plan until it is destroyed.
int plan_upload(Plan* p, void* dst, const void* src, size_t bytes) {
  if (bytes == 0) return MOMMS_OK;
  cudaError_t e;
  if (p->async) {
    const size_t off = p->host_tables.size();
    p->host_tables.resize(off + bytes);
    memcpy(p->host_tables.data() + off, src, bytes);
    (void)off;
    e = cudaSuccess;
  } else {
    e = cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice);
  }
  return e == cudaSuccess ? MOMMS_OK : cuda_fail(e, "plan upload");
}

int plan_zero(Plan* p, void* dst, size_t bytes) {
  if (bytes == 0) return MOMMS_OK;
  cudaError_t e = p->async ? cudaMemsetAsync(dst, 0, bytes, p->stream) : cudaMemset(dst, 0, bytes);
  return e == cudaSuccess ? MOMMS_OK : cuda_fail(e, "plan workspace");
}

int plan_create(const momms_gemm_desc* descs, int count, Plan** out, cudaStream_t async_stream, bool async,
                const char* tight) {
  *out = nullptr;
  if (!descs || count < 0) return fail(MOMMS_ERR_INVALID_ARG, "descs is null or count < 0");
  DeviceState* ds = device_state();
  if (!ds) return MOMMS_ERR_NO_DEVICE;
  for (int i = 0; i < count; ++i) {
    int rc = momms_gemm_validate(&descs[i]);
    if (rc) return fail(rc, "problem %d: %s", i, momms_last_error());
    const momms_gemm_desc& d = descs[i];
    if (d.m == 0 || d.n == 0 || d.k == 0) continue;
    const momms_operand* ops[3] = {&d.a, &d.b, &d.c};
    for (int j = 0; j < 3; ++j)
      if (!packed_of(*ops[j]) && (ops[j]->mem == MOMMS_MEM_HOST || !on_device(ops[j]->ptr)))
        return fail(MOMMS_ERR_INVALID_ARG, "problem %d: plans take device operands only", i);
  }
  Plan* p = new Plan();
  p->device = ds->device;
  p->async = async;
  p->stream = async_stream;
  std::vector<std::pair<void*, std::pair<size_t, size_t>>> pending;  // (dst, (offset, bytes)) of async uploads

  std::vector<int> dlist, slist;
  for (int i = 0; i < count; ++i) {
    const momms_gemm_desc& d = descs[i];
    if (d.m == 0 || d.n == 0 || d.k == 0) continue;
    if (d.precision == MOMMS_PREC_PLAIN && d.dtype == MOMMS_DTYPE_F64) dlist.push_back(i);
    else if (d.precision == MOMMS_PREC_PLAIN) slist.push_back(i);
    else p->other.push_back(PlanProblem{d, d.slices, tight && tight[i]});
  }

  // ---- f64 group ----
  if (!dlist.empty()) {
    using namespace dmma;
    std::vector<grouped::DProblem> probs;
    std::vector<CUtensorMap> maps;
    // the same plan as a single launch of this shape: a problem's result does
    // not depend on the batch it is in; costliest units first
    std::vector<std::pair<F64Plan, int>> order;
    for (int i : dlist) order.push_back({f64_plan(descs[i].m, descs[i].n, descs[i].k, ds->sm_count), i});
    std::sort(order.begin(), order.end(),
              [](const auto& a, const auto& b) { return a.first.unit_cost > b.first.unit_cost; });
    int64_t units = 0, parts = 0, ctrs = 0;
    for (auto& oc : order) {
      const F64Plan& fp = oc.first;
      const momms_gemm_desc& d = descs[oc.second];
      const DevGemm gv = devgemm_of(d);  // packed operands: their column-major copies
      grouped::DProblem P;
      CUtensorMap ma, mb;
      const int rc = dmma_problem(gv, fp, &P, &ma, &mb);
      if (rc) {
        plan_free(p);
        return rc;
      }
      P.unit_begin = units;
      units += fp.units();
      if (P.splits > 1) {
        // offsets until the buffers exist
        P.partials = reinterpret_cast<double*>(parts * sizeof(double));
        P.counters = reinterpret_cast<unsigned*>(ctrs * sizeof(unsigned));
        parts += fp.partial_elems();
        ctrs += fp.tiles();
      }
      probs.push_back(P);
      maps.push_back(ma);
      maps.push_back(mb);
    }
    p->nd = (int)probs.size();
    p->d_units = units;
    void* buf;
    int rc = plan_alloc(p, &buf, probs.size() * sizeof(grouped::DProblem));
    if (!rc) { p->d_probs = static_cast<grouped::DProblem*>(buf); rc = plan_alloc(p, &buf, maps.size() * sizeof(CUtensorMap)); }
    if (!rc) { p->d_maps = static_cast<CUtensorMap*>(buf); rc = plan_alloc(p, &buf, (size_t)parts * 8); }
    if (!rc) { p->d_partials = static_cast<double*>(buf); rc = plan_alloc(p, &buf, (size_t)ctrs * 4); }
    if (!rc) { p->d_counters = static_cast<unsigned*>(buf); rc = plan_alloc(p, &buf, 2 * sizeof(unsigned long long)); }
    if (!rc) p->d_next = static_cast<unsigned long long*>(buf);
    if (rc) { plan_free(p); return rc; }
    for (grouped::DProblem& P : probs)
      if (P.splits > 1) {
        P.partials = p->d_partials + reinterpret_cast<size_t>(P.partials) / sizeof(double);
        P.counters = p->d_counters + reinterpret_cast<size_t>(P.counters) / sizeof(unsigned);
      }
    size_t off = p->host_tables.size();
    rc = plan_upload(p, p->d_probs, probs.data(), probs.size() * sizeof(grouped::DProblem));
    if (!rc && async) pending.push_back({p->d_probs, {off, probs.size() * sizeof(grouped::DProblem)}});
    off = p->host_tables.size();
    if (!rc) rc = plan_upload(p, p->d_maps, maps.data(), maps.size() * sizeof(CUtensorMap));
    if (!rc && async) pending.push_back({p->d_maps, {off, maps.size() * sizeof(CUtensorMap)}});
    if (!rc) rc = plan_zero(p, p->d_counters, (size_t)ctrs * 4);
    if (!rc) rc = plan_zero(p, p->d_next, 2 * sizeof(unsigned long long));
    if (rc) { plan_free(p); return rc; }
  }

  // ---- f32 groups: each problem's tile (tuning table or model) decides its group ----
  if (!slist.empty()) {
    using namespace ffma;
    std::vector<std::pair<double, grouped::SProblem>> items[2];
    for (int i : slist) {
      const momms_gemm_desc& d = descs[i];
      const DevGemm gv = devgemm_of(d);  // packed operands: their column-major copies
      const DevMat& va = gv.a;
      const DevMat& vb = gv.b;
      if (!((va.rs == 1 || va.cs == 1) && (vb.rs == 1 || vb.cs == 1))) {
        plan_free(p);
        return fail(MOMMS_ERR_INVALID_ARG, "problem %d: grouped f32 operands need unit stride along one index", i);
      }
      grouped::SProblem P;
      memset(&P, 0, sizeof(P));
      const bool a_xc = (va.rs == 1) && !(va.cs == 1 && d.m == 1);
      const bool b_xc = (vb.cs == 1) && !(vb.rs == 1 && d.n == 1);
      const int64_t a_ld = a_xc ? va.cs : va.rs, b_ld = b_xc ? vb.rs : vb.cs;
      const bool vec = ((reinterpret_cast<uintptr_t>(va.ptr) | reinterpret_cast<uintptr_t>(vb.ptr)) & 15) == 0 &&
                       a_ld % 4 == 0 && b_ld % 4 == 0;
      P.o = Operands{static_cast<const float*>(va.ptr), va.rs, va.cs, static_cast<const float*>(vb.ptr), vb.rs,
                     vb.cs, d.m, d.n, d.k, a_xc, b_xc, vec};
      P.e = Epi{d.m, d.n, (float)d.alpha, (float)d.beta, static_cast<float*>(d.c.ptr), d.c.rs, d.c.cs};
      const PlainCfg cfg = f32_cfg(d.m, d.n, d.k, ds->sm_count);
      const int TMv = cfg.tile == 1 ? 64 : 128;
      if (!offsets_fit_32(P.o)) p->sg[cfg.tile].wide = true;
      P.tiles_m = (int)ceil_div(d.m, TMv);
      P.tiles_n = (int)ceil_div(d.n, TMv);
      const int64_t kb = ceil_div(d.k, BK);
      const double tile_cost = (double)std::min<int64_t>(d.m, TMv) * std::min<int64_t>(d.n, TMv) * (double)kb;
      P.kb_split = ceil_div(kb, cfg.splits);
      P.splits = (int)ceil_div(kb, P.kb_split);
      items[cfg.tile].push_back({tile_cost / P.splits, P});
    }
    for (int t = 0; t < 2; ++t) {
      if (items[t].empty()) continue;
      const int TMv = t == 1 ? 64 : 128;
      Plan::SGroup& G = p->sg[t];
      std::sort(items[t].begin(), items[t].end(), [](const auto& a, const auto& b) { return a.first > b.first; });
      std::vector<grouped::SProblem> probs;
      int64_t units = 0, parts = 0, ctrs = 0;
      for (auto& it : items[t]) {
        grouped::SProblem P = it.second;
        const int64_t tiles = (int64_t)P.tiles_m * P.tiles_n;
        P.unit_begin = units;
        units += tiles * P.splits;
        if (P.splits > 1) {
          P.part_offset = parts;
          P.counter_offset = ctrs;
          parts += tiles * P.splits * TMv * TMv;
          ctrs += tiles;
        }
        probs.push_back(P);
      }
      G.ns = (int)probs.size();
      G.units = units;
      void* buf;
      int rc = plan_alloc(p, &buf, probs.size() * sizeof(grouped::SProblem));
      if (!rc) { G.probs = static_cast<grouped::SProblem*>(buf); rc = plan_alloc(p, &buf, (size_t)parts * 4); }
      if (!rc) { G.partials = static_cast<float*>(buf); rc = plan_alloc(p, &buf, (size_t)ctrs * 4 + 16); }
      if (!rc) { G.counters = static_cast<unsigned*>(buf); rc = plan_alloc(p, &buf, 2 * sizeof(unsigned long long)); }
      if (!rc) G.next = static_cast<unsigned long long*>(buf);
      if (rc) { plan_free(p); return rc; }
      const size_t off = p->host_tables.size();
      rc = plan_upload(p, G.probs, probs.data(), probs.size() * sizeof(grouped::SProblem));
      if (!rc && async) pending.push_back({G.probs, {off, probs.size() * sizeof(grouped::SProblem)}});
      if (!rc) rc = plan_zero(p, G.counters, (size_t)ctrs * 4 + 16);
      if (!rc) rc = plan_zero(p, G.next, 2 * sizeof(unsigned long long));
      if (rc) { plan_free(p); return rc; }
    }
  }

  // Ozaki problems with a data-chosen slice count: choose once now (one
  // sampled bound on the current operands), so that launches never wait.
  for (PlanProblem& pp : p->other) {
    if (pp.d.precision == MOMMS_PREC_OZAKI && pp.slices == 0) {
      int s = 0;
      int rc = ozaki_choose_slices(pp.d, &s, async ? async_stream : nullptr);
      if (rc) { plan_free(p); return rc; }
      pp.slices = s;
    }
  }
  // Emulated problems that qualify run together: their slice products in one
  // persistent launch (ozaki_batch_*); the rest keep their own sequences.
  {
    std::vector<DevGemm> gs;
    std::vector<int> sl;
    std::vector<size_t> at;
    for (size_t i = 0; i < p->other.size(); ++i) {
      const PlanProblem& pp = p->other[i];
      const DevGemm g = pp.gemm();
      if (pp.d.precision != MOMMS_PREC_OZAKI || !ozaki_batchable(g, pp.slices)) continue;
      gs.push_back(g);
      sl.push_back(pp.slices);
      at.push_back(i);
    }
    const std::vector<char> in = ozaki_batch_members(gs.data(), sl.data(), (int)gs.size());
    std::vector<char> joined(p->other.size(), 0);
    size_t count = 0;
    for (size_t i = 0; i < gs.size(); ++i) {
      if (!in[i]) continue;
      joined[at[i]] = 1;
      gs[count] = gs[i];
      sl[count++] = sl[i];
    }
    int clusters = 0;
    if (count >= 2 && sp_pairs_available(&clusters)) {
      const int rc = ozaki_batch_create(gs.data(), sl.data(), (int)count, async ? async_stream : nullptr, async, &p->ozb);
      if (rc) { plan_free(p); return rc; }
      std::vector<PlanProblem> rest;
      for (size_t i = 0; i < p->other.size(); ++i)
        if (!joined[i]) rest.push_back(p->other[i]);
      p->other = rest;
    }
  }
  // stream-ordered uploads: the host copies live in p->host_tables (no more
  // appends from here on, so the addresses are stable)
  for (auto& pu : pending) {
    cudaError_t e = cudaMemcpyAsync(pu.first, p->host_tables.data() + pu.second.first, pu.second.second,
                                    cudaMemcpyHostToDevice, async_stream);
    if (e != cudaSuccess) {
      plan_free(p);
      return cuda_fail(e, "plan upload");
    }
  }
  *out = p;
  return MOMMS_OK;
}

void plan_destroy(Plan* p) { plan_free(p); }

int plan_launch(Plan* p, cudaStream_t s, int max_sms) {
  DeviceState* ds = device_state();
  if (!ds) return MOMMS_ERR_NO_DEVICE;
  if (ds->device != p->device) return fail(MOMMS_ERR_INVALID_ARG, "plan belongs to device %d", p->device);
  cudaError_t e;
  if (p->nd) {
    const bool capped = max_sms > 0 && max_sms < ds->sm_count;
    KernelTimer kt(MOMMS_KERNEL_DGEMM_DMMA, s);
    auto launch = [&](auto kernel, int groups, int64_t ctas) {
      const int grid = (int)std::min<int64_t>(ceil_div(p->d_units, groups), ctas);
      kernel<<<grid, dmma::THREADS * groups, dmma::smem_bytes(groups), s>>>(p->d_maps, p->d_probs, p->nd, p->d_units,
                                                                            p->d_next, ds->status);
    };
    if (capped) launch(grouped::dgemm_grouped_kernel<dmma::CTAS_PER_SM>, dmma::CTAS_PER_SM, max_sms);
    else launch(grouped::dgemm_grouped_kernel<1>, 1, (int64_t)dmma::CTAS_PER_SM * ds->sm_count);
    note_launch();
    if ((e = launch_status()) != cudaSuccess) return cuda_fail(e, "grouped f64 launch");
  }
  for (int t = 0; t < 2; ++t) {
    const Plan::SGroup& G = p->sg[t];
    if (!G.ns) continue;
    const int sms = (max_sms > 0 && max_sms < ds->sm_count) ? max_sms : ds->sm_count;
    KernelTimer kt(MOMMS_KERNEL_SGEMM_FFMA, s);
    if (t == 1) {
      using T = ffma::Tile<64>;
      const int grid = (int)std::min<int64_t>(G.units, (int64_t)T::CTAS_PER_SM * sms);
      auto k = G.wide ? grouped::sgemm_grouped_kernel<64, uint64_t> : grouped::sgemm_grouped_kernel<64, uint32_t>;
      k<<<grid, T::THREADS, T::SMEM_BYTES, s>>>(G.probs, G.ns, G.units, G.next, G.partials, G.counters);
    } else {
      using T = ffma::Tile<128>;
      const int grid = (int)std::min<int64_t>(G.units, (int64_t)T::CTAS_PER_SM * sms);
      auto k = G.wide ? grouped::sgemm_grouped_kernel<128, uint64_t> : grouped::sgemm_grouped_kernel<128, uint32_t>;
      k<<<grid, T::THREADS, T::SMEM_BYTES, s>>>(G.probs, G.ns, G.units, G.next, G.partials, G.counters);
    }
    note_launch();
    if ((e = launch_status()) != cudaSuccess) return cuda_fail(e, "grouped f32 launch");
  }
  if (p->ozb) {
    const int rc = ozaki_batch_launch(p->ozb, s, max_sms);
    if (rc) return rc;
  }
  for (PlanProblem& pp : p->other) {
    const DevGemm g = pp.gemm();
    int rc;
    if (pp.d.precision == MOMMS_PREC_OZAKI) {
      int used = 0;
      rc = launch_dgemm_ozaki(g, pp.d.target_rel_err, pp.slices, &used, s);
    } else {
      rc = launch_sgemm_tf32x3(g, s);
    }
    if (rc) return rc;
  }
  return MOMMS_OK;
}

}  // namespace momms

// ---------------------------------------------------------------------------
// extern "C"
// ---------------------------------------------------------------------------
extern "C" {

struct momms_plan_s {
  momms::Plan* p;
};

int momms_plan_create(const momms_gemm_desc* descs, int count, momms_plan* out) {
  if (!out) return momms::fail(MOMMS_ERR_INVALID_ARG, "out is null");
  *out = nullptr;
  momms::Plan* p = nullptr;
  int rc = momms::plan_create(descs, count, &p, nullptr, false, nullptr);
  if (rc) return rc;
  *out = new momms_plan_s{p};
  return MOMMS_OK;
}

int momms_plan_launch(momms_plan plan, void* stream) {
  if (!plan) return momms::fail(MOMMS_ERR_INVALID_ARG, "plan is null");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (plan->p->graph) {
    cudaError_t e = cudaGraphLaunch(plan->p->graph, s);
    return e == cudaSuccess ? MOMMS_OK : momms::cuda_fail(e, "cudaGraphLaunch");
  }
  return momms::plan_launch(plan->p, s, 0);
}

int momms_plan_capture(momms_plan plan, void* stream) {
  if (!plan) return momms::fail(MOMMS_ERR_INVALID_ARG, "plan is null");
  momms::Plan* p = plan->p;
  if (p->graph) return MOMMS_OK;
  cudaStream_t s = nullptr;
  cudaError_t e = cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  if (e != cudaSuccess) return momms::cuda_fail(e, "capture stream");
  (void)stream;
  e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
  if (e != cudaSuccess) {
    cudaStreamDestroy(s);
    return momms::cuda_fail(e, "cudaStreamBeginCapture");
  }
  int rc = momms::plan_launch(p, s, 0);
  cudaGraph_t g = nullptr;
  e = cudaStreamEndCapture(s, &g);
  cudaStreamDestroy(s);
  if (rc) {
    if (g) cudaGraphDestroy(g);
    return rc;
  }
  if (e != cudaSuccess) return momms::cuda_fail(e, "cudaStreamEndCapture");
  e = cudaGraphInstantiate(&p->graph, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) {
    p->graph = nullptr;
    return momms::cuda_fail(e, "cudaGraphInstantiate");
  }
  return MOMMS_OK;
}

int momms_plan_destroy(momms_plan plan) {
  if (!plan) return MOMMS_OK;
  momms::plan_free(plan->p);
  delete plan;
  return MOMMS_OK;
}

int momms_gemm_grouped(const momms_gemm_desc* descs, int count, void* stream) {
  momms_plan plan = nullptr;
  int rc = momms_plan_create(descs, count, &plan);
  if (rc) return rc;
  rc = momms_plan_launch(plan, stream);
  cudaError_t e = cudaStreamSynchronize(static_cast<cudaStream_t>(stream));
  if (!rc && e != cudaSuccess) rc = momms::cuda_fail(e, "stream synchronize");
  momms_plan_destroy(plan);
  return rc;
}

}  // extern "C"

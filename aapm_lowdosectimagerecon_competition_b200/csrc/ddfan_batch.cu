// ddfan_batch.cu -- many OS-SART solves advanced together: one launch per
// kernel kind, subset step and vector class over a device work list of every
// solve's CTAs, instead of one launch per solve.
//
// A batched iteration runs subset step k of every solve that has one: the image
// columns of the solves of few slices, the forward projectors (with the fused
// residual) of all those solves in one launch per class (slices per thread;
// thin or not), then the backprojections the same way (the exact adjoint's,
// then the reference's), then FISTA of every solve in one launch pair.  Each
// CTA reads its item {solve's argument block, view row or voxel tile, channel
// block, z-tile} and runs the same kernel body a single solve's launch runs,
// with that solve's arguments, so every solve computes exactly what it computes
// alone.  Small solves
// (a few slices, a few hundred views) that leave most of the GPU idle in a
// launch of their own fill it together.  The iteration is captured as one
// CUDA graph.  No counterpart in the reference, which runs one
// reconstruction per MATLAB call (AAPM_script/OSSART_AAPM.m:85, :92).
#include <algorithm>
#include <climits>
#include <cstdlib>
#include <map>
#include <memory>
#include <tuple>
#include <vector>

#include <cuda_runtime.h>

#include "ddfan.h"
#include "ddfan_kernels.cuh"
#include "ddfan_plan.h"
#include "ddfan_solver.h"

namespace ddfan {

namespace {

enum BatchKind { BK_FWD = 0, BK_ADJ = 1, BK_REF = 2, BK_COL = 3 };

struct BatchLaunch {
  int kind, sv, thin;  // the kernels' class (dd_dispatch)
  size_t items_off, nitems;
  int group;  // the solver group whose chain the launch belongs to
};

// solver groups whose launch chains run side by side (DDFAN_BATCH_GROUPS in
// the environment overrides it)
#ifndef DDFAN_BATCH_GROUPS
#define DDFAN_BATCH_GROUPS 1
#endif

// the work-list kernels' dynamic shared memory on the current device
// (at every batch creation: the attribute belongs to the context)
int batch_prepare_device(int dev) {
  cudaError_t e = cudaSuccess;
  for (const int sv : {8, 4, 1})
    for (const int thin : {0, 1})
      dd_dispatch(sv, thin, [&](auto SV, auto THIN) {
        constexpr int v = decltype(SV)::value;
        constexpr bool t = decltype(THIN)::value;
        if (e == cudaSuccess) e = dd_allow_dyn(k_fwd_dd_batch<v, t>, DdFwdTile<v>::DYN);
        if (e == cudaSuccess) e = dd_allow_dyn(k_back_dd_batch<v, true, t>, DdBackTile<v>::DYN);
        if (e == cudaSuccess) e = dd_allow_dyn(k_back_dd_batch<v, false, t>, DdBackTile<v>::DYN);
      });
  if (e != cudaSuccess)
    return set_err(DDFAN_ERR_CUDA, "batched kernel attributes on device %d: %s", dev, cudaGetErrorString(e));
  return DDFAN_OK;
}

}  // namespace

struct Batch {
  int device = 0;
  std::vector<Solver*> sv;
  std::vector<BatchLaunch> launches;  // one iteration, in order
  DdFwdArgs* d_fargs = nullptr;
  DdBackArgs* d_bargs = nullptr;
  ColArgs* d_cargs = nullptr;
  int4* d_items = nullptr;
  FistaDesc* d_fista = nullptr;
  int nfista = 0;
  size_t fista_max = 0;
  cudaStream_t own = nullptr;
  cudaEvent_t last_use = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t gexec = nullptr;
  int kernel_launches = 0;
  // side streams and events of the solver groups' chains (parallel branches
  // of the captured graph); group g's launches are contiguous in `launches`
  int groups = 1;
  std::vector<cudaStream_t> side;
  std::vector<cudaEvent_t> join;
  cudaEvent_t fork = nullptr;
};

static void batch_free(Batch* b) {
  if (!b) return;
  int prev = -1;
  cudaGetDevice(&prev);
  cudaSetDevice(b->device);
  if (b->own && b->last_use) {
    cudaStreamWaitEvent(b->own, b->last_use, 0);
    cudaStreamSynchronize(b->own);
  }
  if (b->gexec) cudaGraphExecDestroy(b->gexec);
  if (b->graph) cudaGraphDestroy(b->graph);
  void* ptrs[] = {b->d_fargs, b->d_bargs, b->d_cargs, b->d_items, b->d_fista};
  for (void* q : ptrs) dev_free(q, b->own);
  if (b->own) cudaStreamDestroy(b->own);
  if (b->last_use) cudaEventDestroy(b->last_use);
  for (cudaStream_t q : b->side) cudaStreamDestroy(q);
  for (cudaEvent_t q : b->join) cudaEventDestroy(q);
  if (b->fork) cudaEventDestroy(b->fork);
  cudaGetLastError();
  if (prev >= 0) cudaSetDevice(prev);
  delete b;
}

// One launch of the work list on st.
static int batch_launch(Batch& b, const BatchLaunch& L, cudaStream_t st) {
  {
    const int4* it = b.d_items + L.items_off;
    const unsigned n = (unsigned)L.nitems;
    if (L.kind == BK_COL) {
      ProfScope ps(KIND_FWD, st);
      k_columns_batch<<<n, 256, 0, st>>>(b.d_cargs, it);
    } else if (L.kind == BK_FWD) {
      ProfScope ps(KIND_FWD, st);
      dd_dispatch(L.sv, L.thin, [&](auto SV, auto THIN) {
        constexpr int v = decltype(SV)::value;
        k_fwd_dd_batch<v, decltype(THIN)::value><<<n, 256, DdFwdTile<v>::DYN, st>>>(b.d_fargs, it);
      });
    } else {
      ProfScope ps(KIND_BACK_A, st);
      dd_dispatch(L.sv, L.thin, [&](auto SV, auto THIN) {
        constexpr int v = decltype(SV)::value;
        constexpr bool t = decltype(THIN)::value;
        if (L.kind == BK_ADJ) k_back_dd_batch<v, true, t><<<n, 256, DdBackTile<v>::DYN, st>>>(b.d_bargs, it);
        else k_back_dd_batch<v, false, t><<<n, 256, DdBackTile<v>::DYN, st>>>(b.d_bargs, it);
      });
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return set_err(DDFAN_ERR_CUDA, "batched launch (kind %d): %s", L.kind, cudaGetErrorString(e));
  }
  return DDFAN_OK;
}

// The launches of one batched iteration (every solve's next iteration).  With
// several solver groups each group's launches form a chain of their own on a
// side stream forked from st and joined back before FISTA (under capture:
// parallel branches of the graph), so one group's forward projections run
// beside another's backprojections, as separate solves on separate streams
// do; within a group the launches keep the step order.
static int batch_iteration(Batch& b, cudaStream_t st) {
  const bool fork = b.groups > 1 && !b.side.empty();
  cudaError_t e = cudaSuccess;
  if (fork) {
    e = cudaEventRecord(b.fork, st);
    for (size_t t = 0; t < b.side.size() && e == cudaSuccess; ++t) e = cudaStreamWaitEvent(b.side[t], b.fork, 0);
    if (e != cudaSuccess) return set_err(DDFAN_ERR_CUDA, "batch: fork: %s", cudaGetErrorString(e));
  }
  for (const BatchLaunch& L : b.launches) {
    const cudaStream_t q = fork && L.group > 0 ? b.side[L.group - 1] : st;
    const int rc = batch_launch(b, L, q);
    if (rc) return rc;
  }
  if (fork) {
    for (size_t t = 0; t < b.side.size() && e == cudaSuccess; ++t) {
      e = cudaEventRecord(b.join[t], b.side[t]);
      if (e == cudaSuccess) e = cudaStreamWaitEvent(st, b.join[t], 0);
    }
    if (e != cudaSuccess) return set_err(DDFAN_ERR_CUDA, "batch: join: %s", cudaGetErrorString(e));
  }
  if (b.nfista) {
    ProfScope ps(KIND_FISTA, st);
    const int blocks = (int)std::max<size_t>(1, std::min<size_t>((b.fista_max + 255) / 256, 1024));
    k_fista_batch<<<dim3(blocks, b.nfista), 256, 0, st>>>(b.d_fista);
    k_fista_t_batch<<<(b.nfista + 127) / 128, 128, 0, st>>>(b.d_fista, b.nfista);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return set_err(DDFAN_ERR_CUDA, "batched fista: %s", cudaGetErrorString(e));
  }
  return DDFAN_OK;
}

static int batch_create(Batch** out, Solver* const* solvers, int n) {
  *out = nullptr;
  if (!solvers || n < 1) return set_err(DDFAN_ERR_ARG, "batch: no solvers");
  std::unique_ptr<Batch, void (*)(Batch*)> B(new Batch(), batch_free);
  Batch& b = *B;
  for (int i = 0; i < n; ++i) {
    Solver* s = solvers[i];
    if (!s) return set_err(DDFAN_ERR_ARG, "batch: solver %d is null", i);
    if (!s->batchable)
      return set_err(DDFAN_ERR_UNSUPPORTED,
                     "batch: solver %d is not a direct-mode solver with one angle list for all slices", i);
    if (i && s->device != solvers[0]->device)
      return set_err(DDFAN_ERR_ARG, "batch: solvers on devices %d and %d", solvers[0]->device, s->device);
    for (int j = 0; j < i; ++j)
      if (solvers[j] == s) return set_err(DDFAN_ERR_ARG, "batch: solver %d appears twice", i);
    b.sv.push_back(s);
  }
  b.device = solvers[0]->device;
  DeviceGuard g(b.device);
  {
    const int rc = batch_prepare_device(b.device);
    if (rc) return rc;
  }
  int maxsub = 0;
  for (Solver* s : b.sv) maxsub = std::max(maxsub, s->nsub);
  std::vector<DdFwdArgs> fargs;
  std::vector<DdBackArgs> bargs;
  std::vector<ColArgs> cargs;
  std::vector<int> col_of(b.sv.size(), -1);  // each solver's entry in cargs
  std::vector<int4> items;
  // solver groups: largest solves first, dealt round robin
  int G = DDFAN_BATCH_GROUPS;
  if (const char* v = getenv("DDFAN_BATCH_GROUPS")) G = atoi(v);
  G = std::max(1, std::min(G, (int)b.sv.size()));
  b.groups = G;
  std::vector<int> group_of(b.sv.size());
  {
    std::vector<int> order(b.sv.size());
    for (size_t i = 0; i < order.size(); ++i) order[i] = (int)i;
    auto work = [&](int i) { const Solver& s = *b.sv[i]; return (double)s.XN * s.YN * s.Zi * s.PNall; };
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return work(x) > work(y); });
    for (size_t r = 0; r < order.size(); ++r) group_of[order[r]] = (int)(r % G);
  }
  // per group, per step: class -> items, for each kind
  for (int grp = 0; grp < G; ++grp)
  for (int k = 0; k < maxsub; ++k) {
    std::map<std::pair<int, int>, std::vector<int4>> cols, fwd, back_adj, back_ref;  // by class
    for (size_t si = 0; si < b.sv.size(); ++si) {
      if (group_of[si] != grp) continue;
      Solver& s = *b.sv[si];
      if (k >= s.nsub) continue;
      const Plan& p = *s.P;
      const int o = s.off[k], c = s.cnt[k];
      if (c < 1) continue;
      const bool adj = s.back_mode == DDFAN_BACK_ADJ;
      const ViewGeom* vg = s.d_vg + o;
      const double2* fc = s.d_fc + (size_t)o * (s.U + 1);
      const float* cvd = s.d_cvd + (size_t)o * s.U;
      DdResidual r;
      r.y = s.d_y; r.yview = s.d_yview + o; r.rowsum = s.d_rows + (size_t)o * s.U; r.wgt = adj ? cvd : nullptr;
      r.ystride = s.Zi;
      const DdFwdArgs fa = make_fwd_dd_args(p, s.d_x, s.d_xt, vg, fc, cvd, s.d_order + o, c, s.d_ax, s.U + 1, s.Zi, 0, s.Zi, &r);
      if (fa.nvb < 1) continue;
      if (s.d_xt) {
        if (col_of[si] < 0) {
          col_of[si] = (int)cargs.size();
          cargs.push_back(ColArgs{s.d_x, s.d_xt, s.XN, s.YN, s.Zi});
        }
        for (int y = 0; y < (s.YN + 31) / 32; ++y)
          for (int x = 0; x < (s.XN + 31) / 32; ++x) cols[{0, 0}].push_back(make_int4(col_of[si], x, y, 0));
      }
      const int fi = (int)fargs.size();
      fargs.push_back(fa);
      const int ncb = dd_fwd_cblocks(fa);
      // z-tiles outermost and the rest in the single-solve grid's
      // order: the CTAs in flight share one tile's slices, whose image part
      // then stays in L2
      auto& fl = fwd[{fa.sv, fa.thin}];
      for (int zt = 0; zt < fa.nzt; ++zt)
        for (int cb = 0; cb < ncb; ++cb)
          for (int row = 0; row < c; ++row) fl.push_back(make_int4(fi, row, cb, zt));
      BackEpi e{};
      e.out = s.d_x; e.xin = s.d_x; e.colsum = s.d_cols + (size_t)k * s.XN * s.YN;
      e.nonneg = s.nonneg; e.mask = p.has_mask ? p.d_mask : nullptr; e.zlo = 0; e.zhi = s.Zi;
      int rc = check_back_dd(p, s.back_mode);
      if (rc) return rc;
      const DdBackArgs ba = make_back_dd_args(p, s.back_mode, s.d_ax, vg, c, e);
      const int bi = (int)bargs.size();
      bargs.push_back(ba);
      const int tiles = dd_back_tiles(ba);
      auto& lb = (adj ? back_adj : back_ref)[{ba.sv, ba.thin}];
      for (int zt = 0; zt < ba.nzt; ++zt)
        for (int t = 0; t < tiles; ++t) lb.push_back(make_int4(bi, t, zt, 0));
    }
    auto emit = [&](int kind, std::map<std::pair<int, int>, std::vector<int4>>& m) {
      for (auto& kv : m) {
        if (kv.second.empty()) continue;
        BatchLaunch L{kind, kv.first.first, kv.first.second, items.size(), kv.second.size(), grp};
        items.insert(items.end(), kv.second.begin(), kv.second.end());
        b.launches.push_back(L);
      }
    };
    emit(BK_COL, cols);
    emit(BK_FWD, fwd);
    emit(BK_ADJ, back_adj);
    emit(BK_REF, back_ref);
  }
  for (const BatchLaunch& L : b.launches)
    if (L.nitems > (size_t)INT_MAX) return set_err(DDFAN_ERR_UNSUPPORTED, "batch: %zu CTAs in one launch", L.nitems);
  std::vector<FistaDesc> fista;
  for (Solver* s : b.sv)
    if (s->useFISTA) {
      const size_t V = (size_t)s->XN * s->YN * s->Zi;
      fista.push_back(FistaDesc{s->d_x, s->d_xprev, V, s->d_t});
      b.fista_max = std::max(b.fista_max, V);
    }
  b.nfista = (int)fista.size();
  b.kernel_launches = (int)b.launches.size() + (b.nfista ? 2 : 0);
  cudaError_t e = cudaStreamCreateWithFlags(&b.own, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b.last_use, cudaEventDisableTiming);
  if (b.groups > 1) {
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b.fork, cudaEventDisableTiming);
    for (int t = 1; t < b.groups && e == cudaSuccess; ++t) {
      cudaStream_t q = nullptr;
      cudaEvent_t ev = nullptr;
      e = cudaStreamCreateWithFlags(&q, cudaStreamNonBlocking);
      if (e == cudaSuccess) b.side.push_back(q);
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
      if (e == cudaSuccess) b.join.push_back(ev);
    }
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return set_err(DDFAN_ERR_CUDA, "batch: stream/event creation: %s", cudaGetErrorString(e));
  }
  int rc;
  auto up = [&](auto** dst, auto& vec) -> int {
    if (vec.empty()) return DDFAN_OK;
    const size_t bytes = sizeof(vec[0]) * vec.size();
    int r = dev_alloc((void**)dst, bytes, b.own);
    if (r) return r;
    cudaError_t ee = cudaMemcpyAsync(*dst, vec.data(), bytes, cudaMemcpyHostToDevice, b.own);
    if (ee != cudaSuccess) return set_err(DDFAN_ERR_CUDA, "batch: upload: %s", cudaGetErrorString(ee));
    return DDFAN_OK;
  };
  if ((rc = up(&b.d_fargs, fargs)) || (rc = up(&b.d_bargs, bargs)) || (rc = up(&b.d_cargs, cargs)) ||
      (rc = up(&b.d_items, items)) || (rc = up(&b.d_fista, fista)))
    return rc;
  // the pageable sources above are consumed before they go out of scope
  e = cudaStreamSynchronize(b.own);
  if (e != cudaSuccess) return set_err(DDFAN_ERR_CUDA, "batch: upload: %s", cudaGetErrorString(e));
  *out = B.release();
  return DDFAN_OK;
}

}  // namespace ddfan

using namespace ddfan;

extern "C" {

DDFAN_API int ddfan_batch_create(ddfan_batch** out, ddfan_ossart* const* solvers, int n) {
  if (!out) return set_err(DDFAN_ERR_ARG, "out is null");
  Batch* b = nullptr;
  int rc = batch_create(&b, reinterpret_cast<Solver* const*>(solvers), n);
  *out = reinterpret_cast<ddfan_batch*>(b);
  return rc;
}

DDFAN_API void ddfan_batch_destroy(ddfan_batch* b) { batch_free(reinterpret_cast<Batch*>(b)); }

DDFAN_API int ddfan_batch_launches_per_iter(const ddfan_batch* h) {
  const Batch* b = reinterpret_cast<const Batch*>(h);
  return b ? b->kernel_launches : 0;
}

DDFAN_API int ddfan_batch_iterate(ddfan_batch* h, int numOfIter, int use_graph, void* stream) {
  Batch* b = reinterpret_cast<Batch*>(h);
  if (!b || numOfIter < 0) return set_err(DDFAN_ERR_ARG, "batch_iterate: bad argument");
  DeviceGuard g(b->device);
  cudaStream_t st = (cudaStream_t)stream;
  int rc;
  if (!use_graph) {
    for (int it = 0; it < numOfIter; ++it)
      if ((rc = batch_iteration(*b, st))) return rc;
  } else {
    if (!b->gexec) {
      cudaError_t e = cudaStreamBeginCapture(b->own, cudaStreamCaptureModeThreadLocal);
      if (e != cudaSuccess) return set_err(DDFAN_ERR_CUDA, "batch capture: %s", cudaGetErrorString(e));
      rc = batch_iteration(*b, b->own);
      cudaGraph_t gr = nullptr;
      e = cudaStreamEndCapture(b->own, &gr);
      if (rc) {
        if (gr) cudaGraphDestroy(gr);
        return rc;
      }
      if (e != cudaSuccess) return set_err(DDFAN_ERR_CUDA, "batch capture: %s", cudaGetErrorString(e));
      b->graph = gr;
      e = cudaGraphInstantiate(&b->gexec, b->graph, 0);
      if (e != cudaSuccess) return set_err(DDFAN_ERR_CUDA, "batch graph: %s", cudaGetErrorString(e));
    }
    for (int it = 0; it < numOfIter; ++it) {
      cudaError_t e = cudaGraphLaunch(b->gexec, st);
      if (e != cudaSuccess) return set_err(DDFAN_ERR_CUDA, "batch graph launch: %s", cudaGetErrorString(e));
    }
  }
  for (Solver* s : b->sv)
    if ((rc = solver_after_iterations(*s, numOfIter, st))) return rc;
  cudaEventRecord(b->last_use, st);
  return DDFAN_OK;
}

}  // extern "C"

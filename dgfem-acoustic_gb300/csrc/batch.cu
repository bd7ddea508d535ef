// Batched ensemble of independent solver instances (dg_batch_* in
// include/dgfem_gb300.h). No counterpart in the reference, which runs one
// case per process. Here hundreds of
// independent LEE runs (different meshes, orders, sources, mean flows and time
// steps) advanced together so that the GPU is filled even when each instance
// is small.
//
// Instances of one element type (dim, order) are concatenated into one
// disjoint-union mesh and solved by one context whose geometry records carry
// each element's own mean flow and time step. The contexts run their source
// injection, four RK4 stages and observer reductions on their own streams as
// parallel branches of one CUDA graph, eight steps long where the run is.
// Optionally, for 2-D FP32 instances of orders 2-4, every RK stage of all
// instances is one persistent launch of the mixed-order stage kernel
// (stage_multi.cuh), whose blocks take tiles of every order from a work queue.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <exception>
#include <string>
#include <thread>
#include <vector>

#include "bb.cuh"
#include "ctx.h"
#include "dg_internal.cuh"

namespace dgc {
int create_ctx(const dg_mesh_desc* mesh, const dg_phys* phys, int precision, int device, const double* elem_v0,
               const double* elem_scale, dg_ctx** out, std::string* err);
cudaError_t enqueue_step(dg_ctx* c, double dt, bool follows);
bool chained(const dg_ctx* c);
cudaError_t enqueue_inject(dg_ctx* c);
cudaError_t enqueue_finalize(dg_ctx* c, int nparts);
dgk::StageArgs<float> stage_args_f32(dg_ctx* c, int stage, const float* y_in, float* y_out, double dt);
int set_state_elems(dg_ctx* c, const double* u, int64_t e0, int64_t e1);
int ensure_out_cap(dg_ctx* c, int64_t n);
void set_global_error(const std::string& m);
}  // namespace dgc

struct dg_batch {
  struct Group {
    dg_ctx* ctx = nullptr;
    int dim = 0, order = 0, np = 0;
    std::vector<int> inst;            // member instances in order
    // reference-layout staging [4][N], page-locked where that memory can be had:
    // the copy of the whole group runs at the link's rate
    double* state = nullptr;
    int64_t N = 0;
    bool pinned = false;
    bool state_dirty = false, state_valid = false;
    int own_variant = -2;             // kernel selected before one launch per stage took its layout (-2: none)
    cudaEvent_t join = nullptr;
  };
  std::vector<Group> groups;
  std::vector<int> inst_group;
  std::vector<int64_t> inst_elem_off, inst_E;
  std::vector<char> inst_dirty;  // its part of the staging is to go to the device
  // per-instance sources and observers (instance-local dofs)
  struct Src {
    std::vector<int64_t> off{0}, dofs;
    int n = 0;
    int64_t steps = 0;
    std::vector<double> values;  // [steps][n]
  };
  struct Obs {
    std::vector<int64_t> off{0}, dofs;
    std::vector<double> w;
    int n = 0;
  };
  std::vector<Src> src;
  std::vector<Obs> obs;
  bool sources_dirty = true, observers_dirty = true;
  cudaStream_t main = nullptr;
  cudaEvent_t fork = nullptr;
  cudaGraphExec_t graph = nullptr, graph_n = nullptr;  // one step, kBatchSteps steps
  bool chain = false;  // the graphs' steps end with the next step's sources where a group allows it
  // one launch per RK stage for all element orders (2-D FP32, orders 2-4):
  // slot k -> group holding order k + 2 (or -1), the four stages' work-queue
  // counters, the launch's grid
  bool fused_ok = false, fused = false;
  int slot_group[dgk::kMultiOrders] = {-1, -1, -1};
  unsigned* d_queue = nullptr;
  int fused_grid = 0;
  int64_t step = 0, total_dofs = 0;
  std::string err;
};

namespace {

int fail(dg_batch* b, int code, const std::string& m) {
  if (b) b->err = m;
  return code;
}

#define BCK(b, x)                                                                                \
  do {                                                                                           \
    cudaError_t e_ = (x);                                                                        \
    if (e_ != cudaSuccess) return fail((b), DG_ERR_CUDA, std::string("CUDA: ") + cudaGetErrorString(e_)); \
  } while (0)

void drop_graphs(dg_batch* b) {
  if (b->graph) cudaGraphExecDestroy(b->graph), b->graph = nullptr;
  if (b->graph_n) cudaGraphExecDestroy(b->graph_n), b->graph_n = nullptr;
}

// The four variables' planes of n values, by a thread each where they are large:
// a fresh array of the caller's costs as much in page faults as in copying.
void copy_planes(double* dst, int64_t dst_stride, const double* src, int64_t src_stride, int64_t n) {
  auto plane = [=](int q) { std::memcpy(dst + q * dst_stride, src + q * src_stride, n * sizeof(double)); };
  std::thread t[3];
  for (int q = 0; q < 3; ++q) {
    if (n >= 1 << 15) {
      try {
        t[q] = std::thread(plane, q);
        continue;
      } catch (const std::exception&) {  // no thread to be had
      }
    }
    plane(q);
  }
  plane(3);
  for (auto& x : t)
    if (x.joinable()) x.join();
}

// Pushes staged states, sources and observers to the group contexts.
int sync_inputs(dg_batch* b) {
  // (only what was set: after a run the staging of the other instances is old)
  for (auto& g : b->groups)
    if (g.state_dirty) {
      for (size_t j = 0; j < g.inst.size();) {
        size_t k = j;
        while (k < g.inst.size() && b->inst_dirty[g.inst[k]]) ++k;
        if (k > j) {
          const int64_t e0 = b->inst_elem_off[g.inst[j]];
          const int64_t e1 = b->inst_elem_off[g.inst[k - 1]] + b->inst_E[g.inst[k - 1]];
          const int rc = dgc::set_state_elems(g.ctx, g.state, e0, e1);
          if (rc) return fail(b, rc, dg_last_error(g.ctx));
        }
        j = k + 1;
      }
      for (int i : g.inst) b->inst_dirty[i] = 0;
      g.state_dirty = false;
    }
  if (b->sources_dirty) {
    for (auto& g : b->groups) {
      std::vector<int64_t> off{0}, dofs;
      int64_t steps = 0;
      int nsrc = 0;
      for (int i : g.inst) {
        steps = std::max(steps, b->src[i].steps);
        nsrc += b->src[i].n;
      }
      std::vector<double> vals(std::max<int64_t>(steps * nsrc, 1), std::nan(""));
      int col = 0;
      for (int i : g.inst) {
        const auto& s = b->src[i];
        const int64_t base = b->inst_elem_off[i] * g.np;
        for (int k = 0; k < s.n; ++k) {
          for (int64_t t = s.off[k]; t < s.off[k + 1]; ++t) dofs.push_back(base + s.dofs[t]);
          off.push_back((int64_t)dofs.size());
          for (int64_t st = 0; st < s.steps; ++st) vals[st * nsrc + col + k] = s.values[st * s.n + k];
        }
        col += s.n;
      }
      int rc = dg_set_sources(g.ctx, nsrc, off.data(), dofs.data());
      if (!rc) rc = dg_set_source_values(g.ctx, nsrc > 0 ? steps : 0, vals.data());
      if (rc) return fail(b, rc, dg_last_error(g.ctx));
    }
    b->sources_dirty = false;
    drop_graphs(b);
  }
  if (b->observers_dirty) {
    for (auto& g : b->groups) {
      std::vector<int64_t> off{0}, dofs;
      std::vector<double> w;
      int nobs = 0;
      for (int i : g.inst) {
        const auto& o = b->obs[i];
        const int64_t base = b->inst_elem_off[i] * g.np;
        for (int k = 0; k < o.n; ++k) {
          for (int64_t t = o.off[k]; t < o.off[k + 1]; ++t) dofs.push_back(base + o.dofs[t]), w.push_back(o.w[t]);
          off.push_back((int64_t)dofs.size());
        }
        nobs += o.n;
      }
      int rc = dg_set_observers(g.ctx, nobs, off.data(), dofs.data(), w.data());
      if (rc) return fail(b, rc, dg_last_error(g.ctx));
    }
    b->observers_dirty = false;
    drop_graphs(b);
  }
  return DG_OK;
}

// One graph per step with one launch per RK stage for every element order:
// queue counters reset, per-order source injection, the four mixed-order
// stage kernels, per-order residual and observer reductions (all on the
// batch's stream; the group contexts' work is enqueued there).
int build_fused_graph(dg_batch* b) {
  cudaGraph_t graph = nullptr;
  BCK(b, cudaStreamBeginCapture(b->main, cudaStreamCaptureModeThreadLocal));
  cudaError_t err = cudaMemsetAsync(b->d_queue, 0, 4 * sizeof(unsigned), b->main);
  std::vector<cudaStream_t> keep;
  for (auto& g : b->groups) keep.push_back(g.ctx->stream), g.ctx->stream = b->main;
  for (auto& g : b->groups)
    if (err == cudaSuccess) err = dgc::enqueue_inject(g.ctx);
  int* derr = nullptr;
  for (int st = 1; st <= 4 && err == cudaSuccess; ++st) {
    dgk::MultiArgs m{};
    m.ntiles_total = 0;
    m.queue = b->d_queue + (st - 1);
    m.wait_limit = dgk::kWaitRounds;
    for (int k = 0; k < dgk::kMultiOrders; ++k) {
      m.g[k].stage = st;
      m.g[k].ntiles = 0;
      if (b->slot_group[k] < 0) continue;
      dg_ctx* c = b->groups[b->slot_group[k]].ctx;
      const float* in[4] = {(const float*)c->u, (const float*)c->y0, (const float*)c->y1, (const float*)c->y0};
      float* out[4] = {(float*)c->y0, (float*)c->y1, (float*)c->y0, nullptr};
      // every instance's own dt sits in its elements' step scale
      m.g[k] = dgc::stage_args_f32(c, st, in[st - 1], out[st - 1], 1.0);
      m.g[k].ntiles = (int)(c->Epad / dgk::stage_multi_elems_per_tile(k + 2));
      m.ntiles_total += m.g[k].ntiles;
      if (!derr) derr = c->d_err;
    }
    err = dgk::launch_stage_multi(m, b->fused_grid, derr, b->main);
  }
  for (auto& g : b->groups)
    if (err == cudaSuccess) err = dgc::enqueue_finalize(g.ctx, b->fused_grid);
  for (size_t i = 0; i < b->groups.size(); ++i) b->groups[i].ctx->stream = keep[i];
  cudaError_t err2 = cudaStreamEndCapture(b->main, &graph);
  if (err != cudaSuccess) {
    if (graph) cudaGraphDestroy(graph);
    return fail(b, DG_ERR_CUDA, std::string("CUDA (capture): ") + cudaGetErrorString(err));
  }
  BCK(b, err2);
  err = cudaGraphInstantiate(&b->graph, graph, 0);
  cudaGraphDestroy(graph);
  BCK(b, err);
  return DG_OK;
}

// Steps of the longer graph.
constexpr int kBatchSteps = 8;

// A graph of `steps` steps, every group's as a parallel branch: the groups do not
// wait for one another between steps.
int build_order_graph(dg_batch* b, int steps) {
  cudaGraph_t graph = nullptr;
  BCK(b, cudaStreamBeginCapture(b->main, cudaStreamCaptureModeThreadLocal));
  cudaError_t err = cudaEventRecord(b->fork, b->main);
  for (auto& g : b->groups) {
    if (err == cudaSuccess) err = cudaStreamWaitEvent(g.ctx->stream, b->fork, 0);
    // every instance's own dt sits in its elements' step scale
    for (int i = 0; i < steps && err == cudaSuccess; ++i) err = dgc::enqueue_step(g.ctx, 1.0, i > 0);
    if (err == cudaSuccess) err = cudaEventRecord(g.join, g.ctx->stream);
    if (err == cudaSuccess) err = cudaStreamWaitEvent(b->main, g.join, 0);
  }
  cudaError_t err2 = cudaStreamEndCapture(b->main, &graph);
  if (err != cudaSuccess) return fail(b, DG_ERR_CUDA, std::string("CUDA (capture): ") + cudaGetErrorString(err));
  BCK(b, err2);
  err = cudaGraphInstantiate(steps == 1 ? &b->graph : &b->graph_n, graph, 0);
  cudaGraphDestroy(graph);
  BCK(b, err);
  return DG_OK;
}

int build_graph(dg_batch* b, int64_t n_steps) {
  // a run longer than any before gets new result buffers: the graphs hold the
  // old ones' addresses
  int rc = DG_OK;
  bool moved = false;
  for (auto& g : b->groups) {
    const int64_t cap = g.ctx->out_cap;
    if (!rc && (rc = dgc::ensure_out_cap(g.ctx, n_steps))) fail(b, rc, dg_last_error(g.ctx));
    moved |= rc || g.ctx->out_cap != cap;
  }
  if (moved) drop_graphs(b);
  if (rc) return rc;
  b->chain = !b->fused;
  if (b->fused) return b->graph ? DG_OK : build_fused_graph(b);
  if (n_steps >= kBatchSteps && !b->graph_n) rc = build_order_graph(b, kBatchSteps);
  if (!rc && n_steps % kBatchSteps && !b->graph) rc = build_order_graph(b, 1);
  return rc;
}

// One launch per stage works on Bernstein coefficients: a group whose kernel
// was forced to another layout (DGFEM_STAGE_VARIANT) takes them with it and
// its own kernel back without it.
int group_layouts(dg_batch* b) {
  for (auto& g : b->groups) {
    int rc = DG_OK;
    if (b->fused && !g.ctx->bb) {
      g.own_variant = g.ctx->variant;
      rc = dg_tune(g.ctx, dgk::kBBVariant);
    } else if (!b->fused && g.own_variant != -2) {
      rc = dg_tune(g.ctx, g.own_variant);
      g.own_variant = -2;
    }
    if (rc) return fail(b, rc, dg_last_error(g.ctx));
  }
  return DG_OK;
}

int launch_steps(dg_batch* b, int64_t n_steps) {
  for (auto& g : b->groups) {
    int64_t st[3] = {b->step, b->step, b->step + n_steps};
    BCK(b, cudaMemcpyAsync(g.ctx->d_step, st, sizeof(st), cudaMemcpyHostToDevice, b->main));
  }
  for (auto& g : b->groups)
    if (b->chain && dgc::chained(g.ctx)) {
      cudaStream_t own = g.ctx->stream;
      g.ctx->stream = b->main;
      cudaError_t e = dgc::enqueue_inject(g.ctx);
      g.ctx->stream = own;
      BCK(b, e);
    }
  const int64_t many = b->fused ? 0 : n_steps / kBatchSteps;
  for (int64_t i = 0; i < many; ++i) BCK(b, cudaGraphLaunch(b->graph_n, b->main));
  for (int64_t i = many * kBatchSteps; i < n_steps; ++i) BCK(b, cudaGraphLaunch(b->graph, b->main));
  return DG_OK;
}

}  // namespace

extern "C" {

const char* dg_batch_last_error(const dg_batch* b) { return b ? b->err.c_str() : dg_last_error(nullptr); }

int dg_batch_create(int n, const dg_mesh_desc* meshes, const dg_phys* phys, const double* dts, int precision,
                    int device, dg_batch** out) {
  if (!out || n <= 0 || !meshes || !phys || !dts) {
    dgc::set_global_error("dg_batch_create: invalid argument");
    return DG_ERR_ARG;
  }
  *out = nullptr;
  for (int i = 1; i < n; ++i)
    if (phys[i].rho0 != phys[0].rho0 || phys[i].c0 != phys[0].c0) {
      dgc::set_global_error("dg_batch_create: all instances must share rho0 and c0");
      return DG_ERR_ARG;
    }
  for (int i = 0; i < n; ++i)
    if (!(dts[i] > 0)) {
      dgc::set_global_error("dg_batch_create: time steps must be positive");
      return DG_ERR_ARG;
    }
  auto* b = new dg_batch;
  b->inst_group.assign(n, -1);
  b->inst_elem_off.assign(n, 0);
  b->inst_E.assign(n, 0);
  b->inst_dirty.assign(n, 0);
  b->src.assign(n, {});
  b->obs.assign(n, {});
  std::map<std::pair<int, int>, int> gid;
  for (int i = 0; i < n; ++i) {
    auto key = std::make_pair(meshes[i].dim, meshes[i].order);
    if (!gid.count(key)) {
      gid[key] = (int)b->groups.size();
      b->groups.emplace_back();
      b->groups.back().dim = key.first, b->groups.back().order = key.second;
      b->groups.back().np = meshes[i].nodes_per_elem;
    }
    b->inst_group[i] = gid[key];
    b->groups[gid[key]].inst.push_back(i);
  }
  auto bail = [&](int code, const std::string& m) {
    dgc::set_global_error("dg_batch_create: " + m);
    dg_batch_destroy(b);
    return code;
  };
  for (auto& g : b->groups) {
    // disjoint union of the member meshes
    std::vector<double> xyz, v0, scale;
    std::vector<int64_t> en, goff{0}, gnodes;
    std::vector<int> gbc;
    const dg_mesh_desc& m0 = meshes[g.inst[0]];
    const int ngr = m0.n_groups;
    std::vector<std::vector<int64_t>> gn(ngr);
    int64_t node_off = 0, elem_off = 0;
    for (int i : g.inst) {
      const dg_mesh_desc& m = meshes[i];
      if (m.nodes_per_elem != g.np || m.n_groups != ngr) return bail(DG_ERR_ARG, "instances of one element type must have the same boundary group structure");
      for (int k = 0; k < ngr; ++k)
        if (m.group_bc[k] != m0.group_bc[k]) return bail(DG_ERR_ARG, "instances of one element type must use the same BC per group");
      xyz.insert(xyz.end(), m.xyz, m.xyz + 3 * m.n_nodes);
      for (int64_t k = 0; k < m.n_elems * g.np; ++k) en.push_back(m.elem_nodes[k] + node_off);
      for (int k = 0; k < ngr; ++k)
        for (int64_t t = m.group_offsets[k]; t < m.group_offsets[k + 1]; ++t) gn[k].push_back(m.group_nodes[t] + node_off);
      for (int64_t e = 0; e < m.n_elems; ++e) {
        for (int d = 0; d < 3; ++d) v0.push_back(phys[i].v0[d]);
        scale.push_back(dts[i]);
      }
      b->inst_elem_off[i] = elem_off;
      b->inst_E[i] = m.n_elems;
      node_off += m.n_nodes;
      elem_off += m.n_elems;
    }
    for (int k = 0; k < ngr; ++k) {
      gbc.push_back(m0.group_bc[k]);
      gnodes.insert(gnodes.end(), gn[k].begin(), gn[k].end());
      goff.push_back((int64_t)gnodes.size());
    }
    dg_mesh_desc md = m0;
    md.n_nodes = node_off, md.xyz = xyz.data(), md.n_elems = elem_off, md.elem_nodes = en.data();
    md.n_groups = ngr, md.group_bc = gbc.data(), md.group_offsets = goff.data(), md.group_nodes = gnodes.data();
    dg_phys ph = phys[g.inst[0]];
    std::string e;
    int rc = dgc::create_ctx(&md, &ph, precision, device, v0.data(), scale.data(), &g.ctx, &e);
    if (rc) return bail(rc, e);
    g.N = elem_off * g.np;
    g.pinned = cudaMallocHost((void**)&g.state, 4 * g.N * sizeof(double)) == cudaSuccess;
    if (!g.pinned) {
      cudaGetLastError();
      g.state = (double*)std::malloc(4 * g.N * sizeof(double));
      if (!g.state) return bail(DG_ERR_CUDA, "host memory for the state");
    }
    std::memset(g.state, 0, 4 * g.N * sizeof(double));
    b->total_dofs += elem_off * g.np * (g.dim + 1);
    if (cudaEventCreateWithFlags(&g.join, cudaEventDisableTiming) != cudaSuccess) return bail(DG_ERR_CUDA, "event");
  }
  if (cudaStreamCreateWithFlags(&b->main, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming) != cudaSuccess)
    return bail(DG_ERR_CUDA, "stream/event creation failed");
  // one launch per stage for all orders: 2-D FP32 instances of orders 2-4
  b->fused_ok = precision == DG_FP32;
  for (size_t k = 0; k < b->groups.size(); ++k) {
    const auto& g = b->groups[k];
    if (g.dim != 2 || g.order < 2 || g.order > 4 || !dgc::bb_mesh(g.ctx))
      b->fused_ok = false;
    else
      b->slot_group[g.order - 2] = (int)k;
  }
  if (b->fused_ok) {
    const int bps = dgk::stage_multi_blocks_per_sm();
    int64_t tiles = 0;
    int cap = 1 << 30;
    for (auto& g : b->groups) {
      tiles += g.ctx->Epad / dgk::stage_multi_elems_per_tile(g.order);
      cap = std::min(cap, g.ctx->max_grid);  // rows of every order's partial-sum array
    }
    b->fused_grid = (int)std::min<int64_t>(std::min<int64_t>(tiles, (int64_t)bps * b->groups[0].ctx->num_sms), cap);
    if (bps <= 0 || b->fused_grid <= 0 || cudaMalloc(&b->d_queue, 4 * sizeof(unsigned)) != cudaSuccess) {
      cudaGetLastError();
      b->fused_ok = false;
    }
  }
  // One launch per stage only by choice (DGFEM_BATCH_FUSED=1 or
  // dg_batch_set_fused(b, 1)): it runs every order at the registers and shared
  // memory of the largest, and all orders wait for one another at every stage.
  // us per step, one launch -> branches: 2 instances (0.12M unknowns) 39 -> 18,
  // 16 (2.3M) 100 -> 40, 48 (28M) 450 -> 353.
  const char* ev = std::getenv("DGFEM_BATCH_FUSED");
  b->fused = b->fused_ok && ev && std::strcmp(ev, "1") == 0;
  if (group_layouts(b) != DG_OK) return bail(DG_ERR_CUDA, b->err);
  *out = b;
  return DG_OK;
}

int dg_batch_destroy(dg_batch* b) {
  if (!b) return DG_OK;
  drop_graphs(b);
  for (auto& g : b->groups) {
    if (g.join) cudaEventDestroy(g.join);
    if (g.ctx) dg_destroy(g.ctx);
    if (g.pinned) cudaFreeHost(g.state);
    else std::free(g.state);
  }
  if (b->fork) cudaEventDestroy(b->fork);
  if (b->main) cudaStreamDestroy(b->main);
  if (b->d_queue) cudaFree(b->d_queue);
  delete b;
  return DG_OK;
}

int dg_batch_set_fused(dg_batch* b, int on) {
  if (!b) return DG_ERR_ARG;
  if (on && !b->fused_ok)
    return fail(b, DG_ERR_ARG, "one launch per stage needs FP32 2-D straight-sided instances of orders 2-4 only");
  if (b->fused != (on != 0)) {
    b->fused = on != 0;
    drop_graphs(b);
    return group_layouts(b);
  }
  return DG_OK;
}

int dg_batch_fused(const dg_batch* b) { return b && b->fused ? 1 : 0; }

int dg_batch_info(const dg_batch* b, int* n_groups, int64_t* total_dofs) {
  if (!b) return DG_ERR_ARG;
  if (n_groups) *n_groups = (int)b->groups.size();
  if (total_dofs) *total_dofs = b->total_dofs;
  return DG_OK;
}

int dg_batch_set_state(dg_batch* b, int inst, const double* u) {
  if (!b || !u || inst < 0 || inst >= (int)b->inst_group.size()) return DG_ERR_ARG;
  auto& g = b->groups[b->inst_group[inst]];
  const int64_t n = b->inst_E[inst] * g.np, off = b->inst_elem_off[inst] * g.np;
  copy_planes(g.state + off, g.N, u, n, n);
  b->inst_dirty[inst] = 1;
  g.state_dirty = true;
  return DG_OK;
}

int dg_batch_get_state(dg_batch* b, int inst, double* u) {
  if (!b || !u || inst < 0 || inst >= (int)b->inst_group.size()) return DG_ERR_ARG;
  int rc = sync_inputs(b);
  if (rc) return rc;
  auto& g = b->groups[b->inst_group[inst]];
  const int64_t n = b->inst_E[inst] * g.np, off = b->inst_elem_off[inst] * g.np;
  if (!g.state_valid) {
    rc = dg_get_state(g.ctx, g.state);
    if (rc) return fail(b, rc, dg_last_error(g.ctx));
    g.state_valid = true;
  }
  copy_planes(u, n, g.state + off, g.N, n);
  return DG_OK;
}

int dg_batch_set_sources(dg_batch* b, int inst, int n_src, const int64_t* offsets, const int64_t* dofs,
                         int64_t n_steps, const double* values) {
  if (!b || inst < 0 || inst >= (int)b->inst_group.size() || n_src < 0 || n_steps < 0) return DG_ERR_ARG;
  auto& s = b->src[inst];
  const int64_t nd = b->inst_E[inst] * b->groups[b->inst_group[inst]].np;
  s.n = n_src;
  s.steps = n_src > 0 ? n_steps : 0;
  s.off.assign(offsets, offsets + n_src + 1);
  s.dofs.assign(dofs, dofs + (n_src > 0 ? offsets[n_src] : 0));
  for (auto d : s.dofs)
    if (d < 0 || d >= nd) return fail(b, DG_ERR_ARG, "source dof out of range");
  s.values.assign(values, values + s.steps * n_src);
  b->sources_dirty = true;
  return DG_OK;
}

int dg_batch_set_observers(dg_batch* b, int inst, int n_obs, const int64_t* offsets, const int64_t* dofs,
                           const double* weights) {
  if (!b || inst < 0 || inst >= (int)b->inst_group.size() || n_obs < 0) return DG_ERR_ARG;
  auto& o = b->obs[inst];
  const int64_t nd = b->inst_E[inst] * b->groups[b->inst_group[inst]].np;
  o.n = n_obs;
  o.off.assign(offsets, offsets + n_obs + 1);
  int64_t tot = n_obs > 0 ? offsets[n_obs] : 0;
  o.dofs.assign(dofs, dofs + tot);
  o.w.assign(weights, weights + tot);
  for (auto d : o.dofs)
    if (d < 0 || d >= nd) return fail(b, DG_ERR_ARG, "observer dof out of range");
  b->observers_dirty = true;
  return DG_OK;
}

int dg_batch_run(dg_batch* b, int64_t n_steps, double* obs) {
  if (!b || n_steps < 0) return DG_ERR_ARG;
  if (n_steps == 0) return DG_OK;
  int rc = sync_inputs(b);
  if (!rc) rc = build_graph(b, n_steps);
  if (!rc) rc = launch_steps(b, n_steps);
  if (rc) return rc;
  BCK(b, cudaStreamSynchronize(b->main));
  b->step += n_steps;
  for (auto& g : b->groups) {
    g.state_valid = false;
    g.ctx->step = b->step;
  }
  if (obs) {
    // per instance, in instance order: [n_steps][n_obs_i][4]
    std::vector<int64_t> inst_out(b->inst_group.size(), 0);
    int64_t acc = 0;
    for (size_t i = 0; i < b->inst_group.size(); ++i) inst_out[i] = acc, acc += n_steps * b->obs[i].n * 4;
    for (auto& g : b->groups) {
      int nobs = g.ctx->n_obs;
      if (nobs == 0) continue;
      std::vector<double> h(n_steps * nobs * 4);
      BCK(b, cudaMemcpy(h.data(), g.ctx->d_obs, h.size() * sizeof(double), cudaMemcpyDeviceToHost));
      int col = 0;
      for (int i : g.inst) {
        const int ni = b->obs[i].n;
        for (int64_t s = 0; s < n_steps; ++s)
          for (int k = 0; k < ni; ++k)
            for (int c = 0; c < 4; ++c) obs[inst_out[i] + (s * ni + k) * 4 + c] = h[(s * nobs + col + k) * 4 + c];
        col += ni;
      }
    }
  }
  int herr = 0;
  for (auto& g : b->groups) {
    BCK(b, cudaMemcpy(&herr, g.ctx->d_err, sizeof(int), cudaMemcpyDeviceToHost));
    if (herr) {
      BCK(b, cudaMemset(g.ctx->d_err, 0, sizeof(int)));  // the batch stays usable
      return fail(b, DG_ERR_TIMEOUT, "a bounded device wait gave up");
    }
  }
  return DG_OK;
}

int dg_batch_bench(dg_batch* b, int64_t n_steps, double* step_ms) {
  if (!b || n_steps <= 0) return DG_ERR_ARG;
  int rc = sync_inputs(b);
  if (!rc) rc = build_graph(b, n_steps);
  if (rc) return rc;
  cudaEvent_t ev[2];
  for (auto& e : ev) cudaEventCreate(&e);
  cudaEventRecord(ev[0], b->main);
  rc = launch_steps(b, n_steps);
  cudaEventRecord(ev[1], b->main);
  if (!rc && cudaStreamSynchronize(b->main) != cudaSuccess) rc = fail(b, DG_ERR_CUDA, "synchronize failed");
  float tot = 0.f;
  if (!rc) cudaEventElapsedTime(&tot, ev[0], ev[1]);
  for (auto& e : ev) cudaEventDestroy(e);
  if (rc) return rc;
  b->step += n_steps;
  for (auto& g : b->groups) g.state_valid = false, g.ctx->step = b->step;
  if (step_ms) *step_ms = (double)tot / n_steps;
  return DG_OK;
}

}  // extern "C"

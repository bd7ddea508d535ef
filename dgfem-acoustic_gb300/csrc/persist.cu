// Host side of the many-steps kernel (stage_persist.cuh): lists of sources and
// observers by tile, buffers, and the launches of a run.
#include <algorithm>
#include <map>
#include <vector>

#include "bb.cuh"
#include "stage_persist.cuh"

namespace dgk {

// Per step s (blockIdx.x): the residual means from the tiles' sums (blockIdx.y
// 0) and observer blockIdx.y - 1's sample from its (tile, observer) sums, each
// in a fixed order; once per launch of the steps.
constexpr int kSumThreads = 128;
__global__ void __launch_bounds__(kSumThreads)
    k_persist_sums(const double* partials, int ntiles, int nv, double inv_count, double c0sq, double* res,
                   const double* gsum, int groups, const int* obs_first, const int* obs_grp, const double* obs_w,
                   double* obs, int n_obs) {
  __shared__ double red[4][kSumThreads];
  const int64_t s = blockIdx.x;
  const int tid = threadIdx.x;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  if (blockIdx.y == 0) {
    for (int t = tid; t < ntiles; t += kSumThreads)
      for (int q = 0; q < nv; ++q) acc[q] += partials[(s * ntiles + t) * nv + q];
  } else {
    const int o = blockIdx.y - 1;
    for (int k = obs_first[o] + tid; k < obs_first[o + 1]; k += kSumThreads)
      for (int q = 0; q < nv; ++q) acc[q] += gsum[(s * groups + obs_grp[k]) * 4 + q];
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) red[q][tid] = acc[q];
  __syncthreads();
  for (int h = kSumThreads / 2; h > 0; h >>= 1) {
    if (tid < h)
#pragma unroll
      for (int q = 0; q < 4; ++q) red[q][tid] += red[q][tid + h];
    __syncthreads();
  }
  if (blockIdx.y == 0) {
    if (tid < 5) {  // p, p / c0^2, vx, vy, vz
      const double v = red[tid < 2 ? 0 : tid - 1][0];
      res[s * 5 + tid] = (tid == 1 ? v / (c0sq * c0sq) : v) * inv_count;
    }
  } else if (tid < 4) {
    obs[(s * n_obs + blockIdx.y - 1) * 4 + tid] = red[tid][0] / obs_w[blockIdx.y - 1];
  }
}

}  // namespace dgk

namespace dgc {

// Steps per launch: the launch, the tiles' first loads and the sums (about 20 us)
// are spread over them, and the tiles' sums of all of them are kept.
constexpr int kPersistSteps = 64;
constexpr size_t kPersistSums = (size_t)64 << 20;  // bytes of sums, at most (one step's at least)

bool persist_fits(const dg_ctx* c) {
  return c->prec == DG_FP64 && c->Epad / 32 <= (int64_t)dgk::persist_info(c->dim, c->order).blocks_per_sm * c->num_sms;
}

// At order 3 in 3-D the two tiles that an SM holds hold each other up. us per step
// against one launch per stage: 95 / 100 up to a tile per SM, 118 / 124 at 1.1, 129 /
// 125 at 1.2, 144 / 127 at 1.5, 166 / 128 at 1.8. The others pay at every size.
bool persist_pays(const dg_ctx* c) { return !(c->dim == 3 && c->order == 3) || c->Epad / 32 <= c->num_sms; }

namespace {

void free_lists(dg_ctx* c) {
  dg_ctx::Persist& p = c->persist;
  for (void* x : {(void*)p.ints, (void*)p.weights, (void*)p.partials, (void*)p.gsum})
    if (x) cudaFree(x);
  const dg_ctx::Persist old = p;
  p = dg_ctx::Persist();
  p.inputs = old.inputs, p.seq = old.seq;
}

template <typename T>
bool upload(T** dst, const std::vector<T>& v, cudaStream_t s) {
  return cudaMalloc((void**)dst, std::max<size_t>(v.size(), 1) * sizeof(T)) == cudaSuccess &&
         (v.empty() || cudaMemcpyAsync(*dst, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s) == cudaSuccess);
}

bool build(dg_ctx* c) {
  dg_ctx::Persist& p = c->persist;
  const int nt = (int)(c->Epad / 32), n_obs = c->n_obs;
  const int64_t tw = (int64_t)c->nv * c->np * 32;
  // source elements and node slots of each tile (both ascend)
  std::vector<int> sel(nt + 1, 0), el, snode(nt + 1, 0), node;
  for (int64_t e : c->src_elems) ++sel[(e >> 5) + 1], el.push_back((int)(e & 31));
  for (int64_t d : c->src_dof) {
    const int64_t e = d / c->np;
    ++snode[(e >> 5) + 1];
    node.push_back((int)(e & 31) | (int)(d - e * c->np) << 8);
  }
  for (int t = 0; t < nt; ++t) sel[t + 1] += sel[t], snode[t + 1] += snode[t];
  // the observers' entries by tile
  std::map<std::pair<int, int>, std::vector<int64_t>> by_tile;
  std::vector<double> ow(n_obs, 0.0);
  for (int o = 0; o < n_obs; ++o)
    for (int64_t k = c->obs_bb_off[o]; k < c->obs_bb_off[o + 1]; ++k) {
      by_tile[{(int)(c->obs_bb_slot[k] / tw), o}].push_back(k);
      ow[o] += c->obs_bb_w[k];
    }
  std::vector<int> grp(nt + 1, 0), ent(1, 0), word, ofirst(n_obs + 1, 0), ogrp;
  std::vector<double> w;
  std::vector<std::vector<int>> of(n_obs);
  for (auto& kv : by_tile) {
    ++grp[kv.first.first + 1];
    of[kv.first.second].push_back((int)ent.size() - 1);
    for (int64_t k : kv.second) word.push_back((int)(c->obs_bb_slot[k] % tw)), w.push_back(c->obs_bb_w[k]);
    ent.push_back((int)word.size());
  }
  for (int t = 0; t < nt; ++t) grp[t + 1] += grp[t];
  for (int o = 0; o < n_obs; ++o) {
    ogrp.insert(ogrp.end(), of[o].begin(), of[o].end());
    ofirst[o + 1] = (int)ogrp.size();
  }
  p.groups = (int)by_tile.size();
  const size_t part = (size_t)nt * c->nv * sizeof(double), gs = (size_t)p.groups * 4 * sizeof(double);
  p.steps = (int)std::min<size_t>(kPersistSteps, std::max<size_t>(1, kPersistSums / (part + gs)));
  std::vector<int> ints;
  std::vector<size_t> at;
  for (const std::vector<int>* v : {&sel, &el, &snode, &node, &grp, &ent, &word, &ofirst, &ogrp}) {
    at.push_back(ints.size());
    ints.insert(ints.end(), v->begin(), v->end());
  }
  const size_t n_ent = w.size();
  w.insert(w.end(), ow.begin(), ow.end());
  if (!upload(&p.ints, ints, c->stream) || !upload(&p.weights, w, c->stream)) return false;
  if (cudaMalloc((void**)&p.partials, p.steps * part) != cudaSuccess) return false;
  if (gs > 0 && cudaMalloc((void**)&p.gsum, p.steps * gs) != cudaSuccess) return false;
  int** list[9] = {&p.sel_first, &p.sel,      &p.snode_first, &p.snode,  &p.grp_first,
                   &p.ent_first, &p.ent_word, &p.obs_first,   &p.obs_grp};
  for (int i = 0; i < 9; ++i) *list[i] = p.ints + at[i];
  p.obs_w = p.weights + n_ent;
  if (!p.inputs) {
    const size_t bytes = 2 * (size_t)nt * tw * sizeof(dgk::Tagged::W);
    if (cudaMalloc(&p.inputs, bytes) != cudaSuccess) return false;
    if (cudaMemsetAsync(p.inputs, 0, bytes, c->stream) != cudaSuccess) return false;
    p.seq = 1;
  }
  return cudaStreamSynchronize(c->stream) == cudaSuccess;
}

}  // namespace

void persist_free(dg_ctx* c) {
  free_lists(c);
  if (c->persist.inputs) cudaFree(c->persist.inputs);
  c->persist = dg_ctx::Persist();
}

bool persist_ready(dg_ctx* c) {
  if (!c->persist.stale) return true;
  cudaStreamSynchronize(c->stream);
  free_lists(c);
  // gridDim.y of the sums
  if (c->n_obs > 65000 || !build(c)) {
    cudaGetLastError();
    persist_free(c);
    return false;
  }
  c->persist.stale = false;
  return true;
}

cudaError_t persist_run(dg_ctx* c, int64_t n_steps, double dt, int64_t* launched) {
  dg_ctx::Persist& d = c->persist;
  const int nt = (int)(c->Epad / 32);
  const int64_t words = (int64_t)nt * c->nv * c->np * 32;
  dgk::PersistArgs p{};
  p.a = stage_args_f64(c, 0, nullptr, nullptr, dt);
  p.buf[0] = (dgk::Tagged::W*)d.inputs, p.buf[1] = p.buf[0] + words;
  p.E = c->E;
  p.sel_first = d.sel_first, p.sel = d.sel, p.snode_first = d.snode_first, p.snode = d.snode;
  p.soff = c->d_src_off, p.sids = c->d_src_ids, p.sval = c->d_srcval;
  p.nsrc = c->n_src_elems > 0 && c->srcval_steps > 0 ? c->n_src : 0, p.nrows = c->srcval_steps;
  p.Vt = c->bb_dbl + c->bb_iden[0], p.Vit = c->bb_dbl + c->bb_iden[1];
  p.grp_first = d.grp_first, p.ent_first = d.ent_first, p.ent_word = d.ent_word;
  p.ent_w = d.weights, p.groups = d.groups, p.gsum = d.gsum, p.partials = d.partials;
  const double inv_count = 1.0 / (double)(c->E * c->np);
  for (int64_t done = 0; done < n_steps; done += p.steps) {
    p.steps = (int)std::min<int64_t>(d.steps, n_steps - done);
    p.step0 = c->step + done;
    cudaError_t e = cudaSuccess;
    if (d.seq > 0xfffff000u) {  // the numbers start again
      e = cudaMemsetAsync(d.inputs, 0, 2 * words * sizeof(dgk::Tagged::W), c->stream);
      d.seq = 1;
    }
    p.seq = d.seq;
    d.seq += 4 * (uint32_t)p.steps;
    if (e == cudaSuccess) e = dgk::launch_persist(c->dim, c->order, p, nt, c->d_err, c->stream);
    if (e != cudaSuccess) return e;
    *launched = done + p.steps;
    dgk::k_persist_sums<<<dim3(p.steps, 1 + c->n_obs), dgk::kSumThreads, 0, c->stream>>>(
        d.partials, nt, c->nv, inv_count, c->c0sq, c->d_res + done * 5, d.gsum, d.groups, d.obs_first, d.obs_grp,
        d.obs_w, c->d_obs + done * c->n_obs * 4, c->n_obs);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace dgc

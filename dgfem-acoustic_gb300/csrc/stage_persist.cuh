// Many RK4 steps of a small mesh in one launch (sm_103a; the Bernstein-basis
// tile bodies of stage_bb.cuh).
//
// On a mesh whose tiles all fit on the GPU at once a step is bound by latency:
// the launches of its stages, the chain of each tile's phases, and by the FP64
// rate of an SM sub-partition (64 cycles per warp instruction). Here every tile
// of 32 elements has a block of its own, resident for all steps of the launch
// (cooperative launch), with its geometry, state and accumulator in shared
// memory. What blocks exchange is each stage's input, through two global
// buffers in turn, every 4 bytes of it beside a 4-byte sequence number in one
// 8-byte word: a reader polls the words that it needs until all carry the
// stage's number, so that a stage costs one trip through L2 and no fence. (A flag
// per tile, raised after a fence and polled before the loads: 41 instead of 21 us
// per step of 7,200 linear triangles.) A tile is at most one stage ahead of its
// neighbours: it overwrites input k only when it has read their inputs k + 1,
// which they write after they have read input k, and every tile that reads a
// tile is read by it. Polls are bounded (StageArgs::wait_limit); a block that
// gives up sets the error flag and returns, and those that wait for it give up
// in turn.
//
// Sources and observers are the tiles' own work, and since every tile waits for
// its neighbours the slowest tile sets the pace: a block's threads share them.
// Sums per tile and step go to global memory and are added up, in a fixed order,
// by one launch after the steps (k_persist_sums).
//
// FP64, us per step with one launch per stage -> here, up to one tile per SM and
// at the resident limit: 2-D order 1 20 -> 14, 64 -> 53 (8 tiles per SM); order 2
// 29 -> 22, 67 -> 50 (5); order 3 41 -> 33, 96 -> 76 (5); order 4 57 -> 47, 116 ->
// 98 (4); 3-D order 1 34 -> 24, 83 -> 62 (5); order 2 55 -> 49, 97 -> 88 (3);
// order 3 100 -> 95, and beyond one tile per SM slower, 128 -> 166 (persist_pays).
#pragma once
#include <cstdint>

#include "stage_bb.cuh"

namespace dgk {

// A published value: each 4 bytes with the sequence number of its input.
struct Tagged {
  using W = ulonglong2;
  static __device__ __forceinline__ unsigned long long half(int v, uint32_t seq) {
    return (unsigned long long)seq << 32 | (uint32_t)v;
  }
  static __device__ __forceinline__ void st(W* p, double v, uint32_t seq) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(half(__double2loint(v), seq)),
                 "l"(half(__double2hiint(v), seq))
                 : "memory");
  }
  // false: not the input numbered seq yet
  static __device__ __forceinline__ bool ld(const W* p, double& v, uint32_t seq) {
    unsigned long long x, y;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(p) : "memory");
    v = __hiloint2double((int)(uint32_t)y, (int)(uint32_t)x);
    return (uint32_t)(x >> 32) == seq && (uint32_t)(y >> 32) == seq;
  }
};

struct PersistArgs {
  StageArgs<double> a;  // u, snap, geometry, tables, constants (stage unused)
  Tagged::W* buf[2];    // stage inputs published, [ntiles * TW] each
  uint32_t seq;         // number of the first input; no word of the buffers holds it or a later one
  int64_t E;            // elements (the last tile's others are padding)
  int64_t step0;        // global step of the first step here
  int steps;
  // sources: elements and node slots (element in the tile | node << 8) of each
  // tile, the sources covering each slot, their values, V^T and V^-T
  const int *sel_first, *sel, *snode_first, *snode, *soff, *sids;
  const double* sval;
  int nsrc;
  int64_t nrows;
  const double *Vt, *Vit;
  // observer groups (the entries of one observer in one tile) of each tile,
  // entries of each group: word of the coefficient in the tile, weight
  const int *grp_first, *ent_first;
  const int* ent_word;
  const double* ent_w;
  int groups;
  double* gsum;      // [steps][groups][4]
  double* partials;  // [steps][ntiles][NV]
};

// Layout on top of BBCfg's tables and face buffer (one input buffer).
template <int D, int P, int MINB>
struct PersistCfg : BBCfg<double, D, P, 1, MINB> {
  using B = BBCfg<double, D, P, 1, MINB>;
  static constexpr size_t oU = RoundUp<B::bytes, 128>::v;  // state, accumulator
  static constexpr size_t oA = oU + B::YB;
  static constexpr size_t bytes = oA + B::YB;
  // sources are placed between stages, when the face data are free: the changes
  // at their nodes, [NP][32], lie there
  static_assert(B::NF * B::NV * B::NFP >= B::NP, "source scratch");
};

// The environment of a resident tile's body (see BBGlobalEnv).
template <class C>
struct BBLocalEnv {
  static constexpr int CH = C::CH, SN = C::SN, NP = C::NP, NV = C::NV;
  // the trace is polled after the volume term, when it has mostly arrived
  static constexpr bool kTraceLast = true;
  const Tagged::W* in;    // published inputs of this stage
  Tagged::W* out;         // this tile's next input, at this thread's first word
  double *su, *sa, *sy;   // state, accumulator, stage input in shared memory, same
  const double* snap;     // global, same
  uint32_t seq;           // of this stage's input
  int limit, stage;
  bool pub;               // update() publishes the next input
  bool ok = true;
  double x2[CH];

  // as many nodes are polled together as 64 registers hold
  template <int NFP>
  __device__ __forceinline__ void gather(bool in_tile, const double* y_nb, int64_t word, const uint32_t (&w)[4],
                                         double (&up)[NV][NFP]) {
    constexpr int R = 16 / NV;
    auto at = [&](int m) { return (int)((w[m / 4] >> (8 * (m % 4))) & 0xffu) * SN; };
    if (in_tile) {
#pragma unroll
      for (int m = 0; m < NFP; ++m)
#pragma unroll
        for (int q = 0; q < NV; ++q) up[q][m] = y_nb[at(m) + q * C::SQ];
    }
#pragma unroll
    for (int m0 = 0; m0 < NFP; m0 += R) {
      bool got = in_tile;
      // the lanes stay together: those that went ahead would run the fluxes alone
      for (int n = 0; n < limit && !__all_sync(0xffffffffu, got); ++n) {
        if (got) continue;
        got = true;
#pragma unroll
        for (int m = m0; m < m0 + R; ++m)
          if (m < NFP)
#pragma unroll
            for (int q = 0; q < NV; ++q) got &= Tagged::ld(in + word + at(m) + q * C::SQ, up[q][m], seq);
      }
      ok &= got;
    }
  }
  __device__ __forceinline__ bool sync() { return !__syncthreads_or(!ok); }
  __device__ __forceinline__ bool residual() const { return stage == 4; }
  __device__ __forceinline__ void load(int n0) {
    if (stage != 4) return;
#pragma unroll
    for (int i = 0; i < CH; ++i)
      if (n0 + i < NP) x2[i] = snap[(n0 + i) * SN];
  }
  __device__ __forceinline__ void update(int n0, double dte, double (&o)[NP]) {
    const double c = stage == 3 ? dte : 0.5 * dte, c2 = 2.0 * dte;
#pragma unroll
    for (int i = 0; i < CH; ++i)
      if (n0 + i < NP) {
        const int w = (n0 + i) * SN;
        const double k = o[n0 + i], u = su[w];
        double y;
        if (stage == 4) {
          y = u + (sa[w] + dte * k) * (1.0 / 6.0);
          su[w] = y;
          o[n0 + i] = x2[i] - y;
        } else {
          y = u + c * k;
          sa[w] = stage == 1 ? dte * k : sa[w] + c2 * k;
        }
        sy[w] = y;
        if (pub) Tagged::st(out + w, y, seq + 1);
      }
  }
};

template <int D, int P, int MINB>
__global__ void __launch_bounds__(PersistCfg<D, P, MINB>::NT, MINB)
    stage_persist_kernel(const PersistArgs p, int* err) {
  using C = PersistCfg<D, P, MINB>;
  constexpr int LW = C::LW, NV = C::NV;
  extern __shared__ __align__(128) unsigned char sm[];
  int* sFm = reinterpret_cast<int*>(sm + C::oFm);
  unsigned char* sNb = sm + C::oNb;
  double* sY = reinterpret_cast<double*>(sm + C::oY);
  double* sGF = reinterpret_cast<double*>(sm + C::oGF);
  int* sGI = reinterpret_cast<int*>(sm + C::oGI);
  double* sN = reinterpret_cast<double*>(sm + C::oN);
  double* sU = reinterpret_cast<double*>(sm + C::oU);
  double* sA = reinterpret_cast<double*>(sm + C::oA);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int role = (warp + blockIdx.x) % NV;
  const StageArgs<double>& a = p.a;
  const int64_t tile = blockIdx.x;
  const int fw = C::first_word(tid, role);

  const int e0 = p.nsrc > 0 ? p.sel_first[tile] : 0, nel = p.nsrc > 0 ? p.sel_first[tile + 1] - e0 : 0;
  const int k0 = nel > 0 ? p.snode_first[tile] : 0, k1 = nel > 0 ? p.snode_first[tile + 1] : 0;
  const int g0 = p.groups > 0 ? p.grp_first[tile] : 0, g1 = p.groups > 0 ? p.grp_first[tile + 1] : 0;
  // this thread's part of the state in sY
  auto take_state = [&]() {
#pragma unroll
    for (int n = 0; n < C::NP; ++n) sU[fw + n * C::SN] = sY[fw + n * C::SN];
  };
  // The pressure at source nodes before step s, in sY (src/solver.cpp:455-483).
  // With S an element's nodes that an active source covers and v their values,
  // its coefficients become c + V^-1[:, S] (v - V[S, :] c). Every tile waits for
  // the slowest, so all threads share the work: a thread per node of S, then one
  // per coefficient. (A warp per element: 27 instead of 13 us per step where a
  // source covers some twenty elements of order 4, FP32.)
  auto inject = [&](int64_t s) {
    if (s >= 0 && s < p.nrows) {
      for (int i = tid; i < C::NP * LW; i += C::NT) sN[i] = 0.0;
      __syncthreads();
      const double* row = p.sval + s * p.nsrc;
      for (int k = k0 + tid; k < k1; k += C::NT) {
        double v = 0.0;
        bool any = false;
        for (int t = p.soff[k]; t < p.soff[k + 1]; ++t) {
          const double x = row[p.sids[t]];
          if (!isnan(x)) v = x, any = true;
        }
        if (any) {
          const int le = p.snode[k] & 0xff, n = p.snode[k] >> 8;
          double r = v;
#pragma unroll
          for (int j = 0; j < C::NP; ++j) r -= p.Vt[j * C::NP + n] * sY[le * C::SE + j * C::SN];
          sN[n * LW + le] = r;
        }
      }
      __syncthreads();
      for (int t = tid; t < nel * C::NP; t += C::NT) {
        const int le = p.sel[e0 + t % nel], i = t / nel;
        double x = 0.0;
#pragma unroll
        for (int n = 0; n < C::NP; ++n) x += p.Vit[n * C::NP + i] * sN[n * LW + le];
        sY[le * C::SE + i * C::SN] += x;
      }
      __syncthreads();
    }
    take_state();
  };
  // the state as input k
  auto publish = [&](int k) {
    for (int i = tid; i < C::TW; i += C::NT) Tagged::st(p.buf[k & 1] + tile * C::TW + i, sY[i], p.seq + (uint32_t)k);
  };
  // observer sums of this tile after step s: a warp per variable
  auto observe = [&](int s) {
    for (int g = g0; g < g1; ++g) {
      double acc = 0.0;
      for (int k = p.ent_first[g] + lane; k < p.ent_first[g + 1]; k += 32)
        acc += p.ent_w[k] * sY[p.ent_word[k] + warp * C::SQ];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) p.gsum[((int64_t)s * p.groups + g) * 4 + warp] = acc;
    }
  };

  if (a.wait_limit <= 0) {  // no wait may be made, also where a mesh of one tile would need none
    if (tid == 0) atomicOr(err, 1);
    return;
  }
  bb_load_tables<C>(a, sFm, sNb, tid, C::NT);
  for (int i = tid; i < C::GW * LW; i += C::NT) sGF[i] = a.bbF[tile * C::GW * LW + i];
  // a padding element is its own neighbour here: it reads no tile that does
  // not also read its own
  for (int i = tid; i < C::GI * LW; i += C::NT) {
    const int64_t e = tile * LW + i % LW;
    sGI[i] = e < p.E ? a.bbI[tile * C::GI * LW + i] : i < C::NF * LW ? (int)e : 0;
  }
  for (int i = tid; i < C::TW; i += C::NT) sY[i] = a.u[tile * C::TW + i];
  __syncthreads();
  if (nel > 0)
    inject(p.step0);
  else
    take_state();
  publish(0);

  BBRes<double> racc;
  for (int s = 0; s < p.steps; ++s) {
#pragma unroll 1
    for (int st = 1; st <= 4; ++st) {
      const int k = 4 * s + st - 1;
      BBLocalEnv<C> env;
      env.in = p.buf[k & 1];
      env.out = p.buf[(k + 1) & 1] + tile * C::TW + fw;
      env.su = sU + fw, env.sa = sA + fw, env.sy = sY + fw;
      env.snap = a.snap + tile * C::TW + fw;
      env.seq = p.seq + (uint32_t)k, env.limit = a.wait_limit, env.stage = st;
      env.pub = st < 4 || (nel == 0 && s + 1 < p.steps);
      if (!bb_tile_any<C>(a, env, tile, (const double*)sY, (const double*)sGF, (const int*)sGI, sFm, sNb, sN,
                          reinterpret_cast<int*>(sm + C::oX), tid, role, racc)) {
        if (tid == 0) atomicOr(err, 1);
        return;
      }
      __syncthreads();  // the next input is complete
    }
    // residual sums of this step
    {
      double v = racc.get();
      racc = BBRes<double>();
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
      if (lane == 0) p.partials[((int64_t)s * gridDim.x + tile) * NV + role] = v;
    }
    observe(s);
    if (nel > 0 && s + 1 < p.steps) {
      __syncthreads();
      inject(p.step0 + s + 1);
      publish(4 * s + 4);
    }
  }
  for (int i = tid; i < C::TW; i += C::NT) a.u[tile * C::TW + i] = sY[i];
}

template <int D, int P, int MINB>
struct StagePersist {
  using C = PersistCfg<D, P, MINB>;
  static int blocks_per_sm() {
    auto kfn = stage_persist_kernel<D, P, MINB>;
    if (cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::bytes) != cudaSuccess ||
        cudaFuncSetAttribute(kfn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) !=
            cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kfn, C::NT, C::bytes) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return nb;
  }
  static cudaError_t launch(const PersistArgs& p, int grid, int* err, cudaStream_t s) {
    void* args[2] = {const_cast<PersistArgs*>(&p), &err};
    return cudaLaunchCooperativeKernel((const void*)stage_persist_kernel<D, P, MINB>, dim3((unsigned)grid),
                                       dim3(C::NT), args, C::bytes, s);
  }
};

}  // namespace dgk

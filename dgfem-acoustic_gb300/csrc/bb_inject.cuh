// Source injection into elements given by Bernstein coefficients.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

struct dg_ctx;

namespace dgk {

// Word strides of a tile's variables, coefficients and elements, and the words
// of a tile (BBCfg in stage_bb.cuh).
struct Lay {
  int sq, sn, se, tw;
};

// Sources of a context: elements that hold source nodes (elem, their ranges
// eoff of the node slots dof; off/ids: the sources covering each slot), values
// val [nrows][nsrc], the transposed basis matrices V and V^-1.
template <typename T>
struct InjectArgs {
  T* u;
  const int64_t* elem;
  const int* eoff;
  int64_t ne;
  const int64_t* dof;
  const int *off, *ids;
  const double* val;
  int nsrc;
  int64_t nrows;
  int np;
  Lay l;
  const double *Vt, *Vit;
};

constexpr int kInjectThreads = 64, kInjectElems = kInjectThreads / 32;  // a warp per element
inline int64_t bb_inject_blocks(int64_t ne) { return (ne + kInjectElems - 1) / kInjectElems; }

// Source overwrite (src/solver.cpp:455-483) of the elements of block `block`
// with the values of step s. With S the nodes that an active source covers and
// v their values, the element's pressure becomes c + V^-1[:, S] (v - V[S, :] c):
// its nodal values are v at S and unchanged elsewhere.
template <typename T>
__device__ __forceinline__ void bb_inject_block(const InjectArgs<T>& a, int64_t block, int64_t s) {
  __shared__ T sc[kInjectElems][64], sr[kInjectElems][64];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, np = a.np;
  const int64_t i = block * kInjectElems + w;
  if (w >= kInjectElems || i >= a.ne) return;
  if (s < 0 || s >= a.nrows) return;
  const double* row = a.val + s * a.nsrc;
  const int64_t e = a.elem[i];
  T* c = a.u + (e >> 5) * a.l.tw + (e & 31) * a.l.se;
  for (int n = lane; n < np; n += 32) sc[w][n] = c[n * a.l.sn], sr[w][n] = (T)0;
  __syncwarp();
  for (int k = a.eoff[i] + lane; k < a.eoff[i + 1]; k += 32) {
    double v = 0.0;
    bool any = false;
    for (int t = a.off[k]; t < a.off[k + 1]; ++t) {
      const double x = row[a.ids[t]];
      if (!isnan(x)) v = x, any = true;
    }
    if (any) {
      const int n = (int)(a.dof[k] - e * np);
      T r0 = (T)v, r1 = (T)0;
#pragma unroll 4
      for (int j = 0; j < np; ++j) {
        const T p = (T)a.Vt[j * np + n] * sc[w][j];
        if (j & 1)
          r1 -= p;
        else
          r0 -= p;
      }
      sr[w][n] = r0 + r1;
    }
  }
  __syncwarp();
  for (int n = lane; n < np; n += 32) {
    T a0 = (T)0, a1 = (T)0;
#pragma unroll 4
    for (int j = 0; j < np; ++j) {
      const T p = (T)a.Vit[j * np + n] * sr[w][j];
      if (j & 1)
        a1 += p;
      else
        a0 += p;
    }
    c[n * a.l.sn] = sc[w][n] + (a0 + a1);
  }
}

}  // namespace dgk

namespace dgc {
template <typename T>
dgk::InjectArgs<T> bb_inject_args(const dg_ctx* c);
}

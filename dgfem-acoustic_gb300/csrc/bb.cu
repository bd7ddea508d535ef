// Bernstein basis: tables, conversions, source injection, element means
// (bb.cuh). The nodal values at the element's lattice are V c, the
// coefficients V^-1 u; both matrices are sparse (a vertex, edge or face of
// the lattice depends on its own points only), so a conversion is one sparse
// row per coefficient: 3-D p = 4 has 309 entries of 1225.
#include <cmath>
#include <vector>

#include "bb.cuh"
#include "bb_inject.cuh"
#include "stage_bb.cuh"

namespace {

using namespace dgk;

constexpr int LW = 32;

Lay lay(const dg_ctx* c) {
  const int tw = c->nv * c->np * LW;
  return c->prec == DG_FP32 && c->dim == 3 ? Lay{1, 4 * LW, 4, tw} : Lay{c->np * LW, LW, 1, tw};
}

// Reference layout -> tiles, elements e0 to e1 - 1 (e1 = E: and the padding).
// One block per (tile, variable) from e0's tile on: the tile's nodal values through shared memory (the reference layout is
// element-major), one warp per coefficient row.
template <typename T>
__global__ void __launch_bounds__(128) k_ref_to_bb(const double* __restrict__ ref, T* __restrict__ out,
                                                   const int* __restrict__ perm, const int* __restrict__ ptr,
                                                   const int* __restrict__ col, const double* __restrict__ val,
                                                   int64_t E, int np, Lay l, int64_t first, int64_t end) {
  __shared__ double x[35 * (LW + 1)];
  const int64_t tile = first / LW + blockIdx.x, e0 = tile * LW;
  const int q = blockIdx.y, lane = threadIdx.x & 31;
  for (int i = threadIdx.x; i < np * LW; i += blockDim.x) {
    const int e = i / np, n = i - e * np;
    x[perm[n] * (LW + 1) + e] = e0 + e < E ? ref[q * E * np + (e0 + e) * np + n] : 0.0;
  }
  __syncthreads();
  if (e0 + lane < first || (e0 + lane >= end && end < E)) return;
  T* o = out + tile * l.tw + q * l.sq + lane * l.se;
  for (int r = threadIdx.x >> 5; r < np; r += blockDim.x >> 5) {
    double s = 0.0;
#pragma unroll 4
    for (int k = ptr[r]; k < ptr[r + 1]; ++k) s += val[k] * x[col[k] * (LW + 1) + lane];
    o[r * l.sn] = (T)s;
  }
}

// Tiles -> reference layout (variables the state does not carry: zero).
template <typename T>
__global__ void __launch_bounds__(128) k_bb_to_ref(const T* __restrict__ in, double* __restrict__ ref,
                                                   const int* __restrict__ perm, const int* __restrict__ ptr,
                                                   const int* __restrict__ col, const double* __restrict__ val,
                                                   int64_t E, int np, int nv, Lay l) {
  __shared__ double x[35 * LW], y[35 * (LW + 1)];
  const int64_t tile = blockIdx.x, e0 = tile * LW;
  const int q = blockIdx.y, lane = threadIdx.x & 31;
  if (q < nv) {
    const T* p = in + tile * l.tw + q * l.sq;
    for (int i = threadIdx.x; i < np * LW; i += blockDim.x) x[i] = (double)p[(i / LW) * l.sn + (i % LW) * l.se];
    __syncthreads();
    for (int r = threadIdx.x >> 5; r < np; r += blockDim.x >> 5) {
      double s = 0.0;
#pragma unroll 4
      for (int k = ptr[r]; k < ptr[r + 1]; ++k) s += val[k] * x[col[k] * LW + lane];
      y[r * (LW + 1) + lane] = s;
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < np * LW; i += blockDim.x) {
    const int e = i / np, n = i - e * np;
    if (e0 + e < E) ref[q * E * np + (e0 + e) * np + n] = q < nv ? y[perm[n] * (LW + 1) + e] : 0.0;
  }
}

// Source overwrite at the start of a run's step (bb_inject_block).
template <typename T>
__global__ void __launch_bounds__(kInjectThreads) k_inject_bb(const InjectArgs<T> a, const int64_t* step) {
  bb_inject_block<T>(a, blockIdx.x, step[0]);
}

// Element means of p, p/c0^2 and v (src/Mesh.cpp:1196-1212) from the
// coefficients: w holds the mean of each basis function over the nodes.
template <typename T>
__global__ void k_cell_means_bb(const T* __restrict__ u, const double* __restrict__ w, int64_t E, int np, int nv,
                                double c0sq, double* __restrict__ out, int soa, Lay l) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= E) return;
  const T* c = u + (e >> 5) * l.tw + (e & 31) * l.se;
  double m[4] = {0.0, 0.0, 0.0, 0.0};
  for (int q = 0; q < nv; ++q) {
    double s = 0.0;
    for (int n = 0; n < np; ++n) s += w[n] * (double)c[q * l.sq + n * l.sn];
    m[q] = s;
  }
  if (soa) {
    out[e] = m[0], out[E + e] = m[0] / c0sq;
    for (int d = 0; d < 3; ++d) out[2 * E + 3 * e + d] = m[1 + d];
  } else {
    out[e * 5] = m[0], out[e * 5 + 1] = m[0] / c0sq;
    for (int d = 0; d < 3; ++d) out[e * 5 + 2 + d] = m[1 + d];
  }
}

}  // namespace

namespace dgc {

int64_t bb_slot(const dg_ctx* c, int64_t e, int n) {
  const Lay l = lay(c);
  return (e >> 5) * l.tw + n * l.sn + (e & 31) * l.se;
}

int64_t bb_var_stride(const dg_ctx* c) { return lay(c).sq; }

int bb_setup_basis(dg_ctx* c) {
  const int np = c->np, D = c->dim, P = c->order;
  std::vector<double>& V = c->bb_V;
  std::vector<double>& Vi = c->bb_Vinv;
  V.assign((size_t)np * np, 0.0), Vi.assign((size_t)np * np, 0.0);
  std::vector<long double> A((size_t)np * 2 * np, 0.0L);
  for (int i = 0; i < np; ++i) {
    for (int j = 0; j < np; ++j) V[i * np + j] = dgk::bb_value(D, P, i, j), A[(size_t)i * 2 * np + j] = V[i * np + j];
    A[(size_t)i * 2 * np + np + i] = 1.0L;
  }
  // Gauss-Jordan elimination with partial pivoting
  for (int k = 0; k < np; ++k) {
    int piv = k;
    for (int i = k + 1; i < np; ++i)
      if (std::fabs((double)A[(size_t)i * 2 * np + k]) > std::fabs((double)A[(size_t)piv * 2 * np + k])) piv = i;
    for (int j = 0; j < 2 * np; ++j) std::swap(A[(size_t)k * 2 * np + j], A[(size_t)piv * 2 * np + j]);
    const long double d = A[(size_t)k * 2 * np + k];
    for (int j = 0; j < 2 * np; ++j) A[(size_t)k * 2 * np + j] /= d;
    for (int i = 0; i < np; ++i) {
      const long double f = A[(size_t)i * 2 * np + k];
      if (i == k || f == 0.0L) continue;
      for (int j = 0; j < 2 * np; ++j) A[(size_t)i * 2 * np + j] -= f * A[(size_t)k * 2 * np + j];
    }
  }
  // the inverse has V's sparsity: what elimination leaves elsewhere is rounding
  for (int i = 0; i < np; ++i)
    for (int j = 0; j < np; ++j) Vi[i * np + j] = V[i * np + j] != 0.0 ? (double)A[(size_t)i * 2 * np + np + j] : 0.0;
  // device: [0] V, [1] V^-1 as rows, the transposes dense, the means
  std::vector<int> idx;
  std::vector<double> val;
  for (int m = 0; m < 2; ++m) {
    const std::vector<double>& M = m ? Vi : V;
    std::vector<int> ptr(1, 0), col;
    std::vector<double> v;
    for (int i = 0; i < np; ++i) {
      for (int j = 0; j < np; ++j)
        if (M[i * np + j] != 0.0) col.push_back(j), v.push_back(M[i * np + j]);
      ptr.push_back((int)col.size());
    }
    c->bb_iptr[m] = (int)idx.size(), idx.insert(idx.end(), ptr.begin(), ptr.end());
    c->bb_icol[m] = (int)idx.size(), idx.insert(idx.end(), col.begin(), col.end());
    c->bb_ival[m] = (int)val.size(), val.insert(val.end(), v.begin(), v.end());
    c->bb_iden[m] = (int)val.size();
    for (int j = 0; j < np; ++j)
      for (int i = 0; i < np; ++i) val.push_back(M[i * np + j]);
  }
  c->bb_imean = (int)val.size();
  for (int j = 0; j < np; ++j) {
    double s = 0.0;
    for (int i = 0; i < np; ++i) s += V[i * np + j];
    val.push_back(s / np);
  }
  cudaError_t e = dev_alloc(c, (void**)&c->bb_int, idx.size() * sizeof(int));
  if (e == cudaSuccess) e = dev_alloc(c, (void**)&c->bb_dbl, val.size() * sizeof(double));
  if (e == cudaSuccess) e = cudaMemcpyAsync(c->bb_int, idx.data(), idx.size() * sizeof(int), cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(c->bb_dbl, val.data(), val.size() * sizeof(double), cudaMemcpyHostToDevice, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  return e == cudaSuccess ? DG_OK : DG_ERR_CUDA;
}

cudaError_t bb_from_ref(dg_ctx* c, const double* ref, void* out, int64_t e0, int64_t e1) {
  const dim3 grid((unsigned)(((e1 == c->E ? c->Epad : e1) + LW - 1) / LW - e0 / LW), c->nv);
  const int *p = c->bb_int + c->bb_iptr[1], *k = c->bb_int + c->bb_icol[1];
  const double* v = c->bb_dbl + c->bb_ival[1];
  if (c->prec == DG_FP32)
    k_ref_to_bb<float><<<grid, 128, 0, c->stream>>>(ref, (float*)out, c->d_perm, p, k, v, c->E, c->np, lay(c), e0, e1);
  else
    k_ref_to_bb<double><<<grid, 128, 0, c->stream>>>(ref, (double*)out, c->d_perm, p, k, v, c->E, c->np, lay(c), e0, e1);
  return cudaGetLastError();
}

cudaError_t bb_to_ref(dg_ctx* c, const void* in, double* ref) {
  const dim3 grid((unsigned)((c->E + LW - 1) / LW), 4);
  const int *p = c->bb_int + c->bb_iptr[0], *k = c->bb_int + c->bb_icol[0];
  const double* v = c->bb_dbl + c->bb_ival[0];
  if (c->prec == DG_FP32)
    k_bb_to_ref<float><<<grid, 128, 0, c->stream>>>((const float*)in, ref, c->d_perm, p, k, v, c->E, c->np, c->nv, lay(c));
  else
    k_bb_to_ref<double><<<grid, 128, 0, c->stream>>>((const double*)in, ref, c->d_perm, p, k, v, c->E, c->np, c->nv, lay(c));
  return cudaGetLastError();
}

template <typename T>
InjectArgs<T> bb_inject_args(const dg_ctx* c) {
  InjectArgs<T> a{};
  a.u = (T*)c->u, a.elem = c->d_src_elem, a.eoff = c->d_src_eoff, a.ne = c->n_src_elems;
  a.dof = c->d_src_dof, a.off = c->d_src_off, a.ids = c->d_src_ids, a.val = c->d_srcval;
  a.nsrc = c->n_src, a.nrows = c->srcval_steps, a.np = c->np, a.l = lay(c);
  a.Vt = c->bb_dbl + c->bb_iden[0], a.Vit = c->bb_dbl + c->bb_iden[1];
  return a;
}
template InjectArgs<float> bb_inject_args<float>(const dg_ctx*);
template InjectArgs<double> bb_inject_args<double>(const dg_ctx*);

cudaError_t bb_inject(dg_ctx* c) {
  if (c->n_src_elems == 0) return cudaSuccess;
  const unsigned nb = (unsigned)bb_inject_blocks(c->n_src_elems);
  if (c->prec == DG_FP32)
    k_inject_bb<float><<<nb, kInjectThreads, 0, c->stream>>>(bb_inject_args<float>(c), c->d_step);
  else
    k_inject_bb<double><<<nb, kInjectThreads, 0, c->stream>>>(bb_inject_args<double>(c), c->d_step);
  return cudaGetLastError();
}

cudaError_t bb_cell_means(dg_ctx* c, double* out, bool soa) {
  const unsigned nb = (unsigned)((c->E + 127) / 128);
  const double* w = c->bb_dbl + c->bb_imean;
  if (c->prec == DG_FP32)
    k_cell_means_bb<float><<<nb, 128, 0, c->stream>>>((const float*)c->u, w, c->E, c->np, c->nv, c->c0sq, out, soa, lay(c));
  else
    k_cell_means_bb<double><<<nb, 128, 0, c->stream>>>((const double*)c->u, w, c->E, c->np, c->nv, c->c0sq, out, soa, lay(c));
  return cudaGetLastError();
}

}  // namespace dgc

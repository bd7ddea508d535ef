// Bernstein-basis RK4 stage kernel (sm_103a, FP32 and FP64 state, triangles
// and tetrahedra of orders 1..4).
//
// Same semi-discrete equations as the reference's per-stage work
// (src/Mesh.cpp:734-975, src/solver.cpp:38-57, :488-516). The state is held
// as Bernstein coefficients on the element's lattice in place of nodal
// values. On straight-sided elements every operator of the scheme is then
// sparse with small constants (Chan and Warburton, "GPU-accelerated
// Bernstein-Bezier discontinuous Galerkin methods for wave problems", SIAM J.
// Sci. Comput. 39, 2017):
//   * derivative: d/dxi_r of degree P has the degree P-1 coefficients
//     P (c[b+e_r] - c[b+e_0]);
//   * degree elevation P-1 -> P: c[a] = sum_k (a_k / P) g[a-e_k];
//   * lift of a face flux f: layer 0 (the coefficients on the face) is
//     sJ L0 f, L0 the integer stencil E^T E (E: degree elevation P -> P+1 on
//     the face, times P+1), and layer j, at lattice distance j from the face,
//     is -1/(j+1) sum_k (g_k+1) (layer j-1)[g+e_k].
// The volume term is taken in strong form, so that a face's flux is
//   f = n.F(y-) - h = 1/2 n.F(d) - 1/2 s c0 d,  d = y- - y+   (interior)
//   f = (A_n - B) y-                                          (boundary).
// Per variable and element 3-D p = 3 takes about 700 multiply-adds against
// 2000 with the dense nodal operators, p = 4 about 1150 against 5800. FP32
// stages were bound by the shared-memory loads of the dense operators' entries,
// which are compile-time constants here; they are now within a factor of two of
// the memory floor. FP64 runs at 2 operations per clock and SM on GB300 and
// bounds its stages by their count, which the fixed-point sums (bb_tile_fx,
// fx_gradient) quarter. Measured per RK4 step against the nodal kernels' best:
// 196,608 tetrahedra of order 3, FP32, 0.61 -> 0.28 ms (floor 0.19); 131,712 of
// order 4, FP32, 0.61 -> 0.36 (0.21); 24,576 of order 3, FP64, 2.24 -> 0.33
// (0.05); 125,000 triangles of order 4, FP32, 0.14 -> 0.083 (0.067).
//
// Layout: arrays of tiles of 32 elements, [tile][variable][coefficient][32]:
// a warp's lanes are the tile's elements, every load and store of a
// coefficient is one coalesced line or conflict-free shared row (FP32
// tetrahedra: the Q4 layout of BBCfg and bb_tile_q4).
// One block per tile with D+1 warps; warp w is face w in the flux phase and
// variable w in the volume, lift and update phases:
//   1. the tile's stage input and geometry arrive by TMA bulk copies;
//   2. each thread issues the loads of its face's neighbour trace (from the
//      tile itself where the neighbour is in it, else from global memory),
//      then computes its variable's volume term while they are in flight;
//   3. it forms its face's flux, applies L0 and stores it to shared memory;
//   4. it adds its variable's lift of all faces and updates the RK arrays.
// Every mbarrier wait is bounded; on timeout the block records an error,
// drains its own copies (bounded) and stops.
#pragma once
#include <cstdint>
#include <utility>

#include "stage2.cuh"

namespace dgk {

// ---- compile-time lattice arithmetic ----------------------------------------

template <class F, int... I>
__device__ __forceinline__ void bb_for_impl(F&& f, std::integer_sequence<int, I...>) {
  (f(std::integral_constant<int, I>{}), ...);
}
// f(integral_constant<int, 0>) ... f(integral_constant<int, N-1>)
template <int N, class F>
__device__ __forceinline__ void bb_for(F&& f) {
  bb_for_impl(f, std::make_integer_sequence<int, N>{});
}

struct Bary {
  int a[4];  // barycentric lattice coordinates, sum p
};

__host__ __device__ constexpr int bb_np(int d, int p) {
  return d == 0 ? 1 : d == 1 ? p + 1 : d == 2 ? (p + 1) * (p + 2) / 2 : (p + 1) * (p + 2) * (p + 3) / 6;
}
// Index of lattice point (a[1], a[2], a[3]) of degree p, a[1] fastest (the
// internal node order of refelem.h; a face's lattice is the same in d - 1).
__host__ __device__ constexpr int bb_index(int d, int p, const Bary& b) {
  int idx = 0;
  if (d == 3)
    for (int k = 0; k < b.a[3]; ++k) idx += bb_np(2, p - k);
  const int pj = d == 3 ? p - b.a[3] : p;
  if (d >= 2)
    for (int j = 0; j < b.a[2]; ++j) idx += pj - j + 1;
  return d == 0 ? 0 : idx + b.a[1];
}
__host__ __device__ constexpr Bary bb_lattice(int d, int p, int n) {
  Bary b{};
  int r = n;
  if (d == 3)
    while (r >= bb_np(2, p - b.a[3])) r -= bb_np(2, p - b.a[3]), ++b.a[3];
  const int pj = p - b.a[3];
  if (d >= 2)
    while (r >= pj - b.a[2] + 1) r -= pj - b.a[2] + 1, ++b.a[2];
  if (d >= 1) b.a[1] = r;
  b.a[0] = p - b.a[1] - b.a[2] - b.a[3];
  return b;
}
// The same as a type (its members are constants inside nested lambdas too).
template <int DD, int PP, int N>
struct BLat {
  static constexpr Bary b = bb_lattice(DD, PP, N);
};
__host__ __device__ constexpr Bary bb_add(Bary b, int k, int s) {
  b.a[k] += s;
  return b;
}
// Local faces' corners (Gmsh's local face tables, as refelem.cpp) and the
// vertex opposite each face.
__host__ __device__ constexpr int bb_corner(int d, int f, int k) {
  if (d == 2) return k == 0 ? f : (f + 1) % 3;
  const int t[4][3] = {{0, 2, 1}, {0, 1, 3}, {0, 3, 2}, {3, 1, 2}};
  return t[f][k];
}
__host__ __device__ constexpr int bb_opposite(int d, int f) {
  return d == 2 ? (f + 2) % 3 : f == 0 ? 3 : f == 1 ? 2 : f == 2 ? 1 : 0;
}
// Element lattice index of face lattice point g (degree p - j) at distance j
// from face f.
__host__ __device__ constexpr int bb_layer_index(int d, int p, int f, int j, const Bary& g) {
  Bary b{};
  b.a[bb_opposite(d, f)] = j;
  for (int k = 0; k < d; ++k) b.a[bb_corner(d, f, k)] = g.a[k];
  return bb_index(d, p, b);
}
// Bernstein polynomial j of degree p at lattice point i.
__host__ __device__ constexpr double bb_value(int d, int p, int i, int j) {
  const Bary x = bb_lattice(d, p, i), al = bb_lattice(d, p, j);
  double v = 1.0;
  int left = p;
  for (int k = 0; k <= d; ++k) {
    for (int t = 1; t <= al.a[k]; ++t) v = v * (double)(left - al.a[k] + t) / (double)t * (double)x.a[k] / (double)p;
    left -= al.a[k];
  }
  return v;
}

// ---- configuration ------------------------------------------------------------

// NBUF_: stage-input buffers (2: the next tile arrives while this one
// computes; 1: after its flux phase), MINB: blocks per SM that the register
// budget allows for.
template <typename T_, int D_, int P_, int NBUF_, int MINB_>
struct BBCfg {
  using T = T_;
  static constexpr int D = D_, P = P_, NBUF = NBUF_, MINB = MINB_;
  using S = Shape<D_, P_>;
  static constexpr int NP = S::NP, NF = S::NF, NFP = S::NFP, NV = S::NV, NPERM = S::NPERM;
  static constexpr int LW = 32;                 // elements per tile
  static constexpr int NT = LW * NV;            // threads per block
  static constexpr int TW = NV * NP * LW;       // state words of a tile
  // Q4 (FP32, 3-D): the four variables of a coefficient side by side,
  // [tile][coefficient][32][4], else one plane each, [tile][variable][coefficient][32]
  static constexpr bool Q4 = sizeof(T) == 4 && D == 3;
  // packed FP32 arithmetic for two variables in the fluxes and two metric columns
  // in the volume term: 131,712 tetrahedra of order 4 373 -> 360 us per step; at
  // order 3 its register pairs cost more (1.8 %)
  static constexpr bool PACK2 = Q4 && P == 4;
  static constexpr int SQ = Q4 ? 1 : NP * LW, SN = Q4 ? 4 * LW : LW, SE = Q4 ? 4 : 1;  // word strides
  // word in the tile of the first coefficient that a thread owns in the update
  __host__ __device__ static constexpr int first_word(int tid, int role) { return Q4 ? tid : role * NP * LW + (tid & 31); }
  static constexpr int oGV = NF * (D + 1), oG = oGV + D, oS = oG + D * D, GW = oS + 1;  // geometry words
  static constexpr int GI = 2 * NF;             // neighbour, code
  static constexpr int CH = sizeof(T) == 8 ? 6 : P == 4 ? 10 : 7;  // coefficients whose RK operands are in flight together
  static constexpr uint32_t YB = TW * sizeof(T), GB = GW * LW * sizeof(T), IB = GI * LW * 4;
  static constexpr size_t oBar = 0;                                     // NBUF mbarriers
  static constexpr size_t oFm = 64;                                     // int [NF][16]: element word offset of a face node
  static constexpr size_t oNb = oFm + NF * 16 * 4;                      // uchar [NF*NPERM][16]: neighbour node of a face node
  static constexpr size_t oY = RoundUp<oNb + NF * NPERM * 16, 128>::v;  // NBUF x [NV][NP][32]
  static constexpr size_t oGF = oY + (size_t)NBUF * YB;
  static constexpr size_t oGI = oGF + (size_t)NBUF * GB;
  static constexpr size_t oN = oGI + (size_t)NBUF * IB;                 // [NF][NV][NFP][32]
  static constexpr bool FX = sizeof(T) == 8;  // lift and elevation in fixed point (bb_tile_fx)
  // the gradient in fixed point as well (fx_gradient): in 3-D, where the pressure's
  // thread has sixteen products per coefficient, up to order 3; in 2-D it cost
  // registers and gained nothing (order 3: 47.5 -> 51.5 us per step), and neither
  // did the fluxes in 3-D (381 -> 626 us, spilled registers)
  static constexpr bool FXG = FX && D == 3 && P <= 3;
  static constexpr size_t oX = oN + (size_t)NF * NV * NFP * LW * sizeof(T);  // int [NF][NV][32]: exponents (FX)
  static constexpr size_t oR = oX + (FX ? (size_t)NF * NV * LW * 4 : 0);
  static constexpr size_t bytes = oR + NV * NV * sizeof(double);
  static_assert(NF == NV, "a block's warps are faces and variables in turn");
  static_assert(NFP <= 16 && NP <= 64, "tables hold 16 nodes per face");
};

// g . (c[b+e_r] - c[b+e_0]) summed over r. FP32 takes the differences first
// (an error relative to the difference); FP64, whose rate bounds its kernels,
// one multiply-add per coefficient with g_0 = -sum g_r.
template <typename T, int D>
struct BBGrad {
  T g[D], g0;
  __device__ __forceinline__ void done() {
    g0 = -g[0];
#pragma unroll
    for (int r = 1; r < D; ++r) g0 -= g[r];
  }
  // y: one variable's coefficients; n: index of b + e_0, .., b + e_D
  template <int N0, int N1, int N2, int N3, int LW>
  __device__ __forceinline__ T add(T t, const T* y) const {
    const T c0 = y[N0 * LW];
    if constexpr (sizeof(T) == 8) {
      t += g0 * c0;
      t += g[0] * y[N1 * LW];
      t += g[1] * y[N2 * LW];
      if constexpr (D == 3) t += g[2] * y[N3 * LW];
    } else {
      t += g[0] * (y[N1 * LW] - c0);
      t += g[1] * (y[N2 * LW] - c0);
      if constexpr (D == 3) t += g[2] * (y[N3 * LW] - c0);
    }
    return t;
  }
};

// Volume term of variable q into out (strong form, see the file comment).
// y: the tile's stage input at this lane, g: its geometry at this lane.
template <class C, typename T>
__device__ __forceinline__ void bb_volume(const T* y, const T* g, int q, T rhoc2, T inv_rho0, T (&out)[C::NP]) {
  constexpr int D = C::D, P = C::P, NP = C::NP, LW = C::LW;
  BBGrad<T, D> gv;
#pragma unroll
  for (int r = 0; r < D; ++r) gv.g[r] = g[(C::oGV + r) * LW];
  gv.done();
#pragma unroll
  for (int n = 0; n < NP; ++n) out[n] = (T)0;
  auto scatter = [&](auto b_, T t) {
    using L = BLat<D, P - 1, decltype(b_)::value>;
    bb_for<D + 1>([&](auto k_) {
      constexpr int k = decltype(k_)::value;
      constexpr int a = bb_index(D, P, bb_add(L::b, k, 1));
      constexpr int w = L::b.a[k] + 1;
      out[a] -= (T)w * t;
    });
  };
  if (q == 0) {
    BBGrad<T, D> gm[D];
#pragma unroll
    for (int d = 0; d < D; ++d) {
#pragma unroll
      for (int r = 0; r < D; ++r) gm[d].g[r] = rhoc2 * g[(C::oG + r * D + d) * LW];
      gm[d].done();
    }
    bb_for<bb_np(D, P - 1)>([&](auto b_) {
      using L = BLat<D, P - 1, decltype(b_)::value>;
      constexpr int n0 = bb_index(D, P, bb_add(L::b, 0, 1)), n1 = bb_index(D, P, bb_add(L::b, 1, 1)),
                    n2 = bb_index(D, P, bb_add(L::b, 2, 1)), n3 = D == 3 ? bb_index(D, P, bb_add(L::b, 3, 1)) : 0;
      T t = gv.template add<n0, n1, n2, n3, LW>((T)0, y);
#pragma unroll
      for (int d = 0; d < D; ++d) t = gm[d].template add<n0, n1, n2, n3, LW>(t, y + (1 + d) * NP * LW);
      scatter(b_, t);
    });
  } else {
    BBGrad<T, D> gd;
#pragma unroll
    for (int r = 0; r < D; ++r) gd.g[r] = inv_rho0 * g[(C::oG + r * D + q - 1) * LW];
    gd.done();
    const T* yq = y + q * NP * LW;
    bb_for<bb_np(D, P - 1)>([&](auto b_) {
      using L = BLat<D, P - 1, decltype(b_)::value>;
      constexpr int n0 = bb_index(D, P, bb_add(L::b, 0, 1)), n1 = bb_index(D, P, bb_add(L::b, 1, 1)),
                    n2 = bb_index(D, P, bb_add(L::b, 2, 1)), n3 = D == 3 ? bb_index(D, P, bb_add(L::b, 3, 1)) : 0;
      scatter(b_, gd.template add<n0, n1, n2, n3, LW>(gv.template add<n0, n1, n2, n3, LW>((T)0, yq), y));
    });
  }
}

// Value at face node M of the integer stencil L0 = E^T E of a face flux.
template <class C, int M, typename T>
__device__ __forceinline__ T bb_stencil_at(const T (&f)[C::NFP]) {
  constexpr int D = C::D, P = C::P;
  using L = BLat<D - 1, P, M>;
  constexpr int w0 = (L::b.a[0] + 1) * (L::b.a[0] + 1) + (L::b.a[1] + 1) * (L::b.a[1] + 1) +
                     (D == 3 ? (L::b.a[2] + 1) * (L::b.a[2] + 1) : 0);
  T s = (T)w0 * f[M];
  bb_for<D * D>([&](auto ij_) {
    constexpr int i = decltype(ij_)::value / D, j = decltype(ij_)::value % D;
    if constexpr (i != j && L::b.a[j] > 0) {
      constexpr int n = bb_index(D - 1, P, bb_add(bb_add(L::b, i, 1), j, -1));
      constexpr int w = (L::b.a[i] + 1) * L::b.a[j];
      s += (T)w * f[n];
    }
  });
  return s;
}
// the same for two variables at once, in packed FP32 instructions
template <class C, int M>
__device__ __forceinline__ float2 bb_stencil_at(const float2 (&f)[C::NFP]) {
  constexpr int D = C::D, P = C::P;
  using L = BLat<D - 1, P, M>;
  constexpr int w0 = (L::b.a[0] + 1) * (L::b.a[0] + 1) + (L::b.a[1] + 1) * (L::b.a[1] + 1) +
                     (D == 3 ? (L::b.a[2] + 1) * (L::b.a[2] + 1) : 0);
  float2 s = __fmul2_rn(make_float2((float)w0, (float)w0), f[M]);
  bb_for<D * D>([&](auto ij_) {
    constexpr int i = decltype(ij_)::value / D, j = decltype(ij_)::value % D;
    if constexpr (i != j && L::b.a[j] > 0) {
      constexpr int n = bb_index(D - 1, P, bb_add(bb_add(L::b, i, 1), j, -1));
      constexpr int w = (L::b.a[i] + 1) * L::b.a[j];
      s = __ffma2_rn(make_float2((float)w, (float)w), f[n], s);
    }
  });
  return s;
}
template <class C, typename T>
__device__ __forceinline__ void bb_face_stencil(const T (&f)[C::NFP], T* dst) {
  bb_for<C::NFP>([&](auto m_) { dst[decltype(m_)::value * C::LW] = bb_stencil_at<C, decltype(m_)::value>(f); });
}

// Adds layers J .. P of face F's lift to out; prev holds layer J-1's values.
template <class C, int F, int J, typename T>
__device__ __forceinline__ void bb_layers(const T (&prev)[bb_np(C::D - 1, C::P - J + 1)], T (&out)[C::NP]) {
  constexpr int D = C::D, P = C::P;
  if constexpr (J <= P) {
    T cur[bb_np(D - 1, P - J)];
    bb_for<bb_np(D - 1, P - J)>([&](auto g_) {
      using L = BLat<D - 1, P - J, decltype(g_)::value>;
      constexpr int a = bb_layer_index(D, P, F, J, L::b);
      T s = J < P ? (T)0 : out[a];
      bb_for<D>([&](auto k_) {
        constexpr int k = decltype(k_)::value;
        constexpr int n = bb_index(D - 1, P - J + 1, bb_add(L::b, k, 1));
        constexpr double w = -(double)(L::b.a[k] + 1) / (double)(J + 1);
        s += (T)w * prev[n];
      });
      cur[decltype(g_)::value] = s;
      out[a] = J < P ? out[a] + s : s;
    });
    if constexpr (J < P) bb_layers<C, F, J + 1>(cur, out);
  }
}

// Adds the lift of all faces for one variable of one element; sN: its face
// data (node m of face f at f * SF + m * SM).
template <class C, int SF, int SM, typename T>
__device__ __forceinline__ void bb_lift(const T* sN, T (&out)[C::NP]) {
  constexpr int D = C::D, P = C::P;
  bb_for<C::NF>([&](auto f_) {
    constexpr int f = decltype(f_)::value;
    T l0[C::NFP];
#pragma unroll
    for (int m = 0; m < C::NFP; ++m) l0[m] = sN[f * SF + m * SM];
    bb_for<C::NFP>([&](auto m_) {
      constexpr int a = bb_layer_index(D, P, f, 0, bb_lattice(D - 1, P, decltype(m_)::value));
      out[a] += l0[decltype(m_)::value];
    });
    bb_layers<C, f, 1>(l0, out);
  });
}

// Sum over the element's nodes of the squared nodal values of coefficients d.
template <class C, typename T>
__device__ __forceinline__ T bb_nodal_square(const T (&d)[C::NP]) {
  constexpr int D = C::D, P = C::P;
  T sum = (T)0;
  bb_for<C::NP>([&](auto i_) {
    constexpr int i = decltype(i_)::value;
    T v = (T)0;
    bb_for<C::NP>([&](auto j_) {
      constexpr int j = decltype(j_)::value;
      constexpr double w = bb_value(D, P, i, j);
      if constexpr (w != 0.0) v += (T)w * d[j];
    });
    sum += v * v;
  });
  return sum;
}

// Residual sum of a thread's variable. FP32 squares overflow from 1.8e19 on, far
// below the largest finite state: an element whose sum does is summed again
// with its values scaled by 2^-64, into an FP64 remainder, so that the sum is
// non-finite only when the state is.
template <typename T>
struct BBRes {
  T s = (T)0;
  double big = 0.0;
  template <class C>
  __device__ __forceinline__ void add(T (&d)[C::NP]) {
    const T v = bb_nodal_square<C>(d), t = s + v;
    if constexpr (sizeof(T) == 8) {
      s = t;
    } else {
      if (t <= 3.4028234e38f) {
        s = t;
        return;
      }
#pragma unroll
      for (int n = 0; n < C::NP; ++n) d[n] *= 5.421010862427522e-20f;  // 2^-64
      big += (double)s + (double)bb_nodal_square<C>(d) * 3.402823669209385e38;  // 2^128
      s = 0.f;
    }
  }
  __device__ __forceinline__ double get() const { return (double)s + big; }
};

// What a tile's body meets outside the tile, for the kernels that run one
// stage per launch: other tiles' stage input and the RK arrays, in global
// memory. RK operands of CH coefficients of this thread are loaded together
// (the first group before the lift, so that its latency overlaps it), then
// combined with dt*L and stored; in stages 4 and 5 out becomes the residual's
// difference.
//
// The accumulator k1 + 2 k2 + 2 k3 has an array of its own. (The stages' inputs
// hold the same sum, and an FP32 step that forms it from them moves 14 state words
// in place of 18, but only to the spacing of the state: where a step changes the
// state by about that, the sum was off by up to two thirds of it.)
template <class C, class Free>
struct BBGlobalEnv {
  using T = typename C::T;
  static constexpr int CH = C::CH, SN = C::SN, NP = C::NP;
  // the trace's loads come first: their latency overlaps the volume term
  static constexpr bool kTraceLast = false;
  // FP32: this thread's part of the stage input stays in shared memory until the
  // update, where it is u (not with one buffer, which the next tile enters at the
  // barrier)
  static constexpr bool OWN = sizeof(T) == 4 && C::NBUF == 2;
  const StageArgs<T>& a;
  int64_t base;      // this thread's first coefficient in the arrays
  const T* own;      // the same in the tile's stage input
  Free free_inputs;  // called by every thread once the stage input is no longer read
  // FP32: u of all coefficients before the lift, the other operands in groups
  static constexpr int NU = sizeof(T) == 4 ? NP : CH;
  T x0[NU], x1[CH], x2[CH];
  __device__ __forceinline__ BBGlobalEnv(const StageArgs<T>& a_, int64_t b, const T* y, Free f)
      : a(a_), base(b), own(OWN ? y : a_.y_in + b), free_inputs(f) {}
  // Values at the neighbour's face nodes: node m has coefficient (w byte m) of
  // the element whose first word is y_nb in shared memory (in_tile) or word
  // `word` of the stage input.
  template <int NFP>
  __device__ __forceinline__ void gather(bool in_tile, const T* y_nb, int64_t word, const uint32_t (&w)[4],
                                         T (&up)[C::NV][NFP]) {
    const T* nb = in_tile ? y_nb : a.y_in + word;
#pragma unroll
    for (int m = 0; m < NFP; ++m) {
      const T* p = nb + ((w[m / 4] >> (8 * (m % 4))) & 0xffu) * SN;
#pragma unroll
      for (int q = 0; q < C::NV; ++q) up[q][m] = p[q * C::SQ];
    }
  }
  template <int NFP>
  __device__ __forceinline__ void gather(bool in_tile, const float* y_nb, int64_t word, const uint32_t (&w)[4],
                                         float4 (&up)[NFP]) {
    const float* nb = in_tile ? y_nb : a.y_in + word;
#pragma unroll
    for (int m = 0; m < NFP; ++m)
      up[m] = *reinterpret_cast<const float4*>(nb + ((w[m / 4] >> (8 * (m % 4))) & 0xffu) * SN);
  }
  // the face data of the tile are in shared memory
  __device__ __forceinline__ bool sync() {
    __syncthreads();
    free_inputs();
    return true;
  }
  __device__ __forceinline__ bool residual() const { return a.stage >= 4; }
  __device__ __forceinline__ void operands(int n0, T (&x)[CH], const T* p) const {
#pragma unroll
    for (int i = 0; i < CH; ++i)
      if (n0 + i < NP) x[i] = p[(n0 + i) * SN];
  }
  __device__ __forceinline__ void load(int n0) {
    const int stage = a.stage;
    if (stage == 0) return;
    if constexpr (sizeof(T) == 4) {
      // (stages 1 and 5: the stage input is u)
      if (n0 == 0 && !(OWN && (stage == 1 || stage == 5))) {
#pragma unroll
        for (int n = 0; n < NP; ++n) x0[n] = a.u[base + n * SN];
      }
    } else {
      operands(n0, x0, a.u + base);
    }
    if (stage >= 2 && stage <= 4) operands(n0, x1, a.acc + base);
    if (stage >= 4) operands(n0, x2, a.snap + base);
  }
  // u of coefficient n0 + i
  __device__ __forceinline__ T u0(int n0, int i) const {
    if constexpr (sizeof(T) == 4)
      return OWN && (a.stage == 1 || a.stage == 5) ? own[(n0 + i) * SN] : x0[n0 + i];
    else
      return x0[i];
  }
  __device__ __forceinline__ void update(int n0, T dte, T (&out)[NP]) {
    const int stage = a.stage;
    T* yo = a.y_out + base;
    if (stage == 0) {
      T* ko = a.k_out + base;
#pragma unroll
      for (int i = 0; i < CH; ++i)
        if (n0 + i < NP) ko[(n0 + i) * SN] = dte * out[n0 + i];
      return;
    }
    T* ac = a.acc + base;
    if (stage == 1) {
#pragma unroll
      for (int i = 0; i < CH; ++i)
        if (n0 + i < NP) {
          ac[(n0 + i) * SN] = dte * out[n0 + i];
          yo[(n0 + i) * SN] = u0(n0, i) + ((T)0.5 * dte) * out[n0 + i];
        }
    } else if (stage <= 3) {
      const T c = stage == 3 ? dte : (T)0.5 * dte, c2 = (T)2 * dte;
#pragma unroll
      for (int i = 0; i < CH; ++i)
        if (n0 + i < NP) {
          ac[(n0 + i) * SN] = x1[i] + c2 * out[n0 + i];
          yo[(n0 + i) * SN] = u0(n0, i) + c * out[n0 + i];
        }
    } else {
      T* un_ = stage == 4 ? a.u + base : yo;
#pragma unroll
      for (int i = 0; i < CH; ++i)
        if (n0 + i < NP) {
          const T u = u0(n0, i);
          const T un = stage == 4 ? u + (x1[i] + dte * out[n0 + i]) * (T)(1.0 / 6.0) : u + dte * out[n0 + i];
          un_[(n0 + i) * SN] = un;
          out[n0 + i] = x2[i] - un;
        }
    }
  }
};

// A tile's RK operands towards L2.
template <class C, typename T>
__device__ __forceinline__ void prefetch_operands(const StageArgs<T>& a, int64_t tile) {
  if (a.stage == 0) return;
  if (a.u != a.y_in) prefetch_l2(a.u + tile * C::TW, C::YB);
  if (a.stage >= 2 && a.stage <= 4) prefetch_l2(a.acc + tile * C::TW, C::YB);
  if (a.stage >= 4) prefetch_l2(a.snap + tile * C::TW, C::YB);
}

// constants in the working precision (FP32: rounded on the host, a conversion
// per thread and tile runs at the FP64 rate)
template <typename T>
__device__ __forceinline__ T bb_rhoc2(const StageArgs<T>& a) {
  if constexpr (sizeof(T) == 4) return a.f_rhoc2; else return a.ph.rhoc2;
}
template <typename T>
__device__ __forceinline__ T bb_inv_rho0(const StageArgs<T>& a) {
  if constexpr (sizeof(T) == 4) return a.f_inv_rho0; else return a.ph.inv_rho0;
}
template <typename T>
__device__ __forceinline__ T bb_dt(const StageArgs<T>& a) {
  if constexpr (sizeof(T) == 4) return a.f_dt; else return a.dt;
}

// One tile: y, g, gi at this lane in shared memory; env: BBGlobalEnv, or what
// keeps the RK arrays elsewhere. False when env's barrier said to stop.
template <class C, typename T, class Env>
__device__ __forceinline__ bool bb_tile(const StageArgs<T>& a, Env& env, int64_t tile, const T* y, const T* g,
                                        const int* gi, const int* sFm, const unsigned char* sNb, T* sN, int lane,
                                        int role, BBRes<T>& racc) {
  constexpr int NP = C::NP, NF = C::NF, NFP = C::NFP, NV = C::NV, LW = C::LW, D = C::D;
  const T rhoc2 = bb_rhoc2<T>(a), inv_rho0 = bb_inv_rho0<T>(a);
  // ---- this face's neighbour trace ----
  const int nbr = gi[role * LW], code = gi[(NF + role) * LW];
  const bool boundary = code & kCodeBoundary;
  const bool in_tile = boundary || (nbr >> 5) == tile;
  T up[NV][NFP];
  T* sf = sN + role * NV * NFP * LW + lane;  // this thread's face data
  auto trace = [&]() {
    const int slot = (code & kCodeLfMask) * C::NPERM + ((code >> kCodePermShift) & kCodePermMask);
    uint32_t w[4];
    *reinterpret_cast<uint4*>(w) = *reinterpret_cast<const uint4*>(sNb + (boundary ? 0 : slot) * 16);
    env.template gather<NFP>(in_tile, y - lane + (boundary ? lane : (nbr & 31)),
                             (int64_t)(nbr >> 5) * C::TW + (nbr & 31), w, up);
  };
  if constexpr (!Env::kTraceLast) trace();
  // ---- this variable's volume term ----
  T out[NP];
  bb_volume<C>(y, g, role, rhoc2, inv_rho0, out);
  if constexpr (Env::kTraceLast) trace();
  // ---- this face's flux ----
  {
    const T* gf = g + role * (D + 1) * LW;
    T np_[D], nu_[D];
#pragma unroll
    for (int d = 0; d < D; ++d) np_[d] = rhoc2 * gf[d * LW], nu_[d] = inv_rho0 * gf[d * LW];
    const T A = gf[D * LW];
    const int* fm = sFm + role * 16;
    if (boundary) {
      const T* Bg = a.bbM + (int64_t)nbr * NV * NV;
#pragma unroll
      for (int m = 0; m < NFP; ++m) {
        T um[NV];
#pragma unroll
        for (int q = 0; q < NV; ++q) um[q] = y[q * NP * LW + fm[m]];
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          T s = (T)0;
#pragma unroll
          for (int qq = 0; qq < NV; ++qq) s += __ldg(Bg + q * NV + qq) * um[qq];
          up[q][m] = s;
        }
      }
    } else {
#pragma unroll
      for (int m = 0; m < NFP; ++m) {
        T d[NV];
#pragma unroll
        for (int q = 0; q < NV; ++q) d[q] = y[q * NP * LW + fm[m]] - up[q][m];
        T s = A * d[0];
#pragma unroll
        for (int k = 0; k < D; ++k) s += np_[k] * d[1 + k];
        up[0][m] = s;
#pragma unroll
        for (int k = 0; k < D; ++k) up[1 + k][m] = A * d[1 + k] + nu_[k] * d[0];
      }
    }
#pragma unroll
    for (int q = 0; q < NV; ++q) bb_face_stencil<C>(up[q], sf + q * NFP * LW);
  }
  const T dte = bb_dt<T>(a) * g[C::oS * LW];
  if (!env.sync()) return false;
  // ---- this variable's lift and RK update ----
  env.load(0);
  bb_lift<C, NV * NFP * LW, LW>(sN + role * NFP * LW + lane, out);
#pragma unroll
  for (int n0 = 0; n0 < NP; n0 += C::CH) {
    if (n0 > 0) env.load(n0);
    env.update(n0, dte, out);
  }
  if (env.residual()) racc.template add<C>(out);
  return true;
}

// ---- FP64: fixed-point lift and elevation --------------------------------------
//
// GB300 runs 2 FP64 operations per clock and SM, but 128 integer ones. L0, the
// layers of the lift and the degree elevation are combinations with small
// integer weights, so FP64 kernels take them in 64-bit integers: the values
// that enter (a face's fluxes, the gradient's coefficients) are rounded to 53
// bits below the largest exponent among them, every sum is exact but for the
// layers' divisions by 2, 3, 4 and 5 and the alignment of the faces' scales,
// and the result is rounded to FP64 once. Weights grow a value by at most
// (P+1)(P+3) in L0, 5 in the layers and 4 over the faces, 2^9.5 at P = 4, which
// leaves the sign bit. An infinity or NaN makes the whole sum a NaN. 3-D p = 3:
// 180 FP64 operations per thread (with the gradient, see fx_gradient) instead of
// 740.

__device__ __forceinline__ int fx_exponent(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }

// x as a multiple of 2^(E - 1075), E at least its biased exponent, rounded to
// nearest: at most 2^53 in size.
__device__ __forceinline__ long long fx_fix(double x, int E) {
  const int hi = __double2hiint(x), e = (hi >> 20) & 0x7ff;
  unsigned long long m =
      ((unsigned long long)(((unsigned)hi & 0xfffffu) | 0x100000u) << 32) | (unsigned)__double2loint(x);
  if (e == 0) m = 0;  // zero, and subnormal values far below any scale
  const int s = min(E - e, 63);
  m = (m + ((1ull << s) >> 1)) >> s;
  return hi < 0 ? -(long long)m : (long long)m;
}
// v 2^-d, rounded to nearest
__device__ __forceinline__ long long fx_shift(long long v, int d) {
  const int s = min(d, 62);
  return (v + ((1ll << s) >> 1)) >> s;
}
// v rounded to FP64, put together from its bits (two FP64 additions would take
// four times as long)
__device__ __forceinline__ double fx_double(long long v) {
  const unsigned long long m0 = (unsigned long long)(v < 0 ? -v : v);
  const int z = __clzll(m0);
  const unsigned long long m = m0 << (z & 63);
  // 53 bits, rounded; the leading one and a carry add to the exponent
  const unsigned long long b = ((unsigned long long)(1085 - z) << 52) + (m >> 11) + ((m >> 10) & 1);
  return v == 0 ? 0.0 : __longlong_as_double((long long)(b | ((unsigned long long)v & 0x8000000000000000ull)));
}
// 2^(E - 1075); NaN for the exponent of infinities and NaNs. E >= 54.
__device__ __forceinline__ double fx_scale(int E) {
  // 2^(E - 1075) = 2^(E - 1023 - 52): exponent field E - 52
  return E == 0x7ff ? __hiloint2double(0x7ff80000, 0) : __hiloint2double((E - 52) << 20, 0);
}
constexpr int kFxMinExp = 64;  // scales below 2^-1011 are not resolved

template <class C, int M>
__device__ __forceinline__ long long fx_stencil_at(const long long (&f)[C::NFP]) {
  constexpr int D = C::D, P = C::P;
  using L = BLat<D - 1, P, M>;
  constexpr int w0 = (L::b.a[0] + 1) * (L::b.a[0] + 1) + (L::b.a[1] + 1) * (L::b.a[1] + 1) +
                     (D == 3 ? (L::b.a[2] + 1) * (L::b.a[2] + 1) : 0);
  long long s = (long long)w0 * f[M];
  bb_for<D * D>([&](auto ij_) {
    constexpr int i = decltype(ij_)::value / D, j = decltype(ij_)::value % D;
    if constexpr (i != j && L::b.a[j] > 0) {
      constexpr int n = bb_index(D - 1, P, bb_add(bb_add(L::b, i, 1), j, -1));
      constexpr int w = (L::b.a[i] + 1) * L::b.a[j];
      s += (long long)w * f[n];
    }
  });
  return s;
}

// v / N rounded (N = 2, 3, 4, 5)
template <int N>
__device__ __forceinline__ long long fx_div(long long v) {
  if constexpr (N == 2) return (v + 1) >> 1;
  else if constexpr (N == 4) return (v + 2) >> 2;
  else return __mul64hi(v + N / 2, N == 3 ? 0x5555555555555556ll : 0x3333333333333334ll);
}

// Adds layers J .. P of face F's lift to out (bb_layers in integers).
template <class C, int F, int J>
__device__ __forceinline__ void fx_layers(const long long (&prev)[bb_np(C::D - 1, C::P - J + 1)],
                                          long long (&out)[C::NP]) {
  constexpr int D = C::D, P = C::P;
  if constexpr (J <= P) {
    long long cur[bb_np(D - 1, P - J)];
    bb_for<bb_np(D - 1, P - J)>([&](auto g_) {
      using L = BLat<D - 1, P - J, decltype(g_)::value>;
      long long s = 0;
      bb_for<D>([&](auto k_) {
        constexpr int k = decltype(k_)::value;
        constexpr int n = bb_index(D - 1, P - J + 1, bb_add(L::b, k, 1));
        constexpr int w = L::b.a[k] + 1;
        s -= (long long)w * prev[n];
      });
      s = fx_div<J + 1>(s);
      cur[decltype(g_)::value] = s;
      constexpr int a = bb_layer_index(D, P, F, J, L::b);
      out[a] += s;
    });
    if constexpr (J < P) fx_layers<C, F, J + 1>(cur, out);
  }
}

// The gradient's coefficients t (degree P-1) of variable q's volume term: the
// volume term is -elevation(t) (bb_volume without the elevation).
template <class C>
__device__ __forceinline__ void fp64_gradient(const double* y, const double* g, int q, double rhoc2, double inv_rho0,
                                              double (&t)[bb_np(C::D, C::P - 1)]) {
  constexpr int D = C::D, P = C::P, NP = C::NP, LW = C::LW;
  BBGrad<double, D> gv;
#pragma unroll
  for (int r = 0; r < D; ++r) gv.g[r] = g[(C::oGV + r) * LW];
  gv.done();
  BBGrad<double, D> gm[D];
  if (q == 0) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
#pragma unroll
      for (int r = 0; r < D; ++r) gm[d].g[r] = rhoc2 * g[(C::oG + r * D + d) * LW];
      gm[d].done();
    }
  } else {
#pragma unroll
    for (int r = 0; r < D; ++r) gm[0].g[r] = inv_rho0 * g[(C::oG + r * D + q - 1) * LW];
    gm[0].done();
  }
  const double* yq = y + q * NP * LW;
  bb_for<bb_np(D, P - 1)>([&](auto b_) {
    using L = BLat<D, P - 1, decltype(b_)::value>;
    constexpr int n0 = bb_index(D, P, bb_add(L::b, 0, 1)), n1 = bb_index(D, P, bb_add(L::b, 1, 1)),
                  n2 = bb_index(D, P, bb_add(L::b, 2, 1)), n3 = D == 3 ? bb_index(D, P, bb_add(L::b, 3, 1)) : 0;
    double s = gv.template add<n0, n1, n2, n3, LW>(0.0, yq);
    if (q == 0) {
#pragma unroll
      for (int d = 0; d < D; ++d) s = gm[d].template add<n0, n1, n2, n3, LW>(s, y + (1 + d) * NP * LW);
    } else {
      s = gm[0].template add<n0, n1, n2, n3, LW>(s, y);
    }
    t[decltype(b_)::value] = s;
  });
}

// A fixed-point value as two digits, hi 2^29 + lo, both of its sign: sums and
// differences are taken digit by digit, and a product is three 32-bit
// multiply-adds (that of the low digits, 2^-57 of the largest, is left out).
struct FxDigits {
  int hi, lo;
};
// x as a multiple of 2^(E - 1075 - X), below 2^(53 + X) in size
template <int X>
__device__ __forceinline__ FxDigits fx_digits(double x, int E) {
  const int h = __double2hiint(x), e = (h >> 20) & 0x7ff;
  unsigned long long m =
      ((unsigned long long)(((unsigned)h & 0xfffffu) | 0x100000u) << 32) | (unsigned)__double2loint(x);
  if (e == 0) m = 0;
  m = (m << X) >> min(E - e, 63);
  const FxDigits d{(int)(m >> 29), (int)((unsigned)m & 0x1fffffffu)};
  return h < 0 ? FxDigits{-d.hi, -d.lo} : d;
}
// v 2^-d rounded, d of either sign (the caller's value has room to grow)
__device__ __forceinline__ long long fx_scaled(long long v, int d) { return d >= 0 ? fx_shift(v, d) : v << min(-d, 62); }

template <bool FXG>
struct FxPick {
  using type = double;
};
template <>
struct FxPick<true> {
  using type = long long;
};
// The biased exponent that covers values v in units of 2^U, E at least.
template <int N>
__device__ __forceinline__ int fx_top(const long long (&v)[N], int U, int E) {
  unsigned long long m = 0;
#pragma unroll
  for (int n = 0; n < N; ++n) m |= (unsigned long long)(v[n] < 0 ? -v[n] : v[n]);
  return m == 0 ? E : min(max(E, U + 64 - __clzll((long long)m) + 1022), 0x7ff);
}
__device__ __forceinline__ int fx_size(double x) { return __double2hiint(x) & 0x7fffffff; }
__device__ __forceinline__ int fx_group(int m) { return max(m >> 20, kFxMinExp); }  // exponent of the largest fx_size
// The unit of products of state digits (exponent Ey) and metric digits (Eg).
__device__ __forceinline__ int fx_unit(int Ey, int Eg) { return Ey - 1079 + Eg - 1080 + 58; }
// A sum of products of digits.
struct FxSum {
  long long hh = 0, tt = 0;
  __device__ __forceinline__ void add(const FxDigits& d, const FxDigits& g) {
    hh += (long long)d.hi * g.hi;
    tt += (long long)d.hi * g.lo + (long long)d.lo * g.hi;
  }
  __device__ __forceinline__ long long get() const { return hh + ((tt + (1 << 28)) >> 29); }
};

// The gradient's coefficients t (degree P-1) of variable q's volume term, in
// units of 2^U: the volume term is -elevation(t) (bb_volume without the
// elevation). bad: an infinity or NaN among the inputs.
//
// In fixed point too: a variable's coefficients take 57 bits below the largest
// exponent among its own in the element, a metric column 58, so that sums of nine
// products of coefficient differences stay below 2^63. (One scale for all three
// velocity components, and one for the whole metric, let the component along the
// long sides of a thin element drown the one across it: 4.9e-15 in place of 4e-16
// in the pressure's right-hand side at 1000 : 1.) A multiply-add takes an
// SM sub-partition 64 cycles in FP64 and some 10 here, a conversion some 30. us
// per step: 24,576 tetrahedra of order 3 374 -> 327, 48,000 of order 2 352 -> 292,
// 48,000 of order 1 155 -> 142, 7,722 of order 2 67 -> 62.
template <class C>
__device__ __forceinline__ void fx_gradient(const double* y, const double* g, int q, double rhoc2, double inv_rho0,
                                            long long (&t)[bb_np(C::D, C::P - 1)], int& U, bool& bad) {
  constexpr int D = C::D, P = C::P, NP = C::NP, LW = C::LW, NB = bb_np(D, P - 1);
  auto top = [&](const double* c, int m) {
#pragma unroll
    for (int n = 0; n < NP; ++n) m = max(m, fx_size(c[n * LW]));
    return m;
  };
  FxSum sum[NB];
  // adds sum_r G_r (c[b + e_r] - c[b + e_0]) of one variable's coefficients
  auto add = [&](const double* v, int E, const FxDigits (&G)[D]) {
    FxDigits c[NP];
#pragma unroll
    for (int n = 0; n < NP; ++n) c[n] = fx_digits<4>(v[n * LW], E);
    bb_for<NB>([&](auto b_) {
      constexpr int b = decltype(b_)::value;
      using L = BLat<D, P - 1, b>;
      constexpr int n0 = bb_index(D, P, bb_add(L::b, 0, 1));
      bb_for<D>([&](auto r_) {
        constexpr int r = decltype(r_)::value;
        constexpr int n = bb_index(D, P, bb_add(L::b, r + 1, 1));
        sum[b].add(FxDigits{c[n].hi - c[n0].hi, c[n].lo - c[n0].lo}, G[r]);
      });
    });
  };
  // this variable along the mean flow
  FxDigits G[D];
  int m = 0;
#pragma unroll
  for (int r = 0; r < D; ++r) m = max(m, fx_size(g[(C::oGV + r) * LW]));
  const int Ev = fx_group(m), Ey = fx_group(top(y + q * NP * LW, 0));
#pragma unroll
  for (int r = 0; r < D; ++r) G[r] = fx_digits<5>(g[(C::oGV + r) * LW], Ev);
  add(y + q * NP * LW, Ey, G);
#pragma unroll
  for (int b = 0; b < NB; ++b) t[b] = sum[b].get(), sum[b] = FxSum();
  // the velocity's divergence, or the pressure's derivative: every component at
  // the scale of its own values and of its own metric column
  const int nv = q == 0 ? D : 1;
  const double scale = q == 0 ? rhoc2 : inv_rho0;
  auto metric = [&](int v, int r) { return scale * g[(C::oG + r * D + (q == 0 ? v : q - 1)) * LW]; };
  const int U1 = fx_unit(Ey, Ev);
  U = U1;
  bad = max(Ey, Ev) == 0x7ff;
  int Eo[3] = {}, Eg[3] = {};
#pragma unroll
  for (int v = 0; v < D; ++v)
    if (v < nv) {
      m = 0;
#pragma unroll
      for (int r = 0; r < D; ++r) m = max(m, fx_size(metric(v, r)));
      Eo[v] = fx_group(top(y + (q == 0 ? 1 + v : 0) * NP * LW, 0)), Eg[v] = fx_group(m);
      U = max(U, fx_unit(Eo[v], Eg[v]));
      bad |= max(Eo[v], Eg[v]) == 0x7ff;
    }
#pragma unroll
  for (int b = 0; b < NB; ++b) t[b] = fx_shift(t[b], U - U1);
#pragma unroll 1
  for (int v = 0; v < nv; ++v) {
    const int eo = v == 0 ? Eo[0] : v == 1 ? Eo[1] : Eo[2], eg = v == 0 ? Eg[0] : v == 1 ? Eg[1] : Eg[2];
    const int d = U - fx_unit(eo, eg);
#pragma unroll
    for (int r = 0; r < D; ++r) G[r] = fx_digits<5>(metric(v, r), eg);
    add(y + (q == 0 ? 1 + v : 0) * NP * LW, eo, G);
#pragma unroll
    for (int b = 0; b < NB; ++b) t[b] += fx_shift(sum[b].get(), d), sum[b] = FxSum();
  }
}

// One tile of an FP64 state (see above): bb_tile with fluxes and gradient in
// FP64, stencil, lift and elevation in fixed point. sN holds the faces'
// stencil results as integers, sX [NF][NV][32] their exponents.
template <class C, class Env>
__device__ __forceinline__ bool bb_tile_fx(const StageArgs<double>& a, Env& env, int64_t tile, const double* y,
                                           const double* g, const int* gi, const int* sFm, const unsigned char* sNb,
                                           long long* sN, int* sX, int lane, int role, BBRes<double>& racc) {
  constexpr int NP = C::NP, NF = C::NF, NFP = C::NFP, NV = C::NV, LW = C::LW, D = C::D, P = C::P;
  const double rhoc2 = a.ph.rhoc2, inv_rho0 = a.ph.inv_rho0;
  // ---- this face's neighbour trace ----
  const int nbr = gi[role * LW], code = gi[(NF + role) * LW];
  const bool boundary = code & kCodeBoundary;
  const bool in_tile = boundary || (nbr >> 5) == tile;
  double up[NV][NFP];
  auto trace = [&]() {
    const int slot = (code & kCodeLfMask) * C::NPERM + ((code >> kCodePermShift) & kCodePermMask);
    uint32_t w[4];
    *reinterpret_cast<uint4*>(w) = *reinterpret_cast<const uint4*>(sNb + (boundary ? 0 : slot) * 16);
    env.template gather<NFP>(in_tile, y - lane + (boundary ? lane : (nbr & 31)),
                             (int64_t)(nbr >> 5) * C::TW + (nbr & 31), w, up);
  };
  if constexpr (!Env::kTraceLast) trace();
  // boundary faces' coefficients, before they are needed
  const bool any_boundary = __any_sync(0xffffffffu, boundary);
  const bool plain_boundary = !__any_sync(0xffffffffu, boundary && !(code & kCodePlainBoundary));
  double bc[5] = {};
  if (any_boundary && plain_boundary) {
    bc[0] = bc[3] = g[(role * (D + 1) + D) * LW], bc[1] = rhoc2, bc[2] = inv_rho0, bc[4] = 0.0;
    if (boundary)
#pragma unroll
      for (int i = 0; i < 5; ++i) bc[i] = __ldg(a.bbC + (int64_t)nbr * 8 + i);
  }
  // ---- this variable's gradient ----
  using Grad = typename FxPick<C::FXG>::type;
  Grad t[bb_np(D, P - 1)];
  int tU = 0;
  bool bad = false;
  if constexpr (C::FXG)
    fx_gradient<C>(y, g, role, rhoc2, inv_rho0, t, tU, bad);
  else
    fp64_gradient<C>(y, g, role, rhoc2, inv_rho0, t);
  if constexpr (Env::kTraceLast) trace();
  // ---- this face's flux ----
  {
    const double* gf = g + role * (D + 1) * LW;
    double np_[D], nu_[D];
#pragma unroll
    for (int d = 0; d < D; ++d) np_[d] = rhoc2 * gf[d * LW], nu_[d] = inv_rho0 * gf[d * LW];
    const double A = gf[D * LW];
    const int* fm = sFm + role * 16;
    if (any_boundary && plain_boundary) {
      // interior faces and walls in one form (k_bb_geo): 17 FP64 operations per
      // node in 3-D, where a branch each would take 14 and 16
#pragma unroll
      for (int m = 0; m < NFP; ++m) {
        double d[NV];
#pragma unroll
        for (int q = 0; q < NV; ++q) d[q] = y[q * NP * LW + fm[m]] - (boundary ? 0.0 : up[q][m]);
        double s = gf[0] * d[1];
#pragma unroll
        for (int k = 1; k < D; ++k) s += gf[k * LW] * d[1 + k];
        up[0][m] = bc[0] * d[0] + bc[1] * s;
        const double r = bc[2] * d[0] + bc[4] * s;
#pragma unroll
        for (int k = 0; k < D; ++k) up[1 + k][m] = bc[3] * d[1 + k] + gf[k * LW] * r;
      }
    } else if (boundary) {
      const double* Bg = a.bbM + (int64_t)nbr * NV * NV;
#pragma unroll
      for (int m = 0; m < NFP; ++m) {
        double um[NV];
#pragma unroll
        for (int q = 0; q < NV; ++q) um[q] = y[q * NP * LW + fm[m]];
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          double s = 0.0;
#pragma unroll
          for (int qq = 0; qq < NV; ++qq) s += __ldg(Bg + q * NV + qq) * um[qq];
          up[q][m] = s;
        }
      }
    } else {
#pragma unroll
      for (int m = 0; m < NFP; ++m) {
        double d[NV];
#pragma unroll
        for (int q = 0; q < NV; ++q) d[q] = y[q * NP * LW + fm[m]] - up[q][m];
        double s = A * d[0];
#pragma unroll
        for (int k = 0; k < D; ++k) s += np_[k] * d[1 + k];
        up[0][m] = s;
#pragma unroll
        for (int k = 0; k < D; ++k) up[1 + k][m] = A * d[1 + k] + nu_[k] * d[0];
      }
    }
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      int E = kFxMinExp;
#pragma unroll
      for (int m = 0; m < NFP; ++m) E = max(E, fx_exponent(up[q][m]));
      long long f[NFP];
#pragma unroll
      for (int m = 0; m < NFP; ++m) f[m] = fx_fix(up[q][m], E);
      long long* sf = sN + (role * NV + q) * NFP * LW + lane;
      bb_for<NFP>([&](auto m_) { sf[decltype(m_)::value * LW] = fx_stencil_at<C, decltype(m_)::value>(f); });
      sX[(role * NV + q) * LW + lane] = E;
    }
  }
  const double dte = a.dt * g[C::oS * LW];
  if (!env.sync()) return false;
  // ---- this variable's elevation and lift ----
  env.load(0);
  int E = kFxMinExp, ef[NF];
#pragma unroll
  for (int f = 0; f < NF; ++f) ef[f] = sX[(f * NV + role) * LW + lane], E = max(E, ef[f]);
  if constexpr (C::FXG) {
    E = bad ? 0x7ff : fx_top(t, tU, E);
  } else {
#pragma unroll
    for (int b = 0; b < bb_np(D, P - 1); ++b) E = max(E, fx_exponent(t[b]));
  }
  long long acc[NP];
#pragma unroll
  for (int n = 0; n < NP; ++n) acc[n] = 0;
  bb_for<bb_np(D, P - 1)>([&](auto b_) {
    using L = BLat<D, P - 1, decltype(b_)::value>;
    long long v;
    if constexpr (C::FXG)
      v = fx_scaled(t[decltype(b_)::value], E - 1075 - tU);
    else
      v = fx_fix(t[decltype(b_)::value], E);
    bb_for<D + 1>([&](auto k_) {
      constexpr int k = decltype(k_)::value;
      constexpr int n = bb_index(D, P, bb_add(L::b, k, 1));
      constexpr int w = L::b.a[k] + 1;
      acc[n] -= (long long)w * v;
    });
  });
  bb_for<NF>([&](auto f_) {
    constexpr int f = decltype(f_)::value;
    long long l0[NFP];
#pragma unroll
    for (int m = 0; m < NFP; ++m) l0[m] = fx_shift(sN[((f * NV + role) * NFP + m) * LW + lane], E - ef[f]);
    bb_for<NFP>([&](auto m_) {
      constexpr int n = bb_layer_index(D, P, f, 0, bb_lattice(D - 1, P, decltype(m_)::value));
      acc[n] += l0[decltype(m_)::value];
    });
    fx_layers<C, f, 1>(l0, acc);
  });
  // ---- RK update: dt L is acc in units of dt 2^(E - 1075) ----
  double out[NP];
#pragma unroll
  for (int n = 0; n < NP; ++n) out[n] = fx_double(acc[n]);
  const double unit = dte * fx_scale(E);
#pragma unroll
  for (int n0 = 0; n0 < NP; n0 += C::CH) {
    if (n0 > 0) env.load(n0);
    env.update(n0, unit, out);
  }
  if (env.residual()) racc.template add<C>(out);
  return true;
}

// One tile in the Q4 layout (FP32, 3-D). The flux phase is bb_tile's (a warp
// per face, a lane per element) with all variables of a node in one 16-byte
// load: the neighbour trace touches two elements' values per sector instead
// of one value of eight, and takes a quarter of the load instructions. In the
// volume, lift and update phases thread t is variable t & 3 of element t >> 2,
// so that a coefficient of the tile is one contiguous row of the block; the
// coupling of the variables goes through shuffles within an element's four
// lanes (every lane forms t_j = H_j . D u with H_j the metric column that its
// neighbour lane ^ (j+1) needs, zero where it needs none).
template <class C, class Env>
__device__ __forceinline__ bool bb_tile_q4(const StageArgs<float>& a, Env& env, int64_t tile, const float* y,
                                           const float* g, const int* gi, const int* sFm, const unsigned char* sNb,
                                           float* sN, int tid, int role, BBRes<float>& racc) {
  constexpr int NP = C::NP, NF = C::NF, NFP = C::NFP, LW = C::LW, D = C::D, P = C::P, SN = C::SN;
  const float rhoc2 = a.f_rhoc2, inv_rho0 = a.f_inv_rho0;
  const int lane = tid & 31;
  // ---- this face's neighbour trace ----
  const int nbr = gi[role * LW + lane], code = gi[(NF + role) * LW + lane];
  const bool boundary = code & kCodeBoundary;
  const bool in_tile = boundary || (nbr >> 5) == tile;
  float4 up[NFP];
  auto trace = [&]() {
    const int slot = (code & kCodeLfMask) * C::NPERM + ((code >> kCodePermShift) & kCodePermMask);
    uint32_t w[4];
    *reinterpret_cast<uint4*>(w) = *reinterpret_cast<const uint4*>(sNb + (boundary ? 0 : slot) * 16);
    env.template gather<NFP>(in_tile, y + 4 * (boundary ? lane : (nbr & 31)),
                             (int64_t)(nbr >> 5) * C::TW + 4 * (nbr & 31), w, up);
  };
  if constexpr (!Env::kTraceLast) trace();
  // ---- volume term of this thread's variable q of element el ----
  const int q = tid & 3, el = tid >> 2;
  float out[NP];
  {
    float gv[3], H[3][3];
    float2 h01[3], h2v[3];  // PACK2: (H_0, H_1) and (H_2, the metric along the mean flow)
#pragma unroll
    for (int r = 0; r < 3; ++r) gv[r] = g[(C::oGV + r) * LW + el];
#pragma unroll
    for (int j = 0; j < 3; ++j)
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        const float x = g[(C::oG + r * D + j) * LW + el];
        H[j][r] = q == 0 ? inv_rho0 * x : q == j + 1 ? rhoc2 * x : 0.f;
      }
    if constexpr (C::PACK2)
#pragma unroll
      for (int r = 0; r < 3; ++r) h01[r] = make_float2(H[0][r], H[1][r]), h2v[r] = make_float2(H[2][r], gv[r]);
#pragma unroll
    for (int n = 0; n < NP; ++n) out[n] = 0.f;
    const float* yq = y + tid;
    bb_for<bb_np(D, P - 1)>([&](auto b_) {
      using L = BLat<D, P - 1, decltype(b_)::value>;
      constexpr int n0 = bb_index(D, P, bb_add(L::b, 0, 1)), n1 = bb_index(D, P, bb_add(L::b, 1, 1)),
                    n2 = bb_index(D, P, bb_add(L::b, 2, 1)), n3 = bb_index(D, P, bb_add(L::b, 3, 1));
      const float c0 = yq[n0 * SN], d1 = yq[n1 * SN] - c0, d2 = yq[n2 * SN] - c0, d3 = yq[n3 * SN] - c0;
      float t;
      if constexpr (C::PACK2) {
        const float2 e1 = make_float2(d1, d1), e2 = make_float2(d2, d2), e3 = make_float2(d3, d3);
        const float2 a01 = __ffma2_rn(h01[2], e3, __ffma2_rn(h01[1], e2, __fmul2_rn(h01[0], e1)));
        const float2 a2v = __ffma2_rn(h2v[2], e3, __ffma2_rn(h2v[1], e2, __fmul2_rn(h2v[0], e1)));
        t = a2v.y;
        t += __shfl_xor_sync(0xffffffffu, a01.x, 1);
        t += __shfl_xor_sync(0xffffffffu, a01.y, 2);
        t += __shfl_xor_sync(0xffffffffu, a2v.x, 3);
      } else {
        t = gv[0] * d1 + gv[1] * d2 + gv[2] * d3;
#pragma unroll
        for (int j = 0; j < 3; ++j)
          t += __shfl_xor_sync(0xffffffffu, H[j][0] * d1 + H[j][1] * d2 + H[j][2] * d3, j + 1);
      }
      bb_for<D + 1>([&](auto k_) {
        constexpr int k = decltype(k_)::value;
        constexpr int n = bb_index(D, P, bb_add(L::b, k, 1));
        constexpr int w = L::b.a[k] + 1;
        out[n] -= (float)w * t;
      });
    });
  }
  if constexpr (Env::kTraceLast) trace();
  // ---- this face's flux ----
  {
    const float* gf = g + role * (D + 1) * LW + lane;
    const int* fm = sFm + role * 16;
    if constexpr (C::PACK2) {
      float2 f01[NFP], f23[NFP];
      const float* yl = y + 4 * lane;
      if (boundary) {
        const float* Bg = a.bbM + (int64_t)nbr * 16;
#pragma unroll
        for (int m = 0; m < NFP; ++m) {
          const float4 um = *reinterpret_cast<const float4*>(yl + fm[m]);
          float f[4];
#pragma unroll
          for (int v = 0; v < 4; ++v)
            f[v] = __ldg(Bg + v * 4) * um.x + __ldg(Bg + v * 4 + 1) * um.y + __ldg(Bg + v * 4 + 2) * um.z +
                   __ldg(Bg + v * 4 + 3) * um.w;
          f01[m] = make_float2(f[0], f[1]), f23[m] = make_float2(f[2], f[3]);
        }
      } else {
        const float A = gf[D * LW], n0 = gf[0], n1 = gf[LW], n2 = gf[2 * LW];
        const float p0 = rhoc2 * n0, p1 = rhoc2 * n1, p2 = rhoc2 * n2;
        const float2 A2 = make_float2(A, A), c01 = make_float2(p0, inv_rho0 * n0),
                     u12 = make_float2(inv_rho0 * n1, inv_rho0 * n2), neg = make_float2(-1.f, -1.f);
#pragma unroll
        for (int m = 0; m < NFP; ++m) {
          const float4 um = *reinterpret_cast<const float4*>(yl + fm[m]);
          const float2 d01 = __ffma2_rn(neg, make_float2(up[m].x, up[m].y), make_float2(um.x, um.y));
          const float2 d23 = __ffma2_rn(neg, make_float2(up[m].z, up[m].w), make_float2(um.z, um.w));
          f01[m] = __ffma2_rn(c01, make_float2(d01.y, d01.x), __fmul2_rn(A2, d01));
          f01[m].x += p1 * d23.x + p2 * d23.y;
          f23[m] = __ffma2_rn(u12, make_float2(d01.x, d01.x), __fmul2_rn(A2, d23));
        }
      }
      float* sf = sN + role * NFP * SN + 4 * lane;
      bb_for<NFP>([&](auto m_) {
        constexpr int m = decltype(m_)::value;
        const float2 s01 = bb_stencil_at<C, m>(f01), s23 = bb_stencil_at<C, m>(f23);
        *reinterpret_cast<float4*>(sf + m * SN) = make_float4(s01.x, s01.y, s23.x, s23.y);
      });
    } else {
      float f[4][NFP];
      const float* yl = y + 4 * lane;
      if (boundary) {
        const float* Bg = a.bbM + (int64_t)nbr * 16;
#pragma unroll
        for (int m = 0; m < NFP; ++m) {
          const float4 um = *reinterpret_cast<const float4*>(yl + fm[m]);
#pragma unroll
          for (int v = 0; v < 4; ++v)
            f[v][m] = __ldg(Bg + v * 4) * um.x + __ldg(Bg + v * 4 + 1) * um.y + __ldg(Bg + v * 4 + 2) * um.z +
                      __ldg(Bg + v * 4 + 3) * um.w;
        }
      } else {
        const float A = gf[D * LW], n0 = gf[0], n1 = gf[LW], n2 = gf[2 * LW];
        const float p0 = rhoc2 * n0, p1 = rhoc2 * n1, p2 = rhoc2 * n2;
        const float u0 = inv_rho0 * n0, u1 = inv_rho0 * n1, u2 = inv_rho0 * n2;
#pragma unroll
        for (int m = 0; m < NFP; ++m) {
          const float4 um = *reinterpret_cast<const float4*>(yl + fm[m]);
          const float dp = um.x - up[m].x, dx = um.y - up[m].y, dy = um.z - up[m].z, dz = um.w - up[m].w;
          f[0][m] = A * dp + p0 * dx + p1 * dy + p2 * dz;
          f[1][m] = A * dx + u0 * dp;
          f[2][m] = A * dy + u1 * dp;
          f[3][m] = A * dz + u2 * dp;
        }
      }
      float* sf = sN + role * NFP * SN + 4 * lane;
      bb_for<NFP>([&](auto m_) {
        constexpr int m = decltype(m_)::value;
        *reinterpret_cast<float4*>(sf + m * SN) =
            make_float4(bb_stencil_at<C, m>(f[0]), bb_stencil_at<C, m>(f[1]), bb_stencil_at<C, m>(f[2]),
                        bb_stencil_at<C, m>(f[3]));
      });
    }
  }
  const float dte = a.f_dt * g[C::oS * LW + el];
  if (!env.sync()) return false;
  // ---- this variable's lift and RK update ----
  env.load(0);
  bb_lift<C, NFP * SN, SN>(sN + tid, out);
#pragma unroll
  for (int n0 = 0; n0 < NP; n0 += C::CH) {
    if (n0 > 0) env.load(n0);
    env.update(n0, dte, out);
  }
  if (env.residual()) racc.template add<C>(out);
  return true;
}

// The tile body of configuration C (y, g, gi: the tile's buffers).
template <class C, class Env, typename T>
__device__ __forceinline__ bool bb_tile_any(const StageArgs<T>& a, Env& env, int64_t tile, const T* y, const T* g,
                                            const int* gi, const int* sFm, const unsigned char* sNb, T* sN, int* sX,
                                            int tid, int role, BBRes<T>& racc) {
  const int lane = tid & 31;
  if constexpr (C::Q4)
    return bb_tile_q4<C>(a, env, tile, y, g, gi, sFm, sNb, sN, tid, role, racc);
  else if constexpr (C::FX)
    return bb_tile_fx<C>(a, env, tile, y + lane, g + lane, gi + lane, sFm, sNb, reinterpret_cast<long long*>(sN), sX,
                         lane, role, racc);
  else
    return bb_tile<C, T>(a, env, tile, y + lane, g + lane, gi + lane, sFm, sNb, sN, lane, role, racc);
}

// Face tables in shared memory: element word offset of each face node, and
// the neighbour's node for each (its local face, corner permutation).
template <class C, typename T>
__device__ __forceinline__ void bb_load_tables(const StageArgs<T>& a, int* sFm, unsigned char* sNb, int tid, int nt) {
  for (int i = tid; i < C::NF * 16; i += nt)
    sFm[i] = i % 16 < C::NFP ? (int)a.fmask[i / 16 * C::NFP + i % 16] * C::SN : 0;
  for (int i = tid; i < C::NF * C::NPERM * 16; i += nt)
    sNb[i] = i % 16 < C::NFP ? (unsigned char)a.nbrnode[i / 16 * C::NFP + i % 16] : (unsigned char)0;
}

template <typename T, int D, int P, int NBUF, int MINB>
__global__ void __launch_bounds__(BBCfg<T, D, P, NBUF, MINB>::NT, MINB) stage_bb_kernel(const StageArgs<T> a, int* err) {
  using C = BBCfg<T, D, P, NBUF, MINB>;
  extern __shared__ __align__(128) unsigned char sm[];
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + C::oBar);
  int* sFm = reinterpret_cast<int*>(sm + C::oFm);
  unsigned char* sNb = sm + C::oNb;
  T* sY = reinterpret_cast<T*>(sm + C::oY);
  T* sGF = reinterpret_cast<T*>(sm + C::oGF);
  int* sGI = reinterpret_cast<int*>(sm + C::oGI);
  T* sN = reinterpret_cast<T*>(sm + C::oN);
  double* sRed = reinterpret_cast<double*>(sm + C::oR);
  const int tid = threadIdx.x, lane = tid & 31;
  // the pressure's volume term is the longest: its warp is another scheduler's
  // in each block that shares an SM
  const int role = ((tid >> 5) + blockIdx.x) % C::NV;

  auto issue_geometry = [&](int64_t tile, int b) {
    mbar_expect_tx(&bar[b], C::YB + C::GB + C::IB);
    tma_load_1d(sGF + (size_t)b * C::GW * C::LW, a.bbF + tile * C::GW * C::LW, C::GB, &bar[b]);
    tma_load_1d(sGI + (size_t)b * C::GI * C::LW, a.bbI + tile * C::GI * C::LW, C::IB, &bar[b]);
  };
  auto issue_state = [&](int64_t tile, int b) {
    tma_load_1d(sY + (size_t)b * C::TW, a.y_in + tile * C::TW, C::YB, &bar[b]);
    prefetch_operands<C>(a, tile);
  };
  auto issue = [&](int64_t tile, int b) { issue_geometry(tile, b), issue_state(tile, b); };

  if (tid == 0) {
#pragma unroll
    for (int b = 0; b < NBUF; ++b) mbar_init(&bar[b], 1);
    fence_mbar_init();
  }
  // Alternate stages may go through the tiles in opposite directions, so that what
  // the stage before touched last is still in L2. FP32 kernels do, us per step:
  // 196,608 tetrahedra of order 3 (a state of 63 MB) 294 -> 280, 614,400 triangles
  // of order 2 (44 MB) 174 -> 163, 254,016 tetrahedra of order 4 (142 MB) 698 -> 683,
  // 889,056 (498 MB) 2662 -> 2642; 196,608 of order 1, all of whose arrays fit in L2,
  // 77.3 -> 78.4. FP64 kernels, which do not wait for memory, were 0.5 % slower.
  auto tile_at = [&](int i) { return a.reverse ? a.ntiles - 1 - i : i; };
  // what no kernel before this one writes is fetched while they drain
  if (tid == 0 && (int)blockIdx.x < a.ntiles) issue_geometry(tile_at(blockIdx.x), 0);
  bb_load_tables<C>(a, sFm, sNb, tid, C::NT);
  grid_dependency_wait();
  __syncthreads();
  if (tid == 0 && (int)blockIdx.x < a.ntiles) issue_state(tile_at(blockIdx.x), 0);

  BBRes<T> racc;
  bool ok = true;
  int it = 0;
  for (int i = blockIdx.x; i < a.ntiles; i += gridDim.x, ++it) {
    const int tile = tile_at(i);
    const int b = NBUF == 2 ? it & 1 : 0;
    const bool got = mbar_wait(&bar[b], (NBUF == 2 ? it >> 1 : it) & 1, a.wait_limit);
    if (__syncthreads_or(!got)) {  // also: every thread is done with the previous tile
      ok = false;
      if (tid == 0) mbar_wait(&bar[b], (NBUF == 2 ? it >> 1 : it) & 1);  // drained (full limit)
      break;
    }
    const int next = i + gridDim.x;
    auto issue_next = [&]() {
      if (tid == 0 && next < a.ntiles) {
        fence_proxy_async();
        issue(tile_at(next), NBUF == 2 ? b ^ 1 : 0);
      }
    };
    if constexpr (NBUF == 2) issue_next();
    const T* y = sY + (size_t)b * C::TW;
    const T* g = sGF + (size_t)b * C::GW * C::LW;
    const int* gi = sGI + (size_t)b * C::GI * C::LW;
    auto free_inputs = [&]() {
      if constexpr (NBUF == 1) issue_next();
    };
    BBGlobalEnv<C, decltype(free_inputs)> env(a, (int64_t)tile * C::TW + C::first_word(tid, role), y + C::first_word(tid, role),
                                              free_inputs);
    bb_tile_any<C>(a, env, tile, y, g, gi, sFm, sNb, sN, reinterpret_cast<int*>(sm + C::oX), tid, role, racc);
  }
  if (!ok && tid == 0) atomicOr(err, 1);

  if (a.stage >= 4) {
    // block sums per variable: a warp's lanes are one variable's (Q4: each
    // variable's are every fourth lane)
    double v = racc.get();
#pragma unroll
    for (int off = 16; off >= (C::Q4 ? 4 : 1); off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if constexpr (C::Q4) {
      if (lane < 4) sRed[lane * 4 + (tid >> 5)] = v;
    } else {
      if (lane == 0) sRed[role] = v;
    }
    __syncthreads();
    if (tid < 5) {
      // p, p / c0^2, vx, vy, vz
      const int q = tid < 2 ? 0 : tid - 1;
      double s = 0.0;
      if (q < C::NV) {
        if constexpr (C::Q4)
          s = (sRed[q * 4] + sRed[q * 4 + 1]) + (sRed[q * 4 + 2] + sRed[q * 4 + 3]);
        else
          s = sRed[q];
      }
      a.partials[blockIdx.x * 5 + tid] = tid == 1 ? s / (a.c0sq * a.c0sq) : s;
    }
  }
}

template <typename T, int D, int P, int NBUF, int MINB>
struct StageBB {
  using C = BBCfg<T, D, P, NBUF, MINB>;
  static cudaError_t set_attrs() {
    auto kfn = stage_bb_kernel<T, D, P, NBUF, MINB>;
    cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::bytes);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(kfn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    return e;
  }
  static cudaError_t launch(const StageArgs<T>& a, int grid, int* err, cudaStream_t s) {
    static bool configured = false;
    if (!configured) {
      cudaError_t e = set_attrs();
      if (e != cudaSuccess) return e;
      configured = true;
    }
    return launch_kernel(stage_bb_kernel<T, D, P, NBUF, MINB>, dim3((unsigned)grid), C::NT, C::bytes, s, a.pdl != 0,
                         a, err);
  }
  static int blocks_per_sm() {
    if (set_attrs() != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, stage_bb_kernel<T, D, P, NBUF, MINB>, C::NT, C::bytes) !=
        cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return nb;
  }
};

}  // namespace dgk

// Fused passes of the surrogate network (mlp.cu), products on mma.sync with FP32
// activations split into three BF16 values: the whole forward pass in one launch,
// the whole chain of input gradients in one, all weight and bias gradients and the
// loss in one, and the optimiser step with the refresh of every weight copy in one.
//
// A block takes R rows of the batch through every layer with the
// activations in shared memory; the layers' BF16 weights, laid out in the
// order in which the block reads them, arrive as one stream of 32 KB TMA bulk
// copies (64 contraction steps x 256 outputs), several of them in flight
// across layer boundaries, since they depend on nothing the block computes.
// At the surrogate's sizes (0.33 M weights, up to a few thousand rows) one
// GEMM launch per layer left most of the time to launches, serial K loops and
// too few blocks: 18 us per layer at 2000 rows, against 3 us of arithmetic.
//
// The products run as mma.sync m16n8k16 with FP32 accumulation: 16 outputs
// (weights, BF16 as they are) x 8 rows. An FP32 activation enters as the exact
// sum of three BF16 values (8 + 8 + 8 significand bits), so that every product
// is exact. The tensor core rounds its running sum towards zero at every
// instruction, a bias that grows with the chain: the heads' products are
// taken 16 steps at a time from zero and added in FP32 registers (one chain
// over 256 steps left errors of 2.4e-6 in the gradient where the FP32 GEMM had
// 3e-7); the middle and tail products, at most 2^-8 of the sum, stay in a
// chain of their own that is added last. tcgen05 would leave most of its rate idle here: a tile has
// 8 to 32 rows, and its accumulators would travel through tensor memory after
// each of the layers. The same passes on the CUDA cores (packed FP32
// multiply-adds, the contraction split over thread groups) took 21 us at any
// batch up to 600 rows and 53 us at 2000.
#pragma once
#include <cuda_bf16.h>

#include <cstdint>

#include "stage2.cuh"

namespace mlpf {

constexpr int kMaxLayers = 16;
constexpr int kMaxWidth = 1024;  // of any layer (pass_fits in mlp.cu bounds the two buffers together)
constexpr int kKC = 64, kNC = 256;  // contraction steps and outputs of one weight chunk
constexpr uint32_t kChunkBytes = kKC * kNC * 2;
// chunks in flight of a pass with NT groups of 8 rows (what shared memory
// leaves beside the surrogate's activations; BWD: its 512-wide gradients)
__host__ __device__ constexpr int stages(int NT, bool bwd) { return NT == 1 ? 5 : NT == 2 ? 4 : bwd ? 2 : 3; }
constexpr int kCopies = 4;  // bulk copies of a chunk
constexpr int kThreads = 512, kWarps = kThreads / 32;  // that compute
constexpr int kBlock = kThreads + 32;                  // and the warp that issues the weight stream
constexpr int kDwN = 64, kDwK = 32, kDwB = 32, kDwGroups = 4, kDwThreads = 128 * kDwGroups, kLossBlocks = 64;
static_assert(kWarps * 16 == kNC, "a warp per 16 outputs of a block");

__host__ __device__ constexpr int up(int v, int a) { return (v + a - 1) / a * a; }

// Place of weight (contraction step k, output o) in its layer's part of a
// weight stream with kp (padded) steps: blocks of 256 outputs, chunks of 64
// steps, then per 16 steps and 16 outputs the 8 values of each lane of an
// mma.sync A fragment (one 16-byte load).
__host__ __device__ constexpr int64_t weight_pos(int k, int o, int kp) {
  const int kk = k % 16, oo = o % 16;
  const int lane = (oo % 8) * 4 + (kk % 8) / 2, reg = (oo / 8) + 2 * (kk / 8);
  return ((int64_t)(o / kNC) * kp + k / 16 * 16) * kNC + (o % kNC) / 16 * 256 + lane * 8 + reg * 2 + kk % 2;
}

// Stride (BF16 values) of a row of activations of width k: 16 bytes more than
// whole 128-byte lines, so that the 8 rows of an ldmatrix meet distinct banks.
__host__ __device__ constexpr int row_stride(int k) { return up(k, kKC) + 8; }

struct Net {
  int L;
  int w[kMaxLayers + 1];
  const float* b[kMaxLayers];   // biases
  float* X[kMaxLayers + 1];     // layer inputs [rows][w[l]] (training)
  float* Z[kMaxLayers + 1];     // pre-activations, then the gradients with respect to them (training)
  int64_t woff[kMaxLayers], boff[kMaxLayers];  // in the flat parameter vector
  int64_t hoff[kMaxLayers];                    // in the BF16 copy [out][in]
  int64_t toff[kMaxLayers], goff[kMaxLayers];  // in the forward and backward weight streams
};

// Dynamic shared memory of a pass with tiles of R rows: the activations
// (three planes each) alternate between two buffers of up to ka and kb values
// per row.
inline size_t pass_smem(int R, int S, int ka, int kb) {
  return 128 + (size_t)S * kChunkBytes + (size_t)3 * R * (row_stride(ka) + row_stride(kb)) * 2;
}

// The computing threads' barriers (the stream's warp takes no part).
__device__ __forceinline__ void sync_compute() { asm volatile("bar.sync 1, %0;" ::"n"(kThreads) : "memory"); }
__device__ __forceinline__ bool sync_compute_or(bool v) {
  int r;
  asm volatile(
      "{\n.reg .pred p, q;\nsetp.ne.b32 p, %1, 0;\nbar.red.or.pred q, 1, %2, p;\nselp.b32 %0, 1, 0, q;\n}"
      : "=r"(r)
      : "r"((int)v), "n"(kThreads)
      : "memory");
  return r != 0;
}

// The block's stream of weight chunks: `total` chunks per tile, cycled over
// the block's tiles. Chunk i sits in slot i % kStages; full[] counts its
// arrival, empty[] the warps that are done with it. A warp of its own issues:
// with a computing thread as the issuer, the others waited for its warp at the
// end of every layer (5 of 21 us).
template <int kStages>
struct Stream {
  unsigned char* ring;
  uint64_t *full, *empty;
  int slot = 0;  // of the current chunk, and its phase
  uint32_t phase = 0u;

  // The issuing thread's part: n chunks. False when a slot did not come free;
  // returns after every issued chunk has landed.
  __device__ bool produce(const __nv_bfloat16* src, int total, int64_t n) {
    int at = 0, sl = 0, uses = 0;  // next chunk, its slot, how often that slot was used
    bool ok = true;
    for (; n > 0; --n) {
      if (uses > 0 && !dgk::mbar_wait(&empty[sl], (uint32_t)(uses - 1) & 1u)) {
        ok = false;
        break;
      }
      dgk::mbar_expect_tx(&full[sl], kChunkBytes);
      const __nv_bfloat16* g = src + (int64_t)at * (kKC * kNC);
#pragma unroll
      for (int k = 0; k < kCopies; ++k)
        dgk::tma_load_1d(ring + (size_t)sl * kChunkBytes + k * (kChunkBytes / kCopies), g + k * (kKC * kNC / kCopies),
                         kChunkBytes / kCopies, &full[sl]);
      if (++at == total) at = 0;
      if (++sl == kStages) sl = 0, ++uses;
    }
    for (int s = 0; s < kStages; ++s) {
      const int u = uses + (s < sl ? 1 : 0);
      if (u > 0) dgk::mbar_wait(&full[s], (uint32_t)(u - 1) & 1u);
    }
    return ok;
  }
  // the current chunk; false on timeout
  __device__ bool wait() { return dgk::mbar_wait(&full[slot], phase); }
  __device__ const uint4* chunk() const { return reinterpret_cast<const uint4*>(ring + (size_t)slot * kChunkBytes); }
  __device__ void release() {
    __syncwarp();
    if ((threadIdx.x & 31) == 0)
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(dgk::smem_u32(&empty[slot])) : "memory");
    if (++slot == kStages) slot = 0, phase ^= 1u;
  }
};

// Activations: three planes (head, middle, tail) of [R][stride] BF16.
struct Act {
  __nv_bfloat16* p;
  int ld, plane;
  __device__ void put(int r, int k, float v) const {
    // truncated to 8 significand bits each; an infinity keeps its value
    const uint32_t hb = __float_as_uint(v) & 0xffff0000u;
    const float h = __uint_as_float(hb), r1 = h == v ? 0.f : v - h;
    const uint32_t mb = __float_as_uint(r1) & 0xffff0000u;
    const float r2 = r1 - __uint_as_float(mb);
    unsigned short* q = reinterpret_cast<unsigned short*>(p) + r * ld + k;
    q[0] = (unsigned short)(hb >> 16);
    q[plane] = (unsigned short)(mb >> 16);
    q[2 * plane] = (unsigned short)(__float_as_uint(r2) >> 16);
  }
};

template <int kStages>
struct Pass {
  Stream<kStages> st;
  unsigned char *ba, *bb;
  __device__ Pass(unsigned char* sm, int R, int ka) {
    st.full = reinterpret_cast<uint64_t*>(sm);
    st.empty = st.full + kStages;
    st.ring = sm + 128;
    ba = st.ring + (size_t)kStages * kChunkBytes;
    bb = ba + (size_t)3 * R * row_stride(ka) * 2;
    if (threadIdx.x == 0) {
      for (int s = 0; s < kStages; ++s) dgk::mbar_init(&st.full[s], 1), dgk::mbar_init(&st.empty[s], kWarps);
      dgk::fence_mbar_init();
    }
    __syncthreads();
  }
  // the activations of width k in the first (0) or second (1) buffer
  __device__ Act act(int which, int k, int R) const {
    const int ld = row_stride(k);
    return Act{reinterpret_cast<__nv_bfloat16*>(which ? bb : ba), ld, R * ld};
  }
};

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
  const float cdf = 0.5f * (1.f + erff(z * 0.70710678118654752f));
  const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
  return cdf + z * pdf;
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint4& a, uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, "
      "%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
// the same from zero
__device__ __forceinline__ void mma_bf16_0(float (&d)[4], const uint4& a, uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, "
      "%10, %10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(dgk::smem_u32(p)));
}

// One 256-output block of a layer for NT groups of 8 rows: activations x (zero
// past K up to whole chunks) times weights, summed over K. The warp's 16
// outputs: acc[t][..] holds output 16 warp + lane / 4 (+ 8 for the last two) of
// rows 8 t + 2 (lane % 4) (+ 1 for the odd ones). False (in every thread) when
// a chunk did not arrive.
template <int NT, int S>
__device__ __forceinline__ bool layer_block(Pass<S>& p, const Act& x, int K, float (&acc)[NT][4]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // middle and tail products, a chain each where the registers allow it
  constexpr int NCH = NT == 4 ? 1 : 2;
  float c[NCH][NT][4];
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[t][u] = c[0][t][u] = c[NCH - 1][t][u] = 0.f;
  bool ok = true;
  // ldmatrix: lane's row of matrix lane / 8, whose 8 values start at step 8 (lane / 8)
  const __nv_bfloat16* xl = x.p + (lane & 7) * x.ld + (lane >> 3) * 8;
  for (int k0 = 0; k0 < K; k0 += kKC) {
    ok = ok && p.st.wait();
    const uint4* w = p.st.chunk() + warp * 32 + lane;
    // H x 32 steps at a time: one ldmatrix per 8 rows, plane and 32 steps
    constexpr int H = NT == 1 ? 2 : 1;
    static_assert(kKC == 64, "two halves of a chunk");
#pragma unroll
    for (int h0 = 0; h0 < 2; h0 += H) {
      uint4 a[2 * H];
#pragma unroll
      for (int h = 0; h < 2 * H; ++h) a[h] = w[(2 * h0 + h) * (kNC / 16) * 32];
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        uint32_t b[H][3][4];
#pragma unroll
        for (int h = 0; h < H; ++h)
#pragma unroll
          for (int s = 0; s < 3; ++s) ldmatrix4(b[h][s], xl + t * 8 * x.ld + k0 + 32 * (h0 + h) + s * x.plane);
#pragma unroll
        for (int h = 0; h < H; ++h) {
          float d0[4], d1[4];
          mma_bf16_0(d0, a[2 * h], b[h][0][0], b[h][0][1]);
          mma_bf16_0(d1, a[2 * h + 1], b[h][0][2], b[h][0][3]);
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            mma_bf16(c[s % NCH][t], a[2 * h], b[h][1 + s][0], b[h][1 + s][1]);
            mma_bf16(c[s % NCH][t], a[2 * h + 1], b[h][1 + s][2], b[h][1 + s][3]);
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) acc[t][u] = (acc[t][u] + d0[u]) + d1[u];
        }
      }
    }
    p.st.release();
  }
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int u = 0; u < 4; ++u) acc[t][u] += NCH == 2 ? c[0][t][u] + c[NCH - 1][t][u] : c[0][t][u];
  return !sync_compute_or(!ok);
}

// Forward pass of n rows: x [.][w0] (row idx[r] of it when idx is given) to y
// [n][wL]; TRAIN also stores the gathered inputs, every layer's input and
// pre-activation.
template <int NT, bool TRAIN>
__global__ void __launch_bounds__(kBlock, 1) k_forward(const Net net, const __nv_bfloat16* wstream, int chunks,
                                                         const float* __restrict__ x, const int* __restrict__ idx,
                                                         int64_t n, float* __restrict__ y, int ka, int* err) {
  constexpr int R = 8 * NT, S = stages(NT, false);
  extern __shared__ __align__(128) unsigned char sm[];
  Pass<S> p(sm, R, ka);
  const int tid = threadIdx.x, lane = tid & 31;
  const int oc = (tid >> 5) * 16 + (lane >> 2), rc = 2 * (lane & 3);  // this lane's first output and row
  const int64_t tiles = (n + R - 1) / R, mine = (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x;
  if (tid >= kThreads) {
    if (tid == kThreads && !p.st.produce(wstream, chunks, mine * chunks)) atomicOr(err, 1);
    return;
  }
  bool ok = true;
  for (int64_t tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
    const int64_t r0 = tile * R;
    const int K0 = net.w[0], K0p = up(K0, kKC);
    {
      const Act a = p.act(0, K0, R);
      for (int r = tid >> 5; r < R; r += kWarps) {
        const int64_t row = r0 + r;
        const float* xr = x + (row < n ? (idx ? (int64_t)idx[row] : row) : 0) * K0;
        for (int k = lane; k < K0p; k += 32) {
          const float v = row < n && k < K0 ? xr[k] : 0.f;
          a.put(r, k, v);
          if (TRAIN && idx && row < n && k < K0) net.X[0][row * K0 + k] = v;
        }
      }
    }
    sync_compute();
    for (int l = 0; l < net.L && ok; ++l) {
      const int K = net.w[l], N = net.w[l + 1], Np = up(N, kKC);
      const bool last = l == net.L - 1;
      const Act xa = p.act(l & 1, K, R), xn = p.act(~l & 1, N, R);
      for (int n0 = 0; n0 < N && ok; n0 += kNC) {
        float acc[NT][4], bias[2];  // the biases, in flight while the block is summed
#pragma unroll
        for (int h = 0; h < 2; ++h) bias[h] = n0 + oc + 8 * h < N ? net.b[l][n0 + oc + 8 * h] : 0.f;
        ok = layer_block<NT, S>(p, xa, K, acc);
        if (!ok) break;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int o = n0 + oc + 8 * h;
#pragma unroll
          for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int r = 8 * t + rc + u;
              const int64_t row = r0 + r;
              const float z = acc[t][2 * h + u] + bias[h];
              if (last) {
                if (o < N && row < n) y[row * N + o] = z;
              } else if (o < Np) {
                const float a = o < N ? gelu(z) : 0.f;
                xn.put(r, o, a);
                if (TRAIN && o < N && row < n) net.Z[l + 1][row * N + o] = z, net.X[l + 1][row * N + o] = a;
              }
            }
        }
      }
      sync_compute();  // the next layer's inputs are written, this layer's read
    }
  }
  if (tid == 0 && !ok) atomicOr(err, 1);
}

// Gradients with respect to every layer's pre-activation, in place of the
// pre-activations Z[l], from the outputs y and targets t (row idx[r] of t when
// idx is given): dY = 2 (y - t) / (n wL), then layer by layer
// dZ_l = (dZ_{l+1} W_l) GELU'(Z_l).
template <int NT>
__global__ void __launch_bounds__(kBlock, 1) k_backward(const Net net, const __nv_bfloat16* wstream, int chunks,
                                                          const float* __restrict__ y, const float* __restrict__ t_,
                                                          const int* __restrict__ idx, int64_t n, int ka, int* err) {
  constexpr int R = 8 * NT, S = stages(NT, true);
  extern __shared__ __align__(128) unsigned char sm[];
  Pass<S> p(sm, R, ka);
  const int tid = threadIdx.x, lane = tid & 31;
  const int oc = (tid >> 5) * 16 + (lane >> 2), rc = 2 * (lane & 3);
  const int64_t tiles = (n + R - 1) / R, mine = (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x;
  const int NL = net.w[net.L];
  const float sc = 2.f / (float)(n * NL);
  if (tid >= kThreads) {
    if (tid == kThreads && !p.st.produce(wstream, chunks, mine * chunks)) atomicOr(err, 1);
    return;
  }
  bool ok = true;
  for (int64_t tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
    const int64_t r0 = tile * R;
    const int NLp = up(NL, kKC);
    {
      const Act a = p.act(0, NL, R);
      // kWarps / R threads' worth of warps per row where the tile has fewer rows
      constexpr int PR = R < kWarps ? kWarps / R : 1;
      for (int r = (tid >> 5) / PR; r < R; r += kWarps / PR) {
        const int64_t row = r0 + r;
        const float* yr = y + (row < n ? row : 0) * NL;
        const float* tr = t_ + (row < n ? (idx ? (int64_t)idx[row] : row) : 0) * NL;
#pragma unroll 4
        for (int c = lane + 32 * ((tid >> 5) % PR); c < NLp; c += 32 * PR) {
          float d = 0.f;
          if (row < n && c < NL) {
            d = sc * (yr[c] - tr[c]);
            net.Z[net.L][row * NL + c] = d;
          }
          a.put(r, c, d);
        }
      }
    }
    sync_compute();
    for (int l = net.L - 1; l >= 1 && ok; --l) {
      const int K = net.w[l + 1], N = net.w[l], Np = up(N, kKC), turn = net.L - 1 - l;
      const Act xa = p.act(turn & 1, K, R), xn = p.act(~turn & 1, N, R);
      for (int n0 = 0; n0 < N && ok; n0 += kNC) {
        // the pre-activations, in flight while the block is summed
        float z[2][NT][2];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int o = n0 + oc + 8 * h;
              const int64_t row = r0 + 8 * t + rc + u;
              z[h][t][u] = o < N && row < n ? net.Z[l][row * N + o] : 0.f;
            }
        float acc[NT][4];
        ok = layer_block<NT, S>(p, xa, K, acc);
        if (!ok) break;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              const int o = n0 + oc + 8 * h, r = 8 * t + rc + u;
              const int64_t row = r0 + r;
              float d = 0.f;
              if (o < N && row < n) {
                d = acc[t][2 * h + u] * gelu_grad(z[h][t][u]);
                net.Z[l][row * N + o] = d;
              }
              if (o < Np) xn.put(r, o, d);
            }
      }
      sync_compute();
    }
    sync_compute();  // (one layer: the buffer is rewritten by the next tile)
  }
  if (tid == 0 && !ok) atomicOr(err, 1);
}

// Weight and bias gradients of every layer, dW_l = dZ_{l+1}^T X_l and the
// column sums of dZ_{l+1}, and the loss, in one launch: blocks [0, tiles) each
// compute a 64 x 32 tile of one layer's dW (its first column of tiles also the
// bias gradient), the last kLossBlocks blocks the squared error's partial
// sums (FP64), which the last of them to finish adds up in order.
struct DwPlan {
  int first[kMaxLayers + 1];  // first tile of each layer
  int tiles;
};

__global__ void __launch_bounds__(kDwThreads, 1) k_weight_grads(const Net net, const DwPlan plan, int64_t n,
                                                             float* __restrict__ g, const float* __restrict__ y,
                                                             const float* __restrict__ t,
                                                             const int* __restrict__ idx, double* __restrict__ part,
                                                             unsigned* __restrict__ ticket,
                                                             double* __restrict__ loss) {
  __shared__ __align__(16) float sA[2][kDwB][kDwN];
  __shared__ __align__(16) float sB[2][kDwB][kDwK];
  const int tid = threadIdx.x;
  if ((int)blockIdx.x >= plan.tiles) {
    double* sh = reinterpret_cast<double*>(&sA[0][0][0]);
    __shared__ bool lastb;
    const int lb = blockIdx.x - plan.tiles, NL = net.w[net.L];
    double s = 0.0;
    for (int64_t i = lb * (int64_t)kDwThreads + tid; i < n * NL; i += (int64_t)kLossBlocks * kDwThreads) {
      const int64_t row = i / NL;
      const float d = y[i] - t[idx ? (int64_t)idx[row] * NL + (i - row * NL) : i];
      s += (double)d * d;
    }
    for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
    if ((tid & 31) == 0) sh[tid >> 5] = s;
    __syncthreads();
    if (tid == 0) {
      double v = 0.0;
      for (int w = 0; w < kDwThreads / 32; ++w) v += sh[w];
      part[lb] = v;
      __threadfence();
      lastb = atomicAdd(ticket, 1u) == kLossBlocks - 1;
      if (lastb) {
        __threadfence();
        double v2 = 0.0;
        for (int k = 0; k < kLossBlocks; ++k) v2 += __ldcg(part + k);
        *loss = v2 * (1.0 / (double)(n * NL));
        *ticket = 0u;  // for the next launch
      }
    }
    return;
  }
  int l = 0;
  while (l + 1 < net.L && (int)blockIdx.x >= plan.first[l + 1]) ++l;
  const int K = net.w[l], N = net.w[l + 1], kt = (K + kDwK - 1) / kDwK;
  const int tl = blockIdx.x - plan.first[l];
  const int n0 = tl / kt * kDwN, k0 = (tl % kt) * kDwK;
  const float* A = net.Z[l + 1];
  const float* B = net.X[l];
  const bool va = N % 4 == 0, vb = K % 4 == 0;  // rows start on 16-byte boundaries
  auto load = [&](int64_t b0, int s) {
    for (int i = tid; i < kDwB * kDwN / 4; i += kDwThreads) {
      const int b = i / (kDwN / 4), c = (i % (kDwN / 4)) * 4;
      const int64_t row = b0 + b;
      float* dst = &sA[s][b][c];
      if (va && row < n && n0 + c < N) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dgk::smem_u32(dst)), "l"(A + row * N + n0 + c)
                     : "memory");
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) dst[u] = row < n && n0 + c + u < N ? A[row * N + n0 + c + u] : 0.f;
      }
    }
    for (int i = tid; i < kDwB * kDwK / 4; i += kDwThreads) {
      const int b = i / (kDwK / 4), c = (i % (kDwK / 4)) * 4;
      const int64_t row = b0 + b;
      float* dst = &sB[s][b][c];
      if (vb && row < n && k0 + c < K) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dgk::smem_u32(dst)), "l"(B + row * K + k0 + c)
                     : "memory");
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) dst[u] = row < n && k0 + c + u < K ? B[row * K + k0 + c + u] : 0.f;
      }
    }
    dgk::cp_async_commit();
  };
  // kDwGroups groups of threads each sum a quarter of the staged rows; a
  // thread holds 4 of W's rows x 4 of its columns
  const int grp = tid / 128, tm = (tid % 128) / 8, tn = tid % 8;
  float2 acc[4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = make_float2(0.f, 0.f);
  float4 bs = make_float4(0.f, 0.f, 0.f, 0.f);
  const bool bias = k0 == 0 && tn == 0;
  load(0, 0);
  int s = 0;
  for (int64_t b0 = 0; b0 < n; b0 += kDwB, s ^= 1) {
    if (b0 + kDwB < n) {
      load(b0 + kDwB, s ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      dgk::cp_async_wait_all();
    }
    __syncthreads();
#pragma unroll
    for (int b = grp * (kDwB / kDwGroups); b < (grp + 1) * (kDwB / kDwGroups); ++b) {
      const float4 av = *reinterpret_cast<const float4*>(&sA[s][b][tm * 4]);
      const float4 bv = *reinterpret_cast<const float4*>(&sB[s][b][tn * 4]);
      const float2 p0 = make_float2(bv.x, bv.y), p1 = make_float2(bv.z, bv.w);
      const float a[4] = {av.x, av.y, av.z, av.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc[i][0] = __ffma2_rn(make_float2(a[i], a[i]), p0, acc[i][0]);
        acc[i][1] = __ffma2_rn(make_float2(a[i], a[i]), p1, acc[i][1]);
      }
      if (bias) bs.x += av.x, bs.y += av.y, bs.z += av.z, bs.w += av.w;
    }
    __syncthreads();
  }
  // the groups' sums meet in the staging buffers
  float4* red = reinterpret_cast<float4*>(&sA[0][0][0]);
  float4* redb = reinterpret_cast<float4*>(&sB[0][0][0]);
  static_assert((kDwGroups - 1) * 128 * 4 * 16 <= (int)sizeof(sA) + (int)sizeof(sB), "sums must fit");
  constexpr int kInA = (int)sizeof(sA) / (128 * 4 * 16);  // groups whose sums fit in sA
  auto slot = [&](int g, int i) { return g < kInA ? red + (g * 4 + i) * 128 : redb + ((g - kInA) * 4 + i) * 128; };
  if (grp > 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      slot(grp - 1, i)[tid % 128] = make_float4(acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y);
  }
  __syncthreads();
  if (grp == 0) {
#pragma unroll
    for (int g = 0; g < kDwGroups - 1; ++g)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 v = slot(g, i)[tid];
        acc[i][0].x += v.x, acc[i][0].y += v.y, acc[i][1].x += v.z, acc[i][1].y += v.w;
      }
  }
  __syncthreads();
  if (bias && grp > 0) red[(grp - 1) * 16 + tm] = bs;
  __syncthreads();
  if (grp > 0) return;
  if (bias) {
#pragma unroll
    for (int g = 0; g < kDwGroups - 1; ++g) {
      const float4 v = red[g * 16 + tm];
      bs.x += v.x, bs.y += v.y, bs.z += v.z, bs.w += v.w;
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int o = n0 + tm * 4 + i;
    if (o >= N) break;
    const float v[4] = {acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y};
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (k0 + tn * 4 + u < K) g[net.woff[l] + (int64_t)o * K + k0 + tn * 4 + u] = v[u];
    if (bias) g[net.boff[l] + o] = i == 0 ? bs.x : i == 1 ? bs.y : i == 2 ? bs.z : bs.w;
  }
}

// BF16 copies of weight i (layer l, out o, in k): [out][in] and its places in
// the forward and backward streams (their padding stays zero).
__device__ __forceinline__ void put_weight(const Net& net, int l, int o, int k, float v, __nv_bfloat16* wh,
                                           __nv_bfloat16* wt, __nv_bfloat16* wb) {
  const int K = net.w[l], N = net.w[l + 1];
  const __nv_bfloat16 h = __float2bfloat16_rn(v);
  wh[net.hoff[l] + (int64_t)o * K + k] = h;
  wt[net.toff[l] + weight_pos(k, o, up(K, kKC))] = h;
  if (l > 0) wb[net.goff[l] + weight_pos(o, k, up(N, kKC))] = h;
}

// Layer of flat parameter i, and whether it is a weight.
__device__ __forceinline__ int layer_of(const Net& net, int64_t i, bool& weight) {
  int l = 0;
  while (l + 1 < net.L && i >= net.woff[l + 1]) ++l;
  weight = i < net.boff[l];
  return l;
}

__global__ void k_refresh(const Net net, const float* __restrict__ p, int64_t n, __nv_bfloat16* wh, __nv_bfloat16* wt,
                          __nv_bfloat16* wb) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  bool weight;
  const int l = layer_of(net, i, weight);
  if (!weight) return;
  const int64_t r = i - net.woff[l];
  put_weight(net, l, (int)(r / net.w[l]), (int)(r % net.w[l]), p[i], wh, wt, wb);
}

// AdamW step on the FP32 masters (mlp.cu's k_adam) and the refresh of the
// BF16 copies in one pass.
__global__ void k_adam_refresh(const Net net, float* __restrict__ p, const float* __restrict__ g,
                               float* __restrict__ m1, float* __restrict__ m2, int64_t n, float lr, float b1, float b2,
                               float eps, float c1, float c2, float wd, __nv_bfloat16* wh, __nv_bfloat16* wt,
                               __nv_bfloat16* wb) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float a = b1 * m1[i] + (1.f - b1) * gi;
  const float v = b2 * m2[i] + (1.f - b2) * gi * gi;
  m1[i] = a, m2[i] = v;
  const float pn = p[i] - lr * ((a / c1) / (sqrtf(v / c2) + eps) + wd * p[i]);
  p[i] = pn;
  bool weight;
  const int l = layer_of(net, i, weight);
  if (!weight) return;
  const int64_t r = i - net.woff[l];
  put_weight(net, l, (int)(r / net.w[l]), (int)(r % net.w[l]), pn, wh, wt, wb);
}

}  // namespace mlpf

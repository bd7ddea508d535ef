// One persistent launch per RK stage for a batch of 2-D instances of mixed
// order (p = 2, 3, 4): the batched ensemble's stage kernel (FP32 state).
//
// The batch keeps one disjoint-union mesh per element order (batch.cu). This
// kernel advances all of them in one launch: its blocks take tiles from a
// work queue over every order's tiles (an atomic counter; order after order)
// and run each with the Bernstein-basis kernel's per-tile code for that order
// (bb_tile in stage_bb.cuh), 32 elements and three warps per tile at every
// order. The tile buffers are two fixed slots sized for the largest order
// (consecutive queue items may be of different orders; the next item's stage
// input and geometry arrive by TMA while the current one computes), then the
// face-flux buffer, also sized for the largest order. Every wait is bounded;
// after a timeout a block records the error, drains its own copies (bounded)
// and stops taking work.
#pragma once
#include <cstdint>

#include "stage_bb.cuh"

namespace dgk {

using MultiC2 = BBCfg<float, 2, 2, 2, 1>;
using MultiC3 = BBCfg<float, 2, 3, 2, 1>;
using MultiC4 = BBCfg<float, 2, 4, 2, 1>;
constexpr int kMultiNT = MultiC4::NT;
static_assert(MultiC2::NT == kMultiNT && MultiC3::NT == kMultiNT, "every order's tile takes the whole block");
// blocks per SM the register budget is set for
constexpr int kMultiMinBlocks = 5;

struct MultiLayout {
  static constexpr size_t oBar = 0;    // 2 mbarriers
  static constexpr size_t oItem = 32;  // next work item
  static constexpr size_t FM = MultiC4::NF * 16 * 4, NB = MultiC4::NF * MultiC4::NPERM * 16;
  static constexpr size_t oFm = 64;             // 3 x face node tables
  static constexpr size_t oNb = oFm + 3 * FM;   // 3 x neighbour node tables
  static constexpr size_t SLOT = RoundUp<MultiC4::YB + MultiC4::GB + MultiC4::IB, 128>::v;
  static constexpr size_t oSlot = RoundUp<oNb + 3 * NB, 128>::v;  // 2 slots
  static constexpr size_t oN = oSlot + 2 * SLOT;
  static constexpr size_t oR = oN + (size_t)MultiC4::NF * MultiC4::NV * MultiC4::NFP * 32 * 4;
  static constexpr size_t bytes = oR + MultiC4::NV * sizeof(double);
};

// order slot and tile of a work item (items run order after order)
__device__ __forceinline__ int multi_slot(const MultiArgs& m, int item, int* tile) {
  int t = item;
#pragma unroll
  for (int g = 0; g < kMultiOrders; ++g) {
    if (t < m.g[g].ntiles) {
      *tile = t;
      return g;
    }
    t -= m.g[g].ntiles;
  }
  *tile = 0;
  return -1;
}

template <class C>
__device__ __forceinline__ void multi_issue_tile(const StageArgs<float>& a, int64_t tile, unsigned char* slot,
                                                 uint64_t* bar) {
  mbar_expect_tx(bar, C::YB + C::GB + C::IB);
  tma_load_1d(slot, a.y_in + tile * C::TW, C::YB, bar);
  tma_load_1d(slot + C::YB, a.bbF + tile * C::GW * C::LW, C::GB, bar);
  tma_load_1d(slot + C::YB + C::GB, a.bbI + tile * C::GI * C::LW, C::IB, bar);
  prefetch_operands<C>(a, tile);
}

template <class C>
__device__ __forceinline__ void multi_run_tile(const StageArgs<float>& a, int tile, unsigned char* slot, float* sN,
                                               const int* sFm, const unsigned char* sNb, int lane, int role,
                                               BBRes<float>& racc) {
  auto keep = []() {};
  BBGlobalEnv<C, decltype(keep)> env(a, (int64_t)tile * C::TW + C::first_word(lane, role),
                                       reinterpret_cast<const float*>(slot) + C::first_word(lane, role), keep);
  bb_tile_any<C>(a, env, tile, reinterpret_cast<const float*>(slot), reinterpret_cast<const float*>(slot + C::YB),
                 reinterpret_cast<const int*>(slot + C::YB + C::GB), sFm, sNb, sN, (int*)nullptr, lane, role, racc);
}

__global__ void __launch_bounds__(kMultiNT, kMultiMinBlocks) stage_multi_kernel(const MultiArgs m, int* err) {
  using L = MultiLayout;
  extern __shared__ __align__(128) unsigned char sm[];
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + L::oBar);
  int* sItem = reinterpret_cast<int*>(sm + L::oItem);
  auto sFm = [&](int g) { return reinterpret_cast<int*>(sm + L::oFm + g * L::FM); };
  auto sNb = [&](int g) { return sm + L::oNb + g * L::NB; };
  unsigned char* slots = sm + L::oSlot;
  float* sN = reinterpret_cast<float*>(sm + L::oN);
  double* sRed = reinterpret_cast<double*>(sm + L::oR);
  const int tid = threadIdx.x, lane = tid & 31;
  const int role = ((tid >> 5) + blockIdx.x) % MultiC4::NV;
  const int stage = m.g[0].stage;

  auto issue = [&](int item, int b) {
    int tile;
    const int g = multi_slot(m, item, &tile);
    unsigned char* slot = slots + (size_t)b * L::SLOT;
    if (g == 0) multi_issue_tile<MultiC2>(m.g[0], tile, slot, &bar[b]);
    if (g == 1) multi_issue_tile<MultiC3>(m.g[1], tile, slot, &bar[b]);
    if (g == 2) multi_issue_tile<MultiC4>(m.g[2], tile, slot, &bar[b]);
  };

  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_mbar_init();
  }
  if (m.g[0].ntiles > 0) bb_load_tables<MultiC2>(m.g[0], sFm(0), sNb(0), tid, kMultiNT);
  if (m.g[1].ntiles > 0) bb_load_tables<MultiC3>(m.g[1], sFm(1), sNb(1), tid, kMultiNT);
  if (m.g[2].ntiles > 0) bb_load_tables<MultiC4>(m.g[2], sFm(2), sNb(2), tid, kMultiNT);
  // thread 0 claims items one ahead of the prefetch: the queue's atomic
  // round trip overlaps a tile's work instead of delaying the next copy
  int ahead = 0;
  if (tid == 0) {
    const int first = (int)atomicAdd(m.queue, 1u);
    *sItem = first;
    if (first < m.ntiles_total) {
      issue(first, 0);
      ahead = (int)atomicAdd(m.queue, 1u);
    }
  }
  __syncthreads();

  // stage 4: racc holds the residual sum of this thread's variable for order
  // rg; a block's items come in order after order, so each order's row is
  // written once, when the block moves on to the next order or finishes
  // (orders bit-set in wrote)
  BBRes<float> racc;
  int rg = -1;
  unsigned wrote = 0;
  auto put_row = [&](int g, bool zero) {
    double v = zero ? 0.0 : racc.get();
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if (lane == 0) sRed[role] = v;
    __syncthreads();
    if (tid < 5) {
      // p, p / c0^2, vx, vy (vz: none)
      const double c4 = m.g[g].c0sq * m.g[g].c0sq;
      m.g[g].partials[blockIdx.x * 5 + tid] =
          tid == 0 ? sRed[0] : tid == 1 ? sRed[0] / c4 : tid < 4 ? sRed[tid - 1] : 0.0;
    }
    __syncthreads();
    racc = BBRes<float>();
    wrote |= 1u << g;
  };
  bool ok = true;
  for (int it = 0;; ++it) {
    const int item = *sItem;  // written before the barrier inside the previous item
    if (item >= m.ntiles_total) break;
    const int b = it & 1;
    const bool got = mbar_wait(&bar[b], (it >> 1) & 1, m.wait_limit);
    if (__syncthreads_or(!got)) {  // also: every thread is done with the previous item
      ok = false;
      if (tid == 0) mbar_wait(&bar[b], (it >> 1) & 1);  // the only copy in flight, drained (full limit)
      break;
    }
    int tile;
    const int g = multi_slot(m, item, &tile);
    if (stage == 4 && g != rg) {  // block-uniform
      if (rg >= 0) put_row(rg, false);
      rg = g;
    }
    if (tid == 0) {
      fence_proxy_async();
      const int next = ahead;
      *sItem = next;
      if (next < m.ntiles_total) {
        issue(next, b ^ 1);
        ahead = (int)atomicAdd(m.queue, 1u);
      }
    }
    unsigned char* slot = slots + (size_t)b * L::SLOT;
    if (g == 0)
      multi_run_tile<MultiC2>(m.g[0], tile, slot, sN, sFm(0), sNb(0), lane, role, racc);
    else if (g == 1)
      multi_run_tile<MultiC3>(m.g[1], tile, slot, sN, sFm(1), sNb(1), lane, role, racc);
    else
      multi_run_tile<MultiC4>(m.g[2], tile, slot, sN, sFm(2), sNb(2), lane, role, racc);
  }
  if (tid == 0 && !ok) atomicOr(err, 1);

  if (stage == 4) {
    // residual partial sums per order (one row per block in each order's
    // partials array; a block that ran no tile of an order writes zeros)
    if (rg >= 0) put_row(rg, false);
#pragma unroll
    for (int g = 0; g < kMultiOrders; ++g)
      if (m.g[g].ntiles > 0 && !(wrote & (1u << g))) put_row(g, true);
  }
}

}  // namespace dgk

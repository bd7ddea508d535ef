// Instantiations of the Bernstein-basis stage kernel (stage_bb.cuh), FP32 state.
// Variants (stage-input buffers NBUF, blocks per SM the register budget allows
// for) are offered to the context's kernel selection as kBBVariant + k.
#include "stage_bb.cuh"

namespace dgk {

namespace {
// per (dim, order): candidate (NBUF, MINB)
#define DGK_BB_VARIANTS(X) \
  X(2, 1, 2, 16) X(2, 1, 2, 12) X(2, 1, 2, 8)  \
  X(2, 2, 2, 10) X(2, 2, 2, 8) X(2, 2, 2, 6)   \
  X(2, 3, 2, 8) X(2, 3, 2, 7) X(2, 3, 2, 5)    \
  X(2, 4, 2, 6) X(2, 4, 2, 5) X(2, 4, 2, 4)    \
  X(3, 1, 2, 10) X(3, 1, 2, 8) X(3, 1, 2, 6)   \
  X(3, 2, 2, 6) X(3, 2, 2, 5) X(3, 2, 2, 4)    \
  X(3, 3, 2, 4) X(3, 3, 2, 3) X(3, 3, 2, 2)    \
  X(3, 4, 1, 3) X(3, 4, 2, 2) X(3, 4, 1, 2)
}  // namespace

cudaError_t launch_stage_bb(int dim, int order, int variant, const StageArgs<float>& a, int grid, int* err,
                            cudaStream_t s) {
  int k = 0;
#define DGK_BB_LAUNCH(DD, PP, NB, MB)                                           \
  if (dim == DD && order == PP) {                                               \
    if (k == variant) return StageBB<float, DD, PP, NB, MB>::launch(a, grid, err, s); \
    ++k;                                                                        \
  }
  DGK_BB_VARIANTS(DGK_BB_LAUNCH)
#undef DGK_BB_LAUNCH
  return cudaErrorInvalidValue;
}

Stage2Info stage_bb_info_f32(int dim, int order, int variant) {
  int k = 0, n = 0;
#define DGK_BB_COUNT(DD, PP, NB, MB) \
  if (dim == DD && order == PP) ++n;
  DGK_BB_VARIANTS(DGK_BB_COUNT)
#undef DGK_BB_COUNT
#define DGK_BB_INFO(DD, PP, NB, MB)                                                                            \
  if (dim == DD && order == PP) {                                                                              \
    if (k == variant) {                                                                                        \
      using K = StageBB<float, DD, PP, NB, MB>;                                                                  \
      return Stage2Info{K::C::NP, K::C::LW, K::C::NT, (int)K::C::bytes, K::blocks_per_sm(), n};                  \
    }                                                                                                          \
    ++k;                                                                                                       \
  }
  DGK_BB_VARIANTS(DGK_BB_INFO)
#undef DGK_BB_INFO
  return Stage2Info{0, 0, 0, 0, 0, 0};
}

}  // namespace dgk

// Instantiations of the many-steps kernel (stage_persist.cuh).
#include "stage_persist.cuh"

namespace dgk {

// per (dim, order): blocks per SM that the register budget allows for. (3-D, order
// 4: 191 us per step against 190 with one launch per stage, on any number of
// tiles that fit; not built.)
#define DGK_PERSIST(X) \
  X(2, 1, 8) X(2, 2, 6) X(2, 3, 5) X(2, 4, 4) \
  X(3, 1, 5) X(3, 2, 3) X(3, 3, 2)

cudaError_t launch_persist(int dim, int order, const PersistArgs& p, int grid, int* err, cudaStream_t s) {
#define DGK_P_LAUNCH(DD, PP, MB) \
  if (dim == DD && order == PP) return StagePersist<DD, PP, MB>::launch(p, grid, err, s);
  DGK_PERSIST(DGK_P_LAUNCH)
#undef DGK_P_LAUNCH
  return cudaErrorInvalidValue;
}

PersistInfo persist_info(int dim, int order) {
#define DGK_P_INFO(DD, PP, MB)                                       \
  if (dim == DD && order == PP) {                                    \
    using K = StagePersist<DD, PP, MB>;                              \
    return PersistInfo{K::C::NT, (int)K::C::bytes, K::blocks_per_sm()}; \
  }
  DGK_PERSIST(DGK_P_INFO)
#undef DGK_P_INFO
  return PersistInfo{0, 0, 0};
}

}  // namespace dgk

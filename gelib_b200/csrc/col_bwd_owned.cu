// Backward column kernel for calls with few columns (col.h, col_bwd.cuh): walks cut by gradient rows, either gradient or both.
#include "col_bwd.cuh"

namespace gelib_b200 {

cudaError_t col_launch_bwd_owned(const ColArgs& a, const ColPlan& p, cudaStream_t s) {
  return col::launch_bwd<kColBlockBwd, 1, true, true, 384, true>(a, s, p.warps);
}

}  // namespace gelib_b200

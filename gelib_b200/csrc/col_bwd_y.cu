// Backward column kernels, gradient of y alone (col.h, col_bwd.cuh).
#include "col_bwd.cuh"

namespace gelib_b200 {

cudaError_t col_launch_bwd_y(const ColArgs& a, const ColPlan& p, cudaStream_t s) { return col::launch_bwd_k<false, true>(a, p, s); }

}  // namespace gelib_b200

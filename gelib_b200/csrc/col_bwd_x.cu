// Backward column kernels, gradient of x alone (col.h, col_bwd.cuh).
#include "col_bwd.cuh"

namespace gelib_b200 {

cudaError_t col_launch_bwd_x(const ColArgs& a, const ColPlan& p, cudaStream_t s) { return col::launch_bwd_k<true, false>(a, p, s); }

}  // namespace gelib_b200

// Backward column kernels, both gradients, and the entry for all of them (col.h, col_bwd.cuh).
#include "col_bwd.cuh"

namespace gelib_b200 {

cudaError_t col_launch_bwd_x(const ColArgs& a, const ColPlan& p, cudaStream_t s);
cudaError_t col_launch_bwd_y(const ColArgs& a, const ColPlan& p, cudaStream_t s);
cudaError_t col_launch_bwd_owned(const ColArgs& a, const ColPlan& p, cudaStream_t s);

int launch_col_bwd(const VecCall& c, cudaStream_t s, bool* plan_others) {
  static const char* fn = "SO3vec_addCGproduct_back";
  ColArgs a;
  ColPlan plan;
  if (c.xg.empty() && c.yg.empty()) return -1;
  if (!col_setup(c, true, &a, &plan)) return -1;
  if (!plan.dev) return GELIB_CUDA_ERROR;
  *plan_others = plan.plan_others;
  if (a.nsplits == 0 || c.plan_only) return GELIB_OK;
  const bool do_x = !c.xg.empty(), do_y = !c.yg.empty();
  const cudaError_t e = plan.owned     ? col_launch_bwd_owned(a, plan, s)
                        : do_x && do_y ? col::launch_bwd_k<true, true>(a, plan, s)
                        : do_x       ? col_launch_bwd_x(a, plan, s)
                                     : col_launch_bwd_y(a, plan, s);
  if (e != cudaSuccess) return check_cuda(e, fn, "column backward kernel launch");
  count_launch();
  return GELIB_OK;
}

}  // namespace gelib_b200

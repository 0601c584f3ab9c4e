// inst_refine_l32_12.cu -- instantiation of refine_run.cuh for the L32_12 link format.
#include "refine_run.cuh"

namespace rhmc {

template int rb_group_n<L32_12>(rhmc_ctx *, const L32_12 &, int, const double *, const double *, double2 *, const double2 *, int, int, long *, int *, double);

}  // namespace rhmc

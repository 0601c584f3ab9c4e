// inst_refine_l16_12.cu -- instantiation of refine_run.cuh for the L16_12 link format.
#include "refine_run.cuh"

namespace rhmc {

template int rb_group_n<L16_12>(rhmc_ctx *, const L16_12 &, int, const double *, const double *, double2 *, const double2 *, int, int, long *, int *, double);

}  // namespace rhmc

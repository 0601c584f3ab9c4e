// inst_refine_l64_18.cu -- instantiation of refine_run.cuh for the L64_18 link format.
#include "refine_run.cuh"

namespace rhmc {

template int rb_group_n<L64_18>(rhmc_ctx *, const L64_18 &, int, const double *, const double *, double2 *, const double2 *, int, int, long *, int *, double);

}  // namespace rhmc

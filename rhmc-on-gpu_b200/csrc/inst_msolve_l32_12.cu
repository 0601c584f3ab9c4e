// inst_msolve_l32_12.cu -- instantiation of msolve_run.cuh for the L32_12 link format.
#include "msolve_run.cuh"

namespace rhmc {

template int ms_run<L32_12>(rhmc_ctx *, const L32_12 &, const MSolveArgs &, MSolveInfo *);

}  // namespace rhmc

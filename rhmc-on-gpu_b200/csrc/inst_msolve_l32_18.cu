// inst_msolve_l32_18.cu -- instantiation of msolve_run.cuh for the L32_18 link format.
#include "msolve_run.cuh"

namespace rhmc {

template int ms_run<L32_18>(rhmc_ctx *, const L32_18 &, const MSolveArgs &, MSolveInfo *);

}  // namespace rhmc

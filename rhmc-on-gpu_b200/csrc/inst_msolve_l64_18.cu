// inst_msolve_l64_18.cu -- instantiation of msolve_run.cuh for the L64_18 link format.
#include "msolve_run.cuh"

namespace rhmc {

template int ms_run<L64_18>(rhmc_ctx *, const L64_18 &, const MSolveArgs &, MSolveInfo *);

}  // namespace rhmc

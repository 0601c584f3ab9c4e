// inst_msolve_l64_12.cu -- instantiation of msolve_run.cuh for the L64_12 link format.
#include "msolve_run.cuh"

namespace rhmc {

template int ms_run<L64_12>(rhmc_ctx *, const L64_12 &, const MSolveArgs &, MSolveInfo *);

}  // namespace rhmc

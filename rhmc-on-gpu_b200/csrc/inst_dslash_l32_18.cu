// inst_dslash_l32_18.cu -- instantiation of dslash_run.cuh for the L32_18 link format.
#include "dslash_run.cuh"

namespace rhmc {

template cudaError_t dslash_run<L32_18>(rhmc_ctx *, const L32_18 &, int, void *, const void *, size_t, int, const void *, double, double);

}  // namespace rhmc

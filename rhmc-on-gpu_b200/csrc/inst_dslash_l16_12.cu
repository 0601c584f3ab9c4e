// inst_dslash_l16_12.cu -- instantiation of dslash_run.cuh for the L16_12 link format.
#include "dslash_run.cuh"

namespace rhmc {

template cudaError_t dslash_run<L16_12>(rhmc_ctx *, const L16_12 &, int, void *, const void *, size_t, int, const void *, double, double);

}  // namespace rhmc

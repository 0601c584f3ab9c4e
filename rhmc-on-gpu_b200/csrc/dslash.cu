// dslash.cu -- instantiation and dispatch of the Dslash kernels (dslash.cuh).
#include "context.h"
#include "dslash.cuh"
#include "kernels.h"

namespace rhmc {

// one translation unit per link format (dslash_run.cuh, inst_*.cu)
template <class LF>
cudaError_t dslash_run(rhmc_ctx *c, const LF &lf, int p_out, void *out, const void *in, size_t stride, int n, const void *y,
                       double alpha, double beta);
extern template cudaError_t dslash_run<L64_18>(rhmc_ctx *, const L64_18 &, int, void *, const void *, size_t, int, const void *, double, double);
extern template cudaError_t dslash_run<L64_12>(rhmc_ctx *, const L64_12 &, int, void *, const void *, size_t, int, const void *, double, double);
extern template cudaError_t dslash_run<L32_18>(rhmc_ctx *, const L32_18 &, int, void *, const void *, size_t, int, const void *, double, double);
extern template cudaError_t dslash_run<L32_12>(rhmc_ctx *, const L32_12 &, int, void *, const void *, size_t, int, const void *, double, double);
extern template cudaError_t dslash_run<L16_12>(rhmc_ctx *, const L16_12 &, int, void *, const void *, size_t, int, const void *, double, double);

bool fmt_is_f64(int fmt) { return fmt == RHMC_LINKS_F64_18 || fmt == RHMC_LINKS_F64_12; }

// the largest Dslash grid of any configuration (sizes the per-block reduction partials)
int dslash_grid(rhmc_ctx *c) { return grid_for(c->Vh, DSLASH_MIN_BLOCK); }

// FP64 18-real half-Dslash of one spinor in the reference's site-major layout (A64S) onto the
// output sites [k_lo, k_lo + k_count) only, on stream s (the host-buffer entry point pipelines
// its copies against these slabs)
cudaError_t launch_dslash_f64_range(rhmc_ctx *c, cudaStream_t s, int p_out, void *out, const void *in, int k_lo, int k_count)
{
    L64_18 l18;
    cudaError_t e = links_f64_18(c, &l18);
    if (e != cudaSuccess) return e;
    L64_18A lf;
    lf.p = l18.p;
    lf.Vh = l18.Vh;
    DslashArgs<L64_18A, 1> a;
    memset(&a, 0, sizeof(a));
    a.g = c->g;
    a.p_out = p_out;
    a.links = lf;
    a.in = (const double2 *)in;
    a.out = (double2 *)out;
    a.stride = 3 * (size_t)c->Vh;
    a.beta = 0.5;
    a.k_lo = k_lo;
    a.k_count = k_count;
    c->launches++;
    return dslash_launch<L64_18A, 1, false, false, NoFin>(a, k_count, s);
}

cudaError_t launch_dslash(rhmc_ctx *c, int fmt, int p_out, void *out, const void *in, size_t stride, int n,
                          const void *y, double alpha, double beta, double *partials, int *nblocks)
{
    if (partials) return cudaErrorInvalidValue;  // reductions go through the solver's own launches
    if (nblocks) *nblocks = dslash_grid(c);
    cudaError_t e = cudaSuccess;
    switch (fmt) {
    case RHMC_LINKS_F64_18: { L64_18 lf; e = links_f64_18(c, &lf); if (!e) e = dslash_run(c, lf, p_out, out, in, stride, n, y, alpha, beta); break; }
    case RHMC_LINKS_F64_12: { L64_12 lf; e = links_f64_12(c, &lf); if (!e) e = dslash_run(c, lf, p_out, out, in, stride, n, y, alpha, beta); break; }
    case RHMC_LINKS_F32_18: { L32_18 lf; e = links_f32_18(c, &lf); if (!e) e = dslash_run(c, lf, p_out, out, in, stride, n, y, alpha, beta); break; }
    case RHMC_LINKS_F32_12: { L32_12 lf; e = links_f32_12(c, &lf); if (!e) e = dslash_run(c, lf, p_out, out, in, stride, n, y, alpha, beta); break; }
    case RHMC_LINKS_F16_12: { L16_12 lf; e = links_f16_12(c, &lf); if (!e) e = dslash_run(c, lf, p_out, out, in, stride, n, y, alpha, beta); break; }
    default: return cudaErrorInvalidValue;
    }
    return e;
}

}  // namespace rhmc

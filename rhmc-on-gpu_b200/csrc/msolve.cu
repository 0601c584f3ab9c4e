// msolve.cu -- host orchestration of the multi-shift CG (msolve.cuh): workspace, CUDA-graph
// capture of one delayed-update window of iterations, device-flag polling, the FP64-to-FP32
// precision schedule with reliable updates, and the FP64 true residuals.
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "capi_util.h"
#include "context.h"
#include "kernels.h"
#include "msolve.cuh"
#include "solver.h"

namespace rhmc {

int replay_until_stop(rhmc_ctx *c, cudaGraphExec_t exec, cudaStream_t s, const int *stop, long max_rep, long *replays,
                      int *stop_seen, const char *what)
{
    int *hflag = c->hflags;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    cudaError_t ce = cudaEventCreateWithFlags(&ev[0], cudaEventDisableTiming);
    if (ce == cudaSuccess) ce = cudaEventCreateWithFlags(&ev[1], cudaEventDisableTiming);
    long rep = 0;
    bool done = false;
    hflag[0] = hflag[1] = 0;
    for (; ce == cudaSuccess && rep < max_rep && !done; rep++) {
        ce = cudaGraphLaunch(exec, s);
        if (ce != cudaSuccess) break;
        ce = cudaMemcpyAsync(&hflag[rep & 1], stop, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (ce == cudaSuccess) ce = cudaEventRecord(ev[rep & 1], s);
        if (ce == cudaSuccess && rep >= 1) {
            ce = cudaEventSynchronize(ev[(rep - 1) & 1]);
            if (ce == cudaSuccess && hflag[(rep - 1) & 1]) done = true;
        }
    }
    *replays = rep;
    const cudaError_t cs = cudaStreamSynchronize(s);
    if (ce == cudaSuccess) ce = cs;
    if (ce == cudaSuccess && !done && rep > 0) done = hflag[(rep - 1) & 1] != 0;
    for (cudaEvent_t e : ev)
        if (e) cudaEventDestroy(e);
    *stop_seen = done ? 1 : 0;
    if (ce != cudaSuccess) return cuda_fail(ce, what);
    return RHMC_OK;
}

// one translation unit per link format (msolve_run.cuh, inst_*.cu)
template <class LF>
int ms_run(rhmc_ctx *c, const LF &lf, const MSolveArgs &A, MSolveInfo *info);
extern template int ms_run<L64_18>(rhmc_ctx *, const L64_18 &, const MSolveArgs &, MSolveInfo *);
extern template int ms_run<L64_12>(rhmc_ctx *, const L64_12 &, const MSolveArgs &, MSolveInfo *);
extern template int ms_run<L32_18>(rhmc_ctx *, const L32_18 &, const MSolveArgs &, MSolveInfo *);
extern template int ms_run<L32_12>(rhmc_ctx *, const L32_12 &, const MSolveArgs &, MSolveInfo *);

int msolve_shifted(rhmc_ctx *c, int fmt, const MSolveArgs &A, MSolveInfo *info)
{
    if (A.nshift < 1 || A.nshift > MS_MAX_SHIFT) return fail(RHMC_ERR_ARG, "nshift must be in [1, %d]", MS_MAX_SHIFT);
    if (A.nrhs < 1 || A.nrhs > MS_MAX_RHS) return fail(RHMC_ERR_ARG, "nrhs must be in [1, %d]", MS_MAX_RHS);
    cudaError_t e;
    switch (fmt) {
    case RHMC_LINKS_F64_18: { L64_18 lf; e = links_f64_18(c, &lf); if (e) return cuda_fail(e, "links"); return ms_run(c, lf, A, info); }
    case RHMC_LINKS_F64_12: { L64_12 lf; e = links_f64_12(c, &lf); if (e) return cuda_fail(e, "links"); return ms_run(c, lf, A, info); }
    case RHMC_LINKS_F32_18: { L32_18 lf; e = links_f32_18(c, &lf); if (e) return cuda_fail(e, "links"); return ms_run(c, lf, A, info); }
    case RHMC_LINKS_F32_12: { L32_12 lf; e = links_f32_12(c, &lf); if (e) return cuda_fail(e, "links"); return ms_run(c, lf, A, info); }
    default: return fail(RHMC_ERR_ARG, "bad link format %d", fmt);
    }
}

// ------------------------------------------------------------------ true residuals (FP64)
struct ResidSys {
    int rhs[8];
    double coef[8];
};

// partial |b_rhs(j) - coef_j x_j - t_j|^2, j < J, with t_j = -Deo Doe x_j
__global__ void __launch_bounds__(VEC_BLOCK) resid_norm_kernel(int Vh, size_t stride, int J, ResidSys sys,
                                                                const double2 *__restrict__ b, const double2 *__restrict__ x,
                                                                const double2 *__restrict__ t, double *partials)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    double red[8];
#pragma unroll
    for (int j = 0; j < 8; j++) red[j] = 0.0;
    if (k < Vh) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (j >= J) break;
            for (int c = 0; c < 3; c++) {
                const size_t o = (size_t)c * Vh + k;
                const double2 bv = b[sys.rhs[j] * stride + o], xv = x[j * stride + o], tv = t[j * stride + o];
                const double re = bv.x - sys.coef[j] * xv.x - tv.x, im = bv.y - sys.coef[j] * xv.y - tv.y;
                red[j] += re * re + im * im;
            }
        }
    }
    __shared__ double smem[8 * 32];
    block_sum<8>(red, smem);
    if (threadIdx.x == 0)
        for (int j = 0; j < J; j++) partials[(size_t)blockIdx.x * 8 + j] = red[j];
}

int true_residuals(rhmc_ctx *c, int nshift, const double *shifts, int nrhs, const double2 *x, const double2 *b, double *out)
{
    const int Vh = (int)c->Vh;
    const size_t stride = 3 * (size_t)Vh;
    void *h, *t, *part;
    CK(c->ws.get("tr_h", 8 * stride * sizeof(double2), &h));
    CK(c->ws.get("tr_t", 8 * stride * sizeof(double2), &t));
    const int gv = grid_for(c->Vh, VEC_BLOCK);
    CK(c->ws.get("tr_part", (size_t)gv * 8 * sizeof(double), &part));
    std::vector<double> hp((size_t)gv * 8);
    const int total = nrhs * nshift;
    for (int j0 = 0; j0 < total; j0 += 8) {
        const int J = total - j0 < 8 ? total - j0 : 8;
        ResidSys sys;
        for (int j = 0; j < 8; j++) {
            const int q = j0 + (j < J ? j : 0);
            sys.rhs[j] = q / nshift;
            sys.coef[j] = c->mass * c->mass + shifts[q];  // [nrhs][nshift], q = r * nshift + i
        }
        const double2 *xj = x + (size_t)j0 * stride;
        cudaError_t e = launch_dslash(c, RHMC_LINKS_F64_18, 1, h, xj, stride, J, nullptr, 0.0, 0.5, nullptr, nullptr);
        if (e == cudaSuccess) e = launch_dslash(c, RHMC_LINKS_F64_18, 0, t, h, stride, J, nullptr, 0.0, -0.5, nullptr, nullptr);
        if (e != cudaSuccess) return cuda_fail(e, "true_residuals");
        resid_norm_kernel<<<gv, VEC_BLOCK, 0, c->stream>>>(Vh, stride, J, sys, b, xj, (const double2 *)t, (double *)part);
        c->launches++;
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(hp.data(), part, (size_t)gv * 8 * sizeof(double), cudaMemcpyDeviceToHost, c->stream));
        CK(cudaStreamSynchronize(c->stream));
        for (int j = 0; j < J; j++) {
            double s = 0.0;
            for (int g = 0; g < gv; g++) s += hp[(size_t)g * 8 + j];
            out[j0 + j] = s;
        }
    }
    return RHMC_OK;
}

}  // namespace rhmc

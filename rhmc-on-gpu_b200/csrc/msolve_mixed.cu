// msolve_mixed.cu -- the mixed-precision batched multi-shift solver and the extern "C"
// multi-shift entry points.
//
// Mixed mode (no counterpart in the reference, which picks FP32 or FP64 per call by the
// requested residual, lib/Action/Inverter/cu_inverter.cc:45-60):
//   Phase A  multi-shift CG (msolve.cuh) with FP32 links/vectors, all right-hand sides
//            batched (every link load serves every RHS), base operator M^dag M + sigma_min,
//            until every shift reaches tol_A |b| (FP64 scalars and reductions).
//   Phase B  every (RHS, shift) system is refined by FP32 CG inside an FP64 defect correction:
//            once a system's FP32 residual has dropped by a factor delta since its last
//            update it waits; every n_ru iterations the waiting systems add their FP32
//            correction to the FP64 solution, recompute the residual b - (M^dag M + sigma) x
//            in FP64 with FP64 links and restart their FP32 CG from it (keeping the old search
//            direction across the update diverged for kappa ~ 1e5).  A system is finished only
//            when that FP64 true residual is <= the target.  Systems are sorted by shift and
//            refined in batches of up to 8 that share link loads.
// With fmt = RHMC_LINKS_F16_12 phase A runs on FP32 12-real links and phase B's sloppy CG keeps
// its links, residual, search direction and Dslash intermediates in half precision with a
// per-site scale (H16S; the correction accumulates in FP32), which halves its memory traffic.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <chrono>
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

// iterations between reliable updates of the FP32 multi-shift phase
constexpr int MX_RU_ITERS = 32;

// one translation unit per link format (refine_run.cuh, inst_*.cu)
template <class LF>
int rb_group_n(rhmc_ctx *c, const LF &lf, int n, const double *coef, const double *tgt, double2 *xg, const double2 *bg,
               int max_iter, int n_ru, long *iters, int *ru, double ru_delta);
extern template int rb_group_n<L64_18>(rhmc_ctx *, const L64_18 &, int, const double *, const double *, double2 *, const double2 *, int, int, long *, int *, double);
extern template int rb_group_n<L32_18>(rhmc_ctx *, const L32_18 &, int, const double *, const double *, double2 *, const double2 *, int, int, long *, int *, double);
extern template int rb_group_n<L32_12>(rhmc_ctx *, const L32_12 &, int, const double *, const double *, double2 *, const double2 *, int, int, long *, int *, double);
extern template int rb_group_n<L16_12>(rhmc_ctx *, const L16_12 &, int, const double *, const double *, double2 *, const double2 *, int, int, long *, int *, double);

// Refine all (rhs, shift) systems of x (FP64 internal [nrhs][nshift]) to |b - A_sigma x| <= res.
template <class LF>
static int refine_all(rhmc_ctx *c, const LF &lf, int nshift, const double *shifts, int nrhs, double res, int max_iter,
                      double2 *x, const double2 *b, long *iters, int *ru, double ru_delta, int max_batch = RB_MAX,
                      const double *skip_below = nullptr, int *nsys = nullptr)
{
    const size_t stride = 3 * (size_t)c->Vh;
    const size_t v64 = stride * sizeof(double2);
    void *xg, *bg;
    CK(c->ws.get("rb_xg", RB_MAX * v64, &xg));
    CK(c->ws.get("rb_bg", RB_MAX * v64, &bg));
    std::vector<int> order;
    for (int q = 0; q < nshift * nrhs; q++)
        if (!skip_below || skip_below[q] > res) order.push_back(q);
    std::stable_sort(order.begin(), order.end(), [&](int a, int bq) { return shifts[a] < shifts[bq]; });
    if (nsys) *nsys = (int)order.size();
    const double m2 = c->mass * c->mass;
    size_t g0 = 0;
    while (g0 < order.size()) {
        const size_t left = order.size() - g0;
        int n = left >= 8 ? 8 : (left >= 4 ? 4 : (int)left);  // instantiated batch widths
        if (n > max_batch) n = max_batch;
        double coef[RB_MAX], tgt[RB_MAX];
        for (int j = 0; j < n; j++) {
            const int q = order[g0 + j];
            coef[j] = m2 + shifts[q];  // shifts [nrhs][nshift], q = r * nshift + i
            tgt[j] = res;
            CK(cudaMemcpyAsync((double2 *)xg + j * stride, x + (size_t)q * stride, v64, cudaMemcpyDeviceToDevice, c->stream));
            CK(cudaMemcpyAsync((double2 *)bg + j * stride, b + (size_t)(q / nshift) * stride, v64, cudaMemcpyDeviceToDevice,
                               c->stream));
        }
        // iterations between reliable-update stages: a waiting system idles until the next one, and the
        // stage costs a system that needs none only its skipped launches
        const int n_ru = 8;
        int rc = rb_group_n(c, lf, n, coef, tgt, (double2 *)xg, (const double2 *)bg, max_iter, n_ru, iters, ru, ru_delta);
        if (rc) return rc;
        for (int j = 0; j < n; j++) {
            const int q = order[g0 + j];
            CK(cudaMemcpyAsync(x + (size_t)q * stride, (double2 *)xg + j * stride, v64, cudaMemcpyDeviceToDevice, c->stream));
        }
        g0 += n;
    }
    return RHMC_OK;
}

int msolve_mixed(rhmc_ctx *c, int fmt, int nshift, const double *shifts, int nrhs, double res, int max_iter, double tolA,
                 double ru_delta, double2 *x, const double2 *b, rhmc_msolve_info *info)
{
    auto t0 = std::chrono::steady_clock::now();
    std::vector<double> base(nrhs);  // each RHS iterates on its smallest pole
    for (int r = 0; r < nrhs; r++) {
        base[r] = shifts[(size_t)r * nshift];
        for (int i = 1; i < nshift; i++) base[r] = std::min(base[r], shifts[(size_t)r * nshift + i]);
    }
    MSolveArgs A;
    A.nshift = nshift;
    A.nrhs = nrhs;
    A.shift = shifts;
    A.base = base.data();
    A.max_iter = max_iter;
    A.stop_on_frozen = 1;
    A.b = b;
    MSolveInfo mi;
    memset(&mi, 0, sizeof(mi));
    std::vector<double> tgt(nshift);
    std::vector<double> tr;  // FP64 true residuals after the multi-shift phase
    int it_hi[8] = {0};      // iterations of each RHS in the FP64 part of the precision schedule
    int rc;
    const bool f64a = fmt_is_f64(fmt);
    if (f64a) {
        // Phase A in FP64 (compressed links when fmt is 12-real), straight into x
        for (double &t : tgt) t = res;
        A.tgt = tgt.data();
        A.res_base = res;
        A.x = x;
        rc = msolve_shifted(c, fmt, A, &mi);
        if (rc && rc != RHMC_ERR_MAXITER) return rc;
        tr.resize((size_t)nshift * nrhs);
        rc = true_residuals(c, nshift, shifts, nrhs, x, b, tr.data());
        if (rc) return rc;
        for (double &v : tr) v = std::sqrt(v);
    } else {
        // Precision schedule: FP64 (12-real links) until |r| <= tol_A |b| for every RHS, then the
        // same recurrences resumed with FP32 links and base vectors, FP64 shifted vectors and a
        // reliable update of the base system every MX_RU_ITERS iterations, to the final target.
        for (double &t : tgt) t = res;
        A.tgt = tgt.data();
        A.res_base = res;
        A.x = x;
        A.tau = tolA;
        rc = msolve_shifted(c, RHMC_LINKS_F64_12, A, &mi);
        if (rc && rc != RHMC_ERR_MAXITER) return rc;
        for (int r = 0; r < nrhs && r < 8; r++) it_hi[r] = mi.iters[r];
        if (rc == RHMC_OK) {
            A.fresh = 0;
            A.tau = 0.0;
            A.ru_every = MX_RU_ITERS;
            // half refinement follows an FP32 multi-shift on 12-real links
            rc = msolve_shifted(c, fmt == RHMC_LINKS_F16_12 ? RHMC_LINKS_F32_12 : fmt, A, &mi);
            if (rc && rc != RHMC_ERR_MAXITER) return rc;
        }
        tr.resize((size_t)nshift * nrhs);
        rc = true_residuals(c, nshift, shifts, nrhs, x, b, tr.data());
        if (rc) return rc;
        for (double &v : tr) v = std::sqrt(v);
    }
    const double t_a = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    long it_b = 0;
    int ru = 0, nsys = 0;
    // refinement: half links and spinors for F16_12, else FP32 sloppy links of the matching width
    if (fmt == RHMC_LINKS_F16_12) {
        L16_12 lf;
        CK(links_f16_12(c, &lf));
        rc = refine_all(c, lf, nshift, shifts, nrhs, res, max_iter, x, b, &it_b, &ru, ru_delta, RB_MAX,
                        tr.empty() ? nullptr : tr.data(), &nsys);
    } else if (fmt == RHMC_LINKS_F32_18 || fmt == RHMC_LINKS_F64_18) {
        L32_18 lf;
        CK(links_f32_18(c, &lf));
        rc = refine_all(c, lf, nshift, shifts, nrhs, res, max_iter, x, b, &it_b, &ru, ru_delta, RB_MAX,
                        tr.empty() ? nullptr : tr.data(), &nsys);
    } else {
        L32_12 lf;
        CK(links_f32_12(c, &lf));
        rc = refine_all(c, lf, nshift, shifts, nrhs, res, max_iter, x, b, &it_b, &ru, ru_delta, RB_MAX,
                        tr.empty() ? nullptr : tr.data(), &nsys);
    }
    CK(cudaStreamSynchronize(c->stream));
    if (info) {
        info->status = rc;
        for (int r = 0; r < nrhs && r < 8; r++) info->iters[r] = mi.iters[r];
        info->refine_iters = it_b;
        info->reliable_updates = ru;
        info->seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        info->seconds_phase_a = t_a;
        info->systems_refined = nsys;
        for (int r = 0; r < nrhs && r < 8; r++) info->iters_fp64 += f64a ? mi.iters[r] : it_hi[r];
        info->ms_reliable_updates = f64a ? 0 : mi.ru_count;
    }
    return rc;
}

}  // namespace rhmc

using namespace rhmc;

// multi-shift iteration counts of right-hand sides first..first+n-1 into info (the per-RHS
// array holds the first 8; the total and the maximum cover all of them)
static void add_iters(rhmc_msolve_info *info, int first, const int *it, int n)
{
    if (!info) return;
    for (int j = 0; j < n; j++) {
        if (first + j < 8) info->iters[first + j] = it[j];
        info->iters_total += it[j];
        if (it[j] > info->iters_max) info->iters_max = it[j];
    }
}

// sh: the pole sets [nrhs][nshift]
static int msolve_fp64(rhmc_ctx *c, const rhmc_msolve_params *P, const double *sh, double2 *x, const double2 *b,
                       rhmc_msolve_info *info)
{
    const size_t stride = 3 * (size_t)c->Vh;
    std::vector<double> tgt(P->nshift, P->residual), zero(MS_MAX_RHS, 0.0);
    int done = 0, rc = RHMC_OK;
    auto t0 = std::chrono::steady_clock::now();
    while (done < P->nrhs) {
        const int left = P->nrhs - done;
        const int n = left >= 8 ? 8 : (left >= 4 ? 4 : left);
        MSolveArgs A;
        A.nshift = P->nshift;
        A.nrhs = n;
        A.shift = sh + (size_t)done * P->nshift;
        A.base = zero.data();  // the reference iterates on M^dag M itself
        A.tgt = tgt.data();
        A.res_base = P->residual;
        A.max_iter = P->max_iter;
        A.stop_on_frozen = 1;
        A.b = b + (size_t)done * stride;
        A.x = x + (size_t)done * P->nshift * stride;
        MSolveInfo mi;
        memset(&mi, 0, sizeof(mi));
        rc = msolve_shifted(c, P->fmt, A, &mi);
        add_iters(info, done, mi.iters, n);
        if (rc) break;
        done += n;
    }
    long it_b = 0;
    int ru = 0, nsys = 0;
    cudaStreamSynchronize(c->stream);
    const double t_a = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    if (rc == RHMC_OK && P->certify) {
        // FP64 defect correction of every system whose FP64 true residual is above target
        std::vector<double> tr((size_t)P->nshift * P->nrhs);
        rc = true_residuals(c, P->nshift, sh, P->nrhs, x, b, tr.data());
        for (double &v : tr) v = std::sqrt(v);
        if (rc == RHMC_OK) {
            L64_18 lf;
            CK(links_f64_18(c, &lf));
            rc = refine_all(c, lf, P->nshift, sh, P->nrhs, P->residual, P->max_iter, x, b, &it_b, &ru, 0.05, 1, tr.data(), &nsys);
        }
        cudaStreamSynchronize(c->stream);
    }
    if (info) {
        info->status = rc;
        info->refine_iters = it_b;
        info->reliable_updates = ru;
        info->seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        info->seconds_phase_a = t_a;
        info->systems_refined = nsys;
    }
    return rc;
}

// The reference's single-precision path (cuda_shifted_inverter, lib/Cuda/cuda_inverter.cu:647-857):
// the same recurrences with FP32 links and base vectors and FP64 scalars.  The shifted solutions
// and directions are accumulated in FP64 (the reference keeps them in FP32), which removes their
// storage rounding from the true residual; they are written straight into x.
static int msolve_fp32(rhmc_ctx *c, const rhmc_msolve_params *P, const double *sh, double2 *x, const double2 *b,
                       rhmc_msolve_info *info)
{
    const size_t stride = 3 * (size_t)c->Vh;
    std::vector<double> tgt(P->nshift, P->residual), zero(MS_MAX_RHS, 0.0);
    auto t0 = std::chrono::steady_clock::now();
    int done = 0, rc = RHMC_OK;
    while (done < P->nrhs) {
        const int left = P->nrhs - done;
        const int n = left >= 8 ? 8 : (left >= 4 ? 4 : left);
        MSolveArgs A;
        A.nshift = P->nshift;
        A.nrhs = n;
        A.shift = sh + (size_t)done * P->nshift;
        A.base = zero.data();
        A.tgt = tgt.data();
        A.res_base = P->residual;
        A.max_iter = P->max_iter;
        A.stop_on_frozen = 1;
        A.b = b + (size_t)done * stride;
        A.x = x + (size_t)done * P->nshift * stride;
        MSolveInfo mi;
        memset(&mi, 0, sizeof(mi));
        rc = msolve_shifted(c, P->fmt, A, &mi);
        add_iters(info, done, mi.iters, n);
        if (rc) break;
        done += n;
    }
    CK(cudaStreamSynchronize(c->stream));
    if (info) {
        info->status = rc;
        info->seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    }
    return rc;
}

static int msolve_any(rhmc_ctx *c, const rhmc_msolve_params *P, double *x, const double *b, rhmc_msolve_info *info)
{
    if (P->nshift < 1 || P->nshift > MS_MAX_SHIFT) return fail(RHMC_ERR_ARG, "nshift must be in [1, %d]", MS_MAX_SHIFT);
    if (P->nrhs < 1) return fail(RHMC_ERR_ARG, "nrhs must be >= 1");
    if (P->max_iter < 1) return fail(RHMC_ERR_ARG, "max_iter must be >= 1");
    // the pole set of every RHS: rhs_shifts [nrhs][nshift], or shifts for all of them
    std::vector<double> sh((size_t)P->nrhs * P->nshift);
    for (int r = 0; r < P->nrhs; r++)
        for (int i = 0; i < P->nshift; i++)
            sh[(size_t)r * P->nshift + i] = P->rhs_shifts ? P->rhs_shifts[(size_t)r * P->nshift + i] : P->shifts[i];
    for (double v : sh)
        if (!(v >= 0.0)) return fail(RHMC_ERR_ARG, "shifts must be >= 0");
    if (info) memset(info, 0, sizeof(*info));
    if (P->mode == RHMC_MSOLVE_FP64) {
        if (P->fmt != RHMC_LINKS_F64_18 && P->fmt != RHMC_LINKS_F64_12) return fail(RHMC_ERR_ARG, "FP64 mode needs FP64 links");
        return msolve_fp64(c, P, sh.data(), (double2 *)x, (const double2 *)b, info);
    }
    if (P->mode == RHMC_MSOLVE_FP32) {
        if (P->fmt != RHMC_LINKS_F32_18 && P->fmt != RHMC_LINKS_F32_12) return fail(RHMC_ERR_ARG, "FP32 mode needs FP32 links");
        return msolve_fp32(c, P, sh.data(), (double2 *)x, (const double2 *)b, info);
    }
    if (P->mode == RHMC_MSOLVE_MIXED) {
        if (P->fmt < 0 || P->fmt > RHMC_LINKS_F16_12) return fail(RHMC_ERR_ARG, "bad link format %d", P->fmt);
        // the hand-over of the precision schedule: the caller's, or 1e-3 |b| but at most
        // MS_TAU_REACH above the target (negative: automatic)
        const double tolA = P->tol_phase_a > 0 ? P->tol_phase_a : -1e-3;
        const double rud = (P->ru_delta > 0 && P->ru_delta < 1) ? P->ru_delta : 0.05;
        // batches of 8, 4, 3, 2 or 1 right-hand sides (the widths the kernels are built for)
        const size_t stride = 3 * (size_t)c->Vh;
        int done = 0, rc = RHMC_OK;
        rhmc_msolve_info agg, part;
        memset(&agg, 0, sizeof(agg));
        while (done < P->nrhs && rc == RHMC_OK) {
            const int left = P->nrhs - done;
            const int n = left >= 8 ? 8 : (left >= 4 ? 4 : left);
            memset(&part, 0, sizeof(part));
            rc = msolve_mixed(c, P->fmt, P->nshift, sh.data() + (size_t)done * P->nshift, n, P->residual, P->max_iter, tolA, rud,
                              (double2 *)x + (size_t)done * P->nshift * stride, (const double2 *)b + (size_t)done * stride, &part);
            add_iters(&agg, done, part.iters, n);
            agg.refine_iters += part.refine_iters;
            agg.reliable_updates += part.reliable_updates;
            agg.seconds += part.seconds;
            agg.seconds_phase_a += part.seconds_phase_a;
            agg.systems_refined += part.systems_refined;
            agg.iters_fp64 += part.iters_fp64;
            agg.ms_reliable_updates += part.ms_reliable_updates;
            done += n;
        }
        agg.status = rc;
        if (info) *info = agg;
        return rc;
    }
    return fail(RHMC_ERR_ARG, "bad solver mode %d", P->mode);
}

extern "C" {

int rhmc_msolve(rhmc_ctx *c, const rhmc_msolve_params *P, double *x, const double *b, rhmc_msolve_info *info)
{
    if (!c || !P || !x || !b || (!P->shifts && !P->rhs_shifts)) return fail(RHMC_ERR_ARG, "null argument");
    c->ws.in_solve = true;
    c->ws.out_of_memory = false;
    c->window.was_long = false;
    int rc = msolve_any(c, P, x, b, info);
    if (rc == RHMC_ERR_CUDA && c->ws.out_of_memory && c->window.was_long) {
        // Out of memory beside a ring of whole windows: once more with half ones, whose ring is half as
        // long, unless x overlaps b, which then is not what it was.
        const double *xe = x + (size_t)P->nrhs * P->nshift * 6 * c->Vh, *be = b + (size_t)P->nrhs * 6 * c->Vh;
        cudaStreamSynchronize(c->stream);
        c->ws.drop_rings();
        if (xe <= b || be <= x) {
            c->window.half_only = true;
            rc = msolve_any(c, P, x, b, info);
            c->window.half_only = false;
        }
    }
    c->ws.in_solve = false;
    return rc;
}

int rhmc_msolve_window(const rhmc_ctx *c, int *iterations)
{
    if (!c || !iterations) return fail(RHMC_ERR_ARG, "null argument");
    *iterations = c->window.last;
    return RHMC_OK;
}

int rhmc_msolve_one_kernel(rhmc_ctx *c, int enable)
{
    if (!c) return fail(RHMC_ERR_ARG, "null context");
    c->one_kernel = enable != 0;
    return RHMC_OK;
}

int rhmc_msolve_host(rhmc_ctx *c, const rhmc_msolve_params *P, double *x, const double *b, rhmc_msolve_info *info)
{
    if (!c || !P || !x || !b) return fail(RHMC_ERR_ARG, "null argument");
    const size_t stride = 3 * (size_t)c->Vh;
    const size_t nb = (size_t)P->nrhs, nx = (size_t)P->nrhs * P->nshift;
    void *bi, *xi, *tmp;
    CK(c->ws.get("mh_b", nb * stride * sizeof(double2), &bi));
    CK(c->ws.get("mh_x", nx * stride * sizeof(double2), &xi));
    CK(c->ws.get("mh_tmp", (nx > nb ? nx : nb) * stride * sizeof(double2), &tmp));
    CK(cudaMemcpyAsync(tmp, b, nb * stride * sizeof(double2), cudaMemcpyHostToDevice, c->stream));
    launch_spinor_to_internal(c, RHMC_LINKS_F64_18, bi, (const double *)tmp, (int)nb);
    int rc = rhmc_msolve(c, P, (double *)xi, (const double *)bi, info);
    if (rc) return rc;
    launch_spinor_from_internal(c, RHMC_LINKS_F64_18, (double *)tmp, xi, (int)nx);
    CK(cudaMemcpyAsync(x, tmp, nx * stride * sizeof(double2), cudaMemcpyDeviceToHost, c->stream));
    CK(cudaStreamSynchronize(c->stream));
    return RHMC_OK;
}

int rhmc_true_residuals(rhmc_ctx *c, int nshift, const double *shifts, int nrhs, const double *x, const double *b, double *out)
{
    if (!c || !shifts || !x || !b || !out || nshift < 1 || nrhs < 1) return fail(RHMC_ERR_ARG, "bad argument");
    std::vector<double> sh((size_t)nrhs * nshift);
    for (int r = 0; r < nrhs; r++)
        for (int i = 0; i < nshift; i++) sh[(size_t)r * nshift + i] = shifts[i];
    int rc = true_residuals(c, nshift, sh.data(), nrhs, (const double2 *)x, (const double2 *)b, out);
    if (rc) return rc;
    for (int i = 0; i < nshift * nrhs; i++) out[i] = std::sqrt(out[i]);
    return RHMC_OK;
}

}  // extern "C"

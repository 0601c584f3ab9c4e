// refine_run.cuh -- Phase B of the mixed solver (msolve_mixed.cu): the refinement of a batch of
// (RHS, shift) systems by sloppy CG over link format LF inside an FP64 defect correction.  One
// translation unit per link format instantiates rb_group_n (inst_*.cu); msolve_mixed.cu declares
// them extern.
#pragma once
#include <cmath>
#include <cstring>
#include <type_traits>

#include "capi_util.h"
#include "context.h"
#include "kernels.h"
#include "msolve.cuh"
#include "solver.h"

namespace rhmc {

struct ResidCoef {
    double coef[8];  // mass^2 + sigma of each batched system
};

struct RBState {
    int stop;         // every system converged (or failed)
    int status;       // 0 ok, 2 non-finite
    int nsys;
    int first;        // the next reliable update is the initial one (sets p = r)
    int ru_count;
    int iters;        // sloppy iterations performed
    int any_pending;  // some system waits for a reliable update
    int ru_max;       // force an update after this many sloppy iterations
    double delta2;    // update when |r_sloppy|^2 <= delta2 |r at last update|^2
    double tgt[RB_MAX];
    double rr[RB_MAX];     // |r_sloppy|^2
    double rr_ru[RB_MAX];  // |r|^2 at the last reliable update
    double alpha[RB_MAX], beta[RB_MAX];
    double r2true[RB_MAX];
    int conv[RB_MAX];
    int pending[RB_MAX];   // waiting for the next reliable update
    int hold[RB_MAX];      // skipped by the sloppy iteration
    int since[RB_MAX];     // sloppy iterations since the last update
};

// x += xs (FP64 += the sloppy accumulator X), xs = 0, for systems not yet converged
template <int NR, typename X>
__global__ void __launch_bounds__(VEC_BLOCK) rb_accum_kernel(int Vh, size_t stride, double2 *x, X *xs, const RBState *st)
{
    if (*(volatile const int *)&st->stop || !*(volatile const int *)&st->any_pending) return;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= Vh) return;
#pragma unroll
    for (int j = 0; j < NR; j++) {
        if (st->conv[j] || !st->pending[j]) continue;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const size_t o = j * stride + (size_t)c * Vh + k;
            double2 xv = x[o];
            X d = xs[o];
            xv.x += (double)d.x;
            xv.y += (double)d.y;
            x[o] = xv;
            d.x = 0;
            d.y = 0;
            xs[o] = d;
        }
    }
}

template <int NR>
struct FinRU {
    RBState *st;
    __device__ void operator()(const double *tot) const
    {
        if (threadIdx.x != 0) return;
        int all = 1;
        for (int j = 0; j < NR; j++) {
            if (st->conv[j]) continue;
            if (st->pending[j]) {
                const double r2 = tot[j];
                st->pending[j] = 0;
                st->since[j] = 0;
                if (!isfinite(r2)) {
                    st->status = 2;
                    st->conv[j] = 1;
                    continue;
                }
                st->r2true[j] = r2;
                st->rr[j] = r2;
                st->rr_ru[j] = r2;
                if (sqrt(r2) <= st->tgt[j]) st->conv[j] = 1;
            }
            all &= st->conv[j];
        }
        st->first = 0;
        st->ru_count++;
        st->any_pending = 0;
        if (all) st->stop = 1;
    }
};

// r = b - coef*x - t (FP64), rs = r in the sloppy storage S, |r|^2; the search direction is
// restarted from it (p = rs)
template <int NR, class S>
__global__ void __launch_bounds__(VEC_BLOCK) rb_resid_kernel(int Vh, size_t stride, size_t sstride, const double2 *__restrict__ b,
                                                              const double2 *__restrict__ x, const double2 *__restrict__ t,
                                                              typename S::elem *rs, typename S::elem *p, ResidCoef co,
                                                              double *partials, unsigned *ticket, RBState *st)
{
    if (*(volatile const int *)&st->stop || !*(volatile const int *)&st->any_pending) return;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    double red[NR];
#pragma unroll
    for (int j = 0; j < NR; j++) red[j] = 0.0;
    if (k < Vh) {
#pragma unroll
        for (int j = 0; j < NR; j++) {
            if (st->conv[j] || !st->pending[j]) continue;
            vec3<double> r;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const size_t o = j * stride + (size_t)c * Vh + k;
                const double2 bv = b[o], xv = x[o], tv = t[o];
                const double re = bv.x - co.coef[j] * xv.x - tv.x, im = bv.y - co.coef[j] * xv.y - tv.y;
                red[j] += dot2(re, re, im, im);
                r.c[c] = mk<double>(re, im);
            }
            S::template store<double>(rs + j * sstride, Vh, k, r);
            S::template store<double>(p + j * sstride, Vh, k, r);
        }
    }
    FinRU<NR> fin{st};
    reduce_finalize<NR>(red, partials, ticket, fin);
}

template <int NR>
struct FinRBAlpha {
    RBState *st;
    __device__ void operator()(const double *tot) const
    {
        if (threadIdx.x != 0) return;
        for (int j = 0; j < NR; j++) {
            const double pap = tot[j];
            st->hold[j] = st->pending[j];
            const int skip = st->conv[j] || st->hold[j];
            st->alpha[j] = (skip || !(pap > 0.0)) ? 0.0 : st->rr[j] / pap;
            if (!skip && !isfinite(pap)) st->status = 2;
        }
        st->iters++;
    }
};

template <int NR>
struct FinRBBeta {
    RBState *st;
    __device__ void operator()(const double *tot) const
    {
        if (threadIdx.x != 0) return;
        for (int j = 0; j < NR; j++) {
            if (st->conv[j] || st->hold[j]) { st->beta[j] = 0.0; continue; }
            const double rn = tot[j];
            st->beta[j] = (st->rr[j] > 0.0) ? rn / st->rr[j] : 0.0;
            st->rr[j] = rn;
            st->since[j]++;
            // update after a drop by delta (also below the target: ending there, at a tenth of it, took
            // 120 batched iterations instead of 136 for 20 systems at 32^4, but left a mean true residual
            // of 0.298 of the target instead of 0.293), after ru_max iterations, or when the FP32
            // iteration stops making progress (its residual above 4x the last true one)
            if (rn <= st->delta2 * st->rr_ru[j] || st->since[j] >= st->ru_max || !isfinite(rn) || rn > 4.0 * st->rr_ru[j]) {
                st->pending[j] = 1;
                st->any_pending = 1;
            }
        }
    }
};

// xs += alpha p ; rs -= alpha Ap ; |rs|^2  (p, Ap, rs in the sloppy storage S; xs of type X)
template <int NR, class S, typename X>
__global__ void __launch_bounds__(VEC_BLOCK) rb_xr_kernel(int Vh, size_t stride, size_t sstride, X *xs, typename S::elem *rs,
                                                           const typename S::elem *__restrict__ p,
                                                           const typename S::elem *__restrict__ ap, double *partials,
                                                           unsigned *ticket, RBState *st)
{
    typedef typename S::real Rs;
    if (*(volatile const int *)&st->stop) return;
    // tiles of VEC_BLOCK sites walked by a persistent grid (persistent_grid)
    const int ntiles = (Vh + VEC_BLOCK - 1) / VEC_BLOCK;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int k = tile * VEC_BLOCK + threadIdx.x;
        double red[NR];
#pragma unroll
        for (int j = 0; j < NR; j++) red[j] = 0.0;
        if (k < Vh) {
#pragma unroll
            for (int j = 0; j < NR; j++) {
                if (st->conv[j] || st->hold[j]) continue;
                const Rs a = (Rs)st->alpha[j];
                const vec3<Rs> pv = S::template load<Rs>(p + j * sstride, Vh, k),
                               av = S::template load<Rs>(ap + j * sstride, Vh, k);
                vec3<Rs> rv = S::template load<Rs>(rs + j * sstride, Vh, k);
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const size_t o = j * stride + (size_t)c * Vh + k;
                    X xv = xs[o];
                    xv.x += a * pv.c[c].re;
                    xv.y += a * pv.c[c].im;
                    xs[o] = xv;
                    rv.c[c].re -= a * av.c[c].re;
                    rv.c[c].im -= a * av.c[c].im;
                    red[j] += dot2((double)rv.c[c].re, (double)rv.c[c].re, (double)rv.c[c].im, (double)rv.c[c].im);
                }
                S::template store<Rs>(rs + j * sstride, Vh, k, rv);
            }
        }
        reduce_tile<NR>(red, partials, tile);
    }
    FinRBBeta<NR> fin{st};
    reduce_last<NR>(partials, ticket, ntiles * (VEC_BLOCK / RED_CHUNK), fin);
}

// p = rs + beta p
template <int NR, class S>
__global__ void __launch_bounds__(VEC_BLOCK) rb_p_kernel(int Vh, size_t sstride, int down, const typename S::elem *__restrict__ rs,
                                                          typename S::elem *p, const RBState *st)
{
    typedef typename S::real Rs;
    if (*(volatile const int *)&st->stop) return;
    const int k = (down ? gridDim.x - 1 - blockIdx.x : blockIdx.x) * blockDim.x + threadIdx.x;  // rb_xr_kernel went upwards
    if (k >= Vh) return;
#pragma unroll
    for (int j = 0; j < NR; j++) {
        if (st->conv[j] || st->hold[j]) continue;
        const Rs be = (Rs)st->beta[j];
        const vec3<Rs> rv = S::template load<Rs>(rs + j * sstride, Vh, k);
        vec3<Rs> pv = S::template load<Rs>(p + j * sstride, Vh, k);
#pragma unroll
        for (int c = 0; c < 3; c++) {
            pv.c[c].re = rv.c[c].re + be * pv.c[c].re;
            pv.c[c].im = rv.c[c].im + be * pv.c[c].im;
        }
        S::template store<Rs>(p + j * sstride, Vh, k, pv);
    }
}

// ------------------------------------------------------------------ Phase B driver
template <class LF, int NR>
static int rb_group(rhmc_ctx *c, const LF &lf, const double *coef, const double *tgt, double2 *xg, const double2 *bg,
                    int max_iter, int n_ru, long *iters_out, int *ru_out, double ru_delta)
{
    AuxScope aux_scope(c);
    cudaStream_t s_ = c->aux;
    const int Vh = (int)c->Vh;
    const size_t stride = 3 * (size_t)Vh;  // FP64 fields and the accumulator xs
    void *xs, *rs, *p, *ap, *h, *h64, *t64, *stv, *part, *tick;
    typedef typename LF::real Rs;
    typedef typename LF::store S;  // sloppy storage of rs, p, ap, h
    typedef typename S::elem E;
    typedef typename std::conditional<std::is_same<S, F64S>::value, double2, float2>::type X;
    const size_t sstride = (size_t)S::planes * Vh;
    const size_t vs = sstride * sizeof(E), vx = stride * sizeof(X), v64 = stride * sizeof(double2);
    CK(c->ws.get("rb_xs", NR * vx, &xs));
    CK(c->ws.get("rb_rs", NR * vs, &rs));
    CK(c->ws.get("rb_p", NR * vs, &p));
    CK(c->ws.get("rb_ap", NR * vs, &ap));
    CK(c->ws.get("rb_h", NR * vs, &h));
    CK(c->ws.get("rb_h64", NR * v64, &h64));
    CK(c->ws.get("rb_t64", NR * v64, &t64));
    CK(c->ws.get("rb_state", sizeof(RBState), &stv));
    const int gv = grid_for(Vh, VEC_BLOCK);
    CK(c->ws.get("rb_partials", (size_t)red_chunks(Vh) * 2 * NR * sizeof(double), &part));
    CK(c->ws.get("rb_tickets", 4 * sizeof(unsigned), &tick));
    L64_18 l64;
    CK(links_f64_18(c, &l64));
    RBState *st = (RBState *)stv;
    unsigned *tk = (unsigned *)tick;
    double *pt = (double *)part;

    RBState h0;
    memset(&h0, 0, sizeof(h0));
    h0.nsys = NR;
    h0.first = 1;
    h0.any_pending = 1;
    h0.delta2 = ru_delta * ru_delta;
    h0.ru_max = 2000;
    for (int j = 0; j < NR; j++) {
        h0.tgt[j] = tgt[j];
        h0.pending[j] = 1;
    }
    CK(cudaMemcpyAsync(st, &h0, sizeof(h0), cudaMemcpyHostToDevice, s_));
    CK(cudaMemsetAsync(tk, 0, 4 * sizeof(unsigned), s_));
    CK(cudaMemsetAsync(xs, 0, NR * vx, s_));

    ResidCoef co;
    for (int j = 0; j < 8; j++) co.coef[j] = coef[j < NR ? j : 0];

    // FP64 M^dag M pieces of the reliable update
    DslashArgs<L64_18, NR, NoFin> d1;
    memset(&d1, 0, sizeof(d1));
    d1.g = c->g; d1.p_out = 1; d1.links = l64; d1.in = xg; d1.out = (double2 *)h64; d1.stride = stride; d1.beta = 0.5;
    d1.stop = &st->stop;
    d1.run_if = &st->any_pending;
    DslashArgs<L64_18, NR, NoFin> d2 = d1;
    d2.p_out = 0; d2.in = (const double2 *)h64; d2.out = (double2 *)t64; d2.beta = -0.5;
    // sloppy operator
    DslashArgs<LF, NR, NoFin> s1;
    memset(&s1, 0, sizeof(s1));
    s1.g = c->g; s1.p_out = 1; s1.links = lf; s1.in = (const E *)p; s1.out = (E *)h; s1.stride = sstride;
    s1.beta = (Rs)0.5; s1.stop = &st->stop;
    DslashArgs<LF, NR, FinRBAlpha<NR>> s2;
    memset(&s2, 0, sizeof(s2));
    s2.g = c->g; s2.p_out = 0; s2.links = lf; s2.in = (const E *)h; s2.out = (E *)ap; s2.y = (const E *)p;
    s2.stride = sstride; s2.beta = (Rs)-0.5; s2.use_alphas = 1;
    for (int j = 0; j < NR; j++) s2.alphas[j] = (Rs)coef[j];
    s2.partials = pt; s2.ticket = tk + 1; s2.fin.st = st; s2.stop = &st->stop;
    const int down = walk_alternates<LF, NR>(Vh, c->l2_bytes);
    s2.down = down;

    struct Key {
        int kind, link_reals, link_bytes, nr, n_ru, vh;
        const void *links, *links64, *xs, *rs, *p, *ap, *h, *h64, *t64, *st, *pt, *tk, *xg, *bg;
        double coef[RB_MAX];
        cudaStream_t stream;
        int cand[3];  // launch shapes of the captured Dslash instantiations
    } key;
    memset(&key, 0, sizeof(key));
    // launch shapes (tuned now, outside the capture, when unknown)
    key.cand[0] = dslash_candidate<L64_18, NR, false, false>(c->g, l64, s_);
    key.cand[1] = dslash_candidate<LF, NR, false, false>(c->g, lf, s_);
    key.cand[2] = dslash_candidate<LF, NR, true, true>(c->g, lf, s_);
    key.kind = 2; key.link_reals = LF::reals; key.link_bytes = (int)sizeof(typename LF::real); key.nr = NR;
    key.n_ru = n_ru; key.vh = Vh; key.links = lf.p; key.links64 = l64.p; key.xs = xs; key.rs = rs; key.p = p;
    key.ap = ap; key.h = h; key.h64 = h64; key.t64 = t64; key.st = st; key.pt = pt; key.tk = tk; key.xg = xg;
    key.bg = bg; key.stream = s_;
    for (int j = 0; j < NR; j++) key.coef[j] = coef[j];
    const std::string kb = key_bytes(key);
    cudaGraphExec_t exec = c->graphs.find(kb);
    cudaError_t ce = cudaSuccess;
    if (!exec) {
        cudaGraph_t graph;
        CK(cudaStreamBeginCapture(s_, cudaStreamCaptureModeThreadLocal));
        rb_accum_kernel<NR, X><<<gv, VEC_BLOCK, 0, s_>>>(Vh, stride, xg, (X *)xs, st);
        dslash_launch_cand<L64_18, NR, false, false, NoFin>(key.cand[0], d1, Vh, s_);
        dslash_launch_cand<L64_18, NR, false, false, NoFin>(key.cand[0], d2, Vh, s_);
        rb_resid_kernel<NR, S><<<gv, VEC_BLOCK, 0, s_>>>(Vh, stride, sstride, bg, xg, (const double2 *)t64, (E *)rs, (E *)p,
                                                             co, pt, tk, st);
        for (int it = 0; it < n_ru; it++) {
            dslash_launch_cand<LF, NR, false, false, NoFin>(key.cand[1], s1, Vh, s_);
            dslash_launch_cand<LF, NR, true, true, FinRBAlpha<NR>>(key.cand[2], s2, Vh, s_);
            rb_xr_kernel<NR, S, X><<<persistent_grid((const void *)rb_xr_kernel<NR, S, X>, VEC_BLOCK, gv), VEC_BLOCK, 0,
                                     s_>>>(Vh, stride, sstride, (X *)xs, (E *)rs, (const E *)p, (const E *)ap, pt, tk + 2, st);
            rb_p_kernel<NR, S><<<gv, VEC_BLOCK, 0, s_>>>(Vh, sstride, down, (const E *)rs, (E *)p, st);
        }
        ce = cudaStreamEndCapture(s_, &graph);
        if (ce != cudaSuccess) return cuda_fail(ce, "refine capture");
        ce = cudaGraphInstantiate(&exec, graph, 0);
        cudaGraphDestroy(graph);
        if (ce != cudaSuccess) return cuda_fail(ce, "refine instantiate");
        c->graphs.put(kb, exec);
    }

    // the cap in stages of 16 iterations, whatever n_ru: a recomputation still comes (max_iter / 16 + 1) * 16
    // iterations after the first
    const long max_rep = ((long)max_iter / 16 + 1) * 16 / n_ru + 1;
    long rep = 0;
    int seen = 0;
    const int prc = replay_until_stop(c, exec, s_, &st->stop, max_rep, &rep, &seen, "refine loop");
    c->launches += rep * (4 + 4 * (long)n_ru);
    if (prc) return prc;
    RBState hs;
    CK(cudaMemcpy(&hs, st, sizeof(hs), cudaMemcpyDeviceToHost));
    *iters_out += hs.iters;
    *ru_out += hs.ru_count;
    if (hs.status == 2) return fail(RHMC_ERR_NONFINITE, "refinement: non-finite reduction");
    if (!hs.stop) return fail(RHMC_ERR_MAXITER, "refinement: iteration cap %d reached", max_iter);
    return RHMC_OK;
}

template <class LF>
int rb_group_n(rhmc_ctx *c, const LF &lf, int n, const double *coef, const double *tgt, double2 *xg, const double2 *bg,
                      int max_iter, int n_ru, long *iters, int *ru, double ru_delta)
{
    switch (n) {
    case 1: return rb_group<LF, 1>(c, lf, coef, tgt, xg, bg, max_iter, n_ru, iters, ru, ru_delta);
    case 2: return rb_group<LF, 2>(c, lf, coef, tgt, xg, bg, max_iter, n_ru, iters, ru, ru_delta);
    case 3: return rb_group<LF, 3>(c, lf, coef, tgt, xg, bg, max_iter, n_ru, iters, ru, ru_delta);
    case 4: return rb_group<LF, 4>(c, lf, coef, tgt, xg, bg, max_iter, n_ru, iters, ru, ru_delta);
    case 8: return rb_group<LF, 8>(c, lf, coef, tgt, xg, bg, max_iter, n_ru, iters, ru, ru_delta);
    default: return fail(RHMC_ERR_ARG, "bad refinement batch %d", n);
    }
}

}  // namespace rhmc

// msolve.cuh -- multi-shift conjugate gradient on (M^dag M + sigma_i) x_i = b over even sites.
//
// Algorithm: Jegerlehner's multi-shift CG (hep-lat/9612014) exactly as the reference's CPU
// solver runs it (multips_shifted_invert, lib/Action/Inverter/inverter.cc:142-299): x_i = 0,
// r = p = p_i = b; per iteration
//   s = (M^dag M + sigma_0) p, alpha = Re<p,s>, omega = -delta/alpha
//   zeta'''_i = zeta_i zeta''_i omega_prev / (omega gamma (zeta_i - zeta''_i)
//                                               + zeta_i omega_prev (1 - sigma_i omega))
//   omega_i = omega zeta'''_i / zeta''_i ;  x_i -= omega_i p_i
//   r += omega s, lambda = |r|^2, gamma = lambda/delta, p = r + gamma p
//   gamma_i = gamma zeta'''_i omega_i / (zeta''_i omega) ; p_i = zeta'''_i r + gamma_i p_i
//   freeze shift i when sqrt(delta zeta''_i^2) < tgt_i (lagged residual, as inverter.cc:275-279)
// stopping when sqrt(lambda) <= res (inverter.cc:287), when every shift is frozen (the GPU
// solver's criterion, cuda_inverter.cu:777-785) or at max_iter.  sigma_0 is the base shift
// (0 in the reference; the mixed solver uses the smallest pole) and sigma_i are relative to it.
//
// Kernel sequence per iteration (one CUDA graph replays a window of iterations):
//   K1 D_oe:    h = D_oe p                                   (Dslash, NR right-hand sides)
//   K2 D_eo:    s = (m^2+sigma_0) p - D_eo h, Re<p,s>        (Dslash epilogue + FP64 reduction;
//               the last block computes omega, zeta''', omega_i for every RHS)
//   K3 resid:   r += omega s, |r|^2 into the window's ring   (last block: gamma, gamma_i, freezing,
//               convergence, stop flag)
//   K4 update:  p = r + gamma p
// and once per window the flush kernel applies the window's x_i -= omega_i p_i and
// p_i = zeta''' r + gamma_i p_i of every shift, composed from the recorded scalars and residuals.
// Scalars live in device memory (MSState) and never leave the GPU during the solve; the host
// only polls the stop flag between graph replays.
#pragma once
#include <cstddef>

#include "dslash.cuh"
#include "solver.h"

namespace rhmc {

constexpr int MS_MAX_SHIFT = 32;
constexpr int MS_MAX_RHS = 8;
// Iterations per delayed-update window (= iterations per graph replay).  A window reads and writes
// every active shifted vector once (192 bytes per site and system) and costs a ring of MS_WIN
// residuals per right-hand side and two FP64 coefficients per iteration and system.  With 16 poles
// and 4 right-hand sides a solve takes 64.5 ms at 24^3x32 (FP64) and 172 ms at 32^4 (FP32 schedule)
// with 16 iterations per window, 68.8 and 182.7 ms with 8; 32 would not fit the flush's registers.
// A phase runs windows of MS_WIN or, where the larger ring would not leave the rest of a solve its
// memory, MS_WIN / 2 iterations (ms_ring); the kernels take the length as `win`.
constexpr int MS_WIN = 16;
constexpr int VEC_BLOCK = 256;

struct MSRhs {
    double delta, omega, omega_prev, gamma, lambda, alpha, b2;
    double res;        // this phase stops the RHS when sqrt(lambda) <= res
    int iter;          // iterations performed
    int running;       // this iteration updates the RHS
    int running_next;  // still running after this iteration
    int rslot;         // ring slot holding the current residual
    int i0;            // index of the base shift (relative shift 0) among this RHS's poles
    double ru_best;    // smallest true |r|^2 seen at a reliable update
    int ru_stall;      // reliable updates since ru_best last fell by 4x
    double zeta_i[MS_MAX_SHIFT], zeta_ii[MS_MAX_SHIFT], zeta_iii[MS_MAX_SHIFT];
    double omegas[MS_MAX_SHIFT], gammas[MS_MAX_SHIFT];
    int active[MS_MAX_SHIFT];       // shift updated in this iteration
    int active_next[MS_MAX_SHIFT];  // after the freezing test
    double shift[MS_MAX_SHIFT];     // sigma_{r,i} - sigma_{r,0}: this RHS's poles relative to its base
};

// the scalars of each iteration m of the current window, for the delayed shifted updates:
// x_i -= om p_i, then p_i = ze r_m + ga p_i, applied by ms_flush_kernel when act
struct MSHist {
    double om[MS_MAX_SHIFT][MS_WIN], ga[MS_MAX_SHIFT][MS_WIN], ze[MS_MAX_SHIFT][MS_WIN];
    int act[MS_MAX_SHIFT][MS_WIN];
};

struct MSState {
    int stop;     // every RHS finished: K1-K3 skip
    int stop_k4;  // set by the first skipped K1 so that K4 skips from the next iteration on
    int wpos;     // iterations done in the current window (the residual of iteration m is in ring slot m-1)
    int first;    // no window flushed yet: x_i = 0 and p_i = b are not in memory
    const double2 *b;  // the right-hand sides (read by the first flush; not a captured argument, so
                       // that a new b replays the same graph)
    int status;   // 0 ok, 1 iteration cap, 2 non-finite reduction
    int nshift, nrhs, max_iter;
    int stop_on_frozen;             // also stop when every shift is frozen
    double res;                     // base residual target: stop when sqrt(lambda) <= res
    double tau;                     // > 0: this phase stops an RHS once sqrt(lambda) <= tau |b| (a
                                    // later phase in lower precision resumes it)
    double tgt[MS_MAX_SHIFT];       // freezing threshold for sqrt(delta zeta''^2)
    // reliable updates (resumed lower-precision phase): every ru_every windows the base residual
    // is recomputed in FP64 from the FP64 base solution and the base direction re-synchronised
    int ru_every, ru_windows, ru_now, ru_count;
    MSRhs rhs[MS_MAX_RHS];
    MSHist hist[MS_MAX_RHS];  // last: the host exchanges only what comes before it
};
constexpr size_t MS_STATE_HEAD = offsetof(MSState, hist);

// ------------------------------------------------------------------ last-block scalar steps
// The FP32 part of the precision schedule, with its FP64 reliable updates, leaves the shifted
// systems near 1e-7 of the residual at which it took over (a 1e-10 |b| target is met with the
// hand-over at 1e-3 |b|): the automatic hand-over (tau < 0) is therefore placed at most this far
// above the final target, so that deep targets do not leave every system to the refinement.
constexpr double MS_TAU_REACH = 1e7;
// ... but not below 1e-4 |b|: targets at the FP64 rounding floor of the smallest poles leave
// those systems to the refinement whatever the hand-over, and an earlier one only lengthens the
// FP64 part
constexpr double MS_TAU_MIN = 1e-4;

// The scalar steps run in every thread of the reduction's last block, thread r the scalars of
// right-hand side r and one thread per (rhs, shift) the shifted recurrences.  They sit between two
// launches of the solver, so what counts is their chain of dependent L2 accesses: every thread
// loads all it needs before the first barrier, and the values of a right-hand side that the
// (rhs, shift) threads need travel through shared memory.  With thread 0 stepping the right-hand
// sides one after the other (and counting active shifts one by one) FinAlpha and FinLambda took
// 5 us each for one right-hand side with 8 shifts and 8 us for four with 16; now 2 us.
template <int NR>
struct FinInit {
    MSState *st;
    int win;
    __device__ void operator()(const double *tot) const
    {
        __shared__ int s_any;
        if (threadIdx.x == 0) s_any = 0;
        __syncthreads();
        const int ns = st->nshift;
        if (threadIdx.x < NR) {
            MSRhs &q = st->rhs[threadIdx.x];
            const double b2 = tot[threadIdx.x], res = st->res, tau = st->tau;
            q.b2 = b2;
            q.delta = b2;
            q.omega = 1.0;
            q.omega_prev = 1.0;
            q.gamma = 0.0;
            q.lambda = b2;
            q.alpha = 0.0;
            q.iter = 0;
            q.rslot = win - 1;
            // precision schedule: the FP64 part ends at tau |b| (tau > 0), or with tau < 0 at
            // -tau |b| but no more than MS_TAU_REACH above the final target
            const double nb = sqrt(b2);
            q.res = tau > 0.0   ? fmax(res, tau * nb)
                    : tau < 0.0 ? fmax(res, fmax(MS_TAU_MIN * nb, fmin(-tau * nb, MS_TAU_REACH * res)))
                                : res;
            q.running = 1;
            const int go = isfinite(b2) && b2 > 0.0;  // b == 0: x = 0 is exact
            if (!isfinite(b2)) st->status = 2;
            q.running_next = go;
            if (go) atomicOr(&s_any, 1);
        }
        for (int t = threadIdx.x; t < NR * ns; t += blockDim.x) {
            MSRhs &q = st->rhs[t / ns];
            const int i = t % ns;
            q.zeta_i[i] = 1.0;
            q.zeta_ii[i] = 1.0;
            q.zeta_iii[i] = 1.0;
            q.omegas[i] = 0.0;
            q.gammas[i] = 0.0;
            q.active[i] = 1;
            q.active_next[i] = 1;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            st->stop = s_any ? 0 : 1;
            st->stop_k4 = 0;
            st->first = 1;
        }
    }
};

// zeta''' = zeta zeta'' omega_prev / (omega gamma (zeta - zeta'') + zeta omega_prev (1 - sigma omega)), rounded
// one fixed way (see dot2), so that every kernel that steps it gives the same bits
__device__ __forceinline__ double next_zeta(double zi, double zii, double omp, double om, double ga, double sh)
{
    return __dmul_rn(__dmul_rn(zi, zii), omp) /
           dot2(__dmul_rn(om, ga), zi - zii, __dmul_rn(zi, omp), __fma_rn(-sh, om, 1.0));
}

template <int NR>
struct FinAlpha {
    MSState *st;
    __device__ void operator()(const double *tot) const
    {
        __shared__ double s_om[NR], s_omp[NR], s_ga[NR];
        __shared__ int s_run[NR];
        const int ns = st->nshift, wp = st->wpos;
        if (threadIdx.x < NR) {
            MSRhs &q = st->rhs[threadIdx.x];
            const double delta = q.delta, prev = q.omega, alpha = tot[threadIdx.x];
            int run = q.running_next;
            s_ga[threadIdx.x] = q.gamma;
            if (run) {
                q.alpha = alpha;
                if (!isfinite(alpha) || alpha == 0.0) {
                    st->status = 2;
                    st->stop = 1;
                    q.running_next = 0;
                    run = 0;
                } else {
                    const double om = -delta / alpha;
                    q.omega_prev = prev;
                    q.omega = om;
                    s_omp[threadIdx.x] = prev;
                    s_om[threadIdx.x] = om;
                }
            }
            q.running = run;
            s_run[threadIdx.x] = run;
        }
        for (int t0 = 0; t0 < NR * ns; t0 += blockDim.x) {
            const int t = t0 + threadIdx.x, r = t / ns, i = t % ns;
            const bool in = t < NR * ns;
            int an = 0;
            double zi = 1.0, zii = 1.0, sh = 0.0;
            if (in) {
                const MSRhs &q = st->rhs[r];
                an = q.active_next[i];
                zi = q.zeta_i[i];
                zii = q.zeta_ii[i];
                sh = q.shift[i];
            }
            if (t0 == 0) __syncthreads();
            if (!in) continue;
            MSRhs &q = st->rhs[r];
            const int run = s_run[r], act = run ? an : 0;
            st->hist[r].act[i][wp] = act;
            if (!run) continue;
            q.active[i] = act;
            if (!act) continue;
            const double om = s_om[r], omp = s_omp[r];
            const double ziii = next_zeta(zi, zii, omp, om, s_ga[r], sh);
            q.zeta_iii[i] = ziii;
            const double oms = om * ziii / zii;
            q.omegas[i] = oms;
            st->hist[r].om[i][wp] = oms;
        }
    }
};

template <int NR>
struct FinLambda {
    MSState *st;
    __device__ void operator()(const double *tot) const
    {
        __shared__ double s_om[NR], s_ga[NR], s_de[NR];
        __shared__ int s_run[NR], s_nact[NR], s_any;
        const int ns = st->nshift, wp = st->wpos;
        double lambda = 0.0, res = 0.0;
        int run = 0, iter = 0;
        if (threadIdx.x < NR) {
            MSRhs &q = st->rhs[threadIdx.x];
            const double delta = q.delta;
            run = q.running;
            iter = q.iter;
            res = q.res;
            s_om[threadIdx.x] = q.omega;
            s_de[threadIdx.x] = delta;
            s_nact[threadIdx.x] = 0;
            if (threadIdx.x == 0) s_any = 0;
            if (run) {
                lambda = tot[threadIdx.x];
                q.lambda = lambda;
                q.rslot = wp;
                if (!isfinite(lambda)) {
                    st->status = 2;
                    q.running_next = 0;
                    run = 0;
                } else {
                    const double ga = lambda / delta;
                    q.gamma = ga;
                    s_ga[threadIdx.x] = ga;
                }
            }
            s_run[threadIdx.x] = run;
        }
        for (int t0 = 0; t0 < NR * ns; t0 += blockDim.x) {
            const int t = t0 + threadIdx.x, r = t / ns, i = t % ns;
            const bool in = t < NR * ns;
            int act = 0;
            double zii = 1.0, ziii = 1.0, oms = 0.0, tgt = 0.0;
            if (in) {
                const MSRhs &q = st->rhs[r];
                act = q.active[i];
                zii = q.zeta_ii[i];
                ziii = q.zeta_iii[i];
                oms = q.omegas[i];
                tgt = st->tgt[i];
            }
            if (t0 == 0) __syncthreads();
            if (!in || !s_run[r] || !act) continue;
            MSRhs &q = st->rhs[r];
            const double gas = s_ga[r] * ziii * oms / (zii * s_om[r]);
            q.gammas[i] = gas;
            st->hist[r].ga[i][wp] = gas;
            st->hist[r].ze[i][wp] = ziii;
            const double fact = sqrt(s_de[r] * zii * zii);
            const int an = (fact < tgt) ? 0 : 1;
            q.active_next[i] = an;
            q.zeta_i[i] = zii;
            q.zeta_ii[i] = ziii;
            if (an) atomicAdd(&s_nact[r], 1);
        }
        __syncthreads();
        if (run) {  // threads 0..NR-1
            MSRhs &q = st->rhs[threadIdx.x];
            q.delta = lambda;
            q.iter = ++iter;
            int done = (sqrt(lambda) <= res) || (st->stop_on_frozen && s_nact[threadIdx.x] == 0);
            if (!done && iter >= st->max_iter) {
                done = 1;
                if (st->status == 0) st->status = 1;
            }
            q.running_next = !done;
            if (!done) atomicOr(&s_any, 1);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            if (!s_any) st->stop = 1;
            st->wpos = wp + 1;
        }
    }
};

// ------------------------------------------------------------------ vector kernels
template <typename Rv>
struct MSVec {
    typedef typename SpinorT<Rv>::elem E;
};

// Layout of the base vectors (residual ring, p, h, s) of NR right-hand sides in precision Rv:
// FP32 packed P at a time (PackS; a 32-byte element holds 4 right-hand sides of one colour and
// site, 16 bytes 2 of them), so that the Dslash of the batch loads P right-hand sides per
// instruction; plane per RHS (P = 1) for FP64, whose 16-byte plane loads are already wide (its
// packed form, 2 per 32 bytes, was faster for 4 right-hand sides at 32^4 but slower for 2 and 8
// in trajectories), and for batch widths that do not split into packs.  The shifted solutions
// and directions, the right-hand sides b and every caller-visible vector keep the plane layout.
template <typename Rv, int NR>
struct BasePack {
    static constexpr int P = sizeof(Rv) == 4 ? (NR % 4 == 0 ? 4 : (NR % 2 == 0 ? 2 : 1)) : 1;
};

// index, in complex numbers, of RHS j, colour c, site k in a set of NR base vectors
template <typename Rv, int NR>
__host__ __device__ __forceinline__ size_t bidx(int j, int c, int k, int Vh)
{
    constexpr int P = BasePack<Rv, NR>::P;
    return ((size_t)((j / P) * 3 + c) * Vh + k) * P + (j % P);
}

// r_0 = p = b (b FP64 internal), |b|^2.  r_0 goes to the last slot of the residual ring (the slot
// the first iteration reads).  The shifted x_i = 0 and p_i = b are not written: the first window's
// flush starts from them without reading any (MSState::first).
template <typename Rv, int NR>
__global__ void __launch_bounds__(VEC_BLOCK) ms_init_kernel(int Vh, size_t stride, int win, const double2 *__restrict__ b,
                                                             typename MSVec<Rv>::E *ring, typename MSVec<Rv>::E *p,
                                                             double *partials, unsigned *ticket, MSState *st)
{
    typename MSVec<Rv>::E *r = ring + (size_t)(win - 1) * NR * stride;
    typedef typename MSVec<Rv>::E E;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    double red[NR];
#pragma unroll
    for (int j = 0; j < NR; j++) red[j] = 0.0;
    if (k < Vh) {
#pragma unroll
        for (int j = 0; j < NR; j++) {
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const size_t ob = bidx<Rv, NR>(j, c, k, Vh);
                const double2 v = b[j * stride + (size_t)c * Vh + k];
                red[j] += dot2(v.x, v.x, v.y, v.y);
                E e;
                e.x = (Rv)v.x;
                e.y = (Rv)v.y;
                r[ob] = e;
                p[ob] = e;
            }
        }
    }
    FinInit<NR> fin{st, win};
    reduce_finalize<NR>(red, partials, ticket, fin);
}

// r_m = r_{m-1} + omega s (ring slots wpos-1 -> wpos), |r_m|^2 per RHS
template <typename Rv, int NR>
__global__ void __launch_bounds__(VEC_BLOCK) ms_resid_kernel(int Vh, size_t stride, int win, typename MSVec<Rv>::E *ring,
                                                              const typename MSVec<Rv>::E *__restrict__ s, double *partials,
                                                              unsigned *ticket, MSState *st)
{
    typedef typename MSVec<Rv>::E E;
    if (*(volatile int *)&st->stop) return;
    const int wp = *(volatile const int *)&st->wpos;
    const E *rprev = ring + (size_t)ms_prev_slot(wp, win) * NR * stride;
    E *r = ring + (size_t)wp * NR * stride;
    int run[NR];
    Rv om[NR];
#pragma unroll
    for (int j = 0; j < NR; j++) {
        run[j] = st->rhs[j].running;
        om[j] = (Rv)st->rhs[j].omega;
    }
    // tiles of VEC_BLOCK sites walked by a persistent grid (persistent_grid), so the reduction's
    // per-block fence and ticket are paid once per block
    constexpr int P = BasePack<Rv, NR>::P;
    typedef PackIO<Rv, P> IO;
    typedef PackElem<Rv, P> PE;
    const int ntiles = (Vh + VEC_BLOCK - 1) / VEC_BLOCK;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int k = tile * VEC_BLOCK + threadIdx.x;
        double red[NR];
#pragma unroll
        for (int j = 0; j < NR; j++) red[j] = 0.0;
        if (k < Vh) {
#pragma unroll
            for (int q = 0; q < NR / P; q++) {
                int any = 0, all = 1;
#pragma unroll
                for (int i = 0; i < P; i++) {
                    any |= run[q * P + i];
                    all &= run[q * P + i];
                }
                if (!any) continue;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const size_t o = bidx<Rv, NR>(q * P, c, k, Vh) / P;  // pack element
                    cpx<Rv> rv[P], sv[P], keep[P];
                    IO::ld((const PE *)rprev + o, rv);
                    IO::ld((const PE *)s + o, sv);
                    if (!all) IO::ldc((const PE *)r + o, keep);  // a stopped RHS keeps its slot
#pragma unroll
                    for (int i = 0; i < P; i++) {
                        const int j = q * P + i;
                        if (run[j]) {
                            rv[i].re = rv[i].re + om[j] * sv[i].re;
                            rv[i].im = rv[i].im + om[j] * sv[i].im;
                            red[j] += dot2((double)rv[i].re, (double)rv[i].re, (double)rv[i].im, (double)rv[i].im);
                        } else {
                            rv[i] = keep[i];
                        }
                    }
                    IO::st((PE *)r + o, rv);
                }
            }
        }
        reduce_tile<NR>(red, partials, tile);
    }
    FinLambda<NR> fin{st};
    reduce_last<NR>(partials, ticket, ntiles * (VEC_BLOCK / RED_CHUNK), fin);
}

// p = r_m + gamma p (the base search direction; the shifted p_i and x_i are updated once per
// window by ms_flush_kernel)
template <typename Rv, int NR>
__global__ void __launch_bounds__(VEC_BLOCK) ms_update_kernel(int Vh, size_t stride, int win, int down, const typename MSVec<Rv>::E *__restrict__ ring,
                                                               typename MSVec<Rv>::E *p, MSState *st)
{
    typedef typename MSVec<Rv>::E E;
    constexpr int P = BasePack<Rv, NR>::P;
    typedef PackIO<Rv, P> IO;
    typedef PackElem<Rv, P> PE;
    if (*(volatile int *)&st->stop_k4) return;
    const int k = (down ? gridDim.x - 1 - blockIdx.x : blockIdx.x) * blockDim.x + threadIdx.x;  // K3 went upwards
    if (k >= Vh) return;
    // K3 advanced wpos, unless K2 met a non-finite or zero <p,s> and stopped the solve before it: then
    // wpos may still be 0 (the other right-hand sides' p is formed once more and not used)
    const E *r = ring + (size_t)ms_prev_slot(*(volatile const int *)&st->wpos, win) * NR * stride;
#pragma unroll
    for (int q = 0; q < NR / P; q++) {
        int run[P], any = 0;
        Rv g[P];
#pragma unroll
        for (int i = 0; i < P; i++) {
            run[i] = st->rhs[q * P + i].running;
            g[i] = (Rv)st->rhs[q * P + i].gamma;
            any |= run[i];
        }
        if (!any) continue;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const size_t o = bidx<Rv, NR>(q * P, c, k, Vh) / P;  // pack element
            cpx<Rv> rv[P], pv[P];
            IO::ld((const PE *)r + o, rv);
            IO::ldc((const PE *)p + o, pv);
#pragma unroll
            for (int i = 0; i < P; i++)
                if (run[i]) {  // a stopped RHS keeps its direction
                    pv[i].re = rv[i].re + g[i] * pv[i].re;
                    pv[i].im = rv[i].im + g[i] * pv[i].im;
                }
            IO::st((PE *)p + o, pv);
        }
    }
}

// End of a window of wpos iterations with residuals r_0..r_{wpos-1} (ring slots).  Over the window
// the per-iteration updates x_i -= om_m p_i, p_i = ze_m r_m + ga_m p_i compose to
//   x_i = X0_i - cx0 P0_i - sum_m cx_m r_m,   p_i = ca P0_i + sum_m cb_m r_m
// with P0_i, X0_i the vectors at the window start (b and 0 in the first window).  Backwards over
// the window, with D the coefficient of the direction entering iteration m+1 in x and G that in p,
//   cx_m = ze_m D, cb_m = ze_m G, D <- om_m + ga_m D, G <- ga_m G   (frozen iterations skipped)
// and cx0 = D, ca = G at the end.  Warp j of every block derives the coefficients of right-hand
// side j (lane i: shift i) into shared memory and lists its active shifts; then a thread per site
// and right-hand side of a pack (the pack index fastest, so the lanes of a warp read whole packs)
// holds the window's residuals of one colour in registers and streams every active x_i, p_i
// through, the next one's loads issued before the current one's arithmetic.
template <typename Rv, int NR>
__global__ void __launch_bounds__(VEC_BLOCK, 2) ms_flush_kernel(int Vh, int nshift, size_t stride,
                                                                 const typename MSVec<Rv>::E *__restrict__ ring, double2 *ps,
                                                                 double2 *x, unsigned *ticket, MSState *st)
{
    extern __shared__ double2 s_coef[];  // [rhs][nshift][MS_WIN + 1] (cx, cb), entry MS_WIN (cx0, ca)
    __shared__ int s_list[NR][MS_MAX_SHIFT], s_n[NR];  // active shifts, 2 i + (p_i is needed further)
    __shared__ unsigned s_wrote[NR];                   // the window's iterations of a right-hand side, a bit each
    static_assert(NR <= VEC_BLOCK / 32 && MS_MAX_SHIFT <= 32, "a warp per right-hand side, a lane per shift");
    constexpr int P = BasePack<Rv, NR>::P;
    const int rstride = nshift * (MS_WIN + 1) + 1;  // one element of padding: other banks for another RHS
    const int wp = *(volatile const int *)&st->wpos, first = *(volatile const int *)&st->first;
    {
        const int j = threadIdx.x >> 5, i = threadIdx.x & 31;
        if (j < NR) {
            int an = 0;
            unsigned took = 0;  // iterations that updated the shift
            if (i < nshift) {
                const MSHist &hq = st->hist[j];
                double2 *cf = s_coef + (size_t)j * rstride + i * (MS_WIN + 1);
                an = st->rhs[j].active_next[i];
                double D = 0.0, G = 1.0;
                // the window's scalars loaded in batches (entries past wp or of frozen iterations are
                // stale and not used): one L2 latency per batch instead of one per iteration
                constexpr int B = 8;
                static_assert(MS_WIN % B == 0, "whole batches");
#pragma unroll
                for (int m0 = MS_WIN - B; m0 >= 0; m0 -= B) {
                    double om[B], ga[B], ze[B];
                    int act[B];
#pragma unroll
                    for (int m = 0; m < B; m++) {
                        om[m] = hq.om[i][m0 + m];
                        ga[m] = hq.ga[i][m0 + m];
                        ze[m] = hq.ze[i][m0 + m];
                        act[m] = m0 + m < wp ? hq.act[i][m0 + m] : 0;
                    }
#pragma unroll
                    for (int m = B - 1; m >= 0; m--) {
                        cf[m0 + m] = act[m] ? make_double2(ze[m] * D, ze[m] * G) : make_double2(0.0, 0.0);
                        if (act[m]) {
                            D = om[m] + ga[m] * D;
                            G = ga[m] * G;
                            took |= 1u << (m0 + m);
                        }
                    }
                }
                cf[MS_WIN] = make_double2(D, G);
            }
            // p_i is written for every shift still active, also when the RHS stopped in this window:
            // a later phase may resume it from exactly this state.  The first window visits every
            // shift: x_i is in memory only after it.
            const int use = i < nshift && (took || first);
            const unsigned mask = __ballot_sync(0xffffffffu, use), wrote = __reduce_or_sync(0xffffffffu, took);
            if (i == 0) s_wrote[j] = wrote;
            if (use) s_list[j][__popc(mask & ((1u << i) - 1u))] = 2 * i + (an ? 1 : 0);
            if (i == 0) s_n[j] = __popc(mask);
        }
    }
    __syncthreads();
    const long id = (long)blockIdx.x * VEC_BLOCK + threadIdx.x;
    const int k = (int)(id / P), l = (int)(id % P);
    if (k < Vh && (wp > 0 || first)) {
        for (int q = 0; q < NR / P; q++) {
            const int j = q * P + l, n = s_n[j];
            const unsigned wrote = s_wrote[j];
            if (n == 0) continue;
            const double2 *cj = s_coef + (size_t)j * rstride;
#pragma unroll 1
            for (int c = 0; c < 3; c++) {
                const size_t o = (size_t)j * nshift * stride + (size_t)c * Vh + k;
                // only slots that this right-hand side wrote in this window: the others (it was zero, or had
                // stopped) have zero coefficients but may hold anything, also NaN from memory or an older solve
                double2 rv[MS_WIN];
#pragma unroll
                for (int m = 0; m < MS_WIN; m++) {
                    rv[m] = make_double2(0.0, 0.0);
                    if (wrote >> m & 1u) {
                        const typename MSVec<Rv>::E e = __ldg(ring + (size_t)m * NR * stride + bidx<Rv, NR>(j, c, k, Vh));
                        rv[m] = make_double2((double)e.x, (double)e.y);
                    }
                }
                double2 pn, xn = make_double2(0.0, 0.0);
                int en = s_list[j][0];
                if (first) {
                    pn = __ldg(st->b + (size_t)j * stride + (size_t)c * Vh + k);
                } else {
                    pn = ps[o + (size_t)(en >> 1) * stride];
                    xn = x[o + (size_t)(en >> 1) * stride];
                }
                for (int t = 0; t < n; t++) {
                    const int e = en, i = e >> 1;
                    const double2 p0 = pn;
                    double2 xv = xn;
                    if (t + 1 < n) {
                        en = s_list[j][t + 1];
                        if (!first) {
                            pn = ps[o + (size_t)(en >> 1) * stride];
                            xn = x[o + (size_t)(en >> 1) * stride];
                        }
                    }
                    const double2 *cf = cj + i * (MS_WIN + 1);
                    const double2 c0 = cf[MS_WIN];
                    double2 pv;
                    xv.x = xv.x - c0.x * p0.x;
                    xv.y = xv.y - c0.x * p0.y;
                    pv.x = c0.y * p0.x;
                    pv.y = c0.y * p0.y;
#pragma unroll
                    for (int m = 0; m < MS_WIN; m++) {
                        const double2 cm = cf[m];
                        xv.x = xv.x - cm.x * rv[m].x;
                        xv.y = xv.y - cm.x * rv[m].y;
                        pv.x = pv.x + cm.y * rv[m].x;
                        pv.y = pv.y + cm.y * rv[m].y;
                    }
                    x[o + (size_t)i * stride] = xv;
                    if (e & 1) ps[o + (size_t)i * stride] = pv;
                }
            }
        }
    }
    // the last block to get here starts a new window; every thread of a block read wpos and first
    // before the barrier above, so the reset cannot reach one that still needs them
    if (threadIdx.x == 0 && atomicAdd(ticket, 1u) == gridDim.x - 1) {
        *ticket = 0;
        st->wpos = 0;
        st->first = 0;
    }
}

// ------------------------------------------------------------------ precision-scheduled resumption
// The rounding error a sloppy iteration adds to the shifted systems is proportional to the
// residual at that iteration, and the shifted systems never see it corrected (only the base
// system is reliably updated).  So the mixed solver runs its first iterations in FP64, stops each
// right-hand side once |r| <= tau |b|, and resumes the same recurrences (same scalars, same
// shifted vectors) with FP32 base vectors and links: every later error is then tau times smaller.

// One thread: every RHS that has not reached the final target (and still has an active shift)
// runs again; the phase target becomes the final one and a new window starts.
static __global__ void ms_rearm_kernel(MSState *st)
{
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    int any = 0;
    for (int r = 0; r < st->nrhs; r++) {
        MSRhs &q = st->rhs[r];
        q.res = st->res;
        int nact = 0;
        for (int i = 0; i < st->nshift; i++) nact += q.active_next[i];
        const int go = st->status == 0 && isfinite(q.lambda) && q.b2 > 0.0 && sqrt(q.lambda) > st->res && nact > 0;
        q.running_next = go;
        q.ru_best = q.lambda;
        q.ru_stall = 0;
        any |= go;
    }
    st->tau = 0.0;
    st->stop = any ? 0 : 1;
    st->stop_k4 = 0;
    st->wpos = 0;
    st->ru_windows = 0;
    st->ru_now = 0;
}

// The current residual of every RHS (ring slot rslot of the previous phase) into the last slot of
// the new ring, and the base direction p, converted to the new phase's precision.
template <typename Rf, typename Rt, int NR>
__global__ void __launch_bounds__(VEC_BLOCK) ms_convert_kernel(int Vh, size_t stride, const typename MSVec<Rf>::E *__restrict__ ring_f,
                                                                const typename MSVec<Rf>::E *__restrict__ p_f,
                                                                typename MSVec<Rt>::E *ring_t, typename MSVec<Rt>::E *p_t, int win,
                                                                const MSState *st)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= Vh) return;
#pragma unroll
    for (int j = 0; j < NR; j++) {
        const int slot = st->rhs[j].rslot;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const size_t of = bidx<Rf, NR>(j, c, k, Vh), ot = bidx<Rt, NR>(j, c, k, Vh);
            const typename MSVec<Rf>::E rv = ring_f[(size_t)slot * NR * stride + of], pv = p_f[of];
            typename MSVec<Rt>::E a, b;
            a.x = (Rt)rv.x;
            a.y = (Rt)rv.y;
            b.x = (Rt)pv.x;
            b.y = (Rt)pv.y;
            ring_t[(size_t)(win - 1) * NR * stride + ot] = a;
            p_t[ot] = b;
        }
    }
}

// One thread, after the window's flush: decides whether this window ends with a reliable update.
static __global__ void ms_ru_begin_kernel(MSState *st)
{
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    st->ru_now = 0;
    if (st->stop) return;
    st->ru_windows++;
    int any = 0;
    for (int r = 0; r < st->nrhs; r++) any |= st->rhs[r].running_next;
    st->ru_now = any && (st->ru_windows % st->ru_every == 0);
}

// x0[j] = x_{j, i0(j)}: the FP64 base solution of every RHS, contiguous for the FP64 operator
template <int NR>
__global__ void __launch_bounds__(VEC_BLOCK) ms_gather_base_kernel(int Vh, int nshift, size_t stride, const double2 *__restrict__ x,
                                                                    double2 *x0, const MSState *st)
{
    if (!*(volatile const int *)&st->ru_now) return;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= Vh) return;
#pragma unroll
    for (int j = 0; j < NR; j++) {
        const size_t src = (size_t)(j * nshift + st->rhs[j].i0) * stride;
#pragma unroll
        for (int c = 0; c < 3; c++) x0[j * stride + (size_t)c * Vh + k] = x[src + (size_t)c * Vh + k];
    }
}

// A right-hand side whose true base residual has not fallen by 4x (|r| by 2x) over
// MS_RU_STALL reliable updates, or has grown 4x above its best, has reached the rounding floor
// of the FP64 operator: past it the sloppy recurrence only follows rounding noise and diverges.
// It stops there (its solutions as they are) and is left to the refinement that follows.
constexpr int MS_RU_STALL = 16;

template <int NR>
struct FinMsRU {
    MSState *st;
    __device__ void operator()(const double *tot) const
    {
        if (threadIdx.x != 0) return;
        int any = 0;
        for (int r = 0; r < NR; r++) {
            MSRhs &q = st->rhs[r];
            if (!q.running_next) continue;
            if (!isfinite(tot[r])) {
                st->status = 2;
                q.running_next = 0;
                continue;
            }
            q.delta = tot[r];
            q.lambda = tot[r];
            if (tot[r] < 0.25 * q.ru_best) {
                q.ru_best = tot[r];
                q.ru_stall = 0;
            } else if (++q.ru_stall >= MS_RU_STALL || tot[r] > 4.0 * q.ru_best) {
                q.running_next = 0;
            }
            any |= q.running_next;
        }
        for (int r = NR; r < st->nrhs; r++) any |= st->rhs[r].running_next;
        if (!any) st->stop = 1;
        st->ru_count++;
    }
};

// Reliable update of every running RHS: r = b - t with t = (M^dag M + sigma_0) x0 computed in
// FP64 (the true residual of the base system) replaces the window's last residual, and the
// base direction is re-synchronised with the FP64 shifted direction of the base shift (both
// follow the same recurrence; the sloppy copy drifts by rounding).  |r|^2 becomes delta.
template <typename Rv, int NR>
__global__ void __launch_bounds__(VEC_BLOCK) ms_ru_resid_kernel(int Vh, int nshift, size_t stride, int win, const double2 *__restrict__ b,
                                                                 const double2 *__restrict__ t, const double2 *__restrict__ ps,
                                                                 typename MSVec<Rv>::E *ring, typename MSVec<Rv>::E *p,
                                                                 double *partials, unsigned *ticket, MSState *st)
{
    typedef typename MSVec<Rv>::E E;
    if (!*(volatile const int *)&st->ru_now) return;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    double red[NR];
#pragma unroll
    for (int j = 0; j < NR; j++) red[j] = 0.0;
    if (k < Vh) {
#pragma unroll
        for (int j = 0; j < NR; j++) {
            if (!st->rhs[j].running_next) continue;
            const size_t pbase = (size_t)(j * nshift + st->rhs[j].i0) * stride;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const size_t o = j * stride + (size_t)c * Vh + k, ob = bidx<Rv, NR>(j, c, k, Vh);
                const double2 bv = b[o], tv = t[o], pv = ps[pbase + (size_t)c * Vh + k];
                const double re = bv.x - tv.x, im = bv.y - tv.y;
                red[j] += dot2(re, re, im, im);
                E e, f;
                e.x = (Rv)re;
                e.y = (Rv)im;
                f.x = (Rv)pv.x;
                f.y = (Rv)pv.y;
                ring[(size_t)(win - 1) * NR * stride + ob] = e;
                p[ob] = f;
            }
        }
    }
    FinMsRU<NR> fin{st};
    reduce_finalize<NR>(red, partials, ticket, fin);
}

}  // namespace rhmc

// msolve_run.cuh -- one phase of the multi-shift CG over link format LF: workspaces, state, the CUDA
// graph of a window of iterations and its replay.  One translation unit per link format
// instantiates ms_run (inst_*.cu); msolve.cu declares them extern.
#pragma once
#include <cmath>
#include <cstring>
#include <type_traits>

#include "capi_util.h"
#include "context.h"
#include "kernels.h"
#include "msolve.cuh"
#include "msolve_small.cuh"
#include "solver.h"

namespace rhmc {

// workspace slot name of a base vector set in elements of `bytes` bytes
static inline std::string vname(const char *base, size_t bytes) { return std::string(base) + std::to_string(bytes); }

// The host's part of the initial state (what precedes MSState::hist); false when some right-hand
// side does not iterate on one of its own poles.
static inline bool ms_fill(const MSolveArgs &A, MSState &h0)
{
    memset(&h0, 0, MS_STATE_HEAD);
    h0.nshift = A.nshift;
    h0.nrhs = A.nrhs;
    h0.max_iter = A.max_iter;
    h0.stop_on_frozen = A.stop_on_frozen;
    h0.res = A.res_base;
    h0.tau = A.tau;
    h0.first = 1;
    h0.b = (const double2 *)A.b;
    for (int i = 0; i < A.nshift; i++) h0.tgt[i] = A.tgt[i];
    bool own = true;
    for (int r = 0; r < A.nrhs; r++) {
        int i0 = -1;
        for (int i = 0; i < A.nshift; i++) {
            h0.rhs[r].shift[i] = A.shift[(size_t)r * A.nshift + i] - A.base[r];
            if (i0 < 0 && A.shift[(size_t)r * A.nshift + i] == A.base[r]) i0 = i;
        }
        own = own && i0 >= 0;
        h0.rhs[r].i0 = i0 < 0 ? 0 : i0;
    }
    return own;
}

// What a finished phase left in the state (its head) into info; the phase's return code.
static inline int ms_result(const MSState &hs, const MSolveArgs &A, MSolveInfo *info)
{
    if (info) {
        info->status = hs.status;
        info->ru_count = hs.ru_count;
        for (int j = 0; j < A.nrhs; j++) {
            info->iters[j] = hs.rhs[j].iter;
            info->lambda[j] = hs.rhs[j].lambda;
            info->b2[j] = hs.rhs[j].b2;
        }
    }
    if (hs.status == 3) return fail(RHMC_ERR_CUDA, "multi-shift CG: a grid barrier timed out");
    if (hs.status == 2) return fail(RHMC_ERR_NONFINITE, "multi-shift CG: non-finite reduction");
    if (hs.status == 1) return fail(RHMC_ERR_MAXITER, "multi-shift CG: iteration cap %d reached", A.max_iter);
    return RHMC_OK;
}

// The residual ring of a phase, `slot` bytes per iteration, and the iterations per window it allows:
// MS_WIN where the ring is already that long or the device has room for it and for what the rest of a
// solve may still allocate (`later` FP64 spinors of v64 bytes), else half.  Only a ring that must grow asks
// for the free memory, and not when all of it is small (the query costs a new context's first solve a
// millisecond or more); a choice against the longer ring stands until the ring has to grow again.
// Where the estimate proves too low the solve is repeated with half windows (rhmc_msolve).
static inline cudaError_t ms_ring(rhmc_ctx *c, const std::string &name, size_t slot, size_t v64, int later, void **ring, int *win)
{
    const size_t have = c->ws.held(name), want = MS_WIN * slot, rest = later * v64;
    bool &half = c->window.short_ring[name];
    bool whole = have >= want;
    if (!whole && !(half && have >= want / 2) && !c->window.half_only) {
        whole = true;
        size_t free_bytes = 0, total = 0;
        if (want + rest > ((size_t)1 << 28))
            whole = cudaMemGetInfo(&free_bytes, &total) == cudaSuccess && free_bytes + have >= want + rest;
    }
    cudaError_t e = cudaSuccess;
    if (whole) {
        e = c->ws.get(name, want, ring);
        whole = e != cudaErrorMemoryAllocation;
    }
    *win = c->window.last = whole ? MS_WIN : MS_WIN / 2;
    half = !whole;
    if (whole)
        c->window.was_long = true;
    else
        e = c->ws.get(name, want / 2, ring);
    return e;
}

// What a solve may allocate after a phase's ring, in FP64 spinors: true residuals 16, refinement 52, links
// of the refinement 12, and where an FP32 phase follows (tau) its p, h, s and a short ring in FP32.
static inline int ms_later(const MSolveArgs &A) { return 80 + (A.tau != 0.0 ? 6 * A.nrhs + 12 : 0); }

// One phase of the multi-shift CG with links LF: base vectors (residual ring, p, h, s) in the
// links' precision, shifted solutions and directions always FP64.  A fresh phase starts from
// x_i = 0; a resumed phase continues the state a previous FP64 phase left (scalars, shifted
// vectors, and its base vectors converted to this precision), optionally with reliable updates.
template <class LF, int NR>
static int ms_phase(rhmc_ctx *c, const LF &lf, const MSolveArgs &A, MSolveInfo *info)
{
    AuxScope aux_scope(c);
    cudaStream_t s_ = c->aux;
    typedef typename LF::real Rv;
    typedef typename SpinorT<Rv>::elem E;
    const int Vh = (int)c->Vh;
    const size_t stride = 3 * (size_t)Vh;
    const size_t vbytes = stride * sizeof(E), v64 = stride * sizeof(double2);
    const int S = A.nshift;
    const bool ru = A.ru_every > 0;
    if (!A.fresh && sizeof(E) == sizeof(double2)) return fail(RHMC_ERR_ARG, "multi-shift: an FP64 phase cannot resume an FP64 phase");
    void *r, *p, *h, *s, *ps, *stv, *part, *tick;
    CK(c->ws.get(vname("ms_p", sizeof(E)), NR * vbytes, &p));
    CK(c->ws.get(vname("ms_h", sizeof(E)), NR * vbytes, &h));
    CK(c->ws.get(vname("ms_s", sizeof(E)), NR * vbytes, &s));
    CK(c->ws.get("ms_ps", (size_t)NR * S * v64, &ps));
    CK(c->ws.get("ms_state", sizeof(MSState), &stv));
    const int gv = grid_for(Vh, VEC_BLOCK);
    CK(c->ws.get("ms_partials", (size_t)red_chunks(Vh) * 2 * NR * sizeof(double), &part));
    CK(c->ws.get("ms_tickets", 8 * sizeof(unsigned), &tick));
    // ring of the window's residuals [slot][rhs]
    int win;
    CK(ms_ring(c, vname("ms_r", sizeof(E)), NR * vbytes, v64, ms_later(A), &r, &win));
    const int ru_every = (A.ru_every + win - 1) / win;  // in windows
    MSState *st = (MSState *)stv;
    unsigned *tk = (unsigned *)tick;
    double *pt = (double *)part;
    double2 *xs = (double2 *)A.x;
    CK(cudaMemsetAsync(tk, 0, 8 * sizeof(unsigned), s_));

    if (A.fresh) {
        MSState h0;
        if (!ms_fill(A, h0) && ru) return fail(RHMC_ERR_ARG, "multi-shift: reliable updates need the base shift among the poles");
        h0.ru_every = ru_every;
        CK(cudaMemcpyAsync(st, &h0, MS_STATE_HEAD, cudaMemcpyHostToDevice, s_));
        ms_init_kernel<Rv, NR><<<gv, VEC_BLOCK, 0, s_>>>(Vh, stride, win, (const double2 *)A.b, (E *)r, (E *)p, pt, tk, st);
        c->launches++;
        CK(cudaGetLastError());
    } else {
        // resume the FP64 phase's state in this phase's precision (its ring as long as that phase made it)
        void *r64, *p64;
        CK(c->ws.get(vname("ms_r", sizeof(double2)), NR * v64, &r64));
        CK(c->ws.get(vname("ms_p", sizeof(double2)), NR * v64, &p64));
        CK(cudaMemcpyAsync(&st->res, &A.res_base, sizeof(double), cudaMemcpyHostToDevice, s_));
        CK(cudaMemcpyAsync(&st->ru_every, &ru_every, sizeof(int), cudaMemcpyHostToDevice, s_));
        ms_rearm_kernel<<<1, 32, 0, s_>>>(st);
        ms_convert_kernel<double, Rv, NR><<<gv, VEC_BLOCK, 0, s_>>>(Vh, stride, (const double2 *)r64, (const double2 *)p64,
                                                                     (E *)r, (E *)p, win, st);
        c->launches += 2;
        CK(cudaGetLastError());
    }

    // D_oe and D_eo launch arguments, on the base vectors' packed layout (BasePack)
    typedef typename std::conditional<BasePack<Rv, NR>::P == 1, LF, LPack<LF, BasePack<Rv, NR>::P>>::type LFB;
    typedef typename LFB::store::elem EB;
    LFB lfb;
    static_cast<LF &>(lfb) = lf;
    DslashArgs<LFB, NR, NoFin> a1;
    memset(&a1, 0, sizeof(a1));
    a1.g = c->g;
    a1.p_out = 1;
    a1.links = lfb;
    a1.in = (const EB *)p;
    a1.out = (EB *)h;
    a1.stride = stride;
    a1.beta = (Rv)0.5;
    a1.stop = &st->stop;
    a1.stop_set = &st->stop_k4;
    DslashArgs<LFB, NR, FinAlpha<NR>> a2;
    memset(&a2, 0, sizeof(a2));
    a2.g = c->g;
    a2.p_out = 0;
    a2.links = lfb;
    a2.in = (const EB *)h;
    a2.out = (EB *)s;
    a2.y = (const EB *)p;
    a2.stride = stride;
    a2.alpha = (Rv)(c->mass * c->mass + A.base[0]);
    a2.use_alphas = 1;  // every RHS iterates its own base operator M^dag M + base[r]
    for (int rr = 0; rr < NR; rr++) a2.alphas[rr] = (Rv)(c->mass * c->mass + A.base[rr]);
    a2.beta = (Rv)-0.5;
    a2.partials = pt;
    a2.ticket = tk + 1;
    a2.fin.st = st;
    const int down = walk_alternates<LFB, NR>(Vh, c->l2_bytes);
    a2.down = down;
    a2.stop = &st->stop;

    // reliable update: t = (M^dag M + base) x0 with FP64 12-real links, x0 the FP64 base solutions
    L64_12 l64;
    void *x0 = nullptr, *h64 = nullptr, *t64 = nullptr;
    DslashArgs<L64_12, NR, NoFin> u1, u2;
    memset(&u1, 0, sizeof(u1));
    memset(&u2, 0, sizeof(u2));
    if (ru) {
        cudaError_t e = links_f64_12(c, &l64);
        if (e != cudaSuccess) return cuda_fail(e, "links");
        // the FP64 phase's base vectors are free once resumed: they hold x0, D_oe x0 and t
        CK(c->ws.get(vname("ms_p", sizeof(double2)), NR * v64, &x0));
        CK(c->ws.get(vname("ms_h", sizeof(double2)), NR * v64, &h64));
        CK(c->ws.get(vname("ms_s", sizeof(double2)), NR * v64, &t64));
        u1.g = c->g; u1.p_out = 1; u1.links = l64; u1.in = (const double2 *)x0; u1.out = (double2 *)h64; u1.stride = stride;
        u1.beta = 0.5; u1.run_if = &st->ru_now;
        u2 = u1;
        u2.p_out = 0; u2.in = (const double2 *)h64; u2.out = (double2 *)t64; u2.y = (const double2 *)x0; u2.beta = -0.5;
        u2.use_alphas = 1;
        for (int rr = 0; rr < NR; rr++) u2.alphas[rr] = c->mass * c->mass + A.base[rr];
    }

    // shared memory of the flush's coefficients: above the 48 KB default for wide batches of many poles.
    // The limit belongs to the process, so it is always that of the most poles: one of this call's size
    // could be lowered by another context's call between here and the launch.
    const auto coefs = [](int poles) { return (size_t)NR * (poles * (MS_WIN + 1) + 1) * sizeof(double2); };
    const size_t coef_bytes = coefs(S);
    if (coefs(MS_MAX_SHIFT) > 40 * 1024)
        CK(cudaFuncSetAttribute(ms_flush_kernel<Rv, NR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)coefs(MS_MAX_SHIFT)));
    const int chunk = win;  // one graph replay = one delayed-update window
    struct Key {
        int kind, link_reals, link_bytes, nr, chunk, nshift, vh, ru_every;
        const void *links, *links64, *r, *p, *h, *s, *ps, *xs, *pt, *tk, *st, *x0, *h64, *t64, *b;
        double alpha[MS_MAX_RHS];
        cudaStream_t stream;
        int cand[4];  // launch shapes of the captured Dslash instantiations
    } key;
    memset(&key, 0, sizeof(key));
    // launch shapes (tuned now, outside the capture, when unknown)
    key.cand[0] = dslash_candidate<LFB, NR, false, false>(c->g, lfb, s_);
    key.cand[1] = dslash_candidate<LFB, NR, true, true>(c->g, lfb, s_);
    if (ru) {
        key.cand[2] = dslash_candidate<L64_12, NR, false, false>(c->g, l64, s_);
        key.cand[3] = dslash_candidate<L64_12, NR, true, false>(c->g, l64, s_);
    }
    key.kind = 4; key.link_reals = LF::reals; key.link_bytes = (int)sizeof(typename LF::real); key.nr = NR;
    key.chunk = chunk; key.nshift = S; key.vh = Vh; key.ru_every = ru_every; key.links = lf.p; key.r = r; key.p = p;
    key.h = h; key.s = s; key.ps = ps; key.xs = xs; key.pt = pt; key.tk = tk; key.st = st; key.stream = s_;
    if (ru) {
        key.links64 = l64.p; key.x0 = x0; key.h64 = h64; key.t64 = t64; key.b = A.b;
    }
    for (int rr = 0; rr < NR; rr++) key.alpha[rr] = (double)a2.alphas[rr];
    const std::string kb = key_bytes(key);
    cudaError_t ce = cudaSuccess;
    cudaGraphExec_t exec = c->graphs.find(kb);
    if (!exec) {
        cudaGraph_t graph;
        CK(cudaStreamBeginCapture(s_, cudaStreamCaptureModeThreadLocal));
        for (int it = 0; it < chunk; it++) {
            dslash_launch_cand<LFB, NR, false, false, NoFin>(key.cand[0], a1, Vh, s_);
            dslash_launch_cand<LFB, NR, true, true, FinAlpha<NR>>(key.cand[1], a2, Vh, s_);
            ms_resid_kernel<Rv, NR><<<persistent_grid((const void *)ms_resid_kernel<Rv, NR>, VEC_BLOCK, gv), VEC_BLOCK, 0,
                                      s_>>>(Vh, stride, win, (E *)r, (const E *)s, pt, tk + 2, st);
            ms_update_kernel<Rv, NR><<<gv, VEC_BLOCK, 0, s_>>>(Vh, stride, win, down, (const E *)r, (E *)p, st);
        }
        ms_flush_kernel<Rv, NR><<<grid_for((long)Vh * BasePack<Rv, NR>::P, VEC_BLOCK), VEC_BLOCK, coef_bytes, s_>>>(
            Vh, S, stride, (const E *)r, (double2 *)ps, xs, tk + 3, st);
        if (ru) {
            ms_ru_begin_kernel<<<1, 32, 0, s_>>>(st);
            ms_gather_base_kernel<NR><<<gv, VEC_BLOCK, 0, s_>>>(Vh, S, stride, xs, (double2 *)x0, st);
            dslash_launch_cand<L64_12, NR, false, false, NoFin>(key.cand[2], u1, Vh, s_);
            dslash_launch_cand<L64_12, NR, true, false, NoFin>(key.cand[3], u2, Vh, s_);
            ms_ru_resid_kernel<Rv, NR><<<gv, VEC_BLOCK, 0, s_>>>(Vh, S, stride, win, (const double2 *)A.b, (const double2 *)t64,
                                                                  (const double2 *)ps, (E *)r, (E *)p, pt, tk + 4, st);
        }
        ce = cudaStreamEndCapture(s_, &graph);
        if (ce != cudaSuccess) return cuda_fail(ce, "msolve capture");
        ce = cudaGraphInstantiate(&exec, graph, 0);
        cudaGraphDestroy(graph);
        if (ce != cudaSuccess) return cuda_fail(ce, "msolve instantiate");
        c->graphs.put(kb, exec);
    }

    const long max_chunks = (A.max_iter + chunk - 1) / chunk + 2;
    long launched = 0;
    int seen = 0;
    const int prc = replay_until_stop(c, exec, s_, &st->stop, max_chunks, &launched, &seen, "msolve loop");
    c->launches += launched * (chunk * 4 + 1 + (ru ? 5 : 0));
    if (prc) return prc;

    MSState hs;
    CK(cudaMemcpy(&hs, st, MS_STATE_HEAD, cudaMemcpyDeviceToHost));
    if (info) info->graph_replays += launched;
    return ms_result(hs, A, info);
}

// ------------------------------------------------------------------ small lattices
// Blocks of ms_small_kernel<LF, NR, MINB, false> that can be resident at once (0 when the query fails).
template <class LF, int NR, int MINB>
static long ms_small_capacity(int device, size_t smem)
{
    int occ = 0, sms = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, ms_small_kernel<LF, NR, MINB, false>, MS_SMALL_BLOCK, smem) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return (long)occ * sms;
}

// The launch of `groups` clusters of nch blocks; the attribute lives in *attr.
static inline cudaLaunchConfig_t ms_cluster_config(int nch, int groups, size_t smem, cudaStream_t s, cudaLaunchAttribute *attr)
{
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = (unsigned)nch;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nch * groups));
    cfg.blockDim = dim3(MS_SMALL_BLOCK);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// Whether a cluster of nch blocks of the kernel can be scheduled on this device.
template <class LF>
static bool ms_cluster_fits(int nch, size_t smem)
{
    auto kern = ms_small_kernel<LF, 1, 2, true>;
    if (nch > MS_CLUSTER) return false;
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg = ms_cluster_config(nch, 1, smem, nullptr, &attr);
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return n >= 1;
}

template <class LF, int NR, int MINB, bool CL>
static int ms_small_phase(rhmc_ctx *c, const LF &lf, const MSolveArgs &A, MSolveInfo *info)
{
    typedef typename LF::real Rv;
    typedef typename SpinorT<Rv>::elem E;
    cudaStream_t s_ = c->stream;
    const int Vh = (int)c->Vh, n = A.nrhs;
    const size_t stride = 3 * (size_t)Vh, vbytes = stride * sizeof(E), v64 = stride * sizeof(double2);
    void *r, *p, *h, *q, *ps, *stv, *slots;
    CK(c->ws.get(vname("ms_p", sizeof(E)), n * vbytes, &p));
    CK(c->ws.get(vname("ms_h", sizeof(E)), n * vbytes, &h));
    CK(c->ws.get(vname("ms_s", sizeof(E)), n * vbytes, &q));
    CK(c->ws.get("ms_ps", (size_t)n * A.nshift * v64, &ps));
    CK(c->ws.get("ms_state", sizeof(MSState), &stv));
    const int nch = grid_for(Vh, MS_SMALL_BLOCK);
    const size_t slot_bytes = (size_t)(n / NR) * 3 * ms_small_slots(NR, nch) * sizeof(ulonglong2);
    CK(c->ws.get("ms_slots", slot_bytes, &slots));
    int win;
    CK(ms_ring(c, vname("ms_r", sizeof(E)), n * vbytes, v64, ms_later(A), &r, &win));
    MSState *st = (MSState *)stv;

    MSState hs;
    ms_fill(A, hs);
    CK(cudaMemcpyAsync(st, &hs, MS_STATE_HEAD, cudaMemcpyHostToDevice, s_));
    MSSmallArgs<LF> a;
    a.g = c->g;
    a.links = lf;
    a.ring = (E *)r;
    a.p = (E *)p;
    a.q = (E *)q;
    a.h = (E *)h;
    a.ps = (double2 *)ps;
    a.x = (double2 *)A.x;
    a.slots = (ulonglong2 *)slots;
    a.st = st;
    a.nch = nch;
    a.nshift = A.nshift;
    a.nrhs = n;
    a.win = win;
    a.iters = MS_SMALL_ITERS;
    a.init = 1;
    for (int j = 0; j < MS_MAX_RHS; j++) a.alpha[j] = (Rv)(c->mass * c->mass + A.base[j < n ? j : 0]);
    const size_t smem = ms_small_smem(NR, A.nshift);
    for (int any = 1; any;) {
        CK(cudaMemsetAsync(slots, 0, slot_bytes, s_));
        void *args[] = {&a};
        const void *kern = (const void *)ms_small_kernel<LF, NR, MINB, CL>;
        if (CL) {
            cudaLaunchAttribute attr;
            const cudaLaunchConfig_t cfg = ms_cluster_config(nch, n / NR, smem, s_, &attr);
            CK(cudaLaunchKernelExC(&cfg, kern, args));
        } else {
            CK(cudaLaunchCooperativeKernel(kern, dim3((unsigned)(nch * (n / NR))), dim3(MS_SMALL_BLOCK), args, smem, s_));
        }
        c->launches++;
        CK(cudaMemsetAsync(&st->first, 0, sizeof(int), s_));
        CK(cudaMemcpyAsync(&hs, st, MS_STATE_HEAD, cudaMemcpyDeviceToHost, s_));
        CK(cudaStreamSynchronize(s_));
        a.init = 0;
        any = 0;
        for (int j = 0; j < n; j++) any |= hs.rhs[j].running_next;
        if (hs.status >= 2) any = 0;
    }
    return ms_result(hs, A, info);
}

// Runs a fresh phase as one kernel when all its blocks, one per 128 sites and right-hand side, fit on
// the device at once; false when they do not.  Two resident blocks per SM leave the kernel 255
// registers and its neighbour loads in larger batches (4 directions of p and r; 16.1 against
// 17.2 us an iteration on 12^3x24), three (168 registers) take half as many blocks again; then a
// block carries two right-hand sides, which reads the links once for both.  Every size that fits
// is faster than the launches it replaces, us an iteration: 4^4 6.4 against 21, 8^4 9.0 against 21
// (as clusters; 10 to 13 when its 16 blocks meet through L2, depending on where they land),
// 12^4 12.9 against 21, 12^3x24 two right-hand sides 20 against 29, 16^4 one 18 against 26 and two
// 24 against 32, 16^3x26 one 24 against 31 (FP64, 8 to 15 poles).
template <class LF>
static bool ms_small(rhmc_ctx *c, const LF &lf, const MSolveArgs &A, MSolveInfo *info, int *rc)
{
    const long chunks = grid_for(c->Vh, MS_SMALL_BLOCK);
    const size_t s1 = ms_small_smem(1, A.nshift), s2 = ms_small_smem(2, A.nshift);
    if (chunks > 1 && ms_cluster_fits<LF>((int)chunks, s1))
        *rc = ms_small_phase<LF, 1, 2, true>(c, lf, A, info);
    else if (chunks * A.nrhs <= ms_small_capacity<LF, 1, 2>(c->device, s1))
        *rc = ms_small_phase<LF, 1, 2, false>(c, lf, A, info);
    else if (chunks * A.nrhs <= ms_small_capacity<LF, 1, 3>(c->device, s1))
        *rc = ms_small_phase<LF, 1, 3, false>(c, lf, A, info);
    else if (A.nrhs % 2 == 0 && chunks * (A.nrhs / 2) <= ms_small_capacity<LF, 2, 2>(c->device, s2))
        *rc = ms_small_phase<LF, 2, 2, false>(c, lf, A, info);
    else
        return false;
    return true;
}

template <class LF>
int ms_run(rhmc_ctx *c, const LF &lf, const MSolveArgs &A, MSolveInfo *info)
{
    int rc = RHMC_OK;
    if (c->one_kernel && A.fresh && A.ru_every == 0 && ms_small<LF>(c, lf, A, info, &rc)) return rc;
    switch (A.nrhs) {
    case 1: return ms_phase<LF, 1>(c, lf, A, info);
    case 2: return ms_phase<LF, 2>(c, lf, A, info);
    case 3: return ms_phase<LF, 3>(c, lf, A, info);
    case 4: return ms_phase<LF, 4>(c, lf, A, info);
    case 8: return ms_phase<LF, 8>(c, lf, A, info);
    default: return fail(RHMC_ERR_ARG, "nrhs must be 1, 2, 3, 4 or 8 (got %d)", A.nrhs);
    }
}

}  // namespace rhmc

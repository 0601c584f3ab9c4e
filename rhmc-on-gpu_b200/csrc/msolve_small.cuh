// msolve_small.cuh -- the multi-shift CG of msolve.cuh as one persistent kernel, for lattices so small
// that the launches of an iteration cost more than its work.
//
// What bounds such a solve is latency: four launches with two last-block scalar steps take 20 us an
// iteration on a 4^4 lattice and 24 to 29 us on 12^3x24 (one and two right-hand sides), whatever the
// arithmetic; this kernel 6.4 and 16 to 20 us, of which on 12^3x24 half are the exchanges and on 4^4
// two thirds the dependent loads and FP64 chains of the two half-Dslashes.  Here a group of nch
// blocks carries NR right-hand sides through up to `iters` iterations without a launch: one
// 128-site chunk per block, one site per thread, r and p of the thread's own site in registers, and
// three group-wide exchanges an iteration:
//   A  h = D_oe p          with p = r + gamma p_old formed on the fly at every neighbour (which saves
//                          a barrier after the direction update); own p kept and stored
//   B  s = (m^2+sigma_0) p - D_eo h, chunk sums of Re<p,s>
//   C  omega and the shifted recurrences, in every block alike; r += omega s, chunk sums of |r|^2
// and after C gamma, freezing and stopping, again in every block alike (the same sums in the same
// order, so no block needs another's decision).  The shifted vectors are updated once per window
// from the residual ring as ms_flush_kernel does, each thread its own site.
//
// Right-hand sides of different groups share nothing, so each group has its own exchanges.  The chunk
// sums, their order, the Dslash and every update round exactly as in the kernels of msolve.cuh: a
// right-hand side's solution does not depend on which of the two paths solved it.
//
// Co-residency: a group of 2 to MS_CLUSTER chunks is a cluster, which the hardware places as a whole and
// whose barrier needs no limit (no block leaves before the last meeting); larger groups are launched
// cooperatively, and their exchanges give up after MS_SPIN_LIMIT polls, flag MSState::status = 3 and
// every block leaves.
#pragma once
#include <cooperative_groups.h>

#include "msolve.cuh"

namespace rhmc {

constexpr int MS_SMALL_BLOCK = RED_CHUNK;
constexpr unsigned MS_SPIN_LIMIT = 1u << 21;  // about a second
constexpr int MS_SMALL_ITERS = 1024;  // iterations per launch (about 10 ms; whole windows)

constexpr int MS_SLOT_CHUNKS = 32;
constexpr int MS_CLUSTER = 16;  // largest group that runs as a cluster (the non-portable maximum)

// entries of one kind of exchange of a group of nr right-hand sides: slots (or sums) and the counter
__host__ __device__ inline size_t ms_small_slots(int nr, int nch) { return (size_t)nr * nch + 1; }

// dynamic shared memory: the flush's coefficients
inline size_t ms_small_smem(int nr, int nshift) { return (size_t)nr * nshift * (MS_WIN + 1) * sizeof(double2); }

template <class LF>
struct MSSmallArgs {
    typedef typename LF::real R;
    typedef typename SpinorT<R>::elem E;
    Geom g;
    LF links;
    E *ring;           // [slot][rhs][3][Vh]
    E *p, *q;          // the direction, two buffers [rhs][3][Vh]; p holds it on entry and on return
    E *h;              // [rhs][3][Vh]
    double2 *ps, *x;   // [rhs][nshift][3][Vh]
    ulonglong2 *slots; // exchanges: [group][3][ms_small_slots], zero on entry
    MSState *st;
    int nch, nshift, nrhs, win, iters;
    int init;          // 1: start from b (x = 0); 0: continue
    R alpha[MS_MAX_RHS];  // m^2 + base shift
};

// A slot of the exchange below: a value and the number of the exchange it belongs to, written and
// read as one 16-byte access (single-copy atomic), so that a value needs no separate flag.
__device__ __forceinline__ void slot_store(ulonglong2 *s, double v, unsigned long long tag, bool release)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    if (release)
        asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.release.gpu.global.b128 [%0], t; }" ::"l"(s), "l"(b), "l"(tag) : "memory");
    else
        asm volatile("{ .reg .b128 t; mov.b128 t, {%1, %2}; st.relaxed.gpu.global.b128 [%0], t; }" ::"l"(s), "l"(b), "l"(tag) : "memory");
}
__device__ __forceinline__ double slot_load(const ulonglong2 *s, unsigned long long &tag, bool acquire)
{
    unsigned long long b;
    if (acquire)
        asm volatile("{ .reg .b128 t; ld.acquire.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }" : "=l"(b), "=l"(tag) : "l"(s) : "memory");
    else
        asm volatile("{ .reg .b128 t; ld.relaxed.gpu.global.b128 t, [%2]; mov.b128 {%0, %1}, t; }" : "=l"(b), "=l"(tag) : "l"(s) : "memory");
    return __longlong_as_double((long long)b);
}

// Where the blocks of a group meet, one per kind of exchange; `slots` holds ms_small_slots entries.
struct Meeting {
    ulonglong2 *slots;  // [N][nch]; as doubles, the chunk sums of groups that count
    unsigned *count;    // arrivals, in the entry after them
    unsigned target;    // arrivals of the current exchange
    unsigned long long tag;
};

// Group-wide sums of N values per thread, in every thread of every block, added in the order of
// reduce_tile and reduce_last (a zero added to a partial sum changes no bit).  With DATA every store before the exchange is also visible to the
// loads after it (ld.cg) in all blocks of the group, i.e. it is the barrier as well; without, it
// orders nothing but the sums.
//   * up to MS_CLUSTER chunks: the group is a cluster, which meets at its hardware barrier and passes
//     the sums through shared memory;
//   * sums of up to MS_SLOT_CHUNKS chunks: every block publishes its chunk sums in slots that carry the
//     number of the exchange and reads all chunks' slots until they do: one publication and one
//     poll latency (8^4, 16 chunks: 2,200 to 3,900 cycles against 4,500 to 4,900 when counted);
//   * more chunks: all blocks polling all slots queue in L2 (81 chunks: 8,000 cycles; with 16 copies
//     of every slot, or a root block that sums for all, 5,000 to 9,000), so they count arrivals
//     and then read the sums: 4,500 to 4,900 cycles; the barrier alone always counts (2,900).
// Returns false, uniformly over the block, when some block did not arrive in MS_SPIN_LIMIT polls.
__device__ __forceinline__ bool group_arrive(Meeting &w, MSState *st, int ok)
{
    if (threadIdx.x == 0) {
        unsigned polls = 0;
        __threadfence();
        atomicAdd(w.count, 1u);
        while ((int)(*(volatile unsigned *)w.count - w.target) < 0 && ++polls < MS_SPIN_LIMIT) {}
        __threadfence();
        ok = polls < MS_SPIN_LIMIT;
        if (!ok) st->status = 3;
    }
    return __syncthreads_and(ok);
}

// the barrier alone
template <bool CL>
__device__ __forceinline__ bool group_barrier(Meeting &w, int nch, MSState *st)
{
    if constexpr (CL) {
        cooperative_groups::this_cluster().sync();
        return true;
    }
    __syncthreads();
    w.target += nch;
    return nch == 1 || group_arrive(w, st, 1);
}

template <int N, bool DATA, bool CL>
__device__ __forceinline__ bool group_exchange(const double (&v)[N], double (&tot)[N], Meeting &w, int nch, int chunk, MSState *st)
{
    __shared__ double sm[N][MS_SMALL_BLOCK];
    __shared__ double wsum[N][4];
    if constexpr (CL) {
        // every block's chunk sums into every block's shared memory, one array per kind of exchange (a
        // block is past the next exchange's barrier only when all have read this one's)
        __shared__ double peer[N][MS_CLUSTER];
        namespace cg = cooperative_groups;
        cg::cluster_group cl = cg::this_cluster();
        const int ln = threadIdx.x & 31, wd = threadIdx.x >> 5;
#pragma unroll
        for (int j = 0; j < N; j++) sm[j][threadIdx.x] = v[j];
        __syncthreads();
        for (int j = wd; j < N; j += 4) {
            double t = sm[j][ln];
            t += sm[j][ln + 32];
            t += sm[j][ln + 64];
            t += sm[j][ln + 96];
            t = warp_sum(t);
            if (ln < nch) *cl.map_shared_rank(&peer[j][chunk], ln) = t;
        }
        cl.sync();
        // the order of reduce_last: lane t holds chunk t (fewer than 128 chunks: one each), zeros beyond,
        // a shuffle tree, and the sums of the three other warps, which are zero
#pragma unroll
        for (int j = 0; j < N; j++) {
            double t = warp_sum(ln < nch ? peer[j][ln] : 0.0);
            tot[j] = t;
        }
        return true;
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const bool counted = nch > MS_SLOT_CHUNKS;
    double *part = reinterpret_cast<double *>(w.slots);
#pragma unroll
    for (int j = 0; j < N; j++) sm[j][threadIdx.x] = v[j];
    __syncthreads();
    w.tag++;
    w.target += nch;
    for (int j = wid; j < N; j += 4) {
        double t = sm[j][lane];
        t += sm[j][lane + 32];
        t += sm[j][lane + 64];
        t += sm[j][lane + 96];
        t = warp_sum(t);
        if (lane != 0) continue;
        if (nch == 1)
            wsum[j][0] = t;
        else if (counted)
            __stcg(part + (size_t)j * nch + chunk, t);
        else
            slot_store(w.slots + (size_t)j * nch + chunk, t, w.tag, DATA);
    }
    if (nch == 1) {
        __syncthreads();
#pragma unroll
        for (int j = 0; j < N; j++) tot[j] = wsum[j][0];
        return true;
    }
    int ok = 1;
    double acc[N];
#pragma unroll
    for (int j = 0; j < N; j++) acc[j] = 0.0;
    if (counted) {
        __syncthreads();
        ok = group_arrive(w, st, 1);
        for (int i = threadIdx.x; i < nch; i += RED_CHUNK)
#pragma unroll
            for (int j = 0; j < N; j++) acc[j] += __ldcg(part + (size_t)j * nch + i);
    } else {
        unsigned polls = 0;
        for (int i = threadIdx.x; i < nch; i += RED_CHUNK)
#pragma unroll
            for (int j = 0; j < N; j++) {
                unsigned long long t;
                double q = slot_load(w.slots + (size_t)j * nch + i, t, DATA);
                while (t != w.tag && ++polls < MS_SPIN_LIMIT) q = slot_load(w.slots + (size_t)j * nch + i, t, DATA);
                if (t != w.tag) ok = 0;
                acc[j] += q;
            }
        if (!ok) st->status = 3;
    }
#pragma unroll
    for (int j = 0; j < N; j++) acc[j] = warp_sum(acc[j]);
    if (lane == 0)
#pragma unroll
        for (int j = 0; j < N; j++) wsum[j][wid] = acc[j];
    ok = __syncthreads_and(ok);
#pragma unroll
    for (int j = 0; j < N; j++) {
        double t = wsum[j][0];
        t += wsum[j][1];
        t += wsum[j][2];
        t += wsum[j][3];
        tot[j] = t;
    }
    return ok;
}

template <typename R>
__device__ __forceinline__ vec3<R> ldcg3(const typename SpinorT<R>::elem *v, int Vh, int k)
{
    vec3<R> r;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const typename SpinorT<R>::elem a = __ldcg(v + (size_t)c * Vh + k);
        r.c[c] = mk<R>(a.x, a.y);
    }
    return r;
}

template <typename R>
__device__ __forceinline__ void stcg3(typename SpinorT<R>::elem *v, int Vh, int k, const vec3<R> &r)
{
#pragma unroll
    for (int c = 0; c < 3; c++) {
        typename SpinorT<R>::elem a;
        a.x = r.c[c].re;
        a.y = r.c[c].im;
        __stcg(v + (size_t)c * Vh + k, a);
    }
}

// r + g p, rounded as ms_update_kernel does
template <typename R>
__device__ __forceinline__ void direction(vec3<R> &p, const vec3<R> &r, R g)
{
#pragma unroll
    for (int c = 0; c < 3; c++) {
        p.c[c].re = r.c[c].re + g * p.c[c].re;
        p.c[c].im = r.c[c].im + g * p.c[c].im;
    }
}

// CL: the group is a thread-block cluster of nch blocks
template <class LF, int NR, int MINB, bool CL>
__global__ void __launch_bounds__(MS_SMALL_BLOCK, MINB) ms_small_kernel(MSSmallArgs<LF> a)
{
    typedef typename LF::real R;
    typedef typename SpinorT<R>::elem E;
    extern __shared__ double2 s_coef[];  // [NR][nshift][MS_WIN + 1]
    __shared__ double s_om[NR][MS_MAX_SHIFT][MS_WIN], s_ga[NR][MS_MAX_SHIFT][MS_WIN], s_ze[NR][MS_MAX_SHIFT][MS_WIN];
    __shared__ unsigned s_act[NR][MS_WIN];
    __shared__ int s_nact[NR], s_list[NR][MS_MAX_SHIFT], s_n[NR];
    const int Vh = a.g.Vh, ns = a.nshift, nch = a.nch;
    const int group = blockIdx.x / nch, chunk = blockIdx.x % nch, r0 = group * NR;
    const int k = chunk * MS_SMALL_BLOCK + threadIdx.x;
    const bool in = k < Vh;
    const size_t stride = 3 * (size_t)Vh;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    MSState *st = a.st;
    // exchanges after A (barrier), B (Re<p,s>) and C (|r|^2); a block's entries are written again only
    // after an exchange of another kind, which their readers enter after reading them
    Meeting meet[3];
#pragma unroll
    for (int m = 0; m < 3; m++) {
        meet[m].slots = a.slots + (3 * group + m) * ms_small_slots(NR, nch);
        meet[m].count = reinterpret_cast<unsigned *>(meet[m].slots + (size_t)NR * nch);
        meet[m].target = 0;
        meet[m].tag = 0;
    }
    const Site se = site_of(a.g, 0, in ? k : 0), so = site_of(a.g, 1, in ? k : 0);

    // scalars of the group's right-hand sides, in every thread; the shifted ones in lane i of warp r
    double delta[NR], omega[NR], omega_prev[NR], gamma[NR], lambda[NR], alpha[NR], res[NR], b2[NR];
    int run[NR], iter[NR], rslot[NR];
    bool upd[NR];  // p has still to be formed from r and gamma
    const int max_iter = st->max_iter, stop_on_frozen = st->stop_on_frozen;
    int first = a.init, status = 0;
    double zi = 1.0, zii = 1.0, ziii = 1.0, oms = 0.0, gas = 0.0, sh = 0.0, tgt = 0.0;
    int an = 1;
    const bool sl = wid < NR && lane < ns;  // this lane carries a shift
    if (sl) {
        sh = st->rhs[r0 + wid].shift[lane];
        tgt = st->tgt[lane];
    }
    vec3<R> r[NR], p[NR];
#pragma unroll
    for (int j = 0; j < NR; j++) {
        upd[j] = false;
#pragma unroll
        for (int c = 0; c < 3; c++) r[j].c[c] = p[j].c[c] = mk<R>(0, 0);
    }
    if (a.init) {  // r = p = b, |b|^2 (ms_init_kernel, FinInit)
        double red[NR], tot[NR];
#pragma unroll
        for (int j = 0; j < NR; j++) {
            red[j] = 0.0;
            if (in) {
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const double2 v = st->b[(size_t)(r0 + j) * stride + (size_t)c * Vh + k];
                    red[j] += dot2(v.x, v.x, v.y, v.y);
                    r[j].c[c] = p[j].c[c] = mk<R>((R)v.x, (R)v.y);
                }
                stcg3<R>(a.p + (size_t)(r0 + j) * stride, Vh, k, p[j]);
                stcg3<R>(a.ring + ((size_t)(a.win - 1) * a.nrhs + r0 + j) * stride, Vh, k, r[j]);
            }
        }
        if (!group_exchange<NR, true, CL>(red, tot, meet[2], nch, chunk, st)) return;
        const double rs = st->res, tau = st->tau;
#pragma unroll
        for (int j = 0; j < NR; j++) {
            const double nb = sqrt(tot[j]);
            b2[j] = delta[j] = lambda[j] = tot[j];
            omega[j] = omega_prev[j] = 1.0;
            gamma[j] = alpha[j] = 0.0;
            res[j] = tau > 0.0   ? fmax(rs, tau * nb)
                     : tau < 0.0 ? fmax(rs, fmax(MS_TAU_MIN * nb, fmin(-tau * nb, MS_TAU_REACH * rs)))
                                 : rs;
            iter[j] = 0;
            rslot[j] = a.win - 1;
            run[j] = isfinite(tot[j]) && tot[j] > 0.0;  // b == 0: x = 0 is exact
            if (!isfinite(tot[j])) status = 2;
        }
    } else {
#pragma unroll
        for (int j = 0; j < NR; j++) {
            const MSRhs &q = st->rhs[r0 + j];
            b2[j] = q.b2;
            delta[j] = q.delta;
            omega[j] = q.omega;
            omega_prev[j] = q.omega_prev;
            gamma[j] = q.gamma;
            lambda[j] = q.lambda;
            alpha[j] = q.alpha;
            res[j] = q.res;
            run[j] = q.running_next;
            iter[j] = q.iter;
            rslot[j] = q.rslot;
            if (in) {
                r[j] = ldcg3<R>(a.ring + ((size_t)rslot[j] * a.nrhs + r0 + j) * stride, Vh, k);
                p[j] = ldcg3<R>(a.p + (size_t)(r0 + j) * stride, Vh, k);
            }
        }
        if (sl) {
            const MSRhs &q = st->rhs[r0 + wid];
            zi = q.zeta_i[lane];
            zii = q.zeta_ii[lane];
            ziii = q.zeta_iii[lane];
            oms = q.omegas[lane];
            gas = q.gammas[lane];
            an = q.active_next[lane];
        }
        // every block has read the state before one of the group writes it at the end
        if (!group_barrier<CL>(meet[2], nch, st)) return;
    }
    E *pc = a.p, *pn = a.q;  // current and next direction buffer
    int wp = 0;

    for (int it = 0; it <= a.iters; it++) {
        int any = 0;
#pragma unroll
        for (int j = 0; j < NR; j++) any |= run[j];
        const bool leave = !any || it == a.iters;
        // ---- end of a window (or of this launch): the shifted vectors of the thread's own site
        if ((wp > 0 || first) && (wp == a.win || leave)) {
            if (wid < NR) {
                double D = 0.0, G = 1.0;
                int used = 0;
                if (lane < ns) {
                    double2 *cf = s_coef + (size_t)(wid * ns + lane) * (MS_WIN + 1);
                    for (int m = MS_WIN - 1; m >= 0; m--) {
                        const bool act = m < wp && (s_act[wid][m] >> lane & 1u);
                        const double ze = act ? s_ze[wid][lane][m] : 0.0;
                        cf[m] = act ? make_double2(ze * D, ze * G) : make_double2(0.0, 0.0);
                        if (act) {
                            D = s_om[wid][lane][m] + s_ga[wid][lane][m] * D;
                            G = s_ga[wid][lane][m] * G;
                            used = 1;
                        }
                    }
                    cf[MS_WIN] = make_double2(D, G);
                }
                const int use = lane < ns && (used || first);
                const unsigned mask = __ballot_sync(0xffffffffu, use);
                if (use) s_list[wid][__popc(mask & ((1u << lane) - 1u))] = 2 * lane + (an ? 1 : 0);
                if (lane == 0) s_n[wid] = __popc(mask);
            }
            __syncthreads();
            if (in) {
#pragma unroll 1
                for (int jc = 0; jc < 3 * NR; jc++) {
                    const int j = jc / 3, c = jc % 3;
                    double2 rv[MS_WIN];
#pragma unroll
                    for (int m = 0; m < MS_WIN; m++) {
                        rv[m] = make_double2(0.0, 0.0);
                        if (m < wp && s_act[j][m]) {  // a slot this right-hand side wrote (see ms_flush_kernel)
                            const E e = __ldcg(a.ring + ((size_t)m * a.nrhs + r0 + j) * stride + (size_t)c * Vh + k);
                            rv[m] = make_double2((double)e.x, (double)e.y);
                        }
                    }
                    double2 b0 = make_double2(0.0, 0.0);
                    if (first) b0 = st->b[(size_t)(r0 + j) * stride + (size_t)c * Vh + k];
                    const size_t o = (size_t)(r0 + j) * ns * stride + (size_t)c * Vh + k;
                    const double2 *cj = s_coef + (size_t)j * ns * (MS_WIN + 1);
                    const int n = s_n[j];
                    // the next two active shifts' vectors are in flight
                    double2 p1 = b0, p2 = b0, x1 = make_double2(0.0, 0.0), x2 = x1;
                    if (!first) {
                        if (n > 0) {
                            p1 = a.ps[o + (size_t)(s_list[j][0] >> 1) * stride];
                            x1 = a.x[o + (size_t)(s_list[j][0] >> 1) * stride];
                        }
                        if (n > 1) {
                            p2 = a.ps[o + (size_t)(s_list[j][1] >> 1) * stride];
                            x2 = a.x[o + (size_t)(s_list[j][1] >> 1) * stride];
                        }
                    }
                    for (int t = 0; t < n; t++) {
                        const int e = s_list[j][t], i = e >> 1;
                        const double2 p0 = p1;
                        double2 xv = x1, pv;
                        p1 = p2;
                        x1 = x2;
                        if (!first && t + 2 < n) {
                            const size_t oi = o + (size_t)(s_list[j][t + 2] >> 1) * stride;
                            p2 = a.ps[oi];
                            x2 = a.x[oi];
                        }
                        const double2 *cf = cj + i * (MS_WIN + 1);
                        const double2 c0 = cf[MS_WIN];
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
                        a.x[o + (size_t)i * stride] = xv;
                        if (e & 1) a.ps[o + (size_t)i * stride] = pv;
                    }
                }
            }
            __syncthreads();  // the coefficients and the history are free again
            wp = 0;
            first = 0;
        }
        if (leave) break;

        // ---- A: own direction, h = D_oe p on the odd site k
        R g[NR];
        const bool formed = it == 0;  // on entry p is already the direction
#pragma unroll
        for (int j = 0; j < NR; j++) {
            g[j] = (R)gamma[j];
            if (upd[j]) direction(p[j], r[j], g[j]);
        }
        if (in) {
            if (!formed)
#pragma unroll
                for (int j = 0; j < NR; j++) stcg3<R>(pn + (size_t)(r0 + j) * stride, Vh, k, p[j]);
            vec3<R> acc[NR];
#pragma unroll
            for (int j = 0; j < NR; j++)
#pragma unroll
                for (int c = 0; c < 3; c++) acc[j].c[c] = mk<R>(0, 0);
            // the neighbours' p and r of DB directions are loaded together (a branch per direction, or per
            // right-hand side that still runs, would expose one L2 latency each: 7,300 cycles for the
            // eight directions); a stopped right-hand side is carried along and its h not used
            constexpr int DB = NR == 1 && MINB == 2 ? 4 : 2;
#pragma unroll
            for (int d0 = 0; d0 < 8; d0 += DB) {
                vec3<R> v[DB][NR], w[DB][NR];
#pragma unroll
                for (int d = 0; d < DB; d++) {
                    const int kn = neighbour(a.g, so, (d0 + d) >> 1, (d0 + d) & 1 ? -1 : +1);
#pragma unroll
                    for (int j = 0; j < NR; j++) {
                        v[d][j] = ldcg3<R>(pc + (size_t)(r0 + j) * stride, Vh, kn);
                        w[d][j] = ldcg3<R>(a.ring + ((size_t)rslot[j] * a.nrhs + r0 + j) * stride, Vh, kn);
                    }
                }
#pragma unroll
                for (int d = 0; d < DB; d++) {
                    const int mu = (d0 + d) >> 1, back = (d0 + d) & 1;
                    su3m<R> u;
                    if (!back)
                        a.links.load(mu, 1, k, u, eta_of(a.g, so, mu));
                    else
                        a.links.load(mu, 0, neighbour(a.g, so, mu, -1), u, eta_back(a.g, so, mu));
#pragma unroll
                    for (int j = 0; j < NR; j++) {
                        vec3<R> f = v[d][j];
                        direction(f, w[d][j], g[j]);
                        if (!upd[j]) f = v[d][j];
                        if (!back)
                            mv_acc(u, f, acc[j]);
                        else
                            mdv_sub(u, f, acc[j]);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < NR; j++) {
                vec3<R> o;
#pragma unroll
                for (int c = 0; c < 3; c++) o.c[c] = mk<R>((R)0.5 * acc[j].c[c].re, (R)0.5 * acc[j].c[c].im);
                stcg3<R>(a.h + (size_t)(r0 + j) * stride, Vh, k, o);
            }
        }
        if (!formed) {
            E *t = pc;
            pc = pn;
            pn = t;
        }
#pragma unroll
        for (int j = 0; j < NR; j++) upd[j] = run[j];
        if (!group_barrier<CL>(meet[0], nch, st)) return;

        // ---- B: s = (m^2 + sigma_0) p - D_eo h on the even site k, Re<p, s>
        vec3<R> s[NR];
        double red[NR];
#pragma unroll
        for (int j = 0; j < NR; j++) {
            red[j] = 0.0;
#pragma unroll
            for (int c = 0; c < 3; c++) s[j].c[c] = mk<R>(0, 0);
        }
        if (in) {
            constexpr int DB = NR == 1 && MINB == 2 ? 8 : 4;
#pragma unroll
            for (int d0 = 0; d0 < 8; d0 += DB) {
                vec3<R> v[DB][NR];
#pragma unroll
                for (int d = 0; d < DB; d++) {
                    const int kn = neighbour(a.g, se, (d0 + d) >> 1, (d0 + d) & 1 ? -1 : +1);
#pragma unroll
                    for (int j = 0; j < NR; j++) v[d][j] = ldcg3<R>(a.h + (size_t)(r0 + j) * stride, Vh, kn);
                }
#pragma unroll
                for (int d = 0; d < DB; d++) {
                    const int mu = (d0 + d) >> 1, back = (d0 + d) & 1;
                    su3m<R> u;
                    if (!back)
                        a.links.load(mu, 0, k, u, eta_of(a.g, se, mu));
                    else
                        a.links.load(mu, 1, neighbour(a.g, se, mu, -1), u, eta_back(a.g, se, mu));
#pragma unroll
                    for (int j = 0; j < NR; j++) {
                        if (!back)
                            mv_acc(u, v[d][j], s[j]);
                        else
                            mdv_sub(u, v[d][j], s[j]);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < NR; j++) {
                const R al = a.alpha[r0 + j], be = (R)-0.5;
                float tf = 0.f;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    s[j].c[c] = mk<R>(dot2(be, s[j].c[c].re, al, p[j].c[c].re), dot2(be, s[j].c[c].im, al, p[j].c[c].im));
                    site_dot(red[j], tf, p[j].c[c], s[j].c[c]);
                }
                if (sizeof(R) == 4) red[j] = (double)tf;
            }
        }
        double tot[NR];
        if (!group_exchange<NR, false, CL>(red, tot, meet[1], nch, chunk, st)) return;

        // ---- C: omega, the shifted recurrences (FinAlpha), r += omega s, |r|^2
#pragma unroll
        for (int j = 0; j < NR; j++) {
            if (run[j]) {
                alpha[j] = tot[j];
                if (!isfinite(alpha[j]) || alpha[j] == 0.0) {
                    status = 2;
                    run[j] = 0;
                    upd[j] = false;
                } else {
                    omega_prev[j] = omega[j];
                    omega[j] = -delta[j] / alpha[j];
                }
            }
            if (wid == j) {
                const int act = sl && run[j] && an;
                const unsigned mask = __ballot_sync(0xffffffffu, act);
                if (lane == 0) s_act[j][wp] = mask;
                if (act) {
                    const double om = omega[j], omp = omega_prev[j];
                    ziii = next_zeta(zi, zii, omp, om, gamma[j], sh);
                    oms = om * ziii / zii;
                    s_om[j][lane][wp] = oms;
                }
            }
        }
#pragma unroll
        for (int j = 0; j < NR; j++) {
            red[j] = 0.0;
            if (in && run[j]) {
                const R om = (R)omega[j];
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    r[j].c[c].re = r[j].c[c].re + om * s[j].c[c].re;
                    r[j].c[c].im = r[j].c[c].im + om * s[j].c[c].im;
                    red[j] += dot2((double)r[j].c[c].re, (double)r[j].c[c].re, (double)r[j].c[c].im, (double)r[j].c[c].im);
                }
                stcg3<R>(a.ring + ((size_t)wp * a.nrhs + r0 + j) * stride, Vh, k, r[j]);
            }
        }
        if (!group_exchange<NR, true, CL>(red, tot, meet[2], nch, chunk, st)) return;

        // ---- gamma, freezing (FinLambda)
#pragma unroll
        for (int j = 0; j < NR; j++) {
            if (run[j]) {
                lambda[j] = tot[j];
                rslot[j] = wp;
                if (!isfinite(lambda[j])) {
                    status = 2;
                    run[j] = 0;
                    upd[j] = false;
                } else {
                    gamma[j] = lambda[j] / delta[j];
                }
            }
            if (wid == j) {
                int live = 0;
                if (run[j] && (s_act[j][wp] >> lane & 1u)) {
                    gas = gamma[j] * ziii * oms / (zii * omega[j]);
                    s_ga[j][lane][wp] = gas;
                    s_ze[j][lane][wp] = ziii;
                    const double fact = sqrt(delta[j] * zii * zii);
                    an = (fact < tgt) ? 0 : 1;
                    zi = zii;
                    zii = ziii;
                    live = an;
                }
                const unsigned mask = __ballot_sync(0xffffffffu, live);
                if (lane == 0) s_nact[j] = __popc(mask);
            }
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < NR; j++) {
            if (!run[j]) continue;
            delta[j] = lambda[j];
            iter[j]++;
            int done = (sqrt(lambda[j]) <= res[j]) || (stop_on_frozen && s_nact[j] == 0);
            if (!done && iter[j] >= max_iter) {
                done = 1;
                if (status == 0) status = 1;
            }
            run[j] = !done;
        }
        wp++;
    }

    // the direction of the next iteration, and the state, as the kernels of msolve.cuh leave them
#pragma unroll
    for (int j = 0; j < NR; j++) {
        if (upd[j]) direction(p[j], r[j], (R)gamma[j]);
        if (in) stcg3<R>(a.p + (size_t)(r0 + j) * stride, Vh, k, p[j]);
    }
    if (chunk == 0) {
        if (threadIdx.x == 0) {
#pragma unroll
            for (int j = 0; j < NR; j++) {
                MSRhs &q = st->rhs[r0 + j];
                q.b2 = b2[j];
                q.res = res[j];
                q.delta = delta[j];
                q.omega = omega[j];
                q.omega_prev = omega_prev[j];
                q.gamma = gamma[j];
                q.lambda = lambda[j];
                q.alpha = alpha[j];
                q.running = run[j];
                q.running_next = run[j];
                q.iter = iter[j];
                q.rslot = rslot[j];
            }
            if (status) atomicMax(&st->status, status);
        }
        if (sl) {
            MSRhs &q = st->rhs[r0 + wid];
            q.zeta_i[lane] = zi;
            q.zeta_ii[lane] = zii;
            q.zeta_iii[lane] = ziii;
            q.omegas[lane] = oms;
            q.gammas[lane] = gas;
            q.active[lane] = an;
            q.active_next[lane] = an;
        }
    }
}

}  // namespace rhmc

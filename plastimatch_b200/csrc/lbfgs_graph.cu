// The controller of the graph-resident L-BFGS (optimize.cu builds the
// graph): one thread runs the line-search and iteration logic of the
// host-driven loop on the device, between the vector work and the
// evaluations, and steers the graph's conditional nodes -- the while loop
// over trial points and the branch that starts a new line search
// (correction pair, two-loop recursion, dginit).  For small vectors the
// kernels here do the vector work as well.  No scalar leaves the device
// until the run ends.
//
// This file is compiled without floating-point contraction, so the
// controller rounds exactly as the host-driven loop (host code) does.
#include <algorithm>

#include <cooperative_groups.h>

#include "lbfgs_graph.cuh"

namespace b200 {

namespace {

// The step's bracket and the safeguarded trial step (the top of each
// iteration of the Moré-Thuente loop).
__device__ void
pre_trial (LbDev* s)
{
    if (s->brackt) {
        s->stmin = lb_min (s->stx, s->sty);
        s->stmax = lb_max (s->stx, s->sty);
    } else {
        s->stmin = s->stx;
        s->stmax = s->stp + 4.0 * (s->stp - s->stx);
    }
    s->stp = lb_max (s->min_step, lb_min (s->max_step, s->stp));
    if ((s->brackt && ((s->stp <= s->stmin || s->stmax <= s->stp)
             || s->max_linesearch <= s->count + 1 || s->uinfo != 0))
        || (s->brackt && (s->stmax - s->stmin <= s->xtol * s->stmax))) {
        s->stp = s->stx;
    }
}

__device__ void
finish_run (LbDev* s, int status, cudaGraphConditionalHandle h_while)
{
    s->status = status;
    s->done = 1;
    cudaGraphSetConditional (h_while, 0);
}

// Start of a line search: s->dginit is there.
__device__ void
begin_search (LbDev* s, cudaGraphConditionalHandle h_while)
{
    if (s->done) return;
    s->first = 0;
    s->finit = s->f;
    if (s->stp <= 0.0) {
        finish_run (s, LS_BADSTEP, h_while);
        return;
    }
    if (0.0 < s->dginit) {
        finish_run (s, LS_INCREASE, h_while);
        return;
    }
    s->brackt = 0;
    s->stage1 = 1;
    s->uinfo = 0;
    s->count = 0;
    s->dgtest = s->ftol * s->dginit;
    s->width = s->max_step - s->min_step;
    s->prev_width = 2.0 * s->width;
    s->stx = 0.0;
    s->fx = s->finit;
    s->dgx = s->dginit;
    s->sty = 0.0;
    s->fy = s->finit;
    s->dgy = s->dginit;
    pre_trial (s);
}

// After an evaluation: s->dg, s->xx and s->gg are there.
__device__ void
after_eval (LbDev* s, cudaGraphConditionalHandle h_while,
    cudaGraphConditionalHandle h_new)
{
    cudaGraphSetConditional (h_new, 0);
    if (s->done) {
        cudaGraphSetConditional (h_while, 0);
        return;
    }
    // Bspline_score's total (float) as the objective
    s->f = (double) s->total;
    s->last = s->total;
    s->fevals++;
    if (lb_stop_rule (s->max_its, s->max_feval, s->k, s->fevals)) {
        finish_run (s, LS_STOPPED, h_while);
        return;
    }
    const double f = s->f, dg = s->dg;
    const double ftest1 = s->finit + s->stp * s->dgtest;
    ++s->count;
    if (s->brackt && ((s->stp <= s->stmin || s->stmax <= s->stp)
            || s->uinfo != 0)) {
        finish_run (s, LS_ROUNDING, h_while);
        return;
    }
    if (s->stp == s->max_step && f <= ftest1 && dg <= s->dgtest) {
        finish_run (s, LS_MAXSTEP, h_while);
        return;
    }
    if (s->stp == s->min_step && (ftest1 < f || s->dgtest <= dg)) {
        finish_run (s, LS_MINSTEP, h_while);
        return;
    }
    if (s->brackt && (s->stmax - s->stmin) <= s->xtol * s->stmax) {
        finish_run (s, LS_WIDTH, h_while);
        return;
    }
    if (s->max_linesearch <= s->count) {
        finish_run (s, LS_MAXLS, h_while);
        return;
    }
    if (f <= ftest1 && fabs (dg) <= s->gtol * (-s->dginit)) {
        // the line search is done: the iteration's tests, then a new pair
        s->iterations = s->k;
        double xnorm = sqrt (s->xx), gnorm = sqrt (s->gg);
        if (lb_stop_rule (s->max_its, s->max_feval, s->k, s->fevals)) {
            finish_run (s, B200BSP_LBFGS_STOPPED, h_while);
            return;
        }
        if (xnorm < 1.0) xnorm = 1.0;
        if (gnorm / xnorm <= s->epsilon) {
            finish_run (s, B200BSP_LBFGS_CONVERGED, h_while);
            return;
        }
        s->newest = s->end;
        s->bound = s->m < s->k ? s->m : s->k;
        ++s->k;
        s->end = (s->end + 1) % s->m;
        s->stp = 1.0;
        s->newiter = 1;
        cudaGraphSetConditional (h_new, 1);
        return;
    }
    if (s->stage1 && f <= ftest1
        && lb_min (s->ftol, s->gtol) * s->dginit <= dg) {
        s->stage1 = 0;
    }
    if (s->stage1 && ftest1 < f && f <= s->fx) {
        // first stage: work on the modified function f - stp * dgtest
        const double fm = f - s->stp * s->dgtest;
        double fxm = s->fx - s->stx * s->dgtest, fym = s->fy - s->sty * s->dgtest;
        const double dgm = dg - s->dgtest;
        double dgxm = s->dgx - s->dgtest, dgym = s->dgy - s->dgtest;
        s->uinfo = lb_update_interval (&s->stx, &fxm, &dgxm, &s->sty, &fym,
            &dgym, &s->stp, fm, dgm, s->stmin, s->stmax, &s->brackt);
        s->fx = fxm + s->stx * s->dgtest;
        s->fy = fym + s->sty * s->dgtest;
        s->dgx = dgxm + s->dgtest;
        s->dgy = dgym + s->dgtest;
    } else {
        s->uinfo = lb_update_interval (&s->stx, &s->fx, &s->dgx, &s->sty,
            &s->fy, &s->dgy, &s->stp, f, dg, s->stmin, s->stmax, &s->brackt);
    }
    if (s->brackt) {
        if (0.66 * s->prev_width <= fabs (s->sty - s->stx)) {
            s->stp = s->stx + 0.5 * (s->sty - s->stx);
        }
        s->prev_width = s->width;
        s->width = fabs (s->sty - s->stx);
    }
    s->newiter = 0;
    pre_trial (s);
}

// ---- a cluster per step -------------------------------------------------------
//
// For up to LB_CLUSTER_MAX entries the new-line-search branch and the work
// after an evaluation are one launch each, of one cluster whose threads keep
// their share of the vectors in registers: what bounds them is the chain of
// dot products (two a pair kept, each a reduction of the whole vector), so a
// dot product costs one barrier, and the vectors of the next step are
// fetched while this one's sum is on its way.  Four iterations at 64^3 vpr 8
// (3993 entries, one block): 502 us a call; 578 with one block that re-read
// its vectors from L2 for each step, the search's start and the dot
// products after an evaluation in launches of their own.
//
// The cluster grows by doubling from one block to the portable eight at 8
// entries a thread (s, y and d of a pair and the next: 122 registers), then
// a thread takes 16.

namespace cg = cooperative_groups;

constexpr int LBC_THREADS = 512;
constexpr int LBC_WARPS = LBC_THREADS / 32;
constexpr int LBC_MAX_BLOCKS = 8;
constexpr int LBC_MAX_PAIRS = 64;

// One sum's partials of every warp of the cluster; two sets taken in turn,
// since a fast block may write the next sum's while another reads this one's.
struct LbcSums {
    double v[2][3][LBC_MAX_BLOCKS * LBC_WARPS];
};

// The cluster's sums of K values, in every thread, in a fixed order.
template <int K>
__device__ __forceinline__ void
lbc_sum (double (&v)[K], LbcSums& sums, int& set, int nb, int rank)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < K; k++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync (0xffffffffu, v[k], o);
    }
    if (nb == 1) {
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < K; k++) sums.v[set][k][warp] = v[k];
        }
        __syncthreads ();
    } else {
        cg::cluster_group cl = cg::this_cluster ();
        if (lane < nb) {
#pragma unroll
            for (int k = 0; k < K; k++) {
                *cl.map_shared_rank (&sums.v[set][k][rank * LBC_WARPS + warp],
                    lane) = v[k];
            }
        }
        cl.sync ();
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
        double s = 0.0;
        for (int i = lane; i < nb * LBC_WARPS; i += 32) s += sums.v[set][k][i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync (0xffffffffu, s, o);
        v[k] = s;
    }
    set ^= 1;
}

template <int E>
__device__ __forceinline__ void
lbc_load (double (&v)[E], const double* p, long long i0, long long step, long long n)
{
#pragma unroll
    for (int e = 0; e < E; e++) {
        const long long i = i0 + e * step;
        v[e] = i < n ? p[i] : 0.0;
    }
}

// The new-line-search branch: correction pair, the two-loop recursion,
// xp = x, gp = g, dginit = g.d and the search's start.  Blocks of the
// cluster take every nb-th run of LBC_THREADS entries.
template <int E>
__global__ void __launch_bounds__ (LBC_THREADS)
lb_search_cluster_kernel (LbDev* st, cudaGraphConditionalHandle h_while,
    double* S, double* Y, const double* x, double* xp, const double* g,
    double* gp, double* d, double* dsc, long long n)
{
    __shared__ LbcSums sums;
    __shared__ double s_ys[LBC_MAX_PAIRS], s_alpha[LBC_MAX_PAIRS];
    cg::cluster_group cl = cg::this_cluster ();
    const int nb = (int) gridDim.x, rank = (int) blockIdx.x;
    const int m = st->m, newest = st->newest, bound = st->bound, end = st->end;
    const bool first = st->first;
    const long long i0 = (long long) rank * LBC_THREADS + threadIdx.x;
    const long long step = (long long) nb * LBC_THREADS;
    int set = 0;
    for (int k = threadIdx.x; k < m; k += LBC_THREADS) s_ys[k] = dsc[k];
    // (the other blocks' shared memory is there, and s_ys)
    if (nb > 1) cl.sync ();
    else __syncthreads ();
    double dv[E];
    {
        double sv[E], yv[E];
        double yy = 0.0;
        {
            double gv[E];
            lbc_load<E> (gv, g, i0, step, n);
            lbc_load<E> (sv, x, i0, step, n);
            double sum[2] = {0.0, 0.0};
            double* sn = S + (size_t) newest * n;
            double* yn = Y + (size_t) newest * n;
#pragma unroll
            for (int e = 0; e < E; e++) {
                const long long i = i0 + e * step;
                dv[e] = -gv[e];
                if (i < n) {
                    const double xi = sv[e];
                    if (!first) {
                        sv[e] = xi - xp[i];
                        yv[e] = gv[e] - gp[i];
                        sn[i] = sv[e];
                        yn[i] = yv[e];
                    }
                    xp[i] = xi;
                    gp[i] = gv[e];
                }
                if (first || i >= n) {
                    sv[e] = 0.0;
                    yv[e] = 0.0;
                }
                sum[0] += yv[e] * sv[e];
                sum[1] += yv[e] * yv[e];
            }
            if (!first) {
                lbc_sum<2> (sum, sums, set, nb, rank);
                yy = sum[1];
                if (threadIdx.x == 0) s_ys[newest] = sum[0];
                if (threadIdx.x == 0 && rank == 0) {
                    dsc[newest] = sum[0];
                    dsc[2 * m + 1] = yy;
                }
                __syncthreads ();
            }
        }
        if (!first) {
            // the first loop starts at the newest pair, just formed
            int j = end;
            for (int k = 0; k < bound; k++) {
                j = (j + m - 1) % m;
                const int jn = (j + m - 1) % m;
                const bool more = k + 1 < bound;
                double a[1] = {0.0};
#pragma unroll
                for (int e = 0; e < E; e++) a[0] += sv[e] * dv[e];
                if (more) lbc_load<E> (sv, S + (size_t) jn * n, i0, step, n);
                lbc_sum<1> (a, sums, set, nb, rank);
                const double alpha = a[0] / s_ys[j];
                if (threadIdx.x == 0) s_alpha[j] = alpha;
#pragma unroll
                for (int e = 0; e < E; e++) dv[e] -= alpha * yv[e];
                if (more) lbc_load<E> (yv, Y + (size_t) jn * n, i0, step, n);
            }
            const double bv = s_ys[newest] / yy;
#pragma unroll
            for (int e = 0; e < E; e++) dv[e] *= bv;
            // the second one at the oldest, which the registers still hold
            for (int k = 0; k < bound; k++) {
                const int jn = (j + 1) % m;
                const bool more = k + 1 < bound;
                double b[1] = {0.0};
#pragma unroll
                for (int e = 0; e < E; e++) b[0] += yv[e] * dv[e];
                if (more) lbc_load<E> (yv, Y + (size_t) jn * n, i0, step, n);
                lbc_sum<1> (b, sums, set, nb, rank);
                const double av = s_alpha[j] - b[0] / s_ys[j];
#pragma unroll
                for (int e = 0; e < E; e++) dv[e] += av * sv[e];
                if (more) lbc_load<E> (sv, S + (size_t) jn * n, i0, step, n);
                j = jn;
            }
        }
    }
    double gd[1] = {0.0};
#pragma unroll
    for (int e = 0; e < E; e++) {
        const long long i = i0 + e * step;
        if (i < n) {
            d[i] = dv[e];
            gd[0] += g[i] * dv[e];
        }
    }
    lbc_sum<1> (gd, sums, set, nb, rank);
    if (rank == 0 && threadIdx.x == 0) {
        st->dginit = gd[0];
        begin_search (st, h_while);
    }
}

// After an evaluation: g = (double) grad, g.d, x.x and g.g, then the
// controller.
template <int E>
__global__ void __launch_bounds__ (LBC_THREADS)
lb_eval_cluster_kernel (LbDev* st, cudaGraphConditionalHandle h_while,
    cudaGraphConditionalHandle h_new, const float* __restrict__ grad,
    double* __restrict__ g, const double* __restrict__ d,
    const double* __restrict__ x, long long n)
{
    __shared__ LbcSums sums;
    cg::cluster_group cl = cg::this_cluster ();
    const int nb = (int) gridDim.x, rank = (int) blockIdx.x;
    const long long i0 = (long long) rank * LBC_THREADS + threadIdx.x;
    const long long step = (long long) nb * LBC_THREADS;
    int set = 0;
    if (nb > 1) cl.sync ();
    double sum[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int e = 0; e < E; e++) {
        const long long i = i0 + e * step;
        if (i < n) {
            const double gi = (double) grad[i], di = d[i], xi = x[i];
            g[i] = gi;
            sum[0] += gi * di;
            sum[1] += xi * xi;
            sum[2] += gi * gi;
        }
    }
    lbc_sum<3> (sum, sums, set, nb, rank);
    if (rank == 0 && threadIdx.x == 0) {
        st->dg = sum[0];
        st->xx = sum[1];
        st->gg = sum[2];
        after_eval (st, h_while, h_new);
    }
}

// Blocks of the cluster for n entries, E of them a thread.
template <int E>
int
lbc_blocks (long long n)
{
    int nb = 1;
    while ((long long) nb * LBC_THREADS * E < n) nb *= 2;
    return nb;
}

template <typename... P, typename... A>
cudaError_t
lbc_launch (void (*k) (P...), int nb, cudaStream_t st, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3 (nb);
    cfg.blockDim = dim3 (LBC_THREADS);
    cfg.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = nb;
    at.val.clusterDim.y = 1;
    at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx (&cfg, k, args...);
}

constexpr int LBC_FEW = 8, LBC_MANY = 16;              // entries a thread
static_assert (LB_CLUSTER_MAX == LBC_MAX_BLOCKS * LBC_THREADS * LBC_MANY, "");

}  // namespace

cudaError_t
launch_lb_search (LbDev* dst, cudaGraphConditionalHandle h_while, double* S,
    double* Y, const double* x, double* xp, const double* g, double* gp,
    double* d, double* dsc, long long n, cudaStream_t st)
{
    const int nb = lbc_blocks<LBC_FEW> (n);
    if (nb <= LBC_MAX_BLOCKS) {
        return lbc_launch (lb_search_cluster_kernel<LBC_FEW>, nb, st, dst,
            h_while, S, Y, x, xp, g, gp, d, dsc, n);
    }
    return lbc_launch (lb_search_cluster_kernel<LBC_MANY>,
        lbc_blocks<LBC_MANY> (n), st, dst, h_while, S, Y, x, xp, g, gp, d,
        dsc, n);
}

cudaError_t
launch_lb_eval (LbDev* dst, cudaGraphConditionalHandle h_while,
    cudaGraphConditionalHandle h_new, const float* grad, double* g,
    const double* d, const double* x, long long n, cudaStream_t st)
{
    const int nb = lbc_blocks<LBC_FEW> (n);
    if (nb <= LBC_MAX_BLOCKS) {
        return lbc_launch (lb_eval_cluster_kernel<LBC_FEW>, nb, st, dst,
            h_while, h_new, grad, g, d, x, n);
    }
    return lbc_launch (lb_eval_cluster_kernel<LBC_MANY>,
        lbc_blocks<LBC_MANY> (n), st, dst, h_while, h_new, grad, g, d, x, n);
}

__global__ void
lb_begin_search_kernel (LbDev* s, cudaGraphConditionalHandle h_while,
    const double* part, int nparts)
{
    if (blockIdx.x != 0 || threadIdx.x >= 32) return;
    const double dg0 = lb_warp_sum (part + (size_t) LP_DG0 * nparts, nparts);
    if (threadIdx.x != 0) return;
    s->dginit = dg0;
    begin_search (s, h_while);
}

__global__ void
lb_after_eval_kernel (LbDev* s, cudaGraphConditionalHandle h_while,
    cudaGraphConditionalHandle h_new, const double* part, int nparts)
{
    if (blockIdx.x != 0 || threadIdx.x >= 32) return;
    const double dg = lb_warp_sum (part + (size_t) LP_GD * nparts, nparts);
    const double xx = lb_warp_sum (part + (size_t) LP_XX * nparts, nparts);
    const double gg = lb_warp_sum (part + (size_t) LP_GG * nparts, nparts);
    if (threadIdx.x != 0) return;
    s->dg = dg;
    s->xx = xx;
    s->gg = gg;
    after_eval (s, h_while, h_new);
}

}  // namespace b200

// The graph-resident L-BFGS controller kernels (lbfgs_graph.cu).
#pragma once

#include <cuda_runtime.h>

#include "../../include/plastimatch_b200.h"
#include "lbfgs_logic.cuh"

namespace b200 {

// Start of a line search (after the correction pair, the two-loop
// recursion and gp.d): the search's state and its first trial step; ends
// the run (h_while) when the step or the direction is unusable.  dginit is
// the sum of slot LP_DG0 of part (nparts partials per slot).  Launched with
// one warp.
__global__ void lb_begin_search_kernel (LbDev* s,
    cudaGraphConditionalHandle h_while, const double* part, int nparts);

// After an evaluation: g.d, x.x and g.g from slots LP_GD, LP_XX and LP_GG
// of part, then the progress rule, the line search's tests, and either the
// next trial step, a new line search (h_new) or the end of the run
// (h_while).  Launched with one warp.
__global__ void lb_after_eval_kernel (LbDev* s,
    cudaGraphConditionalHandle h_while, cudaGraphConditionalHandle h_new,
    const double* part, int nparts);

// The new-line-search branch, and the work after an evaluation, as one
// launch each; for vectors of at most LB_CLUSTER_MAX entries.
constexpr long long LB_CLUSTER_MAX = 1 << 16;
cudaError_t launch_lb_search (LbDev* dst, cudaGraphConditionalHandle h_while,
    double* S, double* Y, const double* x, double* xp, const double* g,
    double* gp, double* d, double* dsc, long long n, cudaStream_t st);
cudaError_t launch_lb_eval (LbDev* dst, cudaGraphConditionalHandle h_while,
    cudaGraphConditionalHandle h_new, const float* grad, double* g,
    const double* d, const double* x, long long n, cudaStream_t st);

}  // namespace b200

// The line kernel (line.cu): plan, arguments and launch wrappers.
#pragma once

#include "kernels.cuh"

namespace b200 {

// A block is nw warps, each 32 voxels along x in one voxel plane (thread =
// one (x, z) column) of one tile row along z, planes fastest, marching along
// y through ty tiles.
struct LinePlan {
    int nw, gpr;         // warps a block, blocks per tile row along x and z
    int ty, nys;         // tiles a block along y, blocks along y
    int j;               // knot rows a block touches: ty + 3
    int kx;              // tiles a warp touches along x, at most
    int nxs;             // floats per adjoint row: whole tiles (the last
                         // one's voxels beyond the ROI stay zero)
    int nblocks;
    int threads;
    size_t smem;
};

bool line_plan (const BspGeom& g, LinePlan* p, int sm_count);
// Floats of the adjoint rows of a plan.
inline size_t
line_row_elems (const BspGeom& g, const LinePlan& p)
{
    return (size_t) g.roi_dim[2] * p.nys * p.j * 3 * p.nxs;
}

cudaError_t launch_mse_line (const BspGeom& g, const LinePlan& p,
    int grad_mode, const float* fimg, const float* mimg,
    const float4* mgrad4, const float* coeff, const float* luts, float* rows,
    double* score_part, int* count_part, cudaStream_t st);

// Contraction of the adjoint rows into the gradient, score and count over
// the nparts block parts (0: the result block stands, no normalisation), as
// launch_finish_mse otherwise.
cudaError_t launch_line_finish (const BspGeom& g, const LinePlan& p,
    const float* rows, const float* luts, const double* score_part,
    const int* count_part, int nparts, const int* err, DevResult* res,
    DevResult* res_host, float* grad, double* grad64, float* score_out,
    double* score64_out, long long* nvox_out, cudaStream_t st,
    const FinishCombine& cb = FinishCombine ());

} // namespace b200

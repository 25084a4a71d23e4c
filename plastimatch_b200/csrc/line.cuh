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
    int sms;             // of the device
    size_t smem;
    float wy[40];        // y basis table (vpr[1] * 4)
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
    const float* mgrad, const float* coeff, const float* luts, float* rows,
    double* score_part, int* count_part, cudaStream_t st);

// Mattes MI: pass 1 (PVI-8 or Parzen histograms into hist, integer 2^-24
// units, count last) or, for Parzen windows, pass 2 (adjoint rows).
struct LineMi {
    const uint8_t* fbin;
    const uint32_t* mquad;       // PVI-8: launch_bin_quad's image
    int bins;
    const float* lut;            // Parzen pass 2: [fixed bin][moving bin]
    const float* nvf;            //   [1]: 1 / (N delta_m)
    unsigned long long* hist;    // f[B], m[B], j[B*B], count
    bool parzen;
    const float* mimg;           // Parzen: the moving image
    float m_min, m_delta;        // Parzen: moving value -> window centre
};
cudaError_t launch_mi_line (const BspGeom& g, const LinePlan& p,
    bool hist_pass, const LineMi& mi, const float* coeff, const float* luts,
    float* rows, cudaStream_t st);
cudaError_t launch_bin_quad (const int dim[3], const uint8_t* bin,
    uint32_t* quad, cudaStream_t st);

// Dense field (vf) or warped moving image (warped; the other is NULL) over
// the ROI's voxels.
cudaError_t launch_field_line (const BspGeom& g, const LinePlan& p,
    const float* coeff, const float* luts, const float* mimg, float outside,
    float* vf, float* warped, cudaStream_t st);

// Contraction of the adjoint rows into the gradient, score and count over
// the nparts block parts (0: the result block stands, no normalisation), as
// launch_finish_mse otherwise.  behind: the kernel that writes the rows is
// the last work on the stream and nothing else has to be waited for, so that
// this one may be launched before that one has ended.
cudaError_t launch_line_finish (const BspGeom& g, const LinePlan& p,
    const float* rows, const float* luts, const double* score_part,
    const int* count_part, int nparts, const int* err, DevResult* res,
    DevResult* res_host, float* grad, double* grad64, float* score_out,
    double* score64_out, long long* nvox_out, cudaStream_t st,
    const FinishCombine& cb, bool behind);

} // namespace b200

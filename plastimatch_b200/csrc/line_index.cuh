// Arithmetic of the line kernel that the host shares.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define LINE_FN __host__ __device__ __forceinline__
#else
#define LINE_FN inline
#endif

namespace b200 {

// The float 2^23 + i holds the integer i in its low bits: a corner leaves
// line_load's clamp as the bits of such a float per axis, and the bias of all
// three is taken off at once, with the constant that line_corner0 gives.  The
// biased terms pass 2^32 for every image, so all of this is unsigned (modulo
// 2^32); the index itself is below 2^30 (line_plan).
constexpr unsigned LINE_BIAS = 0x4B000000u;

LINE_FN unsigned
line_corner0 (int nx, int ny)
{
    return 0u - LINE_BIAS * (1u + (unsigned) nx * (1u + (unsigned) ny));
}

LINE_FN unsigned
line_corner (const int bits[3], int nx, int ny, unsigned corner0)
{
    return (unsigned) bits[0] + (unsigned) nx * ((unsigned) bits[1]
        + (unsigned) ny * (unsigned) bits[2]) + corner0;
}

// How the rows' contraction is split into blocks: the whole row of knots along
// x where its voxels fit a block (two a thread), else even parts, kxc knots
// each; kzc knots along z, their planes split over `parts` thread rows.
//
// Knots along z and parts: of the splits whose blocks are all resident at once
// (512 threads of 128 registers an SM) the one with the shortest march, a
// block's own tile rows and the 3 beyond them times a latency and its planes.
// Against 2 to 8 knots and 1 to 4 parts by the number of blocks alone (some
// 300), the call took at 131x117x83 vpr 6 1.4 us less, at 200x180x90 vpr
// 7x7x4 with ROIs 3.2 (377 blocks of which 296 were resident), eight uneven
// images 9.  Where no split is resident (512x512x160, `waves`) the row of 8
// knots reads least: 343 us, 347 with 5, 356 with 2; two blocks an SM in 96
// registers, one in 128: 352.
constexpr int LINE_SPLIT_THREADS = 512;          // an SM's, and a block's at most

struct LineSplit {
    int nbx, kxc, kzc, threads, parts;
    bool waves;          // not all blocks are resident at once
};

inline LineSplit
line_finish_split (const int cdims[3], const int vpr[3], int sms)
{
    LineSplit f = {};
    const int most = (2 * LINE_SPLIT_THREADS - 2) / vpr[0] - 3;
    f.nbx = (cdims[0] + most - 1) / most;
    f.kxc = (cdims[0] + f.nbx - 1) / f.nbx;
    f.threads = (((f.kxc + 3) * vpr[0] + 2) / 2 + 31) / 32 * 32;
    double best = 0.0;
    for (int kzc = 1; kzc <= 8; kzc++) {
        const int n = f.nbx * cdims[1] * ((cdims[2] + kzc - 1) / kzc);
        for (int p = 1; p <= vpr[2] && p <= 8; p++) {
            if (p * f.threads > LINE_SPLIT_THREADS
                || n > sms * (LINE_SPLIT_THREADS / (p * f.threads))) break;
            const double cost = (kzc + 3) * (0.6 + 0.2 * ((vpr[2] + p - 1) / p));
            if (f.parts && cost >= best) continue;
            best = cost;
            f.parts = p;
            f.kzc = kzc;
        }
    }
    f.waves = f.parts == 0;
    if (f.waves) {
        f.kzc = 8;
        f.parts = 1;
    }
    return f;
}

// x / d, rounded correctly, with inv the rounded 1 / d: the quotient's exact
// remainder once more (Markstein's theorem, IBM J. Res. Dev. 34(1), 1990).
// d and inv are normal numbers.
LINE_FN float
line_quotient (float x, float d, float inv)
{
    const float q = x * inv;
    return fmaf (fmaf (-q, d, x), inv, q);
}

}  // namespace b200

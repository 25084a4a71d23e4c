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

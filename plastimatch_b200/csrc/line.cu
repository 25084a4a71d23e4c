// The line kernel: the B-spline field, the per-voxel step of a metric and the
// adjoint in one pass of FP32 arithmetic, separable along the three axes.
//
// A thread owns one (x, z) column of a block and marches along y, so
//   field    v(y) = sum_b By(y, b) p_b,  p_b = sum_a Bx(x, a) Cz(b, a),
//            Cz = the coefficients contracted along z, once per block, in
//            shared memory; the window p_0..p_3 lives in registers and takes
//            one new knot row per tile
//   adjoint  g_b += By(y, b) dc(y) in a register window; the knot row that
//            leaves it goes to memory as it is, one value per column and
//            component, and line_finish_kernel contracts those rows along
//            x and z into the gradient
// which leaves 12 multiply-adds per voxel for the field, 12 for the adjoint
// and a few for the other axes, where the 64-tap form takes 192 + 192.
// x runs along the lanes (image loads of a warp are contiguous up to the
// displacement), the y weights are the same for every thread.  Pairs of
// components go through the two-wide FP32 instructions.  The sums of a block
// run in an order of their own: results do not depend on how blocks are
// scheduled.
//
// Measured at 256x256x128, 5 voxels a region, nearest gradient: 66 us and 17
// us for the contraction (one after the other; 82 us a call), where the
// tcgen05 tile kernel takes 160 and 7 us (64x64x64, 8 voxels: 7 + 9, 14.4 us
// a call, against 22 + 5 us; 512x512x160, 10x10x4: 311 + 31, 340 us a call,
// against 800 + 40 us).  The tensor cores' field must be carried through
// shared memory to the x order and their adjoint operand split into bf16
// pairs, which costs more instructions than 24 two-wide multiply-adds.
// What bounds it: 147 instructions a voxel, some 60 of them address and clamp
// arithmetic, at half the issue slots, and the latency of the loads between
// them.  Without any load 47 us, with loads that all hit L1 58 us.
// Prefetching the next rows into L2 or L1, loading a voxel ahead, corners by
// texture gather (105 us) or the gradient from the moving image instead of
// memory (86 us) do not help.
#include <algorithm>
#include <cfloat>
#include <cstring>
#include <type_traits>

#include "bsp_common.cuh"
#include "line.cuh"
#include "line_index.cuh"

namespace b200 {

void basis_lut (float* lut, int vpr);               // runtime.cu

// What a block does at each voxel: MSE with the nearest or the trilinear
// moving gradient; Mattes MI pass 1 (PVI-8 or Parzen histograms) and, for
// Parzen windows, pass 2 (dc/dv from the factor table); the field itself;
// the warped moving image.
enum LineMode {
    LN_MSE_NEAREST, LN_MSE_LINEAR, LN_MI_HIST, LN_PZ_HIST, LN_PZ_GRAD,
    LN_FIELD, LN_WARP
};

constexpr bool
ln_mse (int mode)
{
    return mode == LN_MSE_NEAREST || mode == LN_MSE_LINEAR;
}

constexpr bool
ln_hist (int mode)
{
    return mode == LN_MI_HIST || mode == LN_PZ_HIST;
}

constexpr bool
ln_adjoint (int mode)
{
    return ln_mse (mode) || mode == LN_PZ_GRAD;
}

// dynamic shared memory that needs no attribute beside the static arrays
constexpr size_t LN_PLAIN_SMEM = 40 * 1024;
constexpr int LN_MAX_VPR = 10;           // voxels a region (line_plan)
constexpr int LN_REGS = 64;             // four blocks of eight warps per SM
constexpr int LN_WARPS = 8;             // warps a block (see line_plan)
constexpr double LN_EDGE = 2.5;         // a block's start and end, in voxel rows along y

typedef unsigned long long u64;

struct LineArgs {
    BspGeom g;
    const float* fimg;
    const float* mimg;
    const float* mgrad;  // xyz interleaved
    const float* coeff;
    const float* luts;
    float* rows;         // adjoint rows [z][y block][j][c][nxs]
    double* score_part;
    int* count_part;
    const uint8_t* fbin; // MI: fixed bin per voxel
    const uint32_t* mquad;                  // PVI-8: bins of 2 x 2 moving voxels
    const float* lut;    // Parzen pass 2: [fixed bin][moving bin] factors
    const float* nvf;    //   [1]: 1 / (N delta_m)
    u64* hist;           // pass 1: f[B], m[B], j[B * B], count
    int bins;
    float pz_min, pz_delta, pz_inv;         // moving value -> window centre
    float* out;          // field (xyz per voxel) or warped image
    float outside;
    bool roi_same;       // the moving ROI is a mask on the moving image's grid
    int ty, j, nxs;
    // y weights of each row of a tile, each twice; in the parameter bank,
    // since they are the same for every thread: shared memory would return
    // them to all 32 lanes (four cycles a 16-byte load: 44 instead of 31 L1
    // cycles a voxel, and 8 registers that then spill: 75 against 70 us)
    u64 wy[LN_MAX_VPR][4];
    u64 step_y;          // AXIS: (0, fixed y step)
    u64 morg, mprj;      // AXIS: moving x and y origin and projection
    int mtop[3];         // bits of 2^23 + (dim - 2): the largest corner
    unsigned midx0;      // line_corner0 of the moving image
    unsigned mzero;      // mgrad's triple of zeros, behind the last voxel's
};

__device__ __forceinline__ u64
pk (float lo, float hi)
{
    u64 r;
    asm ("mov.b64 %0, {%1, %2};" : "=l" (r) : "f" (lo), "f" (hi));
    return r;
}

__device__ __forceinline__ float
lo2 (u64 v)
{
    return __uint_as_float ((unsigned) v);
}

__device__ __forceinline__ float
hi2 (u64 v)
{
    return __uint_as_float ((unsigned) (v >> 32));
}

__device__ __forceinline__ u64
fma2 (u64 a, u64 b, u64 c)
{
    u64 r;
    asm ("fma.rn.f32x2 %0, %1, %2, %3;" : "=l" (r) : "l" (a), "l" (b), "l" (c));
    return r;
}

__device__ __forceinline__ u64
mul2 (u64 a, u64 b)
{
    u64 r;
    asm ("mul.rn.f32x2 %0, %1, %2;" : "=l" (r) : "l" (a), "l" (b));
    return r;
}

__device__ __forceinline__ u64
add2 (u64 a, u64 b)
{
    u64 r;
    asm ("add.rn.f32x2 %0, %1, %2;" : "=l" (r) : "l" (a), "l" (b));
    return r;
}

__device__ __forceinline__ u64
sub2 (u64 a, u64 b)
{
    u64 r;
    asm ("sub.rn.f32x2 %0, %1, %2;" : "=l" (r) : "l" (a), "l" (b));
    return r;
}

// A knot row of the field or of the adjoint: x and y components paired.
struct Row {
    u64 xy;
    float z;
};

// Shared memory of a block, in bytes from its start.
struct LineSmem {
    int bx, bz, cz, total;
};

// cz: planes x knots of a block's footprint (line_foot), times its rows.
__host__ __device__ inline LineSmem
line_smem (int vx, int vz, int j, int foot)
{
    LineSmem m;
    m.bx = 0;
    m.bz = m.bx + 32 * vx;
    m.cz = m.bz + 16 * vz;
    m.total = m.cz + 16 * j * foot;
    return m;
}

// Everything a thread keeps while it marches.
template <bool AXIS>
struct Col {
    u64 pos_xy;          // AXIS: world x, y origin
    float pos0[3];       // AXIS: -, -, world z; else origin + i * step
    float kf;            // z index
    int frow;            // fixed-image index of (x, y = 0, z)
    bool live;           // a voxel column of the ROI
};

// One voxel between its loads and its metric.
struct Vox {
    float cr[8], fv;
    float gr[3];
    float w2[3];
    uint32_t mq[2];
    int fb, fidx, clamp;
    int roi;             // moving ROI's mask at the position
    bool ok;
};

// Loads that stay where they are written: all of a voxel's go out before
// anything waits for one.
__device__ __forceinline__ float
ld1 (const float* p)
{
    float v;
    asm volatile ("ld.global.nc.f32 %0, [%1];" : "=f" (v) : "l" (p));
    return v;
}

// The voxel at fixed row fj (row ly of its tile): field, correspondence, loads.
// R: the window's first slot.
template <int MODE, bool AXIS, bool ROI, int R>
__device__ __forceinline__ void
line_load (const LineArgs& a, const Col<AXIS>& col, int fj, u64& jf2,
    int ly, const Row (&p)[4], Vox& v)
{
    const BspGeom& g = a.g;
    const u64* w = a.wy[ly];
    u64 dxy = mul2 (w[0], p[R].xy);
    dxy = fma2 (w[1], p[(R + 1) & 3].xy, dxy);
    dxy = fma2 (w[2], p[(R + 2) & 3].xy, dxy);
    dxy = fma2 (w[3], p[(R + 3) & 3].xy, dxy);
    float dz = lo2 (w[0]) * p[R].z;
    dz = fmaf (lo2 (w[1]), p[(R + 1) & 3].z, dz);
    dz = fmaf (lo2 (w[2]), p[(R + 2) & 3].z, dz);
    dz = fmaf (lo2 (w[3]), p[(R + 3) & 3].z, dz);
    const float jf = lo2 (jf2);
    float fx[3];
    float ma[3];
    if (AXIS) {
        // origin + step * index and the projection with the zero
        // off-diagonal terms dropped (they add exact zeros)
        const u64 f = fma2 (jf2, a.step_y, col.pos_xy);
        fx[0] = lo2 (f);
        fx[1] = hi2 (f);
        fx[2] = col.pos0[2];
        const u64 t = mul2 (sub2 (add2 (f, dxy), a.morg), a.mprj);
        ma[0] = lo2 (t);
        ma[1] = hi2 (t);
        ma[2] = ((fx[2] + dz) - g.morigin[2]) * g.mproj[8];
    } else {
#pragma unroll
        for (int d = 0; d < 3; d++) {
            fx[d] = fmaf (col.kf, g.fstep[3 * d + 2],
                fmaf (jf, g.fstep[3 * d + 1], col.pos0[d]));
        }
        const float t0 = (fx[0] + lo2 (dxy)) - g.morigin[0];
        const float t1 = (fx[1] + hi2 (dxy)) - g.morigin[1];
        const float t2 = (fx[2] + dz) - g.morigin[2];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            ma[d] = t0 * g.mproj[3 * d] + t1 * g.mproj[3 * d + 1]
                + t2 * g.mproj[3 * d + 2];
        }
    }
    jf2 = add2 (jf2, pk (1.f, 1.f));
    bool in = col.live;
    int bits[3], rbits[3];
    v.clamp = 0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        in = in && ma[d] > -0.5f && ma[d] < g.m_hi[d];
        // li_clamp without conversions (see locate_nx): floor in the low
        // mantissa bits of max(ma, 0) + 2^23 rounded down, corner at
        // most dim - 2, fraction saturated to [0, 1]
        bits[d] = __float_as_int (__fadd_rd (fmaxf (ma[d], 0.f), 8388608.f));
        if (ROI) rbits[d] = min (bits[d], a.mtop[d] + 1);
        bits[d] = min (bits[d], a.mtop[d]);
        v.w2[d] = __saturatef (ma[d] - (__int_as_float (bits[d]) - 8388608.f));
        if (MODE == LN_PZ_GRAD && (ma[d] < 0.f || ma[d] >= g.m_fmax[d] + 1.f)) {
            v.clamp |= 1 << d;
        }
    }
    const unsigned mvf = line_corner (bits, g.mdim[0], g.mdim[1], a.midx0);
    const int fidx = col.frow + fj * g.fdim[0];
    v.fidx = fidx;
    if (MODE == LN_FIELD) {
        v.cr[0] = lo2 (dxy);
        v.cr[1] = hi2 (dxy);
        v.cr[2] = dz;
        return;
    }
    v.ok = in;
    if (ROI) {
        // the moving mask's byte goes out with the other loads; where the
        // mask lies on the moving image's own grid its index is the clamped
        // floor of the position (the same operations as inside_roi)
        if (AXIS && a.roi_same) {
            v.roi = __ldg (g.mroi + line_corner (rbits, g.mdim[0], g.mdim[1],
                a.midx0));
        } else {
            const float dd[3] = {lo2 (dxy), hi2 (dxy), dz};
            v.roi = roi_moving_ok (g, fx, dd);
        }
    }
    const int dx = g.mdim[0], dxym = g.mdim[0] * g.mdim[1];
    const unsigned off = mvf * 4u;
    const char* b0 = (const char*) a.mimg;
    const char* b1 = (const char*) (a.mimg + dx);
    const char* b2 = (const char*) (a.mimg + dxym);
    const char* b3 = (const char*) (a.mimg + dxym + dx);
    if (MODE == LN_MSE_NEAREST) {
        unsigned mvr = mvf + (v.w2[0] >= 0.5f ? 1 : 0)
            + (v.w2[1] >= 0.5f ? dx : 0) + (v.w2[2] >= 0.5f ? dxym : 0);
        if (!ROI) mvr = in ? mvr : a.mzero;
        const float* gp = a.mgrad + 3 * (size_t) mvr;
        v.gr[0] = ld1 (gp);
        v.gr[1] = ld1 (gp + 1);
        v.gr[2] = ld1 (gp + 2);
    }
    if (ln_mse (MODE)) v.fv = ld1 (a.fimg + fidx);
    if (ln_hist (MODE) || MODE == LN_PZ_GRAD) v.fb = __ldg (a.fbin + fidx);
    if (MODE == LN_MI_HIST) {
        v.mq[0] = __ldg (a.mquad + mvf);
        v.mq[1] = __ldg (a.mquad + mvf + dxym);
        return;
    }
    v.cr[0] = ld1 ((const float*) (b0 + off));
    v.cr[1] = ld1 ((const float*) (b0 + off) + 1);
    v.cr[2] = ld1 ((const float*) (b1 + off));
    v.cr[3] = ld1 ((const float*) (b1 + off) + 1);
    v.cr[4] = ld1 ((const float*) (b2 + off));
    v.cr[5] = ld1 ((const float*) (b2 + off) + 1);
    v.cr[6] = ld1 ((const float*) (b3 + off));
    v.cr[7] = ld1 ((const float*) (b3 + off) + 1);
}

// Trilinear value (x, then y, then z; the z planes' lerps in pairs, with the
// rounding of trilinear_lerp).
__device__ __forceinline__ float
line_value (const Vox& v)
{
    const u64 wx2 = pk (v.w2[0], v.w2[0]), wy2 = pk (v.w2[1], v.w2[1]);
    const u64 m0 = pk (v.cr[0], v.cr[4]), m1 = pk (v.cr[1], v.cr[5]);
    const u64 m2 = pk (v.cr[2], v.cr[6]), m3 = pk (v.cr[3], v.cr[7]);
    const u64 c0 = fma2 (wx2, sub2 (m1, m0), m0);
    const u64 c1 = fma2 (wx2, sub2 (m3, m2), m2);
    const u64 cc = fma2 (wy2, sub2 (c1, c0), c0);
    return fmaf (v.w2[2], hi2 (cc) - lo2 (cc), lo2 (cc));
}

// dc/dv of one voxel (y weights w) into the window of adjoint rows.
template <int R>
__device__ __forceinline__ void
line_adjoint (const u64* w, u64 cxy, float cz, Row (&q)[4])
{
#pragma unroll
    for (int b = 0; b < 4; b++) {
        Row& o = q[(R + b) & 3];
        o.xy = fma2 (w[b], cxy, o.xy);
        o.z = fmaf (lo2 (w[b]), cz, o.z);
    }
}

// MSE at a loaded voxel and its adjoint.
//
// A voxel outside has read the moving image's border, which may hold
// infinities or NaN, so that a derivative times 0 is not enough: its gradient
// is the triple of zeros (line_load; one select), or its derivative is
// selected (three: 83.9 us a call against 82.1 at 256x256x128 vpr 5, 30.7
// against 26.6 at 131x117x83 vpr 6 oblique, with spills).
template <int MODE, bool ROI, int R>
__device__ __forceinline__ void
line_use (const LineArgs& a, int ly, const Vox& v,
    Row (&q)[4], float& scf, int& cnt)
{
    float diff = line_value (v) - v.fv;
    diff = v.ok ? diff : 0.f;
    scf = fmaf (diff, diff, scf);
    cnt += v.ok ? 1 : 0;
    u64 cxy;
    float cz;
    if (MODE == LN_MSE_NEAREST) {
        cxy = mul2 (pk (diff, diff), pk (v.gr[0], v.gr[1]));
        cz = diff * v.gr[2];
    } else {
        float gd[3];
        trilinear_lerp_grad (a.g, v.w2, v.cr, gd);
        cxy = mul2 (pk (diff, diff), pk (gd[0], gd[1]));
        cz = diff * gd[2];
    }
    if (ROI || MODE == LN_MSE_LINEAR) {
        cxy = v.ok ? cxy : 0ull;
        cz = v.ok ? cz : 0.f;
    }
    line_adjoint<R> (a.wy[ly], cxy, cz, q);
}

// The Parzen window's centre at a loaded voxel (parzen_centre's value).
__device__ __forceinline__ float
line_pz_centre (const LineArgs& a, const Vox& v)
{
    return line_quotient (line_value (v) - a.pz_min, a.pz_delta, a.pz_inv) + 2.f;
}

// Parzen pass 2 at a loaded voxel: 1/(N delta_m) * sum over the window's
// bins of beta3'(k - u) log(p(f, k) / p_m(k)) (slut, shared memory), times
// the world gradient of the trilinear interpolant (proj^T times the index
// gradient; 0 along an axis the clamp holds).  With f = u - floor(u) the
// window's derivative at its four bins is (1-f)^2/2, 2f - 3f^2/2,
// -2s + 3s^2/2 (s = 1-f) and -f^2/2.
template <bool AXIS, int R>
__device__ __forceinline__ void
line_use_pz (const LineArgs& a, int ly, const Vox& v, const float* slut, float scale, Row (&q)[4])
{
    const float u = line_pz_centre (a, v);
    const int k0 = parzen_first_bin (u, a.bins);
    const float f = u - (float) (k0 + 1), s = 1.f - f;
    const float* row = slut + v.fb * a.bins + k0;
    const float sum = (0.5f * s * s) * row[0] + (f * fmaf (-1.5f, f, 2.f)) * row[1]
        + (s * fmaf (1.5f, s, -2.f)) * row[2] - (0.5f * f * f) * row[3];
    float gi[3];
    trilinear_igrad (v.w2, v.cr, v.clamp, gi);
    const float sc = scale * sum;
    const float* p = a.g.mproj;
    float dc[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
        dc[c] = AXIS ? sc * (p[4 * c] * gi[c])
                     : sc * (p[c] * gi[0] + p[3 + c] * gi[1] + p[6 + c] * gi[2]);
        dc[c] = v.ok ? dc[c] : 0.f;         // (as in line_use)
    }
    line_adjoint<R> (a.wy[ly], pk (dc[0], dc[1]), dc[2], q);
}

// Histograms of a block: weights are summed as integers in 2^-24 units (no
// float atomics, any order).  A thread keeps the sums of the bin (pair) its
// last voxels fell into and adds them to shared memory only when the next
// voxel falls into another, the low 13 bits and the rest in 32-bit counters:
// shared 32-bit adds are native.  A block has fewer than 65536 voxels
// (line_plan) and a voxel adds at most seven weights to a bin, so the low
// counter stays below 7 * 65535 * 2^13 < 2^32; all weights of a block's
// voxels together are below 65536 * (2^24 + 8).  (As 16-bit halves, which a
// voxel's further bins overflow, those have to go to the histogram in memory:
// PVI-8 at 256x256x128 vpr 5, 32 bins, noise of 20 in 800 grey levels 6740 us
// a call, 346 with all of them here; on the tile kernel 1031.)
constexpr int LN_HIST_LOW = 13;

struct Run {
    int key;             // joint bin (Parzen: the first of four); -1: none
    uint32_t s[4];       // weights (PVI-8: [0] the weight, [1] the voxels)
};

__device__ __forceinline__ void
hist_add (uint32_t* sh, int nj, int bin, uint32_t w)
{
    atomicAdd (sh + bin, w & ((1u << LN_HIST_LOW) - 1u));
    atomicAdd (sh + nj + bin, w >> LN_HIST_LOW);
}

template <int MODE>
__device__ __forceinline__ void
hist_flush (uint32_t* sh, int B, const Run& r)
{
    const int nj = B * B;
    if (MODE == LN_PZ_HIST) {
#pragma unroll
        for (int j = 0; j < 4; j++) hist_add (sh, nj, r.key + j, r.s[j]);
    } else {
        hist_add (sh, nj, r.key, r.s[0]);
        atomicAdd (sh + 2 * nj + r.key / B, r.s[1]);
    }
}

// Parzen pass 1 at a loaded voxel: the cubic window's four weights at the
// moving value into the fixed bin's row.
__device__ __forceinline__ void
line_use_pz_hist (const LineArgs& a, const Vox& v, uint32_t* sh, Run& r)
{
    if (!v.ok) return;
    const float u = line_pz_centre (a, v);
    const int k0 = parzen_first_bin (u, a.bins);
    const float f = u - (float) (k0 + 1), s = 1.f - f;
    const float f2 = f * f, s2 = s * s;
    const float w0 = s2 * s * (1.f / 6.f), w3 = f2 * f * (1.f / 6.f);
    const float w1 = fmaf (f2, fmaf (0.5f, f, -1.f), 2.f / 3.f);
    const float w2 = fmaf (s2, fmaf (0.5f, s, -1.f), 2.f / 3.f);
    const uint32_t q[4] = {__float2uint_rn (w0 * 16777216.f),
        __float2uint_rn (w1 * 16777216.f), __float2uint_rn (w2 * 16777216.f),
        __float2uint_rn (w3 * 16777216.f)};
    const int key = v.fb * a.bins + k0;
    if (key != r.key) {
        if (r.key >= 0) hist_flush<LN_PZ_HIST> (sh, a.bins, r);
        r.key = key;
#pragma unroll
        for (int j = 0; j < 4; j++) r.s[j] = q[j];
    } else {
#pragma unroll
        for (int j = 0; j < 4; j++) r.s[j] += q[j];
    }
}

// PVI-8 pass 1 at a loaded voxel: the eight corner weights into the joint
// bins of (fixed bin, corner's bin).  The first corner's bin takes part in
// the thread's run, with the voxel's count; corners in other bins (edges of
// structures) go straight to shared memory, those of the first such bin
// together.  Where all eight share one bin their weights add up to one.
__device__ __forceinline__ void
line_use_mi_hist (const LineArgs& a, const Vox& v, uint32_t* sh, Run& r)
{
    if (!v.ok) return;
    const int B = a.bins, nj = B * B;
    const int m0 = v.mq[0] & 255;
    const int key = v.fb * B + m0;
    uint32_t q1 = 16777216u;
    const uint32_t same = (uint32_t) m0 * 0x01010101u;
    if (v.mq[0] != same || v.mq[1] != same) {
        const float* l2 = v.w2;
        const float l1[3] = {1.f - l2[0], 1.f - l2[1], 1.f - l2[2]};
        const float w[8] = {l1[0] * l1[1] * l1[2], l2[0] * l1[1] * l1[2],
            l1[0] * l2[1] * l1[2], l2[0] * l2[1] * l1[2],
            l1[0] * l1[1] * l2[2], l2[0] * l1[1] * l2[2],
            l1[0] * l2[1] * l2[2], l2[0] * l2[1] * l2[2]};
        q1 = __float2uint_rn (w[0] * 16777216.f);
        uint32_t q2 = 0;
        int m2 = -1;
#pragma unroll
        for (int k = 1; k < 8; k++) {
            const int mk = (v.mq[k >> 2] >> (8 * (k & 3))) & 255;
            const uint32_t q = __float2uint_rn (w[k] * 16777216.f);
            if (mk == m0) {
                q1 += q;
            } else if (m2 < 0 || mk == m2) {
                m2 = mk;
                q2 += q;
            } else {
                hist_add (sh, nj, v.fb * B + mk, q);     // a third bin
            }
        }
        if (m2 >= 0) hist_add (sh, nj, v.fb * B + m2, q2);
    }
    if (key != r.key) {
        if (r.key >= 0) hist_flush<LN_MI_HIST> (sh, B, r);
        r.key = key;
        r.s[0] = q1;
        r.s[1] = 1;
    } else {
        r.s[0] += q1;
        r.s[1] += 1;
    }
}

// The warped value with the reference's weight products and sum order
// (LI_VALUE, src/base/interpolate_macros.h:23-38): products ((w_x w_y) w_z) m,
// added corner by corner.
__device__ __forceinline__ float
line_li_value (const Vox& v)
{
    const float* b = v.w2;
    const float a[3] = {1.f - b[0], 1.f - b[1], 1.f - b[2]};
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const float t = __fmul_rn (__fmul_rn (__fmul_rn (k & 1 ? b[0] : a[0],
            k & 2 ? b[1] : a[1]), k & 4 ? b[2] : a[2]), v.cr[k]);
        s = k == 0 ? t : __fadd_rn (s, t);
    }
    return s;
}

template <int MODE, bool AXIS, bool ROI>
__global__ void __maxnreg__ (LN_REGS)
line_kernel (const __grid_constant__ LineArgs a)
{
    extern __shared__ __align__ (16) uint8_t sm[];
    __shared__ double sh_v[LN_WARPS];
    __shared__ int sh_n[LN_WARPS];
    // each thread's own sums
    __shared__ double t_v[ln_mse (MODE) ? 32 * LN_WARPS : 1];
    __shared__ int t_n[ln_mse (MODE) ? 32 * LN_WARPS : 1];
    // (the contraction's blocks may start as this grid's last ones end)
    if (ln_adjoint (MODE)) asm volatile ("griddepcontrol.launch_dependents;");
    if (ln_mse (MODE)) {
        t_v[threadIdx.x] = 0.0;
        t_n[threadIdx.x] = 0;
    }
    const BspGeom& g = a.g;
    const int vx = g.vpr[0], vy = g.vpr[1], vz = g.vpr[2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int W = blockDim.x >> 5;
    const LineSmem m = line_smem (vx, vz, 0, 0);

    // the block: W warp columns (32 voxels along x in one plane) of tile
    // row tz, planes fastest, tiles ty0 .. along y
    const int tz = blockIdx.z;
    const int nz = min (vz, g.roi_dim[2] - tz * vz);
    const int nxw = (g.roi_dim[0] + 31) >> 5;
    const int wc = blockIdx.x * W + warp;
    const int xw0 = blockIdx.x * W / nz;
    const int xw1 = min (blockIdx.x * W + W - 1, nxw * nz - 1) / nz;
    const int x0 = 32 * xw0;
    const int ty0 = blockIdx.y * a.ty;
    const int nt = min (a.ty, g.rdims[1] - ty0);
    const int t0 = x0 / vx;
    const int nkx = xw1 < xw0 ? 0
        : (min (32 * xw1 + 32, g.roi_dim[0]) - 1) / vx - t0 + 4;
    const int nj = nt + 3;

    u64* sbx = (u64*) (sm + m.bx);
    float* sbz = (float*) (sm + m.bz);
    ulonglong2* cz = (ulonglong2*) (sm + m.cz);
    // after the coefficients: the histograms (low and high halves of the
    // joint one, fixed counts) or the factor table
    uint32_t* shist = (uint32_t*) (cz + nz * nj * nkx);
    float* slut = (float*) shist;
    const int nh = 2 * a.bins * a.bins + a.bins;
    if (ln_hist (MODE)) {
        for (int o = threadIdx.x; o < nh; o += blockDim.x) shist[o] = 0u;
    }
    if (MODE == LN_PZ_GRAD) {
        for (int o = threadIdx.x; o < a.bins * a.bins; o += blockDim.x) slut[o] = a.lut[o];
    }
    const float scale = MODE == LN_PZ_GRAD ? a.nvf[1] : 0.f;
    // the block's coefficients contracted along z, for each of its planes;
    // their loads go out before the weights are waited for (256x256x128
    // vpr 5: 82.3 us a call, 83.3 after them)
    const int plane = 3 * g.cdims[0] * g.cdims[1];
    float ck[4][3];
    auto fetch = [&] (int o) {
        const int jj = o / nkx, i = o - jj * nkx;
        const float* c = a.coeff + 3 * ((size_t) (tz * g.cdims[1] + ty0 + jj)
            * g.cdims[0] + t0 + i);
#pragma unroll
        for (int k = 0; k < 4; k++) {
#pragma unroll
            for (int d = 0; d < 3; d++) ck[k][d] = __ldg (c + (size_t) k * plane + d);
        }
    };
    int oc = threadIdx.x;
    if (oc < nj * nkx) fetch (oc);
    for (int o = threadIdx.x; o < 4 * vx; o += blockDim.x) {
        const float w = a.luts[o];
        sbx[o] = pk (w, w);
    }
    for (int o = threadIdx.x; o < 4 * vz; o += blockDim.x) {
        sbz[o] = a.luts[4 * (vx + vy) + o];
    }
    __syncthreads ();
    while (oc < nj * nkx) {
        for (int z = 0; z < nz; z++) {
            const float4 w = *(const float4*) (sbz + 4 * z);
            float v[3];
#pragma unroll
            for (int d = 0; d < 3; d++) {
                v[d] = fmaf (w.w, ck[3][d], fmaf (w.z, ck[2][d],
                    fmaf (w.y, ck[1][d], w.x * ck[0][d])));
            }
            cz[z * nj * nkx + oc] = make_ulonglong2 (pk (v[0], v[1]),
                pk (v[2], 0.f));
        }
        oc += blockDim.x;
        if (oc < nj * nkx) fetch (oc);
    }

    // the thread's column (a lane beyond the ROI stays on valid addresses)
    const bool wlive = wc < nxw * nz;
    const int xw = wlive ? wc / nz : xw0;
    const int zl = wlive ? wc - xw * nz : 0;
    const int xr = min (32 * xw + lane, g.roi_dim[0] - 1);
    const int zr = tz * vz + zl;
    const int kxl = xr / vx - t0;
    const int fi = g.roi_off[0] + xr, fk = g.roi_off[2] + zr;
    Col<AXIS> col;
    col.live = 32 * xw + lane < g.roi_dim[0];
    col.frow = fi + g.fdim[0] * g.fdim[1] * fk;
    col.kf = i2f_small (fk);
    if (AXIS) {
        col.pos_xy = pk (fmaf (i2f_small (fi), g.fstep[0], g.img_origin[0]),
            g.img_origin[1]);
        col.pos0[2] = fmaf (col.kf, g.fstep[8], g.img_origin[2]);
    } else {
#pragma unroll
        for (int d = 0; d < 3; d++) {
            col.pos0[d] = fmaf (i2f_small (fi), g.fstep[3 * d], g.img_origin[d]);
        }
    }
    __syncthreads ();

    const ulonglong2* crow = cz + zl * nj * nkx + kxl;
    const ulonglong2* bxp = (const ulonglong2*) (sbx + 4 * (xr - (xr / vx) * vx));
    Row p[4], q[4];
    // knot row jj of the block's window at the column's x
    auto load_row = [&] (Row& o, int jj) {
        const ulonglong2* c = crow + jj * nkx;
        const ulonglong2 w01 = bxp[0], w23 = bxp[1];
        const ulonglong2 c0 = c[0], c1 = c[1], c2 = c[2], c3 = c[3];
        o.xy = fma2 (w23.y, c3.x, fma2 (w23.x, c2.x, fma2 (w01.y, c1.x,
            mul2 (w01.x, c0.x))));
        o.z = fmaf (lo2 (w23.y), lo2 (c3.y), fmaf (lo2 (w23.x), lo2 (c2.y),
            fmaf (lo2 (w01.y), lo2 (c1.y), lo2 (w01.x) * lo2 (c0.y))));
    };
    // adjoint row r leaves the window
    float* out = !ln_adjoint (MODE) ? nullptr
        : a.rows + ((size_t) zr * gridDim.y + blockIdx.y) * a.j * 3 * a.nxs
        + 32 * xw + lane;
    auto retire = [&] (Row& o) {
        if (col.live) {
            out[0] = lo2 (o.xy);
            out[a.nxs] = hi2 (o.xy);
            out[2 * a.nxs] = o.z;
        }
        out += 3 * a.nxs;
        o.xy = 0ull;
        o.z = 0.f;
    };
#pragma unroll
    for (int b = 0; b < 4; b++) {
        q[b].xy = 0ull;
        q[b].z = 0.f;
    }
    // the fixed row index as a float, twice
    u64 jf2 = pk (i2f_small (g.roi_off[1] + ty0 * vy),
        i2f_small (g.roi_off[1] + ty0 * vy));
    Run run;
    run.key = -1;
    int nvox = 0;
    auto tile = [&] (auto rc, int t) {
        constexpr int R = decltype (rc)::value;
        load_row (p[(R + 3) & 3], t + 3);
        const int y0 = (ty0 + t) * vy;
        const int ny = min (vy, g.roi_dim[1] - y0);
        float scf = 0.f;
        int cnt = 0;
        // the column's fixed mask over the tile, a bit a row; rows that no
        // lane of the warp has inside are skipped
        unsigned inside = ~0u, any = ~0u;
        if (ROI && g.fmask) {
            inside = 0u;
            const uint8_t* fm = g.fmask + col.frow + (g.roi_off[1] + y0) * g.fdim[0];
#pragma unroll 5
            for (int ly = 0; ly < ny; ly++) {
                inside |= (unsigned) (__ldg (fm + ly * g.fdim[0]) & 1) << ly;
            }
            any = __reduce_or_sync (0xffffffffu, inside);
        }
        for (int ly = 0; ly < ny; ly++) {
            Vox v;
            if (ROI) {
                if (!(any >> ly & 1u)) continue;
                const float f = i2f_small (g.roi_off[1] + y0 + ly);
                jf2 = pk (f, f);
            }
            line_load<MODE, AXIS, ROI, R> (a, col, g.roi_off[1] + y0 + ly,
                jf2, ly, p, v);
            if (ROI) v.ok = v.ok && v.roi && (inside >> ly & 1u);
            if constexpr (ln_mse (MODE)) {
                line_use<MODE, ROI, R> (a, ly, v, q, scf, cnt);
            } else if constexpr (MODE == LN_PZ_GRAD) {
                line_use_pz<AXIS, R> (a, ly, v, slut, scale, q);
            } else if constexpr (ln_hist (MODE)) {
                if (MODE == LN_PZ_HIST) line_use_pz_hist (a, v, shist, run);
                else line_use_mi_hist (a, v, shist, run);
                nvox += v.ok ? 1 : 0;
            } else if (col.live) {
                if (MODE == LN_WARP) {
                    a.out[v.fidx] = v.ok ? line_li_value (v) : a.outside;
                } else {
                    float* o = a.out + 3 * (size_t) v.fidx;
                    o[0] = v.cr[0];
                    o[1] = v.cr[1];
                    o[2] = v.cr[2];
                }
            }
        }
        if (ln_mse (MODE)) {
            t_v[threadIdx.x] += (double) scf;
            t_n[threadIdx.x] += cnt;
        }
        if (ln_adjoint (MODE)) retire (q[R]);
    };
    if (wlive) {
        load_row (p[0], 0);
        load_row (p[1], 1);
        load_row (p[2], 2);
        for (int t = 0; t < nt; t++) {
            switch (t & 3) {
            case 0: tile (std::integral_constant<int, 0> (), t); break;
            case 1: tile (std::integral_constant<int, 1> (), t); break;
            case 2: tile (std::integral_constant<int, 2> (), t); break;
            default: tile (std::integral_constant<int, 3> (), t); break;
            }
        }
        // the three rows that are left in the window
        if (ln_adjoint (MODE)) {
            switch (nt & 3) {
            case 0: retire (q[0]); retire (q[1]); retire (q[2]); break;
            case 1: retire (q[1]); retire (q[2]); retire (q[3]); break;
            case 2: retire (q[2]); retire (q[3]); retire (q[0]); break;
            default: retire (q[3]); retire (q[0]); retire (q[1]); break;
            }
        }
    }
    if constexpr (ln_hist (MODE)) {
        const int B = a.bins;
        if (run.key >= 0) hist_flush<MODE> (shist, B, run);
        nvox = __reduce_add_sync (0xffffffffu, nvox);
        if (lane == 0 && nvox) atomicAdd (a.hist + 2 * B + B * B, (u64) nvox);
        __syncthreads ();
        for (int o = threadIdx.x; o < B * B; o += blockDim.x) {
            const u64 w = (u64) shist[o] + ((u64) shist[B * B + o] << LN_HIST_LOW);
            if (w) {
                atomicAdd (a.hist + 2 * B + o, w);
                // the moving histogram: the joint one's column sums
                if (MODE == LN_MI_HIST) atomicAdd (a.hist + B + o % B, w);
            }
        }
        if (MODE == LN_MI_HIST) {
            for (int o = threadIdx.x; o < B; o += blockDim.x) {
                const uint32_t w = shist[2 * B * B + o];
                if (w) atomicAdd (a.hist + o, (u64) w);
            }
        }
    }
    if constexpr (ln_mse (MODE)) {

    // the block's score and count, in warp order
    double sc = t_v[threadIdx.x];
    int cnt = t_n[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        sc += __shfl_down_sync (0xffffffffu, sc, o);
        cnt += __shfl_down_sync (0xffffffffu, cnt, o);
    }
    if (lane == 0) {
        sh_v[warp] = sc;
        sh_n[warp] = cnt;
    }
    __syncthreads ();
    if (threadIdx.x == 0) {
        double v = 0.0;
        int n = 0;
        for (int w = 0; w < W; w++) {
            v += sh_v[w];
            n += sh_n[w];
        }
        const int b = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
        a.score_part[b] = v;
        a.count_part[b] = n;
    }
    }
}

// ---- the rows' contraction ------------------------------------------------
//
// One block per knot row ky, kxc knots along x and kzc knots along z; a
// thread owns two voxel columns x, x + 1 of the block's tiles and marches
// along z (every blockDim.y-th plane), so that every load of a warp is one
// run of a row.  It contracts along z into a register window of four knots;
// the knots that leave it meet in shared memory, where they are contracted
// along x, normalised (MSE) and stored, the block's knots as one run per z
// knot.  The rows come from L2: what bounds it is how many loads are in
// flight.  (The next planes' loads sent out before the last ones are used:
// 88 us a call at 256x256x128 vpr 5 where this takes 83; the registers for
// it leave fewer planes in flight.)  Each block sums the voxel counts for
// its normalisation; the first one writes the result block.
//
// Its launch does not wait for the end of the line kernel's: the blocks
// start as the last of that one's end, fetch the weights and wait there
// (64^3 vpr 8: 14.6 us a call where one after the other takes 18.3).  The
// rows, counts and scores are written during this kernel's lifetime then:
// they are read through L2, never as read-only data.

constexpr int LF_MAX_THREADS = LINE_SPLIT_THREADS;

struct LineFinishArgs {
    BspGeom g;
    const float* rows;
    const float* luts;
    const double* sp;
    const int* cp;
    int nparts;          // 0: no score parts (res holds the result)
    const int* err;
    DevResult* res;
    DevResult* res_host;
    float* grad;
    double* grad64;
    float* score_out;
    double* score64_out;
    long long* nvox_out;
    FinishCombine cb;
    int ty, nys, j, nxs, kxc, kzc;
};

// NZ2: planes of a tile in flight where at most two y blocks reach a row.
// MIN_BLOCKS: blocks an SM holds (2: of at most 320 threads).
template <int NZ2, int MIN_BLOCKS>
__global__ void
__launch_bounds__ (MIN_BLOCKS == 1 ? LF_MAX_THREADS : 320, MIN_BLOCKS)
line_finish_kernel (const __grid_constant__ LineFinishArgs a)
{
    extern __shared__ __align__ (16) float sh[];       // [part][c][kz][voxel]
    __shared__ float4 sbx[64];
    __shared__ ulonglong2 sbz[2 * 64];                 // each weight twice
    __shared__ double sh_v[LF_MAX_THREADS / 32];
    __shared__ int sh_n[LF_MAX_THREADS / 32];
    const BspGeom& g = a.g;
    const int vx = g.vpr[0], vy = g.vpr[1], vz = g.vpr[2];
    const int T = blockDim.x, P = blockDim.y, NT = T * P;
    const int xt = threadIdx.x, part = threadIdx.y, tid = xt + T * part;
    const int kx0 = blockIdx.x * a.kxc, ky = blockIdx.y;
    const int kz0 = blockIdx.z * a.kzc;
    const int nkx = min (a.kxc, g.cdims[0] - kx0);
    const int nkz = min (a.kzc, g.cdims[2] - kz0);
    for (int o = tid; o < vx; o += NT) sbx[o] = *(const float4*) (a.luts + 4 * o);
    for (int o = tid; o < 4 * vz; o += NT) {
        const float w = a.luts[4 * (vx + vy) + o];
        ((u64*) sbz)[o] = pk (w, w);
    }
    __syncthreads ();
    asm volatile ("griddepcontrol.wait;" ::: "memory");

    // tile rows along z that reach the block's knots, y blocks that reach ky
    const int ta = max (0, kz0 - 3), tb = min (g.rdims[2], kz0 + nkz);
    const int y0 = max (0, ky - 3) / a.ty;
    const int y1 = min (g.rdims[1] - 1, ky) / a.ty;
    const int xs = ((kx0 - 3) * vx) & ~1;              // even: 8-byte loads
    const int x = xs + 2 * xt;
    const int nx = (nkx + 3) * vx + 1;                 // voxels of the block
    const bool live = 2 * xt < nx && x >= 0 && x < a.nxs;
    const int hs = a.kzc * 2 * T;
    u64 acc[3][4];
#pragma unroll
    for (int c = 0; c < 3; c++) {
#pragma unroll
        for (int k = 0; k < 4; k++) acc[c][k] = 0ull;
    }
    const size_t zs = (size_t) a.nys * a.j * 3 * a.nxs;          // per plane
    const int ys = (a.j - a.ty) * 3 * a.nxs;                     // per y block
    const float* row0 = a.rows + ((size_t) y0 * a.j + ky - y0 * a.ty) * 3 * a.nxs
        + (live ? x : 0);
    auto leave = [&] (int kz) {
        // knot kz has all its tile rows
        if (kz >= kz0 && kz < kz0 + nkz) {
            float* h = sh + part * 3 * hs + (kz - kz0) * 2 * T + 2 * xt;
#pragma unroll
            for (int c = 0; c < 3; c++) *(u64*) (h + c * hs) = live ? acc[c][0] : 0ull;
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {
            acc[c][0] = acc[c][1];
            acc[c][1] = acc[c][2];
            acc[c][2] = acc[c][3];
            acc[c][3] = 0ull;
        }
    };
    // NB: y blocks that reach ky; NZ planes' loads go out together
    auto march = [&] (auto nc) {
        constexpr int NB = decltype (nc)::value;
        constexpr int NZ = NB <= 2 ? NZ2 : 2;
        const float* p = row0 + (size_t) (ta * vz + part) * zs;
        const size_t step = (size_t) vz * zs, pstep = (size_t) P * zs;
        for (int tz = ta; tz < tb; tz++, p += step) {
            const int nz = min (vz, g.roi_dim[2] - tz * vz);
            const float* r = p;
            for (int z0 = part; z0 < nz; z0 += NZ * P) {
                u64 e[NZ][NB][3];
#pragma unroll
                for (int q = 0; q < NZ; q++) {
                    const bool in = z0 + q * P < nz;
#pragma unroll
                    for (int b = 0; b < NB; b++) {
                        const float* rb = r + b * ys;
#pragma unroll
                        for (int c = 0; c < 3; c++, rb += a.nxs) {
                            e[q][b][c] = in ? __ldcg ((const u64*) rb) : 0ull;
                        }
                    }
                    r += pstep;
                }
#pragma unroll
                for (int q = 0; q < NZ; q++) {
                    const ulonglong2* w = sbz + 2 * min (z0 + q * P, vz - 1);
                    const ulonglong2 w01 = w[0], w23 = w[1];
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        u64 s = e[q][0][c];
#pragma unroll
                        for (int b = 1; b < NB; b++) s = add2 (s, e[q][b][c]);
                        acc[c][0] = fma2 (w01.x, s, acc[c][0]);
                        acc[c][1] = fma2 (w01.y, s, acc[c][1]);
                        acc[c][2] = fma2 (w23.x, s, acc[c][2]);
                        acc[c][3] = fma2 (w23.y, s, acc[c][3]);
                    }
                }
            }
            leave (tz);
        }
    };
    switch (y1 - y0) {
    case 0: march (std::integral_constant<int, 1> ()); break;
    case 1: march (std::integral_constant<int, 2> ()); break;
    case 2: march (std::integral_constant<int, 3> ()); break;
    default: march (std::integral_constant<int, 4> ()); break;
    }
    leave (tb);
    leave (tb + 1);
    leave (tb + 2);
    // The blocks' counts (and on the first block their scores), in index order
    const bool first = blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0;
    {
        double v = 0.0;
        int n32 = 0;
        for (int i0 = tid; i0 < a.nparts; i0 += 4 * NT) {
            int c4[4];
            double s4[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int i = i0 + u * NT;
                c4[u] = i < a.nparts ? __ldcg (a.cp + i) : 0;
                s4[u] = first && i < a.nparts ? __ldcg (a.sp + i) : 0.0;
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                n32 += c4[u];
                v += s4[u];
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            v += __shfl_down_sync (0xffffffffu, v, o);
            n32 += __shfl_down_sync (0xffffffffu, n32, o);
        }
        if ((tid & 31) == 0) {
            sh_v[tid >> 5] = v;
            sh_n[tid >> 5] = n32;
        }
    }
    __syncthreads ();

    long long n_all = 0;
    if (a.nparts > 0) {
        int n32 = 0;
        for (int w = 0; w < NT / 32; w++) n32 += sh_n[w];
        n_all = n32;
    }
    if (first && tid == 0) {
        DevResult r;
        if (a.nparts > 0) {
            double v = 0.0;
            for (int w = 0; w < NT / 32; w++) v += sh_v[w];
            r.raw = v;
            r.num_vox = n_all;
            r.error = a.err ? *a.err : 0;
            r.score = n_all < 1 ? (double) FLT_MAX : v / (double) n_all;
            r.score_f = n_all < 1 ? FLT_MAX : (float) r.score;
            *a.res = r;
        } else {
            r = *a.res;
        }
        if (a.res_host) *a.res_host = r;
        if (a.cb.total_score) {
            // Bspline_score::accumulate then the regulariser's score
            // (src/register/bspline.cxx:595-622), in float
            float total = 0.f;
            total += a.cb.lambda * r.score_f;
            if (a.cb.reg_score) total += (float) *a.cb.reg_score;
            *a.cb.total_score = total;
        }
        if (a.score_out) *a.score_out = r.score_f;
        if (a.score64_out) *a.score64_out = r.score;
        if (a.nvox_out) *a.nvox_out = r.num_vox;
    }
    const double scale = a.nparts == 0 ? 1.0
        : n_all < 1 ? 0.0 : 2.0 / (double) n_all;
    // the parts' sums, into the first
    if (P > 1) {
        for (int o = tid; o < 3 * hs; o += NT) {
            float s = sh[o];
            for (int b = 1; b < P; b++) s += sh[b * 3 * hs + o];
            sh[o] = s;
        }
        __syncthreads ();
    }
    for (int o = tid; o < 3 * nkx * nkz; o += NT) {
        const int q = o / (3 * nkx), i = o - q * (3 * nkx);
        const int kx = i / 3, c = i - 3 * kx;
        // tiles kx - 3 .. kx of the knot, its weight 3 .. 0 of each
        const float* h = sh + c * hs + q * 2 * T + (kx0 - 3 + kx) * vx - xs;
        float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
        for (int u = 0; u < vx; u++) {
            const float4 w = sbx[u];
            s0 = fmaf (w.w, h[u], s0);
            s1 = fmaf (w.z, h[u + vx], s1);
            s2 = fmaf (w.y, h[u + 2 * vx], s2);
            s3 = fmaf (w.x, h[u + 3 * vx], s3);
        }
        double s = (((double) s0 + s1) + s2) + s3;
        s *= scale;
        const size_t at = 3 * ((size_t) ((kz0 + q) * g.cdims[1] + ky)
            * g.cdims[0] + kx0) + i;
        if (a.cb.total_score) {
            // total_grad = 0 + lambda * smetric_grad (float), then the
            // regulariser's double gradient added with one rounding
            const float t = 0.f + a.cb.lambda * (float) s;
            s = a.cb.reg_grad ? (double) (float) ((double) t + a.cb.reg_grad[at])
                              : (double) t;
        }
        if (a.grad) a.grad[at] = (float) s;
        if (a.grad64) a.grad64[at] = s;
    }
}

// ---- host -------------------------------------------------------------------

bool
line_plan (const BspGeom& g, LinePlan* p, int sm_count)
{
    static_assert (sizeof (p->wy) == 16 * LN_MAX_VPR, "y weights");
    // the regions that 10 mm grids give on 1 to 2.5 mm voxels, where it was
    // compared with the tile kernel (1.2 to 2.1 times as fast, 2^18 to 2^25
    // voxels); others stay there
    for (int d = 0; d < 3; d++) {
        if (g.vpr[d] < 3 || g.vpr[d] > LN_MAX_VPR) return false;
    }
    // corner offsets are 32-bit byte counts
    if ((long long) g.mdim[0] * g.mdim[1] * g.mdim[2] >= (1LL << 30)) return false;
    p->nxs = (g.rdims[0] * g.vpr[0] + 3) & ~3;
    // Warps a block: a multiple of four, so that an SM's four schedulers get
    // the same number each (two blocks of ten: 98 us where three of eight
    // take 83); eight, so that a block's coefficients serve more columns
    // (four: 92).
    const int nxw = (g.roi_dim[0] + 31) / 32;
    const int cols = nxw * g.vpr[2];
    p->nw = LN_WARPS;
    p->gpr = (cols + p->nw - 1) / p->nw;
    const int nzl = g.roi_dim[2] - (g.rdims[2] - 1) * g.vpr[2];
    int foot = 0;
    for (int nz : {g.vpr[2], nzl}) {
        // a block's warps span at most this many 32-voxel columns
        const int span = std::min (nxw, (p->nw - 2) / nz + 2);
        const int kx = std::min (g.rdims[0], (32 * span + g.vpr[0] - 2) / g.vpr[0] + 1) + 3;
        foot = std::max (foot, nz * kx);
    }
    p->kx = std::min (g.rdims[0], 32 / g.vpr[0] + 1);
    // Tiles a block along y: an SM's share is whole blocks, and a block's
    // start and end (its z contraction, the three extra rows) cost as much as
    // LN_EDGE voxel rows.
    double best = 0.0;
    p->ty = 0;
    for (int ty = 1; ty <= g.rdims[1]; ty++) {
        const int nys = (g.rdims[1] + ty - 1) / ty;
        if (p->ty && nys == p->nys) continue;
        const long long n = (long long) p->gpr * nys * g.rdims[2];
        // fewer than four blocks on an SM leave its issue slots idle
        const double rate[5] = {0.0, 0.36, 0.63, 0.85, 1.0};
        const long long per_sm = (n + sm_count - 1) / sm_count;
        const double cost = (double) per_sm * (ty + LN_EDGE / g.vpr[1])
            / rate[std::min<long long> (per_sm, 4)];
        const LineSmem m = line_smem (g.vpr[0], g.vpr[2], ty + 3, foot);
        // (fewer than 65536 voxels a block: its histogram counters)
        if (p->ty && (m.total > 48 * 1024 || cost >= best
                || p->nw * 32 * ty * g.vpr[1] > 65535)) continue;
        best = cost;
        p->ty = ty;
        p->nys = nys;
        p->j = ty + 3;
        p->smem = m.total;
    }
    p->threads = 32 * p->nw;
    p->sms = sm_count;
    basis_lut (p->wy, g.vpr[1]);
    p->nblocks = p->gpr * p->nys * g.rdims[2];
    return p->nys < 65536 && g.rdims[2] < 65536 && p->smem <= 200 * 1024;
}

static bool
axis_aligned (const BspGeom& g)
{
    for (int i = 0; i < 3; i++) {
        for (int j = 0; j < 3; j++) {
            if (i != j && (g.fstep[3 * i + j] != 0.f || g.mproj[3 * i + j] != 0.f)) {
                return false;
            }
        }
    }
    return true;
}

static void
line_args (const BspGeom& g, const LinePlan& p, const float* coeff,
    const float* luts, LineArgs& a)
{
    a = LineArgs ();
    a.g = g;
    a.coeff = coeff;
    a.luts = luts;
    a.ty = p.ty;
    a.j = p.j;
    a.nxs = p.nxs;
    auto two = [] (float x, float y) {
        unsigned ux, uy;
        memcpy (&ux, &x, 4);
        memcpy (&uy, &y, 4);
        return (u64) uy << 32 | ux;
    };
    for (int v = 0; v < g.vpr[1]; v++) {
        for (int k = 0; k < 4; k++) {
            a.wy[v][k] = two (p.wy[4 * v + k], p.wy[4 * v + k]);
        }
    }
    a.roi_same = g.mroi != nullptr;
    for (int d = 0; d < 3; d++) {
        a.roi_same = a.roi_same && g.mroi_dim[d] == g.mdim[d]
            && g.mroi_origin[d] == g.morigin[d];
    }
    for (int i = 0; i < 9; i++) {
        a.roi_same = a.roi_same && g.mroi_proj[i] == g.mproj[i];
    }
    a.step_y = two (0.f, g.fstep[4]);
    a.morg = two (g.morigin[0], g.morigin[1]);
    a.mprj = two (g.mproj[0], g.mproj[4]);
    for (int d = 0; d < 3; d++) a.mtop[d] = (int) LINE_BIAS + g.mdim[d] - 2;
    a.mzero = (unsigned) g.mdim[0] * g.mdim[1] * g.mdim[2];
    a.midx0 = line_corner0 (g.mdim[0], g.mdim[1]);
}

template <int MODE, bool AXIS, bool ROI>
static cudaError_t
launch (const LinePlan& p, const LineArgs& a, cudaStream_t st)
{
    const BspGeom& g = a.g;
    auto k = line_kernel<MODE, AXIS, ROI>;
    size_t smem = p.smem;
    if (ln_hist (MODE)) smem += (2 * a.bins * a.bins + a.bins) * sizeof (uint32_t);
    if (MODE == LN_PZ_GRAD) smem += a.bins * a.bins * sizeof (float);
    if (smem > LN_PLAIN_SMEM) {
        cudaError_t e = set_max_dynamic_smem ((const void*) k, (int) smem);
        if (e != cudaSuccess) return e;
    }
    k<<<dim3 (p.gpr, p.nys, g.rdims[2]), p.threads, smem, st>>> (a);
    return cudaGetLastError ();
}

template <int MODE>
static cudaError_t
launch_mode (const LinePlan& p, const LineArgs& a, cudaStream_t st)
{
    const BspGeom& g = a.g;
    const bool axis = axis_aligned (g);
    if constexpr (ln_mse (MODE)) {
        if (g.fmask || g.mroi) {
            return axis ? launch<MODE, true, true> (p, a, st)
                        : launch<MODE, false, true> (p, a, st);
        }
    }
    return axis ? launch<MODE, true, false> (p, a, st)
                : launch<MODE, false, false> (p, a, st);
}

cudaError_t
launch_mse_line (const BspGeom& g, const LinePlan& p, int grad_mode,
    const float* fimg, const float* mimg, const float* mgrad,
    const float* coeff, const float* luts, float* rows, double* score_part,
    int* count_part, cudaStream_t st)
{
    LineArgs a;
    line_args (g, p, coeff, luts, a);
    a.fimg = fimg;
    a.mimg = mimg;
    a.mgrad = mgrad;
    a.rows = rows;
    a.score_part = score_part;
    a.count_part = count_part;
    return grad_mode == 0 ? launch_mode<LN_MSE_NEAREST> (p, a, st)
                          : launch_mode<LN_MSE_LINEAR> (p, a, st);
}

cudaError_t
launch_mi_line (const BspGeom& g, const LinePlan& p, bool hist_pass,
    const LineMi& mi, const float* coeff, const float* luts, float* rows,
    cudaStream_t st)
{
    LineArgs a;
    line_args (g, p, coeff, luts, a);
    a.fbin = mi.fbin;
    a.mquad = mi.mquad;
    a.bins = mi.bins;
    a.lut = mi.lut;
    a.nvf = mi.nvf;
    a.hist = mi.hist;
    a.mimg = mi.mimg;
    a.pz_min = mi.m_min;
    a.pz_delta = mi.m_delta;
    a.pz_inv = 1.f / mi.m_delta;
    a.rows = rows;
    if (!mi.parzen) {
        return hist_pass ? launch_mode<LN_MI_HIST> (p, a, st) : cudaErrorInvalidValue;
    }
    return hist_pass ? launch_mode<LN_PZ_HIST> (p, a, st)
                     : launch_mode<LN_PZ_GRAD> (p, a, st);
}

cudaError_t
launch_field_line (const BspGeom& g, const LinePlan& p, const float* coeff,
    const float* luts, const float* mimg, float outside, float* vf,
    float* warped, cudaStream_t st)
{
    LineArgs a;
    line_args (g, p, coeff, luts, a);
    a.mimg = mimg;
    a.outside = outside;
    a.out = vf ? vf : warped;
    return vf ? launch_mode<LN_FIELD> (p, a, st) : launch_mode<LN_WARP> (p, a, st);
}

// Bins of the 2 x 2 moving voxels from each voxel on (x fastest, a byte
// each): one 4-byte load in place of four of one byte.  A warp takes a row:
// bound by memory, 5 bytes a voxel.
__global__ void
bin_quad_kernel (int nx, int ny, long long rows, const uint8_t* __restrict__ bin,
    uint32_t* __restrict__ quad)
{
    const int nw = gridDim.x * (blockDim.x >> 5);
    for (long long r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
         r < rows; r += nw) {
        const uint8_t* b = bin + r * nx;
        const int dy = r % ny + 1 < ny ? nx : 0;
        for (int x = threadIdx.x & 31; x < nx; x += 32) {
            const int dx = x + 1 < nx ? 1 : 0;
            quad[r * nx + x] = b[x] | (uint32_t) b[x + dx] << 8
                | (uint32_t) b[x + dy] << 16 | (uint32_t) b[x + dy + dx] << 24;
        }
    }
}

cudaError_t
launch_bin_quad (const int dim[3], const uint8_t* bin, uint32_t* quad,
    cudaStream_t st)
{
    bin_quad_kernel<<<1184, 256, 0, st>>> (dim[0], dim[1],
        (long long) dim[1] * dim[2], bin, quad);
    return cudaGetLastError ();
}

cudaError_t
launch_line_finish (const BspGeom& g, const LinePlan& p, const float* rows,
    const float* luts, const double* score_part, const int* count_part,
    int nparts, const int* err, DevResult* res, DevResult* res_host,
    float* grad, double* grad64, float* score_out, double* score64_out,
    long long* nvox_out, cudaStream_t st, const FinishCombine& cb, bool behind)
{
    LineFinishArgs a;
    a.g = g;
    a.rows = rows;
    a.luts = luts;
    a.sp = score_part;
    a.cp = count_part;
    a.nparts = nparts;
    a.err = err;
    a.res = res;
    a.res_host = res_host;
    a.grad = grad;
    a.grad64 = grad64;
    a.score_out = score_out;
    a.score64_out = score64_out;
    a.nvox_out = nvox_out;
    a.cb = cb;
    a.ty = p.ty;
    a.nys = p.nys;
    a.j = p.j;
    a.nxs = p.nxs;
    const LineSplit f = line_finish_split (g.cdims, g.vpr, p.sms);
    const int threads = f.threads, parts = f.parts, nbx = f.nbx;
    a.kxc = f.kxc;
    a.kzc = f.kzc;
    const dim3 grid (nbx, g.cdims[1], (g.cdims[2] + a.kzc - 1) / a.kzc);
    const size_t smem = (size_t) 6 * a.kzc * threads * parts * sizeof (float);
    // the fewest rounds of at most five planes, evenly filled
    const int nz = (g.vpr[2] + parts - 1) / parts;
    const int rounds = (nz + 4) / 5;
    const int most_nz = (nz + rounds - 1) / rounds;
    auto k = line_finish_kernel<5, 1>;
    if (f.waves && threads <= 320 && most_nz <= 4) k = line_finish_kernel<4, 2>;
    else if (most_nz <= 3) k = line_finish_kernel<3, 1>;
    else if (most_nz == 4) k = line_finish_kernel<4, 1>;
    if (smem > LN_PLAIN_SMEM) {
        cudaError_t e = set_max_dynamic_smem ((const void*) k, (int) smem);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3 (threads, parts);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = behind ? 1 : 0;
    return cudaLaunchKernelEx (&cfg, k, a);
}

} // namespace b200

// spatial.cuh -- the clouds in spatial order, with bounds, for exact pruning.
//
// Most pairs of two large clouds cannot matter: a target farther from a source than its nearest one
// is no nearest neighbour, and a pair whose two exponentials are below the smallest normal FP32
// number adds exactly 0 (ex2.approx.ftz flushes it).  To find the pairs that can matter without
// visiting all of them, init sorts each cloud into the cells of a grid along a Hilbert curve, splits
// runs of that order into tiles of 32 points, and keeps a bounding sphere per subgroup of 8, tile, and super tile of
// 32 tiles.  The searches test spheres against
// spheres, then points, and evaluate what is left with the same FP32 operations as the all-pairs
// kernels.  The order inside a cell is arbitrary: no result depends on it.
#pragma once

#include "common.cuh"

namespace dugma {

constexpr int kTile = 32;   // points per tile (one warp: one point per lane)
constexpr int kSub = 8;     // points per subgroup of a tile
constexpr int kSuper = 32;  // tiles of a super tile
constexpr int kRun = 512;   // points of the cell order split into tiles together

// The FP32 flush: 2^x is 0 for x < -126.  1.5 more covers the rounding of the log weights.
constexpr float kFlushExp = 127.5f;

// A point in spatial order: coordinates, a = the exponent it can lose before the flush (kFlushExp +
// log2 of its relative weight), L = a bound on 1 / (smallest eigenvalue of sym(Sigma^-1)) (the
// largest variance; +inf when that matrix is not positive definite, or the weight 0 beside a positive
// determinant; 0 when the point is neglected), and its index in the cloud.
struct __align__(16) SortedPoint {
    float p[3];
    float a;
    float L;
    int idx;
    float pad[2];
};

// Bounding sphere of a tile or subgroup, and its points' largest a and L.
struct __align__(16) Bound {
    float c[3];
    float r;
    float a, L;
    float pad[2];
};

// Squares of less than this are below the normal FP32 numbers, and sqrt_fast makes 0 of them: a bound is at
// least this much, and a radius wider by a few.
constexpr float kLeastReach = 1.1e-19f;

// sqrt on the SFU (PTX sqrt.approx.ftz.f32, relative error 2^-23)
__device__ __forceinline__ float sqrt_fast(float x)
{
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Nearest-neighbour targets, two per record: a = (-y0, -y0', -y1, -y1'), b = (-y2, -y2', j, j')
// (the all-pairs search, whose records are in index order, leaves j, j' zero).
struct __align__(16) NNRec2 {
    float4 a, b;
};

// sqrt(1 + |R^T R - I|_F), rounded up: how much R stretches a length at most
__device__ __forceinline__ float pose_stretch(const double* R, int D)
{
    double f = 0;
    for (int a = 0; a < D; ++a)
        for (int b = 0; b < D; ++b) {
            double v = a == b ? -1.0 : 0.0;
            for (int k = 0; k < D; ++k) v += R[k + D * a] * R[k + D * b];
            f += v * v;
        }
    return __double2float_ru(sqrt(1.0 + sqrt(f)) * (1.0 + 1e-6));
}

// A bound's sphere under y' = R y + t: the centre rounded to FP32, the radius stretched and widened by
// what that rounding, the FP32 distance tests and squares below the normal numbers (both spheres') can lose.
template <int D>
__device__ __forceinline__ float4 posed_sphere(const Bound& b, const double* R, const double* t, float stretch)
{
    float c[3] = {0.f, 0.f, 0.f};
    float size = 0.f;
#pragma unroll
    for (int a = 0; a < D; ++a) {
        double v = t[a];
#pragma unroll
        for (int k = 0; k < D; ++k) v += R[a + D * k] * (double)b.c[k];
        c[a] = __double2float_rn(v);
        size += fabsf(c[a]) + fabsf(b.c[a]) + fabsf(__double2float_rn(t[a]));
    }
    return make_float4(c[0], c[1], c[2], fmaf(b.r, stretch, fmaf(1e-6f, size, 4.f * kLeastReach)));
}

// The place of a point's grid cell along a Hilbert curve through the 2^bits cells per axis (J. Skilling,
// "Programming the Hilbert curve", AIP Conf. Proc. 707, 2004): cells next to each other on it are
// neighbours, so runs of it stay compact.
template <int D>
__device__ __forceinline__ int cell_code(const float* p, const float* lo, float inv, int bits)
{
    const float top = (float)((1 << bits) - 1);
    int x[D];
#pragma unroll
    for (int a = 0; a < D; ++a) x[a] = (int)fminf(fmaxf((p[a] - lo[a]) * inv, 0.f), top);   // (NaN: cell 0)
    for (int q = 1 << (bits - 1); q > 1; q >>= 1)
#pragma unroll
        for (int a = 0; a < D; ++a) {
            if (x[a] & q) {
                x[0] ^= q - 1;
            } else {
                const int t = (x[0] ^ x[a]) & (q - 1);
                x[0] ^= t;
                x[a] ^= t;
            }
        }
#pragma unroll
    for (int a = 1; a < D; ++a) x[a] ^= x[a - 1];
    int t = 0;
    for (int q = 1 << (bits - 1); q > 1; q >>= 1)
        if (x[D - 1] & q) t ^= q - 1;
    int code = 0;
    for (int b = bits - 1; b >= 0; --b)
#pragma unroll
        for (int a = 0; a < D; ++a) code = code << 1 | ((x[a] ^ t) >> b & 1);
    return code;
}

}  // namespace dugma

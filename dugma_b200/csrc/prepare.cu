// prepare.cu -- init-time and per-evaluation prologue kernels.
//
// This file is compiled with -fmad=false: every FP64 expression below is evaluated
// as written (no fused multiply-add), so the FP32 state written by init and the
// FP32 rounding of y' match the CPU oracle bit for bit.
#include <cmath>
#include <cstdio>
#include <cstring>

#include "context.hpp"
#include "spatial.cuh"

namespace dugma {

// ---------------------------------------------------------------------------
// init, both clouds in each launch (blockIdx.y: 0 the sources, 1 the targets):
//   1 init_stats_kernel   per-block sums of the covariance traces, coordinates and squared norms
//   2 init_points_kernel  FP64 -> FP32 conversion (init.cu:192-234) fused with the per-point inverse
//     covariance and |Sigma|^-1/2 (init.cu:22-190): the inverse in FP64 from the FP32-rounded
//     covariance by the adjugate, in the order of the reference's formula, rounded to FP32; det <= 0:
//     all entries 1e5, weight 0 (init.cu:48-57, 86-100).  Also the packed FP32 covariance of the CONV
//     model, the largest weight, the Cholesky factors, and each point's grid cell and place in it.
//   3 cell_scan_kernel    the cells' first positions; beside it, samples of how far points reach
//   4 sort_points_kernel  log2 weights relative to the largest, and the points in cell order
//   5 split_kernel        runs of kRun points in that order split down to tiles at medians
//   6 bounds_kernel       bounding spheres of subgroups, tiles and super tiles; the scalars for the host
// Bound by launch latency up to ~100K points; the six launches do both clouds.
// ---------------------------------------------------------------------------
struct InitCloud {
    const double *P, *C;   // FP64 inputs (staged)
    int n;
    float *p32, *cinv, *w, *cpack, *lw;
    double* ufac;          // nullable: upper Cholesky factor of sym(cinv) per point (packed, FP64); zero
                           // for neglected points and those whose sym(cinv) is not positive definite
    float* L;              // largest variance per point (SortedPoint::L)
    int2* place;           // grid cell and rank in it
    int* hist;             // points per cell, then the cells' first positions
    SortedPoint* pt;
    Bound *tile, *sub, *super;
};
struct InitArgs {
    InitCloud cl[2];
    double* part;          // [2][kInitParts][5] partial sums
    int nb, bits;
    int* counter;          // [0] det <= 0, [2 + cloud] largest weight (float bits), [4 + cloud] weighted
                           // points without a Cholesky factor, [6] largest trace of an inverse covariance
    int* reach;            // per cloud [2][kReachBins] (sample_reach), then the targets' pairs nearer than a grid cell
    double *out, *host;    // kInitOut scalars for the host (host: nullable, mapped)
    double* out_reach;     // and the samples, which go to host + 16
};

// partial sums over contiguous slices, both in fixed order (deterministic): trace, coordinates, |p|^2
__global__ void init_stats_kernel(InitArgs a, int D)
{
    const InitCloud& c = a.cl[blockIdx.y];
    const int per = (c.n + gridDim.x - 1) / gridDim.x;
    const int b0 = blockIdx.x * per, b1 = min(c.n, b0 + per);
    double v[5] = {0, 0, 0, 0, 0};
    for (int i = b0 + threadIdx.x; i < b1; i += blockDim.x)
        for (int q = 0; q < D; ++q) {
            const double x = c.P[(size_t)i * D + q];
            v[0] += c.C[(size_t)i * D * D + q * (D + 1)];
            v[1 + q] += x;
            v[4] += x * x;
        }
    __shared__ double red[8][5];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int q = 0; q < 5; ++q) {
        const double s = warp_sum(v[q]);
        if (lane == 0) red[warp][q] = s;
    }
    __syncthreads();
    if (threadIdx.x < 5) {
        double s = 0;
        for (int w = 0; w < 8; ++w) s += red[w][threadIdx.x];
        a.part[((size_t)blockIdx.y * kInitParts + blockIdx.x) * 5 + threadIdx.x] = s;
    }
}

// The sums of the partials: per cloud the trace sum, the coordinates' sums and that of |p|^2 (every
// block adds them in the same order, so all agree).  At least 8 warps.
__device__ __forceinline__ void init_stats_total(const InitArgs& a, double (&tot)[2][5])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int e = warp; e < 10 && warp < 8; e += 8) {
        double s = 0;
        for (int b = lane; b < a.nb; b += 32) s += a.part[((size_t)(e / 5) * kInitParts + b) * 5 + e % 5];
        s = warp_sum(s);
        if (lane == 0) tot[e / 5][e % 5] = s;
    }
    __syncthreads();
}

// CONV covariance scale: the mean of trace / D over both clouds' covariances, rounded to a power of
// two so that dividing by it is exact in FP32
__device__ __forceinline__ double conv_scale(const InitArgs& a, const double (&tot)[2][5], int D)
{
    const double tr = (tot[0][0] + tot[1][0]) / ((double)D * (a.cl[0].n + a.cl[1].n));
    return (isfinite(tr) && tr > 0) ? exp2(round(log2(tr))) : 1.0;
}

// mean squared distance of a cloud's points to their mean
__device__ __forceinline__ double mean_radius2(const double* tot, int n, int D)
{
    double r2 = tot[4] / n;
    for (int q = 0; q < D; ++q) r2 -= (tot[1 + q] / n) * (tot[1 + q] / n);
    return isfinite(r2) && r2 > 0 ? r2 : 0.0;
}

// the grid of a cloud: cells of 2.5 radii / 2^bits about the mean, points outside in the edge cells
__device__ __forceinline__ float cell_grid(const double* tot, int n, int D, int bits, float* lo)
{
    const double r = sqrt(mean_radius2(tot, n, D));
    for (int q = 0; q < D; ++q) lo[q] = r > 0 ? __double2float_rn(tot[1 + q] / n - 1.25 * r) : 0.f;
    return r > 0 ? __double2float_rn((double)(1 << bits) / (2.5 * r)) : 0.f;
}

// bound on the largest eigenvalue of A^-1 for a positive definite A (packed): the 8-norm of the
// eigenvalues of adj(A) / det(A), less than 3^(1/8) above it (FP64 adjugate, FP32 powers, 1e-5 for their
// rounding).  The 4e-6 of the trace taken off A's smallest eigenvalue covers the rounding of the
// FP32 records made from A and of the quadratic forms.
template <int D>
__device__ __forceinline__ float variance_bound(const double* A)
{
    constexpr int NS = Sym<D>::N;
    float m[6];
    double tr;
    if (D == 3) {
        const double a = A[0], b = A[1], c = A[2], d = A[3], e = A[4], f = A[5];
        const double m0 = b * c - f * f, m3 = e * f - d * c, m4 = d * f - b * e;
        tr = a + b + c;
        const double q = tr / (a * m0 + d * m3 + e * m4);   // scaled by the trace
        m[0] = (float)(m0 * q);
        m[1] = (float)((a * c - e * e) * q);
        m[2] = (float)((a * b - d * d) * q);
        m[3] = (float)(m3 * q);
        m[4] = (float)(m4 * q);
        m[5] = (float)((d * e - a * f) * q);
    } else {
        tr = A[0] + A[1];
        const double q = tr / (A[0] * A[1] - A[2] * A[2]);
        m[0] = (float)(A[1] * q);
        m[1] = (float)(A[0] * q);
        m[2] = (float)(-A[2] * q);
    }
    float top[4];
#pragma unroll
    for (int it = 0; it < 4; ++it) {   // m <- (m / trace)^2, three times
        top[it] = D == 3 ? m[0] + m[1] + m[2] : m[0] + m[1];
        if (it == 3) break;
        const float r = 1.f / top[it];
#pragma unroll
        for (int k = 0; k < NS; ++k) m[k] *= r;
        if (D == 3) {
            const float q0 = m[0] * m[0] + m[3] * m[3] + m[4] * m[4], q1 = m[3] * m[3] + m[1] * m[1] + m[5] * m[5],
                        q2 = m[4] * m[4] + m[5] * m[5] + m[2] * m[2], q3 = m[0] * m[3] + m[3] * m[1] + m[4] * m[5],
                        q4 = m[0] * m[4] + m[3] * m[5] + m[4] * m[2], q5 = m[3] * m[4] + m[1] * m[5] + m[5] * m[2];
            m[0] = q0; m[1] = q1; m[2] = q2; m[3] = q3; m[4] = q4; m[5] = q5;
        } else {
            const float q0 = m[0] * m[0] + m[2] * m[2], q1 = m[1] * m[1] + m[2] * m[2], q2 = m[2] * (m[0] + m[1]);
            m[0] = q0; m[1] = q1; m[2] = q2;
        }
    }
    // of A^-1, in units of 1 / trace(A)
    const double lmax = (double)top[0] * sqrtf(top[1] * sqrtf(top[2] * sqrtf(top[3]))) * (1.0 + 1e-5);
    const double low = (1.0 / lmax - 4e-6) * tr;   // A's smallest eigenvalue, from below
    return low > 0 && isfinite(low) ? __double2float_ru(1.0 / low) : INFINITY;
}

template <int D>
__global__ void __launch_bounds__(256) init_points_kernel(InitArgs ia)
{
    constexpr int NS = Sym<D>::N;
    __shared__ double tot[2][5];
    init_stats_total(ia, tot);
    const InitCloud& cl = ia.cl[blockIdx.y];
    const double* __restrict__ P = cl.P;
    const double* __restrict__ C = cl.C;
    float* __restrict__ w = cl.w;
    const int n = cl.n;
    const double inv_scale = 1.0 / conv_scale(ia, tot, D);
    float lo[3];
    const float inv = cell_grid(tot[blockIdx.y], n, D, ia.bits, lo);
    int wmax = 0, tmax = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float pf[D];
#pragma unroll
        for (int a = 0; a < D; ++a) cl.p32[(size_t)i * D + a] = pf[a] = __double2float_rn(P[(size_t)i * D + a]);
        double a_[D * D];
#pragma unroll
        for (int k = 0; k < D * D; ++k) a_[k] = (double)__double2float_rn(C[(size_t)i * D * D + k]);
#pragma unroll
        for (int k = 0; k < NS; ++k) {
            const int ra = Sym<D>::a(k), rb = Sym<D>::b(k);
            cl.cpack[(size_t)i * NS + k] = __double2float_rn(0.5 * (a_[ra + D * rb] + a_[rb + D * ra]) * inv_scale);
        }
        float o[D * D];
        float wi;
        bool valid;   // det > 0
        if (D == 3) {
            const double a11 = a_[0], a21 = a_[1], a31 = a_[2], a12 = a_[3], a22 = a_[4], a32 = a_[5],
                         a13 = a_[6], a23 = a_[7], a33 = a_[8];
            const double d = a11 * a22 * a33 - a11 * a23 * a32 - a12 * a21 * a33 + a12 * a23 * a31 +
                             a13 * a21 * a32 - a13 * a22 * a31;
            valid = d > 0;
            if (valid) {
                o[0] = __double2float_rn((a22 * a33 - a23 * a32) / d);
                o[1] = __double2float_rn(-(a21 * a33 - a23 * a31) / d);
                o[2] = __double2float_rn((a21 * a32 - a22 * a31) / d);
                o[3] = __double2float_rn(-(a12 * a33 - a13 * a32) / d);
                o[4] = __double2float_rn((a11 * a33 - a13 * a31) / d);
                o[5] = __double2float_rn(-(a11 * a32 - a12 * a31) / d);
                o[6] = __double2float_rn((a12 * a23 - a13 * a22) / d);
                o[7] = __double2float_rn(-(a11 * a23 - a13 * a21) / d);
                o[8] = __double2float_rn((a11 * a22 - a12 * a21) / d);
                wi = __double2float_rn(sqrt(1.0 / d));
            } else {
#pragma unroll
                for (int k = 0; k < 9; ++k) o[k] = 100000.0f;
                wi = 0.0f;
                atomicAdd(ia.counter, 1);
            }
        } else {
            const double a1 = a_[0], a2 = a_[1], a3 = a_[2], a4 = a_[3];
            const double d = a1 * a4 - a2 * a3;
            valid = d > 0;
            if (valid) {
                o[0] = __double2float_rn(a4 / d);
                o[1] = __double2float_rn(-a2 / d);
                o[2] = __double2float_rn(-a3 / d);
                o[3] = __double2float_rn(a1 / d);
                wi = __double2float_rn(sqrt(1.0 / d));
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) o[k] = 100000.0f;
                wi = 0.0f;
                atomicAdd(ia.counter, 1);
            }
        }
#pragma unroll
        for (int k = 0; k < D * D; ++k) cl.cinv[(size_t)i * D * D + k] = o[k];
        w[i] = wi;
        // positive floats order like their bit patterns
        if (wi > 0.0f) {
            float tr = 0.f;
#pragma unroll
            for (int a = 0; a < D; ++a) tr += fabsf(o[a * (D + 1)]);
            wmax = max(wmax, __float_as_int(wi));
            tmax = max(tmax, __float_as_int(tr));
        }
        double pk[NS], u[NS];
#pragma unroll
        for (int k = 0; k < NS; ++k) {
            const int ra = Sym<D>::a(k), rb = Sym<D>::b(k);
            pk[k] = 0.5 * ((double)o[ra + D * rb] + (double)o[rb + D * ra]);
        }
        const bool ok = chol_upper<D>(pk, u);
        if (wi > 0.0f && !ok) atomicAdd(ia.counter + 4 + blockIdx.y, 1);
        if (cl.ufac)
#pragma unroll
            for (int k = 0; k < NS; ++k) cl.ufac[(size_t)i * NS + k] = wi > 0.0f ? u[k] : 0.0;
        // (a weight that is 0 in FP32 beside a positive determinant: no bound; the CONV model has such points' pairs)
        cl.L[i] = wi > 0.0f ? (ok ? variance_bound<D>(pk) : INFINITY) : (valid ? INFINITY : 0.f);
        const int code = cell_code<D>(pf, lo, inv, ia.bits);
        cl.place[i] = make_int2(code, atomicAdd(cl.hist + code, 1));
    }
    // the largest weight (order-independent, so deterministic); log2 is monotonic, so log2 of the
    // largest weight is the largest log2
    wmax = __reduce_max_sync(0xffffffffu, wmax);
    tmax = __reduce_max_sync(0xffffffffu, tmax);
    if ((threadIdx.x & 31) == 0 && wmax > 0) {
        atomicMax(ia.counter + 2 + blockIdx.y, wmax);
        atomicMax(ia.counter + 6, tmax);
    }
}

// Samples of how far a cloud's points reach, for the choice between all pairs and the sparse passes
// (sparse_sigma): for each of kReachPoints points, a warp each, kReachDraws pairs of it with another
// point of its cloud, standing for a target that lies there, and with the largest variance of a point
// of the other cloud.  A pair is in reach where |k| |d|^2 / sig is less than the exponent to the flush
// times that variance, so q = |d|^2 / the variance is binned by octaves, and per bin the sums over the
// points of their pairs below its end, c, and of c (c - 1) are kept: how much a point reaches on average,
// and how unevenly.  Points and pairs are chosen by index and the sums are whole numbers: the same in every init.
template <int D>
__device__ __forceinline__ void sample_reach(const InitArgs& a, int cloud, int block)
{
    __shared__ int count[32][kReachBins];
    __shared__ int sums[2 * kReachBins + 1];
    __shared__ double tot[2][5];
    const InitCloud &c = a.cl[cloud], &o = a.cl[1 - cloud];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tid = threadIdx.x;
    for (int b = lane; b < kReachBins; b += 32) count[warp][b] = 0;
    if (tid < 2 * kReachBins + 1) sums[tid] = 0;
    init_stats_total(a, tot);   // (synchronises)
    float lo[3];
    const float inv = cell_grid(tot[cloud], c.n, D, a.bits, lo);
    auto mix = [](uint32_t x) {   // multiplications by odd numbers and shifts: one to one, and far from regular
        x *= 0x9e3779b1u;
        x ^= x >> 15;
        x *= 0x85ebca6bu;
        return x ^ x >> 13;
    };
    const uint32_t s = 32 * block + warp;
    const int i = (int)((long long)s * c.n / kReachPoints);
    int near = 0;
    if (c.n > 1)
        for (int r = 0; r < kReachDraws / 32; ++r) {
            const uint32_t h = mix(s * kReachDraws + 32 * r + lane + 1);
            int j = i + 1 + (int)__umulhi(h, (uint32_t)c.n - 1);
            if (j >= c.n) j -= c.n;
            const int k = (int)__umulhi(mix(h ^ 0x5bd1e995u), (uint32_t)o.n);
            float d2 = 0.f;
#pragma unroll
            for (int q = 0; q < D; ++q) {
                const float d = c.p32[(size_t)i * D + q] - c.p32[(size_t)j * D + q];
                d2 = d2 + d * d;
            }
            near += d2 * inv * inv < 1.f;
            if (!(c.w[i] > 0.f && o.w[k] > 0.f)) continue;   // (without weight: reaches nothing)
            const int e = (int)(__float_as_uint(d2 / fmaxf(c.L[i], o.L[k])) >> 23);
            atomicAdd(&count[warp][min(max(e - kReachExp, 0), kReachBins - 1)], 1);
        }
    near = (int)__reduce_add_sync(0xffffffffu, (unsigned)near);
    __syncwarp();
    int v[kReachBins / 32], sum = 0;   // this lane's bins, and the bins before them
#pragma unroll
    for (int b = 0; b < kReachBins / 32; ++b) sum += v[b] = count[warp][kReachBins / 32 * lane + b];
    int below = sum;
#pragma unroll
    for (int w = 1; w < 32; w <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, below, w);
        if (lane >= w) below += u;
    }
    below -= sum;
#pragma unroll
    for (int b = 0; b < kReachBins / 32; ++b) {
        below += v[b];
        if (below == 0) continue;
        atomicAdd(&sums[kReachBins / 32 * lane + b], below);
        atomicAdd(&sums[kReachBins + kReachBins / 32 * lane + b], below * (below - 1));
    }
    if (lane == 0) atomicAdd(&sums[2 * kReachBins], near);
    __syncthreads();
    if (tid < 2 * kReachBins && sums[tid]) atomicAdd(a.reach + 2 * kReachBins * cloud + tid, sums[tid]);
    if (tid == 2 * kReachBins && cloud == 1 && sums[tid]) atomicAdd(a.reach + 4 * kReachBins, sums[tid]);
}

// hist[c] <- the points in the cells before c; one block of 1024 threads per cloud.  The blocks behind
// them sample the reach, on SMs that the scan leaves idle.
template <int D>
__global__ void __launch_bounds__(1024) cell_scan_kernel(InitArgs a, int cells)
{
    if (blockIdx.x >= 2) {
        sample_reach<D>(a, blockIdx.x & 1, (int)blockIdx.x / 2 - 1);
        return;
    }
    int* __restrict__ hist = a.cl[blockIdx.x].hist;
    __shared__ int sums[32];
    __shared__ int carry;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < cells; base += 4096) {   // cells is a multiple of 4
        const int e = base + 4 * (int)threadIdx.x;
        int4 v = e < cells ? *reinterpret_cast<const int4*>(hist + e) : make_int4(0, 0, 0, 0);
        const int s = v.x + v.y + v.z + v.w;
        int inc = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        if (lane == 31) sums[warp] = inc;
        __syncthreads();
        if (warp == 0) {
            int t = sums[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= o) t += u;
            }
            sums[lane] = t;
        }
        __syncthreads();
        int off = carry + (warp > 0 ? sums[warp - 1] : 0) + inc - s;
        const int total = sums[31];
        v = make_int4(off, off + v.x, off + v.x + v.y, off + v.x + v.y + v.z);
        if (e < cells) *reinterpret_cast<int4*>(hist + e) = v;
        __syncthreads();
        if (threadIdx.x == 0) carry += total;
        __syncthreads();
    }
}

// lw_i = log2(w_i) - Lmax with Lmax = log2(largest weight) (-inf when no weight is positive), and the
// points to their places in cell order
template <int D>
__global__ void sort_points_kernel(InitArgs ia)
{
    const InitCloud& c = ia.cl[blockIdx.y];
    const int mb = ia.counter[2 + blockIdx.y];
    const double Lm = mb > 0 ? log2((double)__int_as_float(mb)) : -INFINITY;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < c.n; i += gridDim.x * blockDim.x) {
        const float lw = c.w[i] > 0.0f ? __double2float_rn(log2((double)c.w[i]) - Lm) : -INFINITY;
        c.lw[i] = lw;
        const int2 pl = c.place[i];
        SortedPoint s;
        s.p[2] = 0.f;
#pragma unroll
        for (int a = 0; a < D; ++a) s.p[a] = c.p32[(size_t)i * D + a];
        // (the source's weight is no part of the exponent)
        s.a = blockIdx.y == 0 ? (lw > -INFINITY ? kFlushExp : -1.f) : fmaxf(lw + kFlushExp, -1.f);
        s.L = c.L[i];
        s.idx = i;
        s.pad[0] = s.pad[1] = 0.f;
        c.pt[c.hist[pl.x] + pl.y] = s;
    }
}

// Runs of kRun points of the cell order, each split down to its tiles by a block: at every level each
// part is sorted along its longest axis and halved at the median, down to subgroups of 8.  The sorts
// are bitonic on 32-bit keys: 22 bits of the coordinate within its part above the point's number in
// the run, one shuffle a step.  64K points of a surface, tile radius (mean, largest) over the cloud's:
// cell order alone 0.093, 0.63; runs of 256 0.071, 0.50; of 512 0.066, 0.43; of 1024 0.064, 0.45 (and
// twice the time: its sorts meet at block barriers).
template <int D>
__global__ void __launch_bounds__(kRun) split_kernel(InitArgs ia)
{
    const InitCloud& c = ia.cl[blockIdx.y];
    const int base = blockIdx.x * kRun, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n = min(kRun, c.n - base);
    if (n <= 0) return;
    __shared__ float sx[D][kRun];
    __shared__ uint32_t key[kRun];
    __shared__ int ext[2 * D][kRun / 32];
    auto ordered = [](float f) {   // float order as int order
        const int b = __float_as_int(f);
        return b >= 0 ? b : b ^ 0x7fffffff;
    };
    auto unordered = [](int b) { return __int_as_float(b >= 0 ? b : b ^ 0x7fffffff); };
#pragma unroll
    for (int a = 0; a < D; ++a) sx[a][tid] = tid < n ? fminf(fmaxf(c.pt[base + tid].p[a], -1e30f), 1e30f) : 0.f;
    __syncthreads();
    int id = tid;
    for (int S = kRun; S > kSub; S >>= 1) {
        // the longest axis of this thread's part (threads [tid / S * S, + S)) and the part's range on it
        int mn[D], mx[D];
        const bool in = id < n;
#pragma unroll
        for (int a = 0; a < D; ++a) {
            const int v = ordered(sx[a][id]);
            mn[a] = in ? v : 0x7fffffff;
            mx[a] = in ? v : (int)0x80000000;
            if (S >= 32) {
                mn[a] = __reduce_min_sync(0xffffffffu, mn[a]);
                mx[a] = __reduce_max_sync(0xffffffffu, mx[a]);
            } else {
                for (int o = 1; o < S; o <<= 1) {
                    mn[a] = min(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], o));
                    mx[a] = max(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], o));
                }
            }
        }
        if (S > 32) {
            __syncthreads();
            if (lane == 0)
#pragma unroll
                for (int a = 0; a < D; ++a) {
                    ext[2 * a][warp] = mn[a];
                    ext[2 * a + 1][warp] = mx[a];
                }
            __syncthreads();
            const int w = warp / (S / 32) * (S / 32) + lane % (S / 32);   // a warp of this part
#pragma unroll
            for (int a = 0; a < D; ++a) {
                mn[a] = __reduce_min_sync(0xffffffffu, ext[2 * a][w]);
                mx[a] = __reduce_max_sync(0xffffffffu, ext[2 * a + 1][w]);
            }
        }
        int axis = 0;
        float lo = unordered(mn[0]), len = unordered(mx[0]) - lo;
#pragma unroll
        for (int a = 1; a < D; ++a) {
            const float l = unordered(mn[a]), e = unordered(mx[a]) - l;
            if (e > len) { axis = a; lo = l; len = e; }
        }
        static_assert(kRun <= 1024, "10 bits of the key number the run's points");
        // points past the end sort last and stay there
        uint32_t k = 0x3fffffu << 10 | (uint32_t)id;
        if (in) {
            const float f = len > 0.f ? (sx[axis][id] - lo) / len : 0.f;
            k = (uint32_t)(f * 4194302.f) << 10 | (uint32_t)id;
        }
        for (int K = 2; K <= S; K <<= 1)
            for (int j = K >> 1; j > 0; j >>= 1) {
                uint32_t o;
                if (j >= 32) {
                    __syncthreads();
                    key[tid] = k;
                    __syncthreads();
                    o = key[tid ^ j];
                } else {
                    o = __shfl_xor_sync(0xffffffffu, k, j);
                }
                const bool up = ((tid & (S - 1)) & K) == 0, lower = (tid & j) == 0;
                k = up == lower ? min(k, o) : max(k, o);
            }
        id = (int)(k & 1023u);
    }
    SortedPoint p;
    if (tid < n) p = c.pt[base + id];
    __syncthreads();
    if (tid < n) c.pt[base + tid] = p;
}

// one block of 32 warps per super tile, one warp per tile: spheres (about the middle of the points' box)
// of the tile and its four subgroups, then the super tile's around the tiles'
template <int D>
__global__ void __launch_bounds__(1024) bounds_kernel(InitArgs ia)
{
    const InitCloud& c = ia.cl[blockIdx.y];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n_tiles = (c.n + kTile - 1) / kTile;
    const int t = blockIdx.x * kSuper + warp;
    __shared__ Bound s_tile[kSuper];
    if (blockIdx.x * kSuper < n_tiles) {
        const int i = t * kTile + lane;
        const bool in = i < c.n;
        SortedPoint s;
        if (in) s = c.pt[i];
#pragma unroll
        for (int w = kSub; w <= kTile; w *= kTile / kSub) {   // subgroups of 8 lanes, then the tile's 32
            Bound b;
            b.pad[0] = b.pad[1] = 0.f;
            b.c[2] = 0.f;
            float r2 = 0.f;
#pragma unroll
            for (int a = 0; a < D; ++a) {
                float mn = in ? s.p[a] : INFINITY, mx = in ? s.p[a] : -INFINITY;
                for (int o = 1; o < w; o <<= 1) {
                    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                }
                b.c[a] = mn > mx ? 0.f : 0.5f * mn + 0.5f * mx;   // (no points: 0)
                const float d = in ? s.p[a] - b.c[a] : 0.f;
                r2 = fmaf(d, d, r2);
            }
            // a point that is not finite leaves a sphere that holds everything
            float r = in && !(r2 < INFINITY) ? INFINITY : sqrtf(r2) * (1.f + 1e-6f);
            b.a = in ? s.a : -1.f;
            b.L = in ? (s.L >= 0.f ? s.L : INFINITY) : 0.f;
            for (int o = 1; o < w; o <<= 1) {
                r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, o));
                b.a = fmaxf(b.a, __shfl_xor_sync(0xffffffffu, b.a, o));
                b.L = fmaxf(b.L, __shfl_xor_sync(0xffffffffu, b.L, o));
            }
            b.r = r;
            if (w == kSub) {
                if (t < n_tiles && (lane & (kSub - 1)) == 0) c.sub[4 * t + lane / kSub] = b;
            } else if (lane == 0) {
                s_tile[warp] = b;
                if (t < n_tiles) c.tile[t] = b;
            }
        }
        __syncthreads();
        if (warp == 0) {
            const bool have = blockIdx.x * kSuper + lane < n_tiles;
            Bound b = s_tile[lane];
            float d2 = 0.f;
#pragma unroll
            for (int a = 0; a < D; ++a) {
                float mn = have ? b.c[a] : INFINITY, mx = have ? b.c[a] : -INFINITY;
                for (int o = 1; o < 32; o <<= 1) {
                    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                }
                const float m = 0.5f * mn + 0.5f * mx, d = b.c[a] - m;
                d2 = fmaf(d, d, d2);
                b.c[a] = m;
            }
            float r = have ? (d2 < INFINITY ? (sqrtf(d2) + b.r) * (1.f + 1e-6f) : INFINITY) : 0.f;
            b.a = have ? b.a : -1.f;
            b.L = have ? b.L : 0.f;
            for (int o = 1; o < 32; o <<= 1) {
                r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, o));
                b.a = fmaxf(b.a, __shfl_xor_sync(0xffffffffu, b.a, o));
                b.L = fmaxf(b.L, __shfl_xor_sync(0xffffffffu, b.L, o));
            }
            b.r = r;
            if (lane == 0) c.super[blockIdx.x] = b;
        }
    }
    if (blockIdx.x == 0 && blockIdx.y == 0) {   // the scalars for the host
        __shared__ double tot[2][5];
        init_stats_total(ia, tot);
        if (threadIdx.x < kInitOut) {
            const int q = threadIdx.x;
            double v = 0;
            if (q < 2) {
                const int mb = ia.counter[2 + q];
                v = mb > 0 ? log2((double)__int_as_float(mb)) : -INFINITY;
            } else if (q == 2) {
                v = conv_scale(ia, tot, D);
            } else if (q < 6) {
                v = (double)ia.counter[q == 3 ? 0 : q];
            } else if (q == 6) {
                v = (double)__int_as_float(ia.counter[6]);
            } else {
                v = (double)ia.reach[4 * kReachBins];
            }
            ia.out[q] = v;
            if (ia.host) ia.host[q] = v;
        }
        for (int q = threadIdx.x; q < 4 * kReachBins; q += blockDim.x) {
            ia.out_reach[q] = (double)ia.reach[q];
            if (ia.host) ia.host[16 + q] = (double)ia.reach[q];
        }
    }
}

int launch_init(Context& c, const double* X, const double* XC, const double* Y, const double* YC)
{
    const int D = c.D, N = c.N, M = c.M;
    const size_t nd = (size_t)N * D, md = (size_t)M * D;
    const size_t bytes = sizeof(double) * (nd + nd * D + md + md * D);
    if (bytes > c.scratch_bytes) return set_error(DUGMA_ERR_STATE, "init: staging does not fit the scratch region");
    double* tmp = c.scratch;   // the FP64 inputs are staged in the (still unused) scratch region
    double *tX = tmp, *tXC = tX + nd, *tY = tXC + nd * D, *tYC = tY + md;
    cudaStream_t s = c.stream;
    int rc = DUGMA_OK;
    auto ck = [&](cudaError_t e, const char* what) {
        if (e != cudaSuccess && rc == DUGMA_OK)
            rc = set_error(DUGMA_ERR_CUDA, "init: %s failed: %s", what, cudaGetErrorString(e));
    };
    // pageable sources: the driver pipelines these through its own pinned buffers (a
    // host-side copy into a pinned ring of ours measured slower on the B200 host)
    ck(cudaMemcpyAsync(tX, X, sizeof(double) * nd, cudaMemcpyHostToDevice, s), "copy X");
    ck(cudaMemcpyAsync(tXC, XC, sizeof(double) * nd * D, cudaMemcpyHostToDevice, s), "copy X_C");
    ck(cudaMemcpyAsync(tY, Y, sizeof(double) * md, cudaMemcpyHostToDevice, s), "copy Y");
    ck(cudaMemcpyAsync(tYC, YC, sizeof(double) * md * D, cudaMemcpyHostToDevice, s), "copy Y_C");
    // the work counters and, behind them, the cell histograms and the samples of the reach
    ck(cudaMemsetAsync(c.counter, 0, sizeof(int) * (kCounters + 2 * (size_t)c.cells + kReachInts), s), "memset");
    InitArgs a{};
    a.cl[0] = {tX, tXC, N, c.x, c.xinv, c.wx, c.xcov, c.lwx, c.ux, c.init_L, c.init_place, c.hist,
               c.xpt, c.xtile, c.xsub, c.xsuper};
    a.cl[1] = {tY, tYC, M, c.y, c.yinv, c.wy, c.ycov, c.lwy, nullptr, c.init_L + N, c.init_place + N,
               c.hist + c.cells, c.ypt, c.ytile, c.ysub, c.ysuper};
    a.part = c.init_part;
    const int n = std::max(N, M);
    a.nb = std::min(kInitParts, std::max(1, (n + 255) / 256));
    a.bits = c.cell_bits;
    a.counter = c.counter;
    a.reach = c.hist + 2 * (size_t)c.cells;
    a.out = c.out;
    a.host = c.host_dev;
    static_assert(4 * kReachBins <= kMomSlots && 16 + 4 * kReachBins <= kHostDoubles, "staging of the samples");
    a.out_reach = c.mom;
    const dim3 g(std::min((n + 255) / 256, c.num_sms * 8), 2);
    const dim3 gs((n + kTile * kSuper - 1) / (kTile * kSuper), 2);
    init_stats_kernel<<<dim3(a.nb, 2), 256, 0, s>>>(a, D);
    if (D == 3)
        init_points_kernel<3><<<g, 256, 0, s>>>(a);
    else
        init_points_kernel<2><<<g, 256, 0, s>>>(a);
    const int scan_blocks = 2 + 2 * kReachPoints / 32;
    if (D == 3) {
        cell_scan_kernel<3><<<scan_blocks, 1024, 0, s>>>(a, c.cells);
        sort_points_kernel<3><<<g, 256, 0, s>>>(a);
        split_kernel<3><<<dim3((n + kRun - 1) / kRun, 2), kRun, 0, s>>>(a);
        bounds_kernel<3><<<gs, kTile * kSuper, 0, s>>>(a);
    } else {
        cell_scan_kernel<2><<<scan_blocks, 1024, 0, s>>>(a, c.cells);
        sort_points_kernel<2><<<g, 256, 0, s>>>(a);
        split_kernel<2><<<dim3((n + kRun - 1) / kRun, 2), kRun, 0, s>>>(a);
        bounds_kernel<2><<<gs, kTile * kSuper, 0, s>>>(a);
    }
    ck(cudaGetLastError(), "init kernels");
    if (!c.host_dev) {
        ck(cudaMemcpyAsync(c.host, c.out, kInitOut * sizeof(double), cudaMemcpyDeviceToHost, s), "copy back");
        ck(cudaMemcpyAsync(c.host + 16, c.mom, 4 * kReachBins * sizeof(double), cudaMemcpyDeviceToHost, s), "copy back");
    }
    ck(cudaStreamSynchronize(s), "sync");
    if (rc != DUGMA_OK) return rc;
    c.Lmax_x = std::isfinite(c.host[0]) ? c.host[0] : 0.0;
    c.Lmax_y = std::isfinite(c.host[1]) ? c.host[1] : 0.0;
    c.cscale = c.host[2];
    c.nonpd = (int)c.host[3];
    c.x_indef = c.ux ? (int)c.host[4] : N;
    c.y_indef = (int)c.host[5];
    c.inv_trace = (float)c.host[6];
    c.near_y = c.host[7] / (kReachPoints * kReachDraws);
    for (int q = 0; q < 4 * kReachBins; ++q) (&c.reach[0][0][0])[q] = (int)c.host[16 + q];
    return DUGMA_OK;
}

// ---------------------------------------------------------------------------
// Per-evaluation prologue.
//   y records: y' = R y + t in FP64 in the order of update_sig.cu:247-249 / compi.cu:784-786,
//              split into y'hi = float(y'), y'lo = float(y' - y'hi);
//              C'_j = R (s sym(Sigma_y_j^-1)) R^T (compi.cu:757-765) scaled by k = -1/2 log2 e
//              (layout 0: packed as is; layout 1: off-diagonals doubled for the Horner form);
//              lv_j = log2(w_j) - Lmax_y.
//   x records: x_i, lw_i and either k * s * sym(Sigma_x_i^-1) with doubled off-diagonals (Horner
//              form) or, when ux is given, sqrt(|k| s) U_i from the init-time Cholesky factor U_i
//              of sym(Sigma_x_i^-1) (Cholesky form: (sqrt(|k| s) U_i)^T (sqrt(|k| s) U_i) = |k| B_i).
// Rows past N / M are null records (lw = -inf, zero matrices): they contribute exactly 0.
// ---------------------------------------------------------------------------
// source i's record: x, the log2 weight and its matrix, either the Cholesky factor scaled by
// sqrt(-ks) (ux given) or k B in the Horner layout
template <int D>
__device__ __forceinline__ void source_record(int i, const float* __restrict__ x, const float* __restrict__ xinv,
                                              const float* __restrict__ lwx, int N, XRec* __restrict__ xrec,
                                              const double* __restrict__ ux, double ks)
{
    constexpr int NS = Sym<D>::N;
    XRec r;
    float xv[3] = {0, 0, 0}, bp[6] = {0, 0, 0, 0, 0, 0};
    float lw = -INFINITY;
    if (i < N) {
#pragma unroll
        for (int a = 0; a < D; ++a) xv[a] = x[(size_t)i * D + a];
        lw = lwx[i];
        if (lw != -INFINITY && ux) {
            const double r = sqrt(-ks);
#pragma unroll
            for (int k = 0; k < NS; ++k) bp[k] = __double2float_rn(r * ux[(size_t)i * NS + k]);
        } else if (lw != -INFINITY) {
#pragma unroll
            for (int k = 0; k < NS; ++k) {
                const int ra = Sym<D>::a(k), rb = Sym<D>::b(k);
                double b = 0.5 * ((double)xinv[(size_t)i * D * D + ra + D * rb] +
                                  (double)xinv[(size_t)i * D * D + rb + D * ra]);
                double v = ks * b;
                if (ra != rb) v = 2.0 * v;
                bp[k] = __double2float_rn(v);
            }
        }
    }
    r.v0 = make_float4(xv[0], xv[1], xv[2], lw);
    r.v1 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (D == 3) {
        r.v2 = make_float4(bp[0], bp[1], bp[2], bp[3]);
        r.v3 = make_float4(bp[4], bp[5], 0.f, 0.f);
    } else {
        r.v2 = make_float4(bp[0], bp[1], bp[2], 0.f);
        r.v3 = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    xrec[i] = r;
}

template <int D>
__global__ void prologue_kernel(const double* __restrict__ pose, const float* __restrict__ y,
                                const float* __restrict__ yinv, const float* __restrict__ lwy, int M, int M_pad,
                                int ylayout, YRec* __restrict__ yrec, float4* __restrict__ yp32,
                                const float* __restrict__ x, const float* __restrict__ xinv,
                                const float* __restrict__ lwx, int N, int N_pad, XRec* __restrict__ xrec,
                                const double* __restrict__ ux, int* __restrict__ reset_counter, const PoseBlock pv,
                                int use_pv, double* __restrict__ pose_out, int* __restrict__ reset_err,
                                double sparse_below)
{
    pdl_trigger();   // the pair kernel may be scheduled now; it waits for this kernel's writes
    constexpr int NS = Sym<D>::N;
    // the pose pv by value (use_pv; block 0 also writes it to pose_out, if given, for the kernels
    // that follow) or from pose
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (reset_counter) {
            reset_counter[0] = reset_counter[1] = 0;
            reset_counter[4] = (use_pv ? pv.v[kPoseSig] : pose[kPoseSig]) < sparse_below;
        }
        if (reset_err) *reset_err = 0;
        if (use_pv && pose_out)
#pragma unroll
            for (int k = 0; k < kPoseDoubles; ++k) pose_out[k] = pv.v[k];
    }
    double R[9], t[3];
#pragma unroll
    for (int k = 0; k < D * D; ++k) R[k] = use_pv ? pv.v[k] : pose[k];
#pragma unroll
    for (int a = 0; a < D; ++a) t[a] = use_pv ? pv.v[kPoseT + a] : pose[kPoseT + a];
    const double s = 1.0 / (use_pv ? pv.v[kPoseSig] : pose[kPoseSig]);
    const double ks = K_EXP2 * s;
    const int stride = gridDim.x * blockDim.x;
    // one thread per point: [0, M_pad) the targets, [M_pad, M_pad + N_pad) the sources
    for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < M_pad + N_pad; u += stride) {
        if (u >= M_pad) {
            source_record<D>(u - M_pad, x, xinv, lwx, N, xrec, ux, ks);
            continue;
        }
        const int j = u;
        YRec r;
        float hi[3] = {0, 0, 0}, lo[3] = {0, 0, 0}, cp[6] = {0, 0, 0, 0, 0, 0};
        float lv = -INFINITY;
        if (j < M) {
            double yj[3];
#pragma unroll
            for (int a = 0; a < D; ++a) yj[a] = (double)y[(size_t)j * D + a];
#pragma unroll
            for (int a = 0; a < D; ++a) {
                double v = R[a] * yj[0] + R[a + D] * yj[1];
                if (D == 3) v = v + R[a + 6] * yj[2];
                v = v + t[a];
                hi[a] = __double2float_rn(v);
                lo[a] = __double2float_rn(v - (double)hi[a]);
            }
            lv = lwy[j];
            if (lv != -INFINITY) {
                double A[D][D];
#pragma unroll
                for (int r0 = 0; r0 < D; ++r0)
#pragma unroll
                    for (int c0 = 0; c0 < D; ++c0)
                        A[r0][c0] = 0.5 * ((double)yinv[(size_t)j * D * D + r0 + D * c0] +
                                           (double)yinv[(size_t)j * D * D + c0 + D * r0]);
                double T[D][D];   // A R^T
#pragma unroll
                for (int r0 = 0; r0 < D; ++r0)
#pragma unroll
                    for (int c0 = 0; c0 < D; ++c0) {
                        double acc = 0;
#pragma unroll
                        for (int k = 0; k < D; ++k) acc = acc + A[r0][k] * R[c0 + D * k];
                        T[r0][c0] = acc;
                    }
#pragma unroll
                for (int k = 0; k < NS; ++k) {
                    const int ra = Sym<D>::a(k), rb = Sym<D>::b(k);
                    double acc = 0;
#pragma unroll
                    for (int q = 0; q < D; ++q) acc = acc + R[ra + D * q] * T[q][rb];
                    double v = ks * acc;
                    if ((ylayout & 1) && ra != rb) v = 2.0 * v;   // Horner layouts (1, 3)
                    cp[k] = __double2float_rn(v);
                }
            }
        }
        if (ylayout >= 2) {
            // paired layout: this target fills its half of pair record j / 2
            float f[16];
#pragma unroll
            for (int q = 0; q < 16; ++q) f[q] = 0.f;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                f[a] = -hi[a];
                f[4 + a] = -lo[a];
            }
            f[3] = lv;
            f[13] = -lv;
#pragma unroll
            for (int k = 0; k < NS; ++k) f[7 + k] = cp[k];
            float* base = reinterpret_cast<float*>(yrec) + (size_t)(j >> 1) * 32 + (j & 1);
#pragma unroll
            for (int q = 0; q < 16; ++q) base[(q >> 1) * 4 + (q & 1) * 2] = f[q];
        } else {
            r.v0 = make_float4(hi[0], hi[1], hi[2], lv);
            r.v1 = make_float4(lo[0], lo[1], lo[2], 0.f);
            if (D == 3) {
                r.v2 = make_float4(cp[0], cp[1], cp[2], cp[3]);
                r.v3 = make_float4(cp[4], cp[5], 0.f, 0.f);
            } else {
                r.v2 = make_float4(cp[0], cp[1], cp[2], 0.f);
                r.v3 = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            yrec[j] = r;
        }
        // nearest-neighbour records, two targets per 32 bytes with negated coordinates:
        // (-y0 2p, -y0 2p+1, -y1 2p, -y1 2p+1), (-y2 2p, -y2 2p+1, 0, 0); padding targets sit
        // at +inf so that no source ever picks them as a neighbour
        if (yp32) {
            float* pr = reinterpret_cast<float*>(yp32 + 2 * (j / 2));
            const int h = j & 1;
            for (int q = 0; q < 3; ++q) pr[2 * q + h] = j < M ? (q < D ? -hi[q] : 0.f) : -INFINITY;
            pr[6 + h] = 0.f;
        }
    }
}

// the search records of target j (the yp32 layout of prologue_kernel): two targets per 32 bytes,
// coordinates negated, padding targets at +inf.  With pt given, record j is target pt[j].idx (the
// spatial order), its index goes along, and the spheres of the target tiles and, behind them, super
// tiles at this pose go to `sphere`.
// The pose: pv by value (use_pv; block 0 also writes it to pose), else read from pose.
template <int D>
__global__ void nn_prologue_kernel(const PoseBlock pv, int use_pv, double* __restrict__ pose,
                                   const float* __restrict__ y, int M, int M_pad, float4* __restrict__ yp32,
                                   int* __restrict__ reset_counter, int* __restrict__ reset_err,
                                   const SortedPoint* __restrict__ pt, const Bound* __restrict__ tile,
                                   const Bound* __restrict__ super, float4* __restrict__ sphere)
{
    pdl_trigger();   // the search kernel may be scheduled now; it waits for this kernel's writes
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (reset_counter) reset_counter[0] = reset_counter[1] = reset_counter[2] = reset_counter[3] = 0;
        if (reset_err) *reset_err = 0;
        if (use_pv)
#pragma unroll
            for (int k = 0; k < kPoseDoubles; ++k) pose[k] = pv.v[k];
    }
    double R[9], t[3];
#pragma unroll
    for (int k = 0; k < D * D; ++k) R[k] = use_pv ? pv.v[k] : pose[k];
#pragma unroll
    for (int a = 0; a < D; ++a) t[a] = use_pv ? pv.v[kPoseT + a] : pose[kPoseT + a];
    const int stride = gridDim.x * blockDim.x;
    for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < M_pad; j += stride) {
        float hi[3] = {0, 0, 0};
        int id = 0x7fffffff;
        if (j < M) {
            const float* yj32 = pt ? pt[j].p : y + (size_t)j * D;
            if (pt) id = pt[j].idx;
            double yj[3];
#pragma unroll
            for (int a = 0; a < D; ++a) yj[a] = (double)yj32[a];
#pragma unroll
            for (int a = 0; a < D; ++a) {
                double v = R[a] * yj[0] + R[a + D] * yj[1];
                if (D == 3) v = v + R[a + 6] * yj[2];
                v = v + t[a];
                hi[a] = __double2float_rn(v);
            }
        }
        float* pr = reinterpret_cast<float*>(yp32 + 2 * (j / 2));
        const int h = j & 1;
        for (int q = 0; q < 3; ++q) pr[2 * q + h] = j < M ? (q < D ? -hi[q] : 0.f) : -INFINITY;
        pr[6 + h] = pt ? __int_as_float(id) : 0.f;
        if (pt && j < M && j % kTile == 0) {
            const float stretch = pose_stretch(R, D);
            sphere[j / kTile] = posed_sphere<D>(tile[j / kTile], R, t, stretch);
            if (j % (kTile * kSuper) == 0)   // (behind the tiles')
                sphere[(M + kTile - 1) / kTile + j / (kTile * kSuper)] =
                    posed_sphere<D>(super[j / (kTile * kSuper)], R, t, stretch);
        }
    }
}

// One block: the pose block from src (device-visible memory: the mapped pinned staging a captured
// graph reads at each launch) into pose, the error word zeroed.  The kernels that follow read the
// pose from device memory (every block reading the staging over the host link costs more).
__global__ void pose_in_kernel(const double* __restrict__ src, double* __restrict__ pose, int* __restrict__ err)
{
    if (threadIdx.x < kPoseDoubles) pose[threadIdx.x] = src[threadIdx.x];
    if (threadIdx.x == 0 && err) *err = 0;
}

int launch_pose_in(Context& c, const double* src, double* pose_dev, cudaStream_t s, bool reset_err)
{
    pose_in_kernel<<<1, 32, 0, s>>>(src, pose_dev, reset_err ? c.err : nullptr);
    DUGMA_CK(cudaGetLastError());
    return DUGMA_OK;
}

int launch_nn_prologue(Context& c, double* pose_dev, cudaStream_t s, const PoseBlock* pv, int* reset_counter,
                       int* reset_err, bool sorted)
{
    PoseBlock pb{};
    if (pv) pb = *pv;
    const int g = std::min((c.M_pad + 127) / 128, c.num_sms * 8);
    const SortedPoint* pt = sorted ? c.ypt : nullptr;
    auto fn = c.D == 3 ? nn_prologue_kernel<3> : nn_prologue_kernel<2>;
    fn<<<g, 128, 0, s>>>(pb, pv ? 1 : 0, pose_dev, c.y, c.M, c.M_pad, c.yp32, reset_counter, reset_err, pt, c.ytile,
                         c.ysuper, c.ysphere);
    DUGMA_CK(cudaGetLastError());
    return DUGMA_OK;
}

int launch_prologue(Context& c, const double* pose_dev, int ylayout, cudaStream_t s, bool xchol, int* reset_counter,
                    const PoseBlock* pv, double* pose_out, int* reset_err, double sparse_below)
{
    PoseBlock pb{};
    if (pv) pb = *pv;
    if (xchol && (!c.ux || c.x_indef > 0))
        return set_error(DUGMA_ERR_STATE, "Cholesky-form source records need a positive definite factor per source");
    const double* ux = xchol ? c.ux : nullptr;
    const int n = c.M_pad + c.N_pad;
    const int bs = 128;
    const int g = std::min((n + bs - 1) / bs, c.num_sms * 8);
    if (c.D == 3)
        prologue_kernel<3><<<g, bs, 0, s>>>(pose_dev, c.y, c.yinv, c.lwy, c.M, c.M_pad, ylayout, c.yrec, nullptr,
                                            c.x, c.xinv, c.lwx, c.N, c.N_pad, c.xrec, ux, reset_counter, pb,
                                            pv ? 1 : 0, pose_out, reset_err, sparse_below);
    else
        prologue_kernel<2><<<g, bs, 0, s>>>(pose_dev, c.y, c.yinv, c.lwy, c.M, c.M_pad, ylayout, c.yrec, nullptr,
                                            c.x, c.xinv, c.lwx, c.N, c.N_pad, c.xrec, ux, reset_counter, pb,
                                            pv ? 1 : 0, pose_out, reset_err, sparse_below);
    DUGMA_CK(cudaGetLastError());
    return DUGMA_OK;
}

}  // namespace dugma

// sparse.cuh -- one tile of sources against the target records that can reach it (sparse.cu, batch.cu).
#pragma once

#include "bodies.cuh"
#include "context.hpp"
#include "reach.cuh"

namespace dugma {

struct SparseArgs {
    ReachArgs reach;
    const XRec* xrec;      // by source index, Cholesky form
    const YRec2* yrec;     // by target index, pairs
    const float* wx;
    const double* pose;
    double wmax;           // 2^Lmax of the targets' weights
    int n_rec, words;      // records, words of their bitmap
    int tile_shift;        // log2 records per tile (FP32 sum of the energy)
    int chunk_rec;         // records per chunk (FP32 sums of the moments)
    double* rows;          // [N][8] contributions by source index
    double* dx;            // nullable: [N][D]
};

constexpr int kSparseChunk = 1024;  // most records a chunk may have (32 words of the bitmap)
constexpr int kSparseBatch = 8;     // records loaded together
// shared memory: reach tests, then per warp two batches of records, the chunk's list and the FP64 sums
// (there, and not in registers, so that 24 warps fit an SM: 67 us at 64K against 78 with 16 of them)
template <int NW>
struct SparseShape {
    static constexpr size_t kRec = NW * 2 * kSparseBatch * sizeof(YRec2), kList = NW * kSparseChunk * sizeof(uint16_t),
                            kSums = NW * 13 * 32 * sizeof(double);
    static constexpr size_t kFixed = (sizeof(ReachShared) + 15) / 16 * 16 + kRec + kList + kSums;
};

// The tile `group` of 32 sources, by the block's NW warps; the caller has zeroed the bitmap behind
// SparseShape::kFixed bytes of smem.
template <int D, bool GRAD, int NW>
__device__ __forceinline__ void sparse_tile(const SparseArgs& a, int group, unsigned char* smem)
{
    using S = SparseShape<NW>;
    using Body = PackedBody<D, 1, GRAD, true>;
    constexpr int NS = Sym<D>::N, NV = Body::NV;
    ReachShared& sh = *reinterpret_cast<ReachShared*>(smem);
    unsigned char* work = smem + (sizeof(ReachShared) + 15) / 16 * 16;
    uint32_t* bits = reinterpret_cast<uint32_t*>(smem + S::kFixed);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float(*rec)[kSparseBatch * 32] = reinterpret_cast<float(*)[kSparseBatch * 32]>(work) + 2 * warp;
    uint16_t* list = reinterpret_cast<uint16_t*>(work + S::kRec) + kSparseChunk * warp;

    const int pos = group * kTile + lane;
    const bool in = pos < a.reach.st.n;
    const int i = a.reach.st.pt[in ? pos : 0].idx;
    const bool marked = find_reach<D, NW, true>(a.reach, group, bits, sh);
    if (!__syncthreads_or(marked)) {   // nothing reaches these sources
        if (warp == 0 && in) {
#pragma unroll
            for (int v = 0; v < NV; ++v) a.rows[(size_t)i * 8 + v] = 0.0;
            if (GRAD && a.dx)
#pragma unroll
                for (int q = 0; q < D; ++q) a.dx[(size_t)i * D + q] = 0.0;
        }
        return;
    }
    Body body;
    {
        float x[3], b[6];
        load_xrec<D>(a.xrec[i], x, b);
#pragma unroll
        for (int q = 0; q < D; ++q) body.X[0][q] = make_float2(x[q], x[q]);
#pragma unroll
        for (int q = 0; q < NS; ++q) body.B[0][q] = make_float2(b[q], b[q]);
    }
    body.zero_all();
    // E, sum e1 u, sum e2 z, sum e2 z z^T per source
    double(*sums)[13][32] = reinterpret_cast<double(*)[13][32]>(work + S::kRec + S::kList);
#pragma unroll
    for (int q = 0; q < 13; ++q) sums[warp][q][lane] = 0.0;
    const float* recs = reinterpret_cast<const float*>(a.yrec);
    for (int base = warp * a.chunk_rec; base < a.n_rec; base += NW * a.chunk_rec) {
        // the chunk's marked records, ascending
        const int nw = (min(a.chunk_rec, a.n_rec - base) + 31) / 32;
        uint32_t w = lane < nw ? bits[base / 32 + lane] : 0u;
        if (!__any_sync(0xffffffffu, w != 0)) continue;
        int at = __popc(w);
        const int own = at;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, at, o);
            if (lane >= o) at += u;
        }
        const int n = __shfl_sync(0xffffffffu, at, 31);
        at -= own;
        while (w) {
            list[at++] = (uint16_t)(32 * lane + __ffs(w) - 1);
            w &= w - 1;
        }
        __syncwarp();
        float v[kSparseBatch];
        auto fetch = [&](int b) {
#pragma unroll
            for (int k = 0; k < kSparseBatch; ++k)
                v[k] = recs[(size_t)(base + list[min(b + k, n - 1)]) * 32 + lane];
        };
        fetch(0);
        int tile = list[0] >> a.tile_shift;
        for (int b = 0, buf = 0; b < n; b += kSparseBatch, buf ^= 1) {
#pragma unroll
            for (int k = 0; k < kSparseBatch; ++k) rec[buf][32 * k + lane] = v[k];
            __syncwarp();
            if (b + kSparseBatch < n) fetch(b + kSparseBatch);
            const YRec2* r = reinterpret_cast<const YRec2*>(rec[buf]);
            const int m = min(kSparseBatch, n - b);
            for (int k = 0; k < m; ++k) {
                const int t = list[b + k] >> a.tile_shift;
                if (t != tile) {
                    body.fold();
                    tile = t;
                }
                body.consume(r[k], 0);
            }
        }
        body.fold();
        if (GRAD) {
#pragma unroll
            for (int q = 0; q < D; ++q) {
                sums[warp][1 + q][lane] += (double)body.S1[0][q].x + (double)body.S1[0][q].y;
                sums[warp][4 + q][lane] += (double)body.D2[0][q].x + (double)body.D2[0][q].y;
                body.S1[0][q] = body.D2[0][q] = make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int q = 0; q < NS; ++q) {
                sums[warp][7 + q][lane] += (double)body.Q2[0][q].x + (double)body.Q2[0][q].y;
                body.Q2[0][q] = make_float2(0.f, 0.f);
            }
        }
        __syncwarp();   // (the list is rewritten)
    }
    // the warps' sums, in order
    sums[warp][0][lane] = body.E64[0];
    __syncthreads();
    if (warp > 0 || !in) return;
    auto total = [&](int q) {
        double s = sums[0][q][lane];
#pragma unroll
        for (int u = 1; u < NW; ++u) s += sums[u][q][lane];
        return s;
    };
    const double sg = 1.0 / a.pose[kPoseSig];
    const double wt = (double)a.wx[i] * (D == 3 ? sg * sg * sg : sg * sg) * a.wmax;
    double acc[NV], dx[3] = {0, 0, 0};
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = 0.0;
    acc[0] = wt * total(0);
    if constexpr (GRAD) if (acc[0] != 0.0) {   // (no term, no moments)
        double s1[3], d2[3], q2[6];
#pragma unroll
        for (int q = 0; q < D; ++q) {
            s1[q] = total(1 + q);
            d2[q] = total(4 + q);
        }
#pragma unroll
        for (int q = 0; q < NS; ++q) q2[q] = total(7 + q);
        double t[3] = {0, 0, 0};
#pragma unroll
        for (int q = 0; q < D; ++q) t[q] = a.pose[kPoseT + q];
        chol_contract<D>(wt, body.B[0], body.X[0], t, s1, d2, q2, acc, dx);
    }
    if (GRAD && a.dx)
#pragma unroll
        for (int q = 0; q < D; ++q) a.dx[(size_t)i * D + q] = dx[q];
#pragma unroll
    for (int v = 0; v < NV; ++v) a.rows[(size_t)i * 8 + v] = acc[v];
}

}  // namespace dugma

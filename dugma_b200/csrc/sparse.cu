// sparse.cu -- the REF energy and its adjoint over the pairs that can count.
//
// Where the covariances follow the point spacing, all but a few of a source's pairs have both
// exponentials below the FP32 flush (reach.cuh), and the all-pairs kernels spend their time adding
// zeros.  Here a block takes one tile of 32 sources in spatial order (one per lane, the same in its
// warps), marks the target records that can reach one of them, and evaluates those alone.
//
// The sums are those of the all-pairs kernels, term for term: a source's records are taken in index
// order, its energy summed in FP32 over each of their tiles and its moments over each of their chunks,
// by the same body on the same records; the terms left out are exact zeros.  Chunks are split over
// the warps (chunk c to warp c mod their number), the chunks' sums added in FP64 per source, and the sources'
// contributions to E and the gradient go to rows by source index that a second kernel adds in fixed
// order, so neither the spatial order nor the schedule shows in a result.
//
// Bound by the latency and issue slots of the search: the tests of super tiles, tiles and points are
// some 10K instructions a tile of sources, the few dozen records after it (loaded 8 ahead, coalesced,
// and broadcast from shared memory) less.  Measured on one B200, adjoint kernel, all pairs -> here:
// 65536 x 65536 harmonic 6300 -> 40 us; 240000 x 240000 depth views 83500 -> 354 us; 16384 x 16384 sphere
// 370 -> 25 us; 20011 x 20011 in 2D 370 -> 18 us.
#include <algorithm>
#include <cmath>
#include <mutex>

#include "sparse.cuh"

namespace dugma {

// Eight warps a tile: one problem's few heavy tiles (outliers, edges of a depth map) end the launch.  2 / 4 / 8
// warps, adjoint kernel on one B200 (before the packed tests of reach.cuh): 65536 x 65536 73 / 54 / 48 us; 240000
// depth 627 / 490 / 411; 6000 with outliers - / 23 / 17.5; 2D 20011 - / 18.5 / 16.
constexpr int kSparseWarps = 8;
template <int D, bool GRAD, int NW>
__global__ void __launch_bounds__(32 * NW, 24 / NW) sparse_kernel(SparseArgs a, const int* go)
{
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t* bits = reinterpret_cast<uint32_t*>(smem + SparseShape<NW>::kFixed);
    pdl_trigger();   // a dependent of the prologue; the rows' sum is one of this kernel
    for (int w = threadIdx.x; w < a.words; w += 32 * NW) bits[w] = 0;
    pdl_wait();
    if (go && !*go) return;   // (nullable: nothing is done unless set)
    sparse_tile<D, GRAD, NW>(a, blockIdx.x, smem);
}

// out[v] = sum of rows[i][v]: per-block partials over contiguous slices, then the block that finishes
// last adds the partials, all in fixed order (deterministic).  host_out as in reduce_items_kernel.
__global__ void __launch_bounds__(256) reduce_rows_kernel(const double* rows, int n, int nv, double* part, int* ticket,
                                                          double* out, double* host_out, const int* err,
                                                          const int* go)
{
    pdl_wait();
    if (go && !*go) return;
    __shared__ double red[8][8];
    __shared__ bool last;
    const int v = threadIdx.x & 7, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto block_total = [&](double s) {   // threads 0..7: the block's sum of value v
        s += __shfl_xor_sync(0xffffffffu, s, 8);
        s += __shfl_xor_sync(0xffffffffu, s, 16);
        __syncthreads();
        if (lane < 8) red[warp][lane] = s;
        __syncthreads();
        if (threadIdx.x < 8) {
            s = red[0][v];
            for (int w = 1; w < 8; ++w) s += red[w][v];
        }
        return s;
    };
    const int per = (n + gridDim.x - 1) / gridDim.x;
    const int b0 = blockIdx.x * per, b1 = min(n, b0 + per);
    double s = 0;
    if (v < nv)
#pragma unroll 8
        for (int i = b0 + (threadIdx.x >> 3); i < b1; i += 32) s += rows[(size_t)i * 8 + v];
    s = block_total(s);
    if (threadIdx.x < 8) part[blockIdx.x * 8 + v] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    s = 0;
    for (int b = threadIdx.x >> 3; b < (int)gridDim.x; b += 32) s += __ldcg(part + b * 8 + v);
    s = block_total(s);
    if (threadIdx.x < nv) {
        out[v] = s;
        if (host_out) host_out[v] = s;
    }
    if (threadIdx.x == 0 && host_out) host_out[nv] = (double)*err;
}

// the rows c.scratch holds (N x 8) into out_dev; the blocks' partials go behind them
int reduce_rows(Context& c, int nv, double* out_dev, cudaStream_t s, double* host_out, const int* go)
{
    double* rows = c.scratch;
    DUGMA_CK(launch_dependent(c.pdl, reduce_rows_kernel, std::min(kRowBlocks, (c.N + 255) / 256), 256, 0, s,
                              (const double*)rows, c.N, nv, rows + (size_t)c.N * 8, c.counter + 1, out_dev, host_out,
                              (const int*)c.err, go));
    return DUGMA_OK;
}

// Which of a context's evaluations go this way: those with a sigma below this (0: none).  With f the share
// of a surface that a pair of mean variance v reaches, f = 127.5 sig v / (4 |k| r^2) for clouds of radius
// r (r^2: mean squared distance to the mean, of the smaller one), an evaluation is sparse where f is
// under `most`, a line drawn from timings of both ways at 1000 - 32000 points on six kinds of cloud, f
// from 5e-4 to 0.2 (one B200, us a call, all pairs / sparse; the outliers' clouds, whose variances differ
// most, cross first):
//   energy_grad 3000: 46 / 47-52 at any f;  4500: 91 / 52-82 at 6e-3, 91 / 69-145 at 0.02;  16000:
//     487 / 94-304 at 6e-3, 487 / 146-611 at 0.02;  32000: 1608 / 162-736, 1608 / 319-1740
//   compi 4500: 96 / 68-83 at 2e-3, 96 / 77-106 at 6e-3;  6500: 141 / 104-140 at 6e-3;  16000: 622 /
//     154-432 at 6e-3, 622 / 246-877 at 0.02
//   CONV 4500: 121 / 83-96 at 5e-4;  6500: 171 / 121-145 at 2e-3;  16000: 762 / 198-427 at 2e-3,
//     762 / 281-828 at 6e-3
//   batches, many problems at once: 700 points 246 / 162-213 at 6e-3, 246 / 192-267 at 0.02;  1000: 417 /
//     264-362 at 0.02, 417 / 340-552 at 0.06;  8000: 837 / 276-561 at 0.02
double sparse_sigma(const Context& c, SparseUse use)
{
    if (c.x_indef > 0 || c.y_indef > 0 || !c.ux || !c.xpt || c.no_alloc || c.all_pairs || c.M > kSparseMaxTargets)
        return 0.0;
    const double pairs = (double)c.N * c.M, grow = std::pow(std::max(1.0, pairs / 4e7), 1.0 / 6);
    double most = 0.0;
    switch (use) {
    case SparseUse::energy: most = pairs < 12e6 ? 0.0 : (pairs < 2e7 ? 2e-3 : 6e-3 * grow); break;
    case SparseUse::coef: most = pairs < kSparseCoefMinPairs || c.N > kSparseMaxTargets ? 0.0 : (pairs < 4e7 ? 2e-3 : 6e-3 * grow); break;
    case SparseUse::conv: most = pairs < 2e7 ? 0.0 : (pairs < 4e7 ? 5e-4 : 2e-3 * grow); break;
    case SparseUse::batch: most = pairs < 4e5 ? 0.0 : (pairs < 1e6 ? 6e-3 : 2e-2); break;
    }
    const double v = (c.trace_x + c.trace_y) / (2.0 * c.D), r2 = std::min(c.rho2_x, c.rho2_y);
    const double s = most * 4.0 * r2 * -K_EXP2 / ((double)kFlushExp * v);
    return s > 0 && std::isfinite(s) ? s : 0.0;
}

template <int D, bool GRAD>
static int sparse_impl(Context& c, const double* pose_dev, int tile_rec, int chunk_rec, double* out_dev,
                       double* dEdx_dev, cudaStream_t s, double* host_out, const int* go)
{
    constexpr int NW = kSparseWarps;
    static std::mutex mu;
    static bool done[64];
    const size_t most = SparseShape<NW>::kFixed + kSparseMaxTargets / 64 * sizeof(uint32_t);
    {
        std::lock_guard<std::mutex> lk(mu);
        if (c.dev < 64 && !done[c.dev]) {
            DUGMA_CK(cudaFuncSetAttribute(sparse_kernel<D, GRAD, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)most));
            done[c.dev] = true;
        }
    }
    const size_t rows = (size_t)c.N * 8;
    DUGMA_RET(c.ensure_scratch(sizeof(double) * (rows + kRowBlocks * 8)));
    SparseArgs a{};
    a.reach = {{c.xpt, c.xtile, c.xsub, c.xsuper, c.N}, {c.ypt, c.ytile, c.ysub, c.ysuper, c.M}, pose_dev, c.inv_trace};
    a.xrec = c.xrec;
    a.yrec = reinterpret_cast<const YRec2*>(c.yrec);
    a.wx = c.wx;
    a.pose = pose_dev;
    a.wmax = std::exp2(c.Lmax_y);
    a.n_rec = c.M_pad / 2;
    a.words = (a.n_rec + 31) / 32;
    while (1 << a.tile_shift < tile_rec) ++a.tile_shift;
    a.chunk_rec = chunk_rec;
    a.rows = c.scratch;
    a.dx = dEdx_dev;
    const int grid = (c.N + kTile - 1) / kTile;
    DUGMA_RET(timing_begin(c, s));
    DUGMA_CK(launch_dependent(c.pdl, sparse_kernel<D, GRAD, NW>, grid, 32 * NW,
                              SparseShape<NW>::kFixed + sizeof(uint32_t) * a.words, s, a, go));
    DUGMA_RET(timing_end(c, s));
    return reduce_rows(c, GRAD ? 1 + (D == 3 ? 6 : 3) : 1, out_dev, s, host_out, go);
}

int sparse_launch(Context& c, const double* pose_dev, bool grad, int tile_rec, int chunk_rec, double* out_dev,
                  double* dEdx_dev, cudaStream_t s, double* host_out, const int* go)
{
    if (chunk_rec > kSparseChunk || chunk_rec % 32 || tile_rec < 32 || (tile_rec & (tile_rec - 1)))
        return set_error(DUGMA_ERR_STATE, "sparse evaluation: chunks of %d records, tiles of %d", chunk_rec, tile_rec);
    auto fn = c.D == 3 ? (grad ? sparse_impl<3, true> : sparse_impl<3, false>)
                       : (grad ? sparse_impl<2, true> : sparse_impl<2, false>);
    return fn(c, pose_dev, tile_rec, chunk_rec, out_dev, dEdx_dev, s, host_out, go);
}

}  // namespace dugma

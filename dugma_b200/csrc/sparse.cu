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

// Which of a context's evaluations go this way: those with a sigma below a line (0: none) where the
// modelled times of both ways meet.  All pairs: t0 + tp N M + tn (N + M).  The sparse pass, with f the
// share of pairs in reach at that sigma (init's samples, sample_reach) and g the same of the points that
// reach more (weighted by what they reach):
//   s0 + sn (N + M) + |(a N C(f), b C(g))|,     C(f) = M (F + y G)
//   F = min(1, u f, (f^(1/e) + (32/N)^(1/e))^e)                     records that one tile of 32 sources marks
//   G = min(1, x (f^(1/e) + (32/N)^(1/e) + (32/M)^(1/e))^e)         tiles that it searches
// a N C: all blocks at the GPU's rate; b C: one block alone, which is what few sources and uneven densities
// come down to.  The coefficients search from both sides.  A batch's problems fill the GPU together: only
// the terms in N and M count.
// The constants are fits to calls timed both ways on one B200 (us): 12 kinds of cloud (surfaces, volumes,
// curves, discs, outliers, points at one place, clusters of 1 % of the radius), 1000 - 64000 points, and 64
// - 4000 against 20000 - 600000 either way round, f from 1e-4 to 0.35; batches of 8 and 192 evaluations,
// 250 - 8000 points.  Of 2562 cases a use, slower than all pairs by more than 10 % with these lines: at most
// gradient 40 (worst 1.6 times), energy 54 (2.5), CONV 29 (1.7), compi 41 (1.7), batch 13 of 702 (1.4),
// nearly all of them clusters; by the mean variance over the mean squared radius alone, which knows neither of clusters nor
// of few sources, 360 - 470 of 1575 (worst 92 times).
struct SparseCost {
    double t0, tp, tn;                        // all pairs
    double s0, sn, a, b, y, x, u, e;          // the sparse pass
    double margin;                            // sparse where its time is below this share of all pairs'
};
static const SparseCost& sparse_cost(SparseUse use, int D)
{
    static const SparseCost cost[kSparseUses][2] = {
        {{31.2, 9.73e-7, 9.6e-5, 29.1, 3.6e-4, 2.32e-6, 0.0187, 0.0904, 5.01, 6.09, 2.0, 0.95},
         {31.2, 1.59e-6, 9.6e-5, 30.0, 4.46e-4, 3.28e-6, 0.0186, 0.134, 3.33, 10.9, 3.0, 0.95}},
        {{25.9, 5.83e-7, 1.48e-4, 28.6, 3.05e-4, 2.07e-6, 0.0173, 0.0871, 4.9, 4.48, 1.76, 1.0},
         {25.9, 9.12e-7, 1.48e-4, 31.7, 3.63e-4, 2.96e-6, 0.0193, 0.0905, 3.44, 8.44, 3.0, 1.0}},
        {{50.7, 1.54e-6, 1.64e-4, 50.2, 2.27e-4, 3.92e-6, 0.0245, 0.419, 1.95, 11.6, 2.71, 0.95},
         {50.7, 2.75e-6, 1.64e-4, 54.6, 2.93e-4, 5.78e-6, 0.029, 0.526, 3.09, 11.1, 3.0, 0.95}},
        {{43.2, 1.03e-6, 1.93e-3, 32.4, 1.06e-3, 1.5e-6, 0.0215, 0.129, 2.1, 9.37, 3.0, 0.9},
         {43.2, 1.83e-6, 1.93e-3, 33.9, 2.03e-3, 3.36e-6, 0.0377, 0.0904, 3.41, 7.96, 3.0, 0.9}},
        {{0, 7.76e-7, 1.54e-4, 0, 5.12e-5, 8.85e-7, 0, 2.0, 1.0, 1.0, 1.61, 0.85},
         {0, 1.45e-6, 1.54e-4, 0, 3.53e-5, 3.19e-6, 0, 0.483, 2.36, 3.95, 1.88, 0.85}},
    };
    return cost[(int)use][D == 3];
}

// f and g where q < 2^x is in reach; the sampled sums are interpolated between octaves as powers of q
static void reach_shares(const Context& c, double x, double* f, double* g)
{
    const double u = std::min(std::max(x + (127 - kReachExp) - 1.0, 0.0), kReachBins - 2.0);   // (bin b ends at 2^(b - 43))
    const int b = (int)u;
    double share[2], uneven = 0.0;
    for (int k = 0; k < 2; ++k) {
        double at[2], two[2];
        for (int q = 0; q < 2; ++q) {
            const int n = c.reach[k][0][b + q];
            at[q] = std::log((n + 0.25) / (kReachPoints * kReachDraws));
            two[q] = n > 0 ? c.reach[k][1][b + q] / ((kReachDraws - 1.0) * n) : 0.0;
        }
        share[k] = std::exp(at[0] + (u - b) * (at[1] - at[0]));
        uneven = std::max(uneven, two[0] + (u - b) * (two[1] - two[0]));
    }
    *f = std::sqrt(share[0] * share[1]);   // (pairs of two clouds: at most this, by Cauchy-Schwarz)
    *g = std::max(uneven, *f);
}

struct SparseTime {
    const SparseCost& t;
    const bool both_sides;
    const double N, M, r, pn, pm;
    SparseTime(const SparseCost& cost, SparseUse use, double n, double m)
        : t(cost), both_sides(use == SparseUse::coef), N(n), M(m), r(1.0 / cost.e),
          pn(std::pow(std::min(1.0, 32.0 / n), r)), pm(std::pow(std::min(1.0, 32.0 / m), r))
    {
    }
    double block(double h, double p_st, double m) const   // C(h)
    {
        const double p = std::pow(h, r);
        const double F = std::min({1.0, t.u * h, std::pow(p + p_st, t.e)});
        const double G = std::min(1.0, t.x * std::pow(p + pn + pm, t.e));
        return m * (F + t.y * G);
    }
    double at(double f, double g) const
    {
        double all = N * block(f, pn, M), one = t.b > 0 ? block(g, pn, M) : 0.0;
        if (both_sides) {
            all += M * block(f, pm, N);
            one = std::max(one, block(g, pm, N));
        }
        return t.s0 + t.sn * (N + M) + std::hypot(t.a * all, t.b * one);
    }
};

double sparse_sigma(const Context& c, SparseUse use)
{
    if (c.x_indef > 0 || c.y_indef > 0 || !c.ux || !c.xpt || c.no_alloc || c.all_pairs || c.M > kSparseMaxTargets)
        return 0.0;
    const double N = c.N, M = c.M;
    if (use != SparseUse::batch && N * M < kSparseMinPairs) return 0.0;
    if (use == SparseUse::coef && (N * M < kSparseCoefMinPairs || c.N > kSparseMaxTargets)) return 0.0;
    if (use == SparseUse::batch && N * M < kSparseBatchMinPairs) return 0.0;
    double& line = c.sparse_line[(int)use];
    if (line >= 0) return line;
    const SparseCost& t = sparse_cost(use, c.D);
    const double limit = t.margin * (t.t0 + t.tp * N * M + t.tn * (N + M));
    const SparseTime time(t, use, N, M);
    auto sparse_at = [&](double x) {
        double f, g;
        reach_shares(c, x, &f, &g);
        return time.at(f, g) < limit;
    };
    double lo = kReachExp - 127 + 1.0, hi = lo + kReachBins - 2.0;   // log2 of q; the time grows with it
    if (!sparse_at(lo)) return line = 0.0;
    if (sparse_at(hi)) {
        lo = hi;
    } else {
        for (int k = 0; k < 13; ++k) {   // (to 1 %)
            const double x = 0.5 * (lo + hi);
            (sparse_at(x) ? lo : hi) = x;
        }
    }
    return line = std::exp2(lo) * -K_EXP2 / (double)kFlushExp;   // q < 127.5 sig / |k|
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

// nn.cu -- exact nearest neighbours and sigma (the update_sig plugin).
//
// The reference computes, for every x_i, min_j |x_i - (R y_j + t)|^2 / D quantised to
// 1e-6 as an unsigned int with shared and global atomicMin, then a FP32 tree sum
// (update_sig.cu:181-269, 272-315, 384-385).  Here:
//   y'_j = float(FP64(R y_j + t))               (update_sig.cu:247-252, written by the prologue)
//   d    = x_i - y'_j in FP32,  d2 = fmaf(dz,dz, fmaf(dy,dy, dx*dx))
// Target records hold two targets each, coordinates negated (d = x + (-y') is the same FP32
// value), interleaved so that the search kernels evaluate both with f32x2 operations.
//   the k smallest (d2, j) in lexicographic order are kept in registers (ties -> lowest j)
// All rows: the pruned search in spatial order (nn_prune_kernel).  Row ranges, pinned shapes and very uneven
// sizes (nn_pruned): all pairs, the targets streamed by bulk copy like the energy kernels and target chunks merged in
// index order afterwards.  Either is exact and deterministic.  sigma is then
//   exact:      sum_i d2min_i / (D N) in FP64
//   quantised:  sum_i rn_u32(fl32(d2min_i / D) * 1e6) / 1e6 / N   (the reference's value)
#include <cmath>

#include "context.hpp"
#include "pairs.cuh"
#include "spatial.cuh"

namespace dugma {

template <int D, int IPT_, int K>
struct NNBody {
    using StreamRec = NNRec2;
    static constexpr int IPT = IPT_;
    static constexpr int NV = 1;
    float2 X[IPT][D];   // source coordinates, duplicated in both halves
    float bd[IPT][K];
    int bi[IPT][K];
    int row[IPT];

    __device__ void setup(const PairArgs&) {}
    __device__ void load_src(const PairArgs& a, int ii, int i)
    {
        const float* xs = static_cast<const float*>(a.xrec);
        row[ii] = i < a.i_end ? i : -1;
#pragma unroll
        for (int q = 0; q < D; ++q) {
            const float v = i < a.i_end ? xs[(size_t)i * D + q] : 0.f;
            X[ii][q] = make_float2(v, v);
        }
    }
    __device__ void zero_all()
    {
#pragma unroll
        for (int ii = 0; ii < IPT; ++ii)
#pragma unroll
            for (int q = 0; q < K; ++q) { bd[ii][q] = INFINITY; bi[ii][q] = 0x7fffffff; }
    }
    // both targets of a record in one f32x2 sequence (per half the FP32 operations of the
    // reference: d = x + (-y'), d2 = fmaf(dz,dz, fmaf(dy,dy, dx*dx))), then one test per source
    // of the nearer of the two against its k-th distance; the rare insertions take the targets
    // in index order, so ties keep the lower j
    __device__ __forceinline__ void consume(const NNRec2& r, int jp)
    {
        const float2 n0 = make_float2(r.a.x, r.a.y), n1 = make_float2(r.a.z, r.a.w), n2 = make_float2(r.b.x, r.b.y);
        float2 dd[IPT];
        bool hit = false;
#pragma unroll
        for (int ii = 0; ii < IPT; ++ii) {
            const float2 d0 = fadd2(X[ii][0], n0), d1 = fadd2(X[ii][1], n1);
            if (D == 3) {
                const float2 d2 = fadd2(X[ii][2], n2);
                dd[ii] = ffma2(d2, d2, ffma2(d1, d1, fmul2(d0, d0)));
            } else {
                dd[ii] = ffma2(d1, d1, fmul2(d0, d0));
            }
            hit |= fminf(dd[ii].x, dd[ii].y) < bd[ii][K - 1];
        }
        // one branch per record for all the sources: the distance arithmetic above stays
        // branch-free and schedules like the distance-only kernel
        if (hit) {
#pragma unroll
            for (int ii = 0; ii < IPT; ++ii) {
                insert(ii, dd[ii].x, 2 * jp);
                insert(ii, dd[ii].y, 2 * jp + 1);
            }
        }
    }
    __device__ __forceinline__ void insert(int ii, float dd, int j)
    {
        if (!(dd < bd[ii][K - 1])) return;
        // sorted insertion; strict comparisons keep the earlier index first on ties
#pragma unroll
        for (int q = K - 1; q > 0; --q) {
            const bool shift = dd < bd[ii][q - 1];
            const bool place = !shift && dd < bd[ii][q];
            bd[ii][q] = shift ? bd[ii][q - 1] : (place ? dd : bd[ii][q]);
            bi[ii][q] = shift ? bi[ii][q - 1] : (place ? j : bi[ii][q]);
        }
        if (dd < bd[ii][0]) { bd[ii][0] = dd; bi[ii][0] = j; }
    }
    __device__ void fold() {}
    __device__ void finish(const PairArgs& a, int jc, double (&)[NV])
    {
        // partial lists for this target chunk: h_part as [n_jc][rows][K] (d2 float, idx int) pairs
        const int rows = a.i_end - a.i0;
        float2* out = reinterpret_cast<float2*>(a.h_part);
#pragma unroll
        for (int ii = 0; ii < IPT; ++ii) {
            if (row[ii] < 0) continue;
            float2* o = out + ((size_t)jc * rows + (row[ii] - a.i0)) * K;
#pragma unroll
            for (int q = 0; q < K; ++q) o[q] = make_float2(bd[ii][q], __int_as_float(bi[ii][q]));
        }
    }
};

// Nearest squared distance only (sigma): both targets of a record in one f32x2 sequence, the
// same FP32 operations as NNBody, a running minimum per half.
template <int D, int IPT_>
struct NNMinBody {
    using StreamRec = NNRec2;
    static constexpr int IPT = IPT_;
    static constexpr int NV = 1;
    float2 X[IPT][D];
    float2 bd[IPT];
    int row[IPT];

    __device__ void setup(const PairArgs&) {}
    __device__ void load_src(const PairArgs& a, int ii, int i)
    {
        const float* xs = static_cast<const float*>(a.xrec);
        row[ii] = i < a.i_end ? i : -1;
#pragma unroll
        for (int q = 0; q < D; ++q) {
            const float v = i < a.i_end ? xs[(size_t)i * D + q] : 0.f;
            X[ii][q] = make_float2(v, v);
        }
    }
    __device__ void zero_all()
    {
#pragma unroll
        for (int ii = 0; ii < IPT; ++ii) bd[ii] = make_float2(INFINITY, INFINITY);
    }
    __device__ __forceinline__ void consume(const NNRec2& r, int)
    {
        const float2 n0 = make_float2(r.a.x, r.a.y), n1 = make_float2(r.a.z, r.a.w), n2 = make_float2(r.b.x, r.b.y);
#pragma unroll
        for (int ii = 0; ii < IPT; ++ii) {
            const float2 d0 = fadd2(X[ii][0], n0), d1 = fadd2(X[ii][1], n1);
            float2 dd;
            if (D == 3) {
                const float2 d2 = fadd2(X[ii][2], n2);
                dd = ffma2(d2, d2, ffma2(d1, d1, fmul2(d0, d0)));
            } else {
                dd = ffma2(d1, d1, fmul2(d0, d0));
            }
            bd[ii].x = fminf(bd[ii].x, dd.x);
            bd[ii].y = fminf(bd[ii].y, dd.y);
        }
    }
    __device__ void fold() {}
    __device__ void finish(const PairArgs& a, int jc, double (&)[NV])
    {
        const int rows = a.i_end - a.i0;
        float2* out = reinterpret_cast<float2*>(a.h_part);
#pragma unroll
        for (int ii = 0; ii < IPT; ++ii) {
            if (row[ii] < 0) continue;
            out[(size_t)jc * rows + (row[ii] - a.i0)] = make_float2(fminf(bd[ii].x, bd[ii].y), __int_as_float(0));
        }
    }
};

// merge the per-chunk sorted lists in chunk (= index) order
template <int K>
__global__ void nn_merge_kernel(const float2* __restrict__ part, int n_jc, int rows, int k_out, int* __restrict__ idx,
                                float* __restrict__ d2, float* __restrict__ dmin)
{
    pdl_trigger();   // a dependent of the search kernel; the sigma sums (if any) dependents of this one
    pdl_wait();
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        float bd[K];
        int bi[K];
#pragma unroll
        for (int q = 0; q < K; ++q) { bd[q] = INFINITY; bi[q] = 0x7fffffff; }
        for (int c = 0; c < n_jc; ++c) {
            const float2* p = part + ((size_t)c * rows + r) * K;
            for (int e = 0; e < K; ++e) {
                const float dd = p[e].x;
                const int j = __float_as_int(p[e].y);
                if (!(dd < bd[K - 1])) break;   // lists are sorted: nothing further can enter
#pragma unroll
                for (int q = K - 1; q > 0; --q) {
                    const bool shift = dd < bd[q - 1];
                    const bool place = !shift && dd < bd[q];
                    bd[q] = shift ? bd[q - 1] : (place ? dd : bd[q]);
                    bi[q] = shift ? bi[q - 1] : (place ? j : bi[q]);
                }
                if (dd < bd[0]) { bd[0] = dd; bi[0] = j; }
            }
        }
        if (idx)
            for (int q = 0; q < k_out; ++q) {
                idx[(size_t)r * k_out + q] = bi[q];
                d2[(size_t)r * k_out + q] = bd[q];
            }
        if (dmin) dmin[r] = bd[0];
    }
}

// ---------------------------------------------------------------------------
// The pruned search: one block per tile of 32 sources (one per lane, the same in each of its NW
// warps), the targets' tiles split round-robin over the warps.  A warp first searches the tile nearest
// to one of the sources' subgroups, then each of its tiles whose super tile and whose own sphere are
// not farther than the worst of the lanes' k-th distances (group against sphere, then sources
// against sphere), the warps sharing each lane's best k-th distance.  The distances are the FP32
// operations of the all-pairs kernels and ties go to the lowest index, so the results are theirs bit
// for bit: a tile is skipped only when every target in it is strictly farther, with 1e-5 to spare for
// the roundings of the tests (and a sphere or source that is not finite skips nothing).
// Bound by latency, a chain of dependent tile searches: a source needs 7-12 tiles of 32 targets instead
// of all.  So a tile is brought in by one coalesced load (16 bytes a lane) that overlaps the search
// before it and is then broadcast from shared memory (32 uniform loads from L2 took twice as long),
// eight warps share the tiles of a group where a block per SM is all there is, and where many spheres
// pass the group's test they are filtered 32 at a time against the sources, not one by one.
// Measured on one B200, all pairs -> pruned: nearest distance 65536 x 65536 922 -> 29 us (update_sig
// 931 -> 52 us a call), 4501 x 3907 9.5 -> 8.2 us and no merge or sums after it (26 -> 8.2 us); 8 nearest
// of 30000 x 28001 660 -> 53 us.  The all-pairs kernels stay for row ranges and pinned shapes.
// ---------------------------------------------------------------------------
struct PruneArgs {
    const SortedPoint* xpt;
    const Bound *xtile, *xsub;
    const NNRec2* rec;       // targets in spatial order at the pose
    const float4* sphere;    // their tiles and, behind them, super tiles
    int N, n_tiles, n_super, k_out;
    int* idx;                // [N][k_out], by source index; with d2
    float* d2;
    float* dmin;             // [N], or, for the quantised sigma alone:
    unsigned long long* qsum;   // its integer sum (zeroed; any order gives the same)
    int* ticket;                // blocks done (zeroed); the last one writes sigma
    double *out, *host_out, *pose_sig;   // as sigma_kernel's
    const int* err;
};

// the reference's term of sigma: rn_u32(fl32(d2min / D) * 1e6)
__device__ __forceinline__ unsigned quantised(float d2, int D)
{
    return __float2uint_rn(__fmul_rn(__fdiv_rn(d2, (float)D), 1000000.0f));
}

// the quantised sigma of n sources, rounded to float as update_sig returns it
__device__ __forceinline__ double quantised_sigma(unsigned long long sum, int n)
{
    return (double)__double2float_rn((double)sum / 1e6 / (double)n);
}

template <int D>
__device__ __forceinline__ float dist2(const float* p, const float4& c)
{
    const float dx = p[0] - c.x, dy = p[1] - c.y;
    float d = fmaf(dy, dy, dx * dx);
    if (D == 3) {
        const float dz = p[2] - c.z;
        d = fmaf(dz, dz, d);
    }
    return d;
}

// certainly farther than `bound`?  d2: squared distance to a sphere's centre, r: the radii to take off
// (NaN and inf: no)
__device__ __forceinline__ bool beyond(float d2, float r, float bound)
{
    const float q = r + bound;
    return d2 * (1.f - 1e-5f) > q * q;
}

// K = 0: the nearest squared distance only; else sorted lists of the K nearest
template <int D, int K, int NW>
__global__ void __launch_bounds__(32 * NW) nn_prune_kernel(PruneArgs a)
{
    constexpr int KL = K > 0 ? K : 1;
    constexpr unsigned long long kNone = (unsigned long long)0x7f800000u << 32 | 0x7fffffffu;
    __shared__ __align__(8) int s_bound[kTile];         // bounds on the lanes' k-th distances (float bits)
    __shared__ int s_best[kTile];                       // K = 0: the squared distances
    __shared__ int s_first[NW];
    __shared__ __align__(8) float s_x[3][kTile];        // minus the sources
    __shared__ __align__(16) float4 s_rec[NW][2][kTile];   // two tiles of records per warp
    __shared__ unsigned long long s_list[K > 0 ? NW - 1 : 1][KL][kTile];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int pos = blockIdx.x * kTile + lane;
    const bool in = pos < a.N;
    pdl_trigger();
    // (the sources are init's, not the prologue's)
    SortedPoint s = a.xpt[in ? pos : 0];
    const Bound g = a.xtile[blockIdx.x];
    float2 X[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) X[q] = make_float2(s.p[q], s.p[q]);
    float best = in ? INFINITY : -1.f;      // K = 0; a lane without a source takes nothing
    unsigned long long list[KL];            // K > 0: (distance bits, index), ascending
#pragma unroll
    for (int q = 0; q < KL; ++q) list[q] = in ? kNone : 0ull;
    float bound = best;
    if (warp == 0) {
        s_best[lane] = s_bound[lane] = __float_as_int(bound);
#pragma unroll
        for (int q = 0; q < 3; ++q) s_x[q][lane] = in ? -s.p[q] : 1e18f;   // (out of every sphere's reach)
    }
    pdl_wait();
    __syncthreads();

    auto insert = [&](unsigned long long key) {
        if (!(key < list[KL - 1])) return;
#pragma unroll
        for (int q = 0; q < KL; ++q) {
            const unsigned long long o = list[q];
            const bool lt = key < o;
            list[q] = lt ? key : o;
            key = lt ? o : key;
        }
    };
    auto key_of = [](float dd, float j) {
        return (unsigned long long)__float_as_uint(dd) << 32 | __float_as_uint(j);
    };
    const float4* rec4 = reinterpret_cast<const float4*>(a.rec);
    int buf = 0;
    // the tile whose records the warp holds in v (one float4 a lane)
    auto search = [&](float4 v) {
        float4* r = s_rec[warp][buf];
        buf ^= 1;
        r[lane] = v;
        __syncwarp();
        float2 nearest = make_float2(best, best);
        // only what can still be among the K nearest (the others' lists count too); an infinite distance, as
        // NaN, is none
        const float cut = fminf(bound * bound * (1.f + 1e-5f), 3.402823466e38f);
#pragma unroll 4
        for (int e = 0; e < kTile / 2; ++e) {
            const float4 ra = r[2 * e], rb = r[2 * e + 1];
            const float2 d0 = fadd2(X[0], make_float2(ra.x, ra.y)), d1 = fadd2(X[1], make_float2(ra.z, ra.w));
            float2 dd;
            if (D == 3) {
                const float2 d2 = fadd2(X[2], make_float2(rb.x, rb.y));
                dd = ffma2(d2, d2, ffma2(d1, d1, fmul2(d0, d0)));
            } else {
                dd = ffma2(d1, d1, fmul2(d0, d0));
            }
            if constexpr (K == 0) {
                nearest.x = fminf(nearest.x, dd.x);
                nearest.y = fminf(nearest.y, dd.y);
            } else {
                const float top = fminf(cut, __uint_as_float((unsigned)(list[KL - 1] >> 32)));
                if (dd.x <= top) insert(key_of(dd.x, rb.z));
                if (dd.y <= top) insert(key_of(dd.y, rb.w));
            }
        }
        if constexpr (K == 0) best = fminf(nearest.x, nearest.y);
        const float kth = K == 0 ? best : __uint_as_float((unsigned)(list[KL - 1] >> 32));
        // (distances order like their bits; -1 comes first)
        if (in) atomicMin(&s_bound[lane], __float_as_int(fmaxf(sqrt_fast(kth) * (1.f + 1e-6f), kLeastReach)));
        bound = __int_as_float(*(volatile int*)&s_bound[lane]);
    };

    const float4* super = a.sphere + a.n_tiles;
    // lane = sphere: can any source still need it?  (many spheres at a time, one test each per source, in packed FP32
    // on two sources: update_sig 65536 x 65536 33.5 -> 29.5 us, 240000 depth points 135 -> 116, k = 8 at 30000 83 -> 75)
    auto filter = [&](float4 c, bool go) {
        bool any = false;
        const float2 w2 = make_float2(c.w, c.w), less = make_float2(1.f - 1e-5f, 1.f - 1e-5f);
#pragma unroll 4
        for (int q = 0; q < kTile; q += 2) {
            const long long b2 = *(const volatile long long*)&s_bound[q];
            const int2 b = make_int2((int)b2, (int)(b2 >> 32));
            const float2 d0 = fadd2(make_float2(c.x, c.x), *(const float2*)&s_x[0][q]);
            const float2 d1 = fadd2(make_float2(c.y, c.y), *(const float2*)&s_x[1][q]);
            float2 d = ffma2(d1, d1, fmul2(d0, d0));
            if (D == 3) {
                const float2 d2 = fadd2(make_float2(c.z, c.z), *(const float2*)&s_x[2][q]);
                d = ffma2(d2, d2, d);
            }
            d = fmul2(d, less);   // (beyond, twice)
            const float2 r = fadd2(w2, make_float2(__int_as_float(b.x), __int_as_float(b.y)));
            const float2 rr = fmul2(r, r);
            any |= !(d.x > rr.x);
            any |= !(d.y > rr.y);
        }
        return __ballot_sync(0xffffffffu, go && any);
    };
    auto refresh = [&]() {   // this lane's bound, and the worst of the group's
        bound = __int_as_float(*(volatile int*)&s_bound[lane]);
        return __int_as_float(__reduce_max_sync(0xffffffffu, __float_as_int(bound)));
    };
    // a warp's tiles of up to NW super tiles at a time: fn(lane's tile or -1, its sphere)
    constexpr int TPW = kSuper / NW;
    auto each_tile = [&](unsigned mask, int sbase, auto&& fn) {
        while (mask) {
            int mine = -1;
#pragma unroll
            for (int k = 0; k < NW; ++k) {
                const int bit = __ffs(mask) - 1;   // -1: none left
                mask &= mask - 1;
                if (k == lane / TPW) mine = bit;
            }
            int t = mine < 0 ? -1 : (sbase + mine) * kSuper + (lane % TPW) * NW + warp;
            if (t >= a.n_tiles) t = -1;
            fn(t, a.sphere[t < 0 ? 0 : t]);
        }
    };

    // The warp's first tile: the one nearest to subgroup warp % 4, in the super tile nearest to it (of
    // eight warps, the nearest even one and the nearest odd one); the same tile only once.
    {
        const Bound h = a.xsub[4 * blockIdx.x + warp % 4];
        unsigned near = 0xffffffffu;
        int s0 = 0;
        for (int u = lane; u < a.n_super; u += 32) {
            const unsigned key = __float_as_uint(dist2<D>(h.c, super[u]));
            if (key < near) { near = key; s0 = u; }
        }
        unsigned least = __reduce_min_sync(0xffffffffu, near);
        unsigned who = __ballot_sync(0xffffffffu, near == least);
        s0 = __shfl_sync(0xffffffffu, s0, __ffs(who) - 1);
        int t0 = s0 * kSuper + lane;
        const bool own = t0 < a.n_tiles && (NW == 4 || lane % 2 == warp / 4);
        near = own ? __float_as_uint(dist2<D>(h.c, a.sphere[t0])) : 0xffffffffu;
        least = __reduce_min_sync(0xffffffffu, near);
        who = __ballot_sync(0xffffffffu, own && near == least);
        t0 = who ? s0 * kSuper + __ffs(who) - 1 : -1;
        if (lane == 0) s_first[warp] = t0;
        const float4 v = rec4[(size_t)max(t0, 0) * kTile + lane];
        __syncthreads();
        bool dup = t0 < 0;
        for (int k = 0; k < warp; ++k) dup |= s_first[k] == t0;
        if (!dup) search(v);
        __syncthreads();   // (every warp's first bounds)
    }
    // the others
    for (int base = 0; base < a.n_super; base += 32) {
        const int u = min(base + lane, a.n_super - 1);
        const float4 cs = super[u];
        const float worst = refresh();
        const bool go = base + lane < a.n_super && !beyond(dist2<D>(g.c, cs), cs.w + g.r, worst);
        unsigned mask = __ballot_sync(0xffffffffu, go);
        if (__popc(mask) > 2 * NW) mask = filter(cs, go);
        each_tile(mask, base, [&](int t, float4 c) {
            const float worst_now = refresh();
            bool need = t >= 0 && !beyond(dist2<D>(g.c, c), c.w + g.r, worst_now);
#pragma unroll
            for (int k = 0; k < NW; ++k) need &= t != s_first[k];
            unsigned todo = __ballot_sync(0xffffffffu, need);
            if (__popc(todo) > 3) todo = filter(c, need);
            if (!todo) return;
            int from = __ffs(todo) - 1;
            float4 v = rec4[(size_t)__shfl_sync(0xffffffffu, t, from) * kTile + lane];
            while (todo) {
                const float4 cu = make_float4(__shfl_sync(0xffffffffu, c.x, from), __shfl_sync(0xffffffffu, c.y, from),
                                              __shfl_sync(0xffffffffu, c.z, from), __shfl_sync(0xffffffffu, c.w, from));
                todo &= todo - 1;
                const float4 vu = v;
                from = todo ? __ffs(todo) - 1 : from;
                const int tn = __shfl_sync(0xffffffffu, t, from);
                if (todo) v = rec4[(size_t)tn * kTile + lane];   // the next one, meanwhile
                if (__any_sync(0xffffffffu, in && !beyond(dist2<D>(s.p, cu), cu.w, bound))) search(vu);
            }
        });
    }
    // the warps' results
    if constexpr (K == 0)
        atomicMin(&s_best[lane], __float_as_int(best));
    else if (warp > 0)
#pragma unroll
        for (int q = 0; q < KL; ++q) s_list[warp - 1][q][lane] = list[q];
    __syncthreads();
    if (warp > 0) return;
    if constexpr (K == 0) {
        const float d2 = __int_as_float(s_best[lane]);
        if (!a.qsum) {
            if (in) a.dmin[s.idx] = d2;
            return;
        }
        const unsigned q = in ? quantised(d2, D) : 0u;
        const unsigned lo = __reduce_add_sync(0xffffffffu, q & 0xffffu), hi = __reduce_add_sync(0xffffffffu, q >> 16);
        if (lane == 0) {
            atomicAdd(a.qsum, ((unsigned long long)hi << 16) + lo);
            __threadfence();
            if (atomicAdd(a.ticket, 1) == (int)gridDim.x - 1) {
                __threadfence();
                const double sig = quantised_sigma(__ldcg(a.qsum), a.N);
                a.out[1] = sig;
                if (a.pose_sig) a.pose_sig[kPoseSig] = sig;
                if (a.host_out) {
                    a.host_out[1] = sig;
                    a.host_out[2] = (double)*a.err;
                }
            }
        }
    } else if (in) {
        for (int w = 0; w < NW - 1; ++w)
            for (int q = 0; q < KL; ++q) insert(s_list[w][q][lane]);
#pragma unroll
        for (int q = 0; q < KL; ++q)
            if (q < a.k_out) {
                a.idx[(size_t)s.idx * a.k_out + q] = (int)(unsigned)list[q];
                a.d2[(size_t)s.idx * a.k_out + q] = __uint_as_float((unsigned)(list[q] >> 32));
            }
    }
}

// sigma from the nearest squared distances: per-block partials over contiguous slices (fixed
// order), then the block that finishes last sums the partials (fixed order too, so the result is
// deterministic); ticket was zeroed by the search prologue.  n_all: the sources, or 0 for the partial
// sums of a row range.  host_out (optional, mapped pinned memory) receives out[0..1] and the error
// word at [2]; pose_sig (optional) a device pose block whose sig becomes out[1].
__global__ void __launch_bounds__(256) sigma_kernel(const float* dmin, int n, int D, int n_all, double* pe,
                                                    unsigned long long* pq, int* ticket, double* out,
                                                    double* host_out, const int* err, double* pose_sig)
{
    pdl_trigger();   // a dependent of the search
    pdl_wait();
    __shared__ double s_exact[8];
    __shared__ unsigned long long s_q[8];
    __shared__ bool s_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    auto block_total = [&](double& se, unsigned long long& sq) {   // (in thread 0)
        se = warp_sum(se);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        __syncthreads();
        if (lane == 0) {
            s_exact[warp] = se;
            s_q[warp] = sq;
        }
        __syncthreads();
        if (threadIdx.x == 0)
            for (int w = 1; w < 8; ++w) {
                se += s_exact[w];
                sq += s_q[w];
            }
    };
    const int per = (n + gridDim.x - 1) / gridDim.x;
    const int b0 = blockIdx.x * per, b1 = min(n, b0 + per);
    double se = 0;
    unsigned long long sq = 0;
    for (int i = b0 + threadIdx.x; i < b1; i += blockDim.x) {
        const float v = dmin[i];
        se += (double)v;
        sq += (unsigned long long)quantised(v, D);
    }
    block_total(se, sq);
    if (threadIdx.x == 0) {
        pe[blockIdx.x] = se;
        pq[blockIdx.x] = sq;
        __threadfence();
        s_last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    se = 0;
    sq = 0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x) {
        se += __ldcg(pe + i);
        sq += __ldcg(pq + i);
    }
    block_total(se, sq);
    if (threadIdx.x == 0) {
        double o0, o1;
        if (n_all > 0) {
            o0 = se / ((double)D * n_all);
            o1 = quantised_sigma(sq, n_all);
        } else {   // the partial sums of a row range: sum d2min, and the sum of the quantised terms
            o0 = se;
            o1 = (double)sq;
        }
        out[0] = o0;
        out[1] = o1;
        if (pose_sig) pose_sig[kPoseSig] = o1;
        if (host_out) {
            host_out[0] = o0;
            host_out[1] = o1;
            host_out[2] = (double)*err;
        }
    }
}

template <class Body, int NT, int TJ>
__global__ void __launch_bounds__(NT) nn_kernel(PairArgs a)
{
    Body body;
    run_pairs<Body, NT, TJ, 4>(a, body);
}


struct NNVariant {
    KernelShape shape;   // tj counts records of two targets; ipt is the k = 1 sources per thread
    KernelFn k1;
    KernelFn k8;
    int ipt8;            // sources per thread of the k <= 8 kernel
    KernelFn k16;
    int ipt16;           // sources per thread of the k <= 16 kernel
    KernelFn kmin;       // nearest distance only (sigma)
};

template <int D>
static const std::vector<NNVariant>& nn_variants()
{
    static const std::vector<NNVariant> v = {
        {{4, 128, 64}, nn_kernel<NNBody<D, 4, 1>, 128, 64>, nn_kernel<NNBody<D, 2, 8>, 128, 64>, 2,
         nn_kernel<NNBody<D, 1, 16>, 128, 64>, 1, nn_kernel<NNMinBody<D, 4>, 128, 64>},
        {{8, 128, 64}, nn_kernel<NNBody<D, 8, 1>, 128, 64>, nn_kernel<NNBody<D, 1, 8>, 128, 64>, 1,
         nn_kernel<NNBody<D, 2, 16>, 128, 64>, 2, nn_kernel<NNMinBody<D, 8>, 128, 64>},
        {{4, 256, 64}, nn_kernel<NNBody<D, 4, 1>, 256, 64>, nn_kernel<NNBody<D, 2, 8>, 256, 64>, 2,
         nn_kernel<NNBody<D, 1, 16>, 256, 64>, 1, nn_kernel<NNMinBody<D, 4>, 256, 64>},
    };
    return v;
}

std::vector<KernelShape> nn_shapes()
{
    std::vector<KernelShape> s;
    for (auto& v : nn_variants<3>()) s.push_back(v.shape);
    return s;
}

template <int D, int NW>
static void (*prune_kernel(int K))(PruneArgs)
{
    return K == 0 ? nn_prune_kernel<D, 0, NW>
                  : (K == 1 ? nn_prune_kernel<D, 1, NW>
                            : (K == 8 ? nn_prune_kernel<D, 8, NW> : nn_prune_kernel<D, 16, NW>));
}

// The pruned search takes all rows, but for one neighbour where its blocks are too few to fill the GPU while each
// has a long chain of spheres and tiles (few sources), or where there is too little to prune for one block per 32
// sources to pay (few targets).  update_sig on one B200, us a call, all pairs / pruned, points of a surface:
//   targets  20000:  32 sources 49 / 60, 128 36 / 46, 512 38 / 32;   65000: 128 52 / 66, 512 53 / 43
//            200000: 128 77 / 128, 512 80 / 73;   600000: 128 143 / 406, 512 146 / 214, 1000 203 / 176
//   sources  200000: 32 targets 36 / 39, 128 38 / 42, 512 57 / 43;   600000: 32 54 / 66, 128 51 / 75, 512 103 / 77
// Targets of which a quarter of the pairs share a grid cell are in a poor order, and few sources find their
// tiles late: a cluster with 95 % of the points, 65000 targets: 1000 sources 60 / 98, 4000 96 / 80;  600000: 1000 205 / 836,
// 2000 330 / 769, 4000 570 / 585.
// With 8 neighbours the pruned search is the faster one at these sizes too (600000 targets: 2.8-14 times).
bool nn_pruned(const Context& c, int k, const KernelShape* force, int rows)
{
    if (force || c.nn_pinned || (rows >= 0 && rows != c.N)) return false;
    const bool few = c.N <= 256 || c.M / 800 >= c.N || (c.near_y > 0.25 && c.N < 4000);
    return k > 1 || !((c.M >= 16384 && few) || (c.M <= 256 && c.N >= 262144));
}

// Runs the search; dmin_dev (nullable) receives the nearest squared distance per source.
// Source rows [i0, i1) (i1 < 0: all); idx/d2 rows are relative to i0, dmin is indexed absolutely.
// The search: the targets' search records (the nearest-neighbour prologue, which also zeroes the
// work counters, and the error word when reset_err; the pose by value when pv, or read from
// pose_src), then the pruned search in spatial order or (nn_pruned) the all-pairs kernel and the
// merge of its per-chunk lists.  quant: the pruned search also sums the quantised sigma (SigmaOpts) into out_dev[1].
static int nn_run(Context& c, double* pose_dev, int k, int* idx_dev, float* d2_dev, float* dmin_dev,
                  cudaStream_t s, const KernelShape* force, int i0 = 0, int i1 = -1, const PoseBlock* pv = nullptr,
                  const double* pose_src = nullptr, bool reset_err = false, const SigmaOpts* quant = nullptr,
                  double* out_dev = nullptr)
{
    if (i1 < 0) i1 = c.N;
    const int rows = i1 - i0;
    if (pose_src) {
        DUGMA_RET(launch_pose_in(c, pose_src, pose_dev, s, reset_err));
        reset_err = false;
    }
    const bool pruned = nn_pruned(c, k, force, rows);
    c.last_search = pruned;
    DUGMA_RET(launch_nn_prologue(c, pose_dev, s, pv, c.counter, reset_err ? c.err : nullptr, pruned));
    if (pruned) {
        const int K = !idx_dev ? 0 : (k <= 1 ? 1 : (k <= 8 ? 8 : 16));
        const int nx = (c.N + kTile - 1) / kTile;
        constexpr int kSpan = kTile * kSuper;
        const PruneArgs a{c.xpt, c.xtile, c.xsub, reinterpret_cast<const NNRec2*>(c.yp32), c.ysphere, c.N,
                          (c.M + kTile - 1) / kTile, (c.M + kSpan - 1) / kSpan, k, idx_dev, d2_dev, dmin_dev,
                          quant ? reinterpret_cast<unsigned long long*>(c.counter + 2) : nullptr, c.counter + 1, out_dev,
                          quant ? quant->host_out : nullptr, quant ? quant->pose_sig : nullptr, c.err};
        // eight warps a group up to two groups per SM, else four
        const bool wide = nx <= 2 * c.num_sms;
        auto fn = wide ? (c.D == 3 ? prune_kernel<3, 8>(K) : prune_kernel<2, 8>(K))
                       : (c.D == 3 ? prune_kernel<3, 4>(K) : prune_kernel<2, 4>(K));
        TimingHold hold(c, false);
        DUGMA_RET(timing_begin(c, s));
        DUGMA_CK(launch_dependent(c.pdl, fn, nx, wide ? 256 : 128, 0, s, a));
        DUGMA_RET(timing_end(c, s));
        return DUGMA_OK;
    }
    const KernelShape want = force ? *force : c.shape_nn;
    const auto& vars = c.D == 3 ? nn_variants<3>() : nn_variants<2>();
    const NNVariant* v = &vars[0];
    for (auto& cand : vars)
        if (cand.shape.ipt == want.ipt && cand.shape.nt == want.nt && cand.shape.tj == want.tj) v = &cand;
    const int K = k <= 1 ? 1 : (k <= 8 ? 8 : 16);
    // only the nearest distance wanted (sigma): the packed distance-only kernel
    const bool min_only = K == 1 && !idx_dev && !d2_dev;
    KernelFn fn = min_only ? v->kmin : (K == 1 ? v->k1 : (K == 8 ? v->k8 : v->k16));
    KernelShape sh = v->shape;
    // the k = 8 / 16 kernels may keep fewer sources per thread (see the variant table)
    if (K == 8) sh.ipt = v->ipt8;
    if (K == 16) sh.ipt = v->ipt16;
    if (K > 1) {
        // every target chunk restarts the sorted lists, and a list insertion (taken by some lane
        // of a warp far more often than by one thread) costs the whole warp ~4K instructions:
        // few long chunks, just enough items to fill the GPU about once
        const int n_ib = (rows + sh.ipt * sh.nt - 1) / (sh.ipt * sh.nt);
        const int want_jc = std::max(1, (4 * c.num_sms + n_ib - 1) / n_ib);
        sh.min_chunk = std::max(1, (c.M_pad / 2 + want_jc - 1) / want_jc);
    }
    double* hp = nullptr;
    int n_jc = 0;
    TimingHold hold(c, false);
    DUGMA_RET(launch_pair_variant(c, fn, sh, c.x, c.yp32, (size_t)c.M_pad / 2, 1, 0.0, pose_dev, i0, i1, nullptr,
                                  nullptr, &hp, K, &n_jc, s, nullptr, true));
    const int g = std::min((rows + 255) / 256, c.num_sms * 8);
    const float2* part = reinterpret_cast<const float2*>(hp);
    float* dm = dmin_dev ? dmin_dev + i0 : nullptr;
    if (K == 1)
        DUGMA_CK(launch_dependent(c.pdl, nn_merge_kernel<1>, g, 256, 0, s, part, n_jc, rows, k, idx_dev, d2_dev, dm));
    else if (K == 8)
        DUGMA_CK(launch_dependent(c.pdl, nn_merge_kernel<8>, g, 256, 0, s, part, n_jc, rows, k, idx_dev, d2_dev, dm));
    else
        DUGMA_CK(launch_dependent(c.pdl, nn_merge_kernel<16>, g, 256, 0, s, part, n_jc, rows, k, idx_dev, d2_dev, dm));
    return DUGMA_OK;
}

int launch_nn(Context& c, double* pose_dev, int k, int* idx_dev, float* d2_dev, cudaStream_t s,
              const KernelShape* force)
{
    if (k < 1 || k > 16 || k > c.M) return set_error(DUGMA_ERR_ARG, "k = %d must be in [1, min(16, M)]", k);
    return nn_run(c, pose_dev, k, idx_dev, d2_dev, nullptr, s, force);
}

int launch_sigma(Context& c, double* pose_dev, double* out_dev, cudaStream_t s, int i0, int i1, const SigmaOpts& o)
{
    const bool whole = i1 < 0;
    if (whole) i1 = c.N;
    const int rows = i1 - i0;
    const bool quant = !o.exact && whole && nn_pruned(c, 1);
    DUGMA_RET(nn_run(c, pose_dev, 1, nullptr, nullptr, c.dmin, s, nullptr, i0, i1, o.pose_value, o.pose_src,
                     o.reset_err, quant ? &o : nullptr, out_dev));
    if (quant) return DUGMA_OK;
    // partials in the scratch region (the search's chunk lists there are merged by now, in stream order)
    const int nb = std::max(1, std::min(2 * c.num_sms, (rows + 511) / 512));
    DUGMA_RET(c.ensure_scratch(sizeof(double) * 2 * (size_t)nb));
    double* pe = c.scratch;
    unsigned long long* pq = reinterpret_cast<unsigned long long*>(c.scratch + nb);
    DUGMA_CK(launch_dependent(c.pdl, sigma_kernel, nb, 256, 0, s, (const float*)(c.dmin + i0), rows, c.D,
                              whole ? c.N : 0, pe, pq, c.counter + 1, out_dev, o.host_out, (const int*)c.err,
                              o.pose_sig));
    return DUGMA_OK;
}

}  // namespace dugma

// reach.cuh -- which streamed points can reach a group of stationary ones.
//
// A pair's two terms are 2^(lv_j - |k| d^T C'_j d) and 2^(lv_j - |k| d^T B_i d), and ex2.approx.ftz
// flushes a result below 2^-126 to 0.  With L a bound on the largest variance behind either matrix
// (SortedPoint::L, x sig), both exponents are at most lv_j - |k| |d|^2 / (sig max(L_i, L_j)), so a pair with
//     |d|^2 > (sig / |k|) a_j max(L_i, L_j),     a_j = lv_j + 127.5
// adds exactly +0 to every sum the kernels keep, and leaving it out changes no bit.
//
// find_reach marks, for one tile of 32 stationary points, the records (pairs of streamed points by
// index) of which a point passes that test for some stationary point: super tiles against the
// tile's four subgroups, tiles against them, points against them, then points against points.
// CONV: the pair's matrix is the sum of both covariances, so the test is |d|^2 > (sig / |k|) cut (L_i + L_j).
// The last of these is most of the work (32 x 32 tests a tile), so it runs in packed FP32 on two stationary
// points at a time, with sig / |k| and its room already in their L, and leaves overflow to the spheres' test:
// 11 instructions a pair of tests against 32.  Adjoint kernel at 65536 x 65536: 53 -> 40 us, compi's 94 -> 62, CONV's
// 76 -> 52, 240000 depth points 493 -> 417, 24 x 8 poses 518 -> 457.
// The tests run in FP32 with room for their rounding, for that of the evaluation (in L, see variance_bound)
// and for what a pose that is no exact rotation stretches.  What is not finite, or so large that the
// evaluation could overflow, is marked.
#pragma once

#include "spatial.cuh"

namespace dugma {

struct ReachSide {
    const SortedPoint* pt;
    const Bound *tile, *sub, *super;
    int n;
};

struct ReachArgs {
    ReachSide st, sm;      // stationary, streamed
    const double* pose;
    float inv_trace;       // largest trace of an inverse covariance (overflow limit)
    float cut, big;        // CONV: the exponent that leaves nothing, and the variance beyond which nothing
                           // is left out (conv.cu)
};

// Super tiles (of 1024 points) beyond which the block shares their tests.  Adjoint kernel on one B200, each warp
// all / shared: 240000 depth points (235) 418 -> 354 us, compi 673 -> 623; 65536 points (64) 40 us either way; below,
// the two barriers cost up to 1 us of 25.
constexpr int kReachShare = 64;
static_assert(kSparseMaxTargets / kTile <= 65536, "a tile's number takes 16 bits");

struct ReachShared {
    float4 xy[kTile / 2], zl[kTile / 2];   // points by pairs: -x -x' -y -y', -z -z' and L L' (scaled)
    float2 a[kTile / 2], slack[kTile / 2];
    float4 sub[4];         // centre, radius
    float2 sa[4];          // a, L
    int n_super;
    uint16_t super[256];   // super tiles that reach the tile, of the 32 NW tested together
};

// R y + t in FP32 (stretch, Lscale: how much R can stretch a length and a variance)
struct PoseF {
    float R[9], t[3], tsize;
    float stretch, Lscale;
};

template <int D>
__device__ __forceinline__ PoseF pose_f32(const double* pose)
{
    PoseF p;
    p.tsize = 0.f;
#pragma unroll
    for (int a = 0; a < D; ++a) {
#pragma unroll
        for (int b = 0; b < D; ++b) p.R[a + D * b] = (float)pose[a + D * b];
        p.t[a] = (float)pose[kPoseT + a];
        p.tsize += fabsf(p.t[a]);
    }
    float f = 0.f;   // |R^T R - I|_F^2
#pragma unroll
    for (int a = 0; a < D; ++a)
#pragma unroll
        for (int b = 0; b < D; ++b) {
            float v = a == b ? -1.f : 0.f;
#pragma unroll
            for (int k = 0; k < D; ++k) v = fmaf(p.R[k + D * a], p.R[k + D * b], v);
            f = fmaf(v, v, f);
        }
    // |R v| lies between sqrt(1 - dev) |v| and sqrt(1 + dev) |v| (2e-6 for the FP32 products)
    const float dev = fmaf(sqrtf(f), 1.f + 1e-6f, 2e-6f);
    p.stretch = sqrtf(1.f + dev) * (1.f + 1e-6f);
    p.Lscale = dev < 0.5f ? (1.f + 1e-6f) / (1.f - dev) : INFINITY;
    return p;
}

// position and, in w, the size its rounding error scales with
template <int D>
__device__ __forceinline__ float4 move_f32(const PoseF& p, const float* y)
{
    float v[3] = {0.f, 0.f, 0.f};
    float size = p.tsize;
#pragma unroll
    for (int a = 0; a < D; ++a) {
        float s = p.t[a];
#pragma unroll
        for (int k = 0; k < D; ++k) s = fmaf(p.R[a + D * k], y[k], s);
        v[a] = s;
        size += fabsf(s) + fabsf(y[a]);
    }
    return make_float4(v[0], v[1], v[2], size);
}

template <int D>
__device__ __forceinline__ float dist2_f32(const float4& p, const float4& q)
{
    const float dx = p.x - q.x, dy = p.y - q.y;
    float d = fmaf(dy, dy, dx * dx);
    if (D == 3) {
        const float dz = p.z - q.z;
        d = fmaf(dz, dz, d);
    }
    return d;
}

// The records that reach tile `group` of the stationary side, into bits (shared, one per record; all
// 32 NW threads; the caller zeroes bits before and synchronises after).  True for a lane that marked any.  POSE_SM: the streamed side is
// the targets' (moved by the pose), else the stationary side is.
template <int D, int NW, bool POSE_SM, bool CONV = false>
__device__ __forceinline__ bool find_reach(const ReachArgs& a, int group, uint32_t* bits, ReachShared& sh)
{
    constexpr int TPW = kSuper / NW;
    static_assert(NW == 2 || NW == 4 || NW == 8, "36 threads and more set the tile up");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const PoseF P = pose_f32<D>(a.pose);
    const float sigk = (float)(a.pose[kPoseSig] * (1.0 / -K_EXP2)) * (1.f + 1e-6f);
    // beyond this squared distance a form could overflow, and 0 x inf is no 0
    const float d2max = CONV ? 1e20f : fminf(1e36f * sigk / (a.inv_trace + 1e-30f), 1e30f);
    // the squared distance beyond which a pair of these a and L counts nothing
    auto reach2 = [&](float a0, float L0, float a1, float L1) {
        return CONV ? (L0 + L1 < a.big ? sigk * a.cut * (L0 + L1) : INFINITY) : sigk * fminf(a0, a1) * fmaxf(L0, L1);
    };
    // a point's L for the tests of point against point: x sig / |k|, and the room of those tests
    auto scaled = [&](float L) {
        return CONV ? (L < 0.5f * a.big ? sigk * a.cut * 1.002f * L : INFINITY) : sigk * 1.002f * L;
    };
    // a sphere or point as the tests see it
    auto place = [&](const float* c, float& r, bool posed) {
        float4 q = make_float4(c[0], c[1], D == 3 ? c[2] : 0.f, 0.f);
        if (posed) {
            q = move_f32<D>(P, c);
            r = fmaf(r, P.stretch, 1e-6f * q.w);
        }
        return q;
    };
    if (threadIdx.x < kTile) {
        const int i = group * kTile + lane;
        SortedPoint s = a.st.pt[i < a.st.n ? i : 0];
        float slack = 0.f;
        const float4 q = place(s.p, slack, !POSE_SM);
        const bool in = i < a.st.n;
        const int p = lane >> 1, h = lane & 1;
        (h ? sh.xy[p].y : sh.xy[p].x) = -q.x;
        (h ? sh.xy[p].w : sh.xy[p].z) = -q.y;
        (h ? sh.zl[p].y : sh.zl[p].x) = -q.z;
        // a lane without a point, and a point without weight (a = -1), reaches nothing
        (h ? sh.zl[p].w : sh.zl[p].z) = CONV && !in ? -INFINITY : scaled(POSE_SM ? s.L : s.L * P.Lscale);
        (h ? sh.a[p].y : sh.a[p].x) = in ? s.a : -1.f;
        (h ? sh.slack[p].y : sh.slack[p].x) = 1001.f * slack * slack;
    } else if (threadIdx.x < kTile + 4) {
        const Bound b = a.st.sub[4 * group + lane];
        float r = b.r;
        float4 q = place(b.c, r, !POSE_SM);
        q.w = r;
        sh.sub[lane] = q;
        sh.sa[lane] = make_float2(b.a, POSE_SM ? b.L : b.L * P.Lscale);
    } else if (threadIdx.x == kTile + 4) {
        sh.n_super = 0;
    }
    __syncthreads();
    // can something at q (radius r, a, L) reach a point of the subgroups in `of`?  one bit each, and bit 4 where
    // a distance is too large to tell (no point of the other subgroups is then beyond d2max)
    auto subs = [&](const float4& q, float r, float aa, float L, unsigned of) {
        unsigned m = 0;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            if (!(of >> s & 1u)) continue;
            const float4 c = sh.sub[s];
            const float2 e = sh.sa[s];
            const float T = reach2(aa, L, e.x, e.y);
            const float rr = r + c.w, reach = fmaf(sqrt_fast(fmaxf(T, 0.f)), 1.f + 2e-6f, rr);
            const float d2 = dist2_f32<D>(q, c);
            const bool near = d2 < 0.2f * d2max && rr * rr < 0.2f * d2max;
            const bool out = d2 * (1.f - 1e-5f) > reach * reach && near;
            m |= (unsigned)!out << s | (unsigned)!near << 4;
        }
        return m;
    };
    bool marked = false;
    const int n_tiles = (a.sm.n + kTile - 1) / kTile, n_super = (n_tiles + kSuper - 1) / kSuper;
    // Each warp tests all super tiles; where they are many a thread tests one, and the block goes on with a list of
    // those that reach (two barriers).
    const bool share = n_super > kReachShare;
    for (int base = 0; base < n_super; base += share ? 32 * NW : 32) {
        const int u = base + (share ? (int)threadIdx.x : lane);
        bool go = u < n_super;
        if (go) {
            const Bound b = a.sm.super[u];
            float r = b.r;
            const float4 q = place(b.c, r, POSE_SM);
            go = subs(q, r, b.a, POSE_SM ? b.L * P.Lscale : b.L, 15u) != 0;
        }
        unsigned mask = __ballot_sync(0xffffffffu, go);
        int listed = 0;
        if (share) {
            if (base) {   // (the last list has been read)
                __syncthreads();
                if (threadIdx.x == 0) sh.n_super = 0;
                __syncthreads();
            }
            int at = 0;
            if (lane == 0 && mask) at = atomicAdd(&sh.n_super, __popc(mask));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(mask & ((1u << lane) - 1u));
            if (go) sh.super[at] = (uint16_t)threadIdx.x;
            __syncthreads();
            listed = sh.n_super;
            mask = 0;
        }
        // the warp's tiles of up to NW super tiles at a time
        for (int first = 0; mask || first < listed; first += NW) {
            int mine = -1;
            if (share) {
                if (first + lane / TPW < listed) mine = sh.super[first + lane / TPW];
            } else {
#pragma unroll
                for (int k = 0; k < NW; ++k) {
                    const int bit = __ffs(mask) - 1;   // -1: none left
                    mask &= mask - 1;
                    if (k == lane / TPW) mine = bit;
                }
            }
            const int t = (base + mine) * kSuper + (lane % TPW) * NW + warp;
            unsigned reached = 0;   // the subgroups a tile reaches
            if (mine >= 0 && t < n_tiles) {
                const Bound b = a.sm.tile[t];
                float r = b.r;
                const float4 q = place(b.c, r, POSE_SM);
                reached = subs(q, r, b.a, POSE_SM ? b.L * P.Lscale : b.L, 15u);
            }
            unsigned todo = __ballot_sync(0xffffffffu, reached != 0);
            while (todo) {   // lane = point of the tile
                const uint32_t e = __shfl_sync(0xffffffffu, (uint32_t)t | reached << 16, __ffs(todo) - 1);
                todo &= todo - 1;
                const int j = (int)(e & 0xffffu) * kTile + lane;
                unsigned m = 0;
                SortedPoint s{};
                float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
                float L = 0.f, slack = 0.f;
                if (j < a.sm.n) {
                    s = a.sm.pt[j];
                    q = place(s.p, slack, POSE_SM);
                    L = POSE_SM ? s.L * P.Lscale : s.L;
                    m = subs(q, slack, s.a, L, e >> 16);
                    slack = 1001.f * slack * slack;
                    L = scaled(L);
                }
                bool hit = m >> 4;
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    if (!__any_sync(0xffffffffu, m >> g & 1u)) continue;
                    bool near = false;
#pragma unroll
                    for (int p = g * (kSub / 2); p < (g + 1) * (kSub / 2); ++p) {   // two of its points
                        const float4 xy = sh.xy[p], zl = sh.zl[p];
                        const float2 dx = fadd2(make_float2(q.x, q.x), make_float2(xy.x, xy.y));
                        const float2 dy = fadd2(make_float2(q.y, q.y), make_float2(xy.z, xy.w));
                        float2 d2 = ffma2(dy, dy, fmul2(dx, dx));
                        if (D == 3) {
                            const float2 dz = fadd2(make_float2(q.z, q.z), make_float2(zl.x, zl.y));
                            d2 = ffma2(dz, dz, d2);
                        }
                        // (d - slack)^2 > T follows from d^2 > 1.001 T + 1001 slack^2
                        const float2 room = POSE_SM ? make_float2(slack, slack) : sh.slack[p];
                        float2 T;
                        if constexpr (CONV) {
                            T = fadd2(fadd2(make_float2(L, L), make_float2(zl.z, zl.w)), room);
                        } else {
                            const float2 pa = sh.a[p];
                            T = ffma2(make_float2(fminf(s.a, pa.x), fminf(s.a, pa.y)),
                                     make_float2(fmaxf(L, zl.z), fmaxf(L, zl.w)), room);
                        }
                        near |= !(d2.x > T.x);
                        near |= !(d2.y > T.y);
                    }
                    hit |= near && (m >> g & 1u);
                }
                if (hit) atomicOr(&bits[s.idx >> 6], 1u << (s.idx >> 1 & 31));
                marked |= hit;
            }
        }
    }
    return marked;
}

}  // namespace dugma

// lbm_fast_pairs.cuh - two x-adjacent cells per thread for the FP32/FP16 two-kernel step.
//
// Populations move between HBM and registers as 2-element vectors (float2 / half2), so one
// warp request covers 64 cells of a direction plane (256 B FP32, 128 B FP16) instead of 32.
// With scalar FP16 loads each request carried 64 B while the collision arithmetic spread
// the requests out in time, and the loads waited about three times as long as FP32 loads
// for the same instruction count; vector requests give FP16 the FP32 request size.
//
// A pull along x shifts the pair by one element: it is assembled from the two aligned
// vectors that hold it.  Cells whose source lies outside the lattice (the x faces for the
// cell at the face, every direction with an out-of-range y or z source) take the scalar
// pull with the reference's boundary rule, so the values are those of the one-cell path.
// The per-cell arithmetic is the same inline functions, on both cells at once (f2).
#pragma once

#include "lbm_fast_cells.cuh"

namespace lbm {

template <class S> struct Vec2;
template <> struct Vec2<float> {
    __device__ static __forceinline__ float2 ld(const float* p, long long i) {
        return __ldg(reinterpret_cast<const float2*>(p + i));
    }
    __device__ static __forceinline__ void st(float* p, long long i, float a, float b) {
        *reinterpret_cast<float2*>(p + i) = make_float2(a, b);
    }
    // two values already in the storage type
    __device__ static __forceinline__ void st_raw(float* p, long long i, float a, float b) { st(p, i, a, b); }
};
template <> struct Vec2<__half> {
    __device__ static __forceinline__ float2 ld(const __half* p, long long i) {
        const unsigned int w = __ldg(reinterpret_cast<const unsigned int*>(p + i));
        return __half22float2(__halves2half2(__ushort_as_half((unsigned short)(w & 0xFFFFu)),
                                             __ushort_as_half((unsigned short)(w >> 16))));
    }
    __device__ static __forceinline__ void st(__half* p, long long i, float a, float b) {
        // each half rounds as __float2half_rn does in the one-cell path
        const unsigned int lo = __half_as_ushort(__float2half_rn(a)), hi = __half_as_ushort(__float2half_rn(b));
        *reinterpret_cast<unsigned int*>(p + i) = lo | (hi << 16);
    }
    // two values already in the storage type
    __device__ static __forceinline__ void st_raw(__half* p, long long i, __half a, __half b) {
        *reinterpret_cast<unsigned int*>(p + i) = (unsigned int)__half_as_ushort(a) | ((unsigned int)__half_as_ushort(b) << 16);
    }
};

__device__ __forceinline__ float2 ldf2(const float* p, long long i) { return __ldg(reinterpret_cast<const float2*>(p + i)); }
__device__ __forceinline__ void stf2(float* p, long long i, float a, float b) {
    *reinterpret_cast<float2*>(p + i) = make_float2(a, b);
}

// Values of direction a pulled into cells (i0, .) and (i0+1, .) from the source row that
// starts at `row` (the row of (sj, sk) in plane a), both sources inside the lattice in x.
template <int Q, class S>
__device__ __forceinline__ float2 vec_pull_row(const Geo& g, const S* __restrict__ p, int a, int i0, long long row) {
    const int ex = Lat<Q>::ex(a);
    if (ex == 0) return Vec2<S>::ld(p, row + i0);
    if (ex == 1) {  // sources i0-1 and i0
        const float2 lo = Vec2<S>::ld(p, row + (i0 > 0 ? i0 - 2 : 0));
        const float2 hi = Vec2<S>::ld(p, row + i0);
        return make_float2(lo.y, hi.x);
    }
    // ex == -1: sources i0+1 and i0+2
    const float2 lo = Vec2<S>::ld(p, row + i0);
    const float2 hi = Vec2<S>::ld(p, row + (i0 + 2 < g.nx ? i0 + 2 : i0));
    return make_float2(lo.y, hi.x);
}

template <int Q, class S, class LOAD>
__device__ __forceinline__ float2 pull_flow_pair(const Geo& g, const S* __restrict__ p, int a, int i0, int j, int k,
                                                 long long c0, long long n, LOAD load) {
    const int ex = Lat<Q>::ex(a), ey = Lat<Q>::ey(a), ez = Lat<Q>::ez(a);
    const int sj = j - ey, sk = k - ez;
    const bool yz = (ey == 0 || (sj >= 0 && sj < g.ny)) && (ez == 0 || (sk >= 0 && sk < g.nz));
    float2 v = make_float2(0.0f, 0.0f);
    if (yz) v = vec_pull_row<Q, S>(g, p, a, i0, (long long)a * n + (long long)g.nx * ((long long)sj + (long long)g.ny * sk));
    if (!yz || (ex == 1 && i0 == 0)) v.x = pull_flow<Q, float>(g, a, i0, j, k, c0, load);
    if (!yz || (ex == -1 && i0 + 2 >= g.nx)) v.y = pull_flow<Q, float>(g, a, i0 + 1, j, k, c0 + 1, load);
    return v;
}

template <int QT, class S, class LOAD>
__device__ __forceinline__ float2 pull_thermal_pair(const Geo& g, const S* __restrict__ p, int a, int i0, int j, int k,
                                                    long long c0, long long n, LOAD load) {
    const int ex = Lat<QT>::ex(a), ey = Lat<QT>::ey(a), ez = Lat<QT>::ez(a);
    const int sj = j - ey, sk = k - ez;
    const bool yz = (ey == 0 || (sj >= 0 && sj < g.ny)) && (ez == 0 || (sk >= 0 && sk < g.nz));
    float2 v = make_float2(0.0f, 0.0f);
    if (yz) v = vec_pull_row<QT, S>(g, p, a, i0, (long long)a * n + (long long)g.nx * ((long long)sj + (long long)g.ny * sk));
    if (!yz || (ex == 1 && i0 == 0)) v.x = pull_thermal<QT, float>(g, a, i0, j, k, c0, load);
    if (!yz || (ex == -1 && i0 + 2 >= g.nx)) v.y = pull_thermal<QT, float>(g, a, i0 + 1, j, k, c0 + 1, load);
    return v;
}

// flow_cell_2k (not FIRST) for the cells c0 = (i0, j, k) and c0 + 1.
template <int D, class S>
__device__ __forceinline__ void flow_pair_2k(const Geo& g, const PhysF& P, const FastArgs<S>& A, const S* __restrict__ fin,
                                             const S* __restrict__ gin, S* __restrict__ fout, long long c0, int i0, int j,
                                             int k) {
    constexpr int Q = (D == 2) ? 9 : 19, QT = (D == 2) ? 5 : 7;
    const long long n = g.ncell;
    auto lf = [&](int a, long long cc) { return ldS(fin, a * n + cc); };
    auto lg = [&](int a, long long cc) { return ldS(gin, a * n + cc); };
    f2 d[Q], ts = make_f2(0.0f, 0.0f);
#pragma unroll
    for (int a = 0; a < Q; ++a) {
        const float2 v = pull_flow_pair<Q, S>(g, fin, a, i0, j, k, c0, n, lf);
        d[a] = make_f2(v.x, v.y);
    }
#pragma unroll
    for (int a = 0; a < QT; ++a) {
        const float2 e = pull_thermal_pair<QT, S>(g, gin, a, i0, j, k, c0, n, lg);
        ts = vadd(ts, make_f2(e.x, e.y));
    }
    const float2 lag = ldf2(A.lag_in, c0);
    const f2 Fy = steady_flow<D>(d, steady_lag<D>(make_f2(lag.x, lag.y), P), ts, P);
    if (D == 2) stf2(A.lag_out, c0, f2_lo(Fy), f2_hi(Fy));
    S h0[Q], h1[Q];
    round_pair<Q>(d, h0, h1, P.sr != 0, sr_seed(*A.tick, c0, 0), sr_seed(*A.tick, c0 + 1, 0));
#pragma unroll
    for (int a = 0; a < Q; ++a) Vec2<S>::st_raw(fout, a * n + c0, h0[a], h1[a]);
}

// thermal_cell_end (not FIRST) for the cells c0 and c0 + 1.
template <int D, class S>
__device__ __forceinline__ void thermal_pair_end(const PhysF& P, const FastArgs<S>& A, const f2* d, f2* e,
                                                 long long c0) {
    const float2 bx = ldf2(A.Bin0, c0), by = ldf2(A.Bin1, c0);
    const float2 bz = D == 3 ? ldf2(A.Bin2, c0) : make_float2(0.0f, 0.0f);
    const float2 lag = D == 2 ? ldf2(A.lag_in, c0) : make_float2(0.0f, 0.0f);
    f2 B[3] = {make_f2(bx.x, bx.y), make_f2(by.x, by.y), make_f2(bz.x, bz.y)};
    const f2 T = steady_thermal<D>(d, e, make_f2(lag.x, lag.y), B, P);
    stf2(A.Bout0, c0, f2_lo(B[0]), f2_hi(B[0]));
    stf2(A.Bout1, c0, f2_lo(B[1]), f2_hi(B[1]));
    if (D == 3) {
        stf2(A.Bout2, c0, f2_lo(B[2]), f2_hi(B[2]));
        stf2(A.lag_out, c0, f2_lo(T), f2_hi(T));
    }
}

// thermal_cell_2k (not FIRST) for the cells c0 and c0 + 1.
template <int D, class S>
__device__ __forceinline__ void thermal_pair_2k(const Geo& g, const PhysF& P, const FastArgs<S>& A,
                                                const S* __restrict__ fin, const S* __restrict__ gin, S* __restrict__ gout,
                                                long long c0, int i0, int j, int k) {
    constexpr int Q = (D == 2) ? 9 : 19, QT = (D == 2) ? 5 : 7;
    const long long n = g.ncell;
    auto lf = [&](int a, long long cc) { return ldS(fin, a * n + cc); };
    auto lg = [&](int a, long long cc) { return ldS(gin, a * n + cc); };
    f2 d[Q], e[QT];
#pragma unroll
    for (int a = 0; a < Q; ++a) {
        const float2 v = pull_flow_pair<Q, S>(g, fin, a, i0, j, k, c0, n, lf);
        d[a] = make_f2(v.x, v.y);
    }
#pragma unroll
    for (int a = 0; a < QT; ++a) {
        const float2 v = pull_thermal_pair<QT, S>(g, gin, a, i0, j, k, c0, n, lg);
        e[a] = make_f2(v.x, v.y);
    }
    thermal_pair_end<D, S>(P, A, d, e, c0);
    S h0[QT], h1[QT];
    round_pair<QT>(e, h0, h1, P.sr != 0, sr_seed(*A.tick, c0, 1), sr_seed(*A.tick, c0 + 1, 1));
#pragma unroll
    for (int a = 0; a < QT; ++a) Vec2<S>::st_raw(gout, a * n + c0, h0[a], h1[a]);
}

}  // namespace lbm

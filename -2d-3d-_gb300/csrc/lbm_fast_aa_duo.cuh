// lbm_fast_aa_duo.cuh - the in-place (AA) sweeps of the FP32/FP16 forms with two cells per thread,
// 32 apart (lbm_fast_duo.cuh), for lattices without periodic faces and 32-bit indices.
//
// The layouts are those of lbm_device.cuh.  An even sweep reads the cells' own slots and writes
// the opposite ones; an odd sweep pulls from the swapped layout and pushes.  Across a wall both
// stay inside the cell, so pull and push are one select per direction on the index.  The other
// array, read only, is in the layout that a regular sequence of steps leaves: swapped beside an
// odd flow sweep and beside an even thermal sweep (the flow sweep of the same step ran before).
#pragma once

#include "lbm_fast_duo.cuh"

namespace lbm {

// Slot that the push of direction a from a cell fills (aa_push on walls).
template <int Q, int AT>
__device__ __forceinline__ int push_index(const Geo& g, int n, int a, int i, int j, int k, int c) {
    const int ex = Lat<Q>::ex(a), ey = Lat<Q>::ey(a), ez = Lat<Q>::ez(a);
    const int back = Lat<Q>::opp(a) * n + c;
    int at = a * n + c + ex + g.nx * (ey + g.ny * ez);
    if (AT != kInner && ex != 0) at = (ex > 0 ? i == g.nx - 1 : i == 0) ? back : at;
    if (AT == kFaces && ey != 0) at = (ey > 0 ? j == g.ny - 1 : j == 0) ? back : at;
    if (AT == kFaces && ez != 0) at = (ez > 0 ? k == g.nz - 1 : k == 0) ? back : at;
    return at;
}

// One set read from the cells' own slots of the streamed layout; thermal values that were pushed
// (raw) take the constant-temperature wall rule.
template <int Q, bool TH, class S>
__device__ __forceinline__ void duo_own_set(const Geo& g, const S* f, const Duo& t, bool raw, f2* d) {
    const int n = (int)g.ncell;
    decltype(ld_raw(f)) x[2][Q];
#pragma unroll
    for (int a = 0; a < Q; ++a) {
        x[0][a] = ld_raw(cell_ptr<Q>(f, a * n, t.c[0]));
        x[1][a] = ld_raw(cell_ptr<Q>(f, a * n, t.c[1]));
    }
    PullRule r = pull_rule<TH>(g);
    if (!raw) r.cx = r.cy = false;
#pragma unroll
    for (int a = 0; a < Q; ++a) {
        float v[2] = {raw_value(x[0][a]), raw_value(x[1][a])};
        if (TH) {
#pragma unroll
            for (int h = 0; h < 2; ++h) v[h] = wall_value<Q, true>(g, r, a, t.i[h], t.j[h], v[h]);
        }
        d[a] = make_f2(v[0], v[1]);
    }
}

template <int Q, bool TH, bool SWAPPED, class S>
__device__ __forceinline__ void duo_layout_set(const Geo& g, const S* f, const Duo& t, bool raw, f2* d) {
    if (!SWAPPED) duo_own_set<Q, TH, S>(g, f, t, raw, d);
    else if (t.inner) duo_pull_set<Q, TH, kInner, S, true>(g, f, t, d);
    else if (t.rows) duo_pull_set<Q, TH, kRows, S, true>(g, f, t, d);
    else duo_pull_set<Q, TH, kFaces, S, true>(g, f, t, d);
}

template <int Q>
__device__ __forceinline__ void duo_round(const f2* v, float* h0, float* h1, const PhysF&, unsigned long long, const Duo&,
                                          unsigned) {
#pragma unroll
    for (int a = 0; a < Q; ++a) {
        h0[a] = f2_lo(v[a]);
        h1[a] = f2_hi(v[a]);
    }
}
template <int Q>
__device__ __forceinline__ void duo_round(const f2* v, __half* h0, __half* h1, const PhysF& P, unsigned long long tick,
                                          const Duo& t, unsigned kind) {
    float x[Q];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
#pragma unroll
        for (int a = 0; a < Q; ++a) x[a] = w ? f2_hi(v[a]) : f2_lo(v[a]);
        round_cell<Q>(x, w ? h1 : h0, P.sr != 0, sr_seed(tick, t.c[w], kind));
    }
}

// The sweep's new values into the array: pushed (odd) or into the opposite own slots (even).
template <int Q, bool ODD, class S>
__device__ __forceinline__ void duo_aa_store(const Geo& g, S* f, const Duo& t, const f2* v, const PhysF& P,
                                             unsigned long long tick, unsigned kind) {
    const int n = (int)g.ncell;
    S h[2][Q];
    duo_round<Q>(v, h[0], h[1], P, tick, t, kind);
    if (!ODD) {
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            if (!t.in[w]) continue;
#pragma unroll
            for (int a = 0; a < Q; ++a) *cell_ptr<Q>(f, Lat<Q>::opp(a) * n, t.c[w]) = h[w][a];
        }
    } else if (t.inner) {
#pragma unroll
        for (int a = 0; a < Q; ++a) {
            S* p = cell_ptr<Q>(f, push_index<Q, kInner>(g, n, a, 0, 0, 0, 0), t.c[0]);
            p[0] = h[0][a];
            if (t.in[1]) p[32] = h[1][a];
        }
    } else {
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            if (!t.in[w]) continue;
            if (t.rows) {
#pragma unroll
                for (int a = 0; a < Q; ++a)
                    f[push_index<Q, kRows>(g, n, a, t.i[w], t.j[w], t.k[w], t.c[0] + 32 * w)] = h[w][a];
            } else {
#pragma unroll
                for (int a = 0; a < Q; ++a)
                    f[push_index<Q, kFaces>(g, n, a, t.i[w], t.j[w], t.k[w], t.c[0] + 32 * w)] = h[w][a];
            }
        }
    }
}

// aa_flow_cell and aa_thermal_cell (not FIRST) for both cells.
template <int D, class S, bool ODD>
__device__ __forceinline__ void aa_flow_duo(const Geo& g, const PhysF& P, const FastArgs<S>& A, S* f,
                                            const S* gs, bool raw, const Duo& t, unsigned long long tick) {
    constexpr int Q = (D == 2) ? 9 : 19, QT = (D == 2) ? 5 : 7;
    if (!t.in[0]) return;
    f2 d[Q], e[QT], ts = make_f2(0.0f, 0.0f);
    duo_layout_set<Q, false, ODD, S>(g, f, t, false, d);
    duo_layout_set<QT, true, ODD, S>(g, gs, t, raw, e);
    const f2 lag = steady_lag<D>(duo_load(A.lag_in, t), P);
#pragma unroll
    for (int a = 0; a < QT; ++a) ts = vadd(ts, e[a]);
    const f2 Fy = steady_flow<D>(d, lag, ts, P);
    if (D == 2) duo_store(A.lag_out, t, Fy);
    duo_aa_store<Q, ODD, S>(g, f, t, d, P, tick, 0);
}

template <int D, class S, bool ODD>
__device__ __forceinline__ void aa_thermal_duo(const Geo& g, const PhysF& P, const FastArgs<S>& A,
                                               const S* fs, S* gg, bool raw, const Duo& t,
                                               unsigned long long tick) {
    constexpr int Q = (D == 2) ? 9 : 19, QT = (D == 2) ? 5 : 7;
    if (!t.in[0]) return;
    f2 d[Q], e[QT];
    duo_layout_set<Q, false, !ODD, S>(g, fs, t, false, d);
    duo_layout_set<QT, true, ODD, S>(g, gg, t, raw, e);
    f2 B[3] = {duo_load(A.Bin0, t), duo_load(A.Bin1, t), D == 3 ? duo_load(A.Bin2, t) : make_f2(0.0f, 0.0f)};
    const f2 T = steady_thermal<D>(d, e, D == 2 ? duo_load(A.lag_in, t) : make_f2(0.0f, 0.0f), B, P);
    duo_store(A.Bout0, t, B[0]);
    duo_store(A.Bout1, t, B[1]);
    if (D == 3) {
        duo_store(A.Bout2, t, B[2]);
        duo_store(A.lag_out, t, T);
    }
    duo_aa_store<QT, ODD, S>(g, gg, t, e, P, tick, 1);
}

}  // namespace lbm

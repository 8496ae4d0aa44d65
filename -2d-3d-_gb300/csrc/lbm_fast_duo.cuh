// lbm_fast_duo.cuh - two cells per thread, 32 apart in lattice order, for the FP32/FP16
// two-kernel step (two buffers).
//
// A warp covers 64 consecutive cells: lane l holds cells c and c + 32.  Every access of a warp is
// a run of 32 consecutive values as in the one-cell kernels, whatever the row length (no
// alignment to keep, no x shift to assemble), the second cell's address is the first's plus a
// constant, and the arithmetic runs on both cells at once (f2).  A warp off every face reads
// at fixed distances, one whose rows lie off the y and z faces selects for the x faces, and one that
// holds a cell of a y or z face row selects for all.  Only the loads are inside that choice.
// The first of the three took index arithmetic out of kernels whose integer pipe was 48% busy
// (GB300, us per step before / after: FP16 2D 2050x1025 44.7 / 42.7, 256^3 605 / 598, 384^3 in
// place 2195 / 2145; FP32 is bound by HBM and unchanged; 60 2D FP32 lattices together 262 / 248).
// 32-bit indices: narrow_index.
#pragma once

#include "lbm_fast_cells.cuh"

namespace lbm {

struct Duo {
    int c[2];     // the cells
    bool in[2];   // whether the lane has them
    int i[2], j[2], k[2];
    bool rows;    // every cell of the warp lies on a row off the y and z faces
    bool inner;   // every cell of the warp lies off every face
};

// Cells c0 and c0 + 32 of a lane (called by whole warps), those below `end`.  A cell beyond the
// lattice is read as its last one and not stored.  OWN (in-place sweeps, where that cell's slots
// are being written): a lane without a second cell repeats its first, and one without a first
// takes no part.
template <bool OWN = false>
__device__ __forceinline__ Duo duo_at(const Geo& g, int c0, int end) {
    Duo t;
    const int last = (int)g.ncell - 1;
    t.in[0] = c0 < end;
    t.in[1] = c0 + 32 < end;
    t.c[0] = min(c0, last);
    t.c[1] = min(c0 + 32, last);
    const int r = t.c[0] / g.nx;
    t.i[0] = t.c[0] - r * g.nx;
    t.k[0] = g.nz > 1 ? r / g.ny : 0;
    t.j[0] = r - t.k[0] * g.ny;
    if (g.nx >= 32) {  // the second cell lies on the same row or the next
        const bool w = t.i[0] + 32 >= g.nx;
        t.i[1] = t.i[0] + 32 - (w ? g.nx : 0);
        const int j = t.j[0] + (w ? 1 : 0);
        t.j[1] = j == g.ny ? 0 : j;
        t.k[1] = t.k[0] + (j == g.ny ? 1 : 0);
    } else {
        const int r1 = t.c[1] / g.nx;
        t.i[1] = t.c[1] - r1 * g.nx;
        t.k[1] = g.nz > 1 ? r1 / g.ny : 0;
        t.j[1] = r1 - t.k[1] * g.ny;
    }
    if (c0 + 32 > last) {
        t.c[1] = OWN ? t.c[0] : last;
        t.i[1] = OWN ? t.i[0] : g.nx - 1;
        t.j[1] = OWN ? t.j[0] : g.ny - 1;
        t.k[1] = OWN ? t.k[0] : g.nz - 1;
    }
    const bool off = row_off_faces(g, t.j[0], t.k[0]) && row_off_faces(g, t.j[1], t.k[1]);
    const bool xoff = t.i[0] > 0 && t.i[0] < g.nx - 1 && t.i[1] > 0 && t.i[1] < g.nx - 1;
    t.rows = __all_sync(0xFFFFFFFFu, off);
    t.inner = __all_sync(0xFFFFFFFFu, off && xoff);
    return t;
}
// The cells of block `block` of a single-lattice launch (ncell / 256 blocks of 128 threads, rounded up).
template <bool OWN = false>
__device__ __forceinline__ Duo duo_cells(const Geo& g, int block) {
    return duo_at<OWN>(g, (block * (int)blockDim.x + (int)(threadIdx.x & ~31u)) * 2 + (int)(threadIdx.x & 31u),
                       (int)g.ncell);
}

// A stored population as loaded, and its value.  Not read-only loads: the kernel before may still
// be writing when this one starts (lbm_launch.cuh).
__device__ __forceinline__ float ld_raw(const float* p) { return *p; }
__device__ __forceinline__ unsigned short ld_raw(const __half* p) { return *reinterpret_cast<const unsigned short*>(p); }
__device__ __forceinline__ float raw_value(float x) { return x; }
__device__ __forceinline__ float raw_value(unsigned short x) { return __half2float(__ushort_as_half(x)); }

// Element c of the array that begins `shift` elements after p.  In 3D as an address that all threads
// share and a 32-bit offset that serves every direction (n * sizeof(S) < 2^32).  GB300, us per step
// with shift + c as one index / so: 96^3 FP16 33.6 / 32.3, 256^3 FP16 589 / 580, 384^3 FP16 2010 / 1959,
// in place 2130 / 2105, FP32 unchanged; 2D 2050x1025 FP16 41.7 / 43.2, so not there.
template <int Q, class S>
__device__ __forceinline__ S* cell_ptr(S* p, int shift, int c) {
    if (Q == 9 || Q == 5) return p + (shift + c);
    return (S*)((char*)(p + shift) + (size_t)((unsigned)c * (unsigned)sizeof(S)));
}

// The wall rule of a constant-temperature face on a pulled thermal value.
template <int QT, bool FACES>
__device__ __forceinline__ float wall_value(const Geo& g, const PullRule& r, int a, int i, int j, float v) {
    const int ex = Lat<QT>::ex(a), ey = Lat<QT>::ey(a);
    if (ex != 0 && r.cx) {
        const float w = -v + (float)(ex > 0 ? g.bcT_lo[0] : g.bcT_hi[0]);
        return (ex > 0 ? i == 0 : i == g.nx - 1) ? w : v;
    }
    if (FACES && ey != 0 && r.cy) {
        const float w = -v + (float)(ey > 0 ? g.bcT_lo[1] : g.bcT_hi[1]);
        return (ey > 0 ? j == 0 : j == g.ny - 1) ? w : v;
    }
    return v;
}

// Where the cells of a warp lie: off every face, on rows off the y and z faces, anywhere.  In the
// first two the second cell is the first plus 32 (the lattice's last cell lies on a face row), so
// its values are read at a constant distance, and off the faces no index is selected.
constexpr int kInner = 0, kRows = 1, kFaces = 2;

// The Q populations of one set pulled into both cells.
template <int Q, bool TH, int AT, class S, bool SWAP = false>
__device__ __forceinline__ void duo_pull_set(const Geo& g, const S* f, const Duo& t, f2* d) {
    const int n = (int)g.ncell;
    const PullRule r = pull_rule<TH>(g);
    decltype(ld_raw(f)) x[2][Q];
#pragma unroll
    for (int a = 0; a < Q; ++a) {
        if (AT == kInner || (AT == kRows && Lat<Q>::ex(a) == 0)) {
            const S* p = cell_ptr<Q>(f, (SWAP ? Lat<Q>::opp(a) : a) * n
                                         - (Lat<Q>::ex(a) + g.nx * (Lat<Q>::ey(a) + g.ny * Lat<Q>::ez(a))), t.c[0]);
            x[0][a] = ld_raw(p);
            x[1][a] = ld_raw(p + 32);
        } else {
#pragma unroll
            for (int h = 0; h < 2; ++h)
                x[h][a] = ld_raw(f + pull_index<Q, AT == kFaces, SWAP>(g, n, r, a, t.i[h], t.j[h], t.k[h],
                                                                      AT == kFaces ? t.c[h] : t.c[0] + 32 * h));
        }
    }
#pragma unroll
    for (int a = 0; a < Q; ++a) {
        float v[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            v[h] = raw_value(x[h][a]);
            if (TH && AT != kInner) v[h] = wall_value<Q, AT == kFaces>(g, r, a, t.i[h], t.j[h], v[h]);
        }
        d[a] = make_f2(v[0], v[1]);
    }
}
template <int Q, int QT, class S>
__device__ __forceinline__ void duo_pull(const Geo& g, const S* f, const S* gs, const Duo& t,
                                         f2* d, f2* e) {
    if (t.inner) {
        duo_pull_set<Q, false, kInner, S>(g, f, t, d);
        duo_pull_set<QT, true, kInner, S>(g, gs, t, e);
    } else if (t.rows) {
        duo_pull_set<Q, false, kRows, S>(g, f, t, d);
        duo_pull_set<QT, true, kRows, S>(g, gs, t, e);
    } else {
        duo_pull_set<Q, false, kFaces, S>(g, f, t, d);
        duo_pull_set<QT, true, kFaces, S>(g, gs, t, e);
    }
}

__device__ __forceinline__ f2 duo_load(const float* p, const Duo& t) { return make_f2(p[t.c[0]], p[t.c[1]]); }
__device__ __forceinline__ void duo_store(float* p, const Duo& t, f2 v) {
    if (t.in[0]) p[t.c[0]] = f2_lo(v);
    if (t.in[1]) p[t.c[1]] = f2_hi(v);
}

// The Q new populations v of both cells, rounded as round_cell rounds each cell's.
template <int Q>
__device__ __forceinline__ void duo_store_pops(float* out, int n, const Duo& t, const f2* v, const PhysF&, unsigned long long,
                                               unsigned) {
    if (t.in[0]) {
#pragma unroll
        for (int a = 0; a < Q; ++a) {
            float* p = cell_ptr<Q>(out, a * n, t.c[0]);
            p[0] = f2_lo(v[a]);
            if (t.in[1]) p[32] = f2_hi(v[a]);
        }
    }
}
template <int Q>
__device__ __forceinline__ void duo_store_pops(__half* out, int n, const Duo& t, const f2* v, const PhysF& P,
                                               unsigned long long tick, unsigned kind) {
    float x[Q];
    __half h[2][Q];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
#pragma unroll
        for (int a = 0; a < Q; ++a) x[a] = w ? f2_hi(v[a]) : f2_lo(v[a]);
        round_cell<Q>(x, h[w], P.sr != 0, sr_seed(tick, t.c[w], kind));
    }
    if (t.in[0]) {
#pragma unroll
        for (int a = 0; a < Q; ++a) {
            __half* p = cell_ptr<Q>(out, a * n, t.c[0]);
            p[0] = h[0][a];
            if (t.in[1]) p[32] = h[1][a];
        }
    }
}

// The step counter inside the step's own kernels, without a launch to advance it: the flow kernel
// reads ticks[0] and one thread copies it to ticks[1]; the thermal kernel reads ticks[1] and one
// thread writes the advanced count to ticks[0], so no kernel writes the word that its blocks read.
__device__ __forceinline__ unsigned long long flow_tick(unsigned long long* ticks, bool one) {
    const unsigned long long n = ticks[0];
    if (one) ticks[1] = n;
    return n;
}
__device__ __forceinline__ unsigned long long thermal_tick(unsigned long long* ticks, bool one) {
    const unsigned long long n = ticks[1];
    if (one) ticks[0] = n + 1ULL;
    return n;
}

// flow_cell_2k and thermal_cell_2k (not FIRST) for both cells.
template <int D, class S>
__device__ __forceinline__ void flow_duo_2k(const Geo& g, const PhysF& P, const FastArgs<S>& A, const S* fin,
                                            const S* gin, S* fout, const Duo& t,
                                            unsigned long long tick) {
    constexpr int Q = (D == 2) ? 9 : 19, QT = (D == 2) ? 5 : 7;
    f2 d[Q], e[QT], ts = make_f2(0.0f, 0.0f);
    duo_pull<Q, QT, S>(g, fin, gin, t, d, e);
    const f2 lag = steady_lag<D>(duo_load(A.lag_in, t), P);
#pragma unroll
    for (int a = 0; a < QT; ++a) ts = vadd(ts, e[a]);
    const f2 Fy = steady_flow<D>(d, lag, ts, P);
    if (D == 2) duo_store(A.lag_out, t, Fy);
    duo_store_pops<Q>(fout, (int)g.ncell, t, d, P, tick, 0);
}

template <int D, class S>
__device__ __forceinline__ void thermal_duo_2k(const Geo& g, const PhysF& P, const FastArgs<S>& A,
                                               const S* fin, const S* gin,
                                               S* gout, const Duo& t, unsigned long long tick) {
    constexpr int Q = (D == 2) ? 9 : 19, QT = (D == 2) ? 5 : 7;
    f2 d[Q], e[QT];
    duo_pull<Q, QT, S>(g, fin, gin, t, d, e);
    f2 B[3] = {duo_load(A.Bin0, t), duo_load(A.Bin1, t), D == 3 ? duo_load(A.Bin2, t) : make_f2(0.0f, 0.0f)};
    const f2 T = steady_thermal<D>(d, e, D == 2 ? duo_load(A.lag_in, t) : make_f2(0.0f, 0.0f), B, P);
    duo_store(A.Bout0, t, B[0]);
    duo_store(A.Bout1, t, B[1]);
    if (D == 3) {
        duo_store(A.Bout2, t, B[2]);
        duo_store(A.lag_out, t, T);
    }
    duo_store_pops<QT>(gout, (int)g.ncell, t, e, P, tick, 1);
}

}  // namespace lbm

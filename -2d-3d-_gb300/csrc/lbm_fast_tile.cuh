// lbm_fast_tile.cuh - the FP32/FP16 step of a 2D lattice in one launch, two cells per thread.
//
// A block runs the flow collisions of its tile and of the ring of cells around it, keeps the new
// populations in shared memory, and runs the thermal collisions of the tile from there.  The flow
// populations are written and not read again and the thermal ones are pulled once: 136 B per cell
// in FP32 where the two kernels move 189.  Cells of the ring are collided by the neighbouring
// blocks as well, with the same arithmetic and random bits, so the values are the two kernels'.
//
// A warp holds one row of 64 cells: lane l the columns l and l + 32.  Off the lattice's faces the
// pulls, from memory and from shared memory, are at fixed distances.
#pragma once

#include "lbm_fast_duo.cuh"
#include "lbm_tile2d.h"

namespace lbm {

// The two cells of lane `lane` in row `row` of tile `tile` (columns tile_column, tile_line).  Returns
// the first cell's index had the row no end; the second's is 32 more.
__host__ __device__ __forceinline__ int tile_cells(const Geo& g, const TilePlan& tp, int tile, int row, int lane, Duo& t) {
    const int ty = tile / tp.ntx, tx = tile - ty * tp.ntx;
    const int y = ty * tp.th + row - tp.oy, x = tx * tp.tw + lane - tp.ox;
    const int j = tile_line(g, y);
    const bool mine = row >= tp.oy && row < tp.oy + tp.th && y < g.ny;
    for (int h = 0; h < 2; ++h) {
        const int l = lane + 32 * h, xi = x + 32 * h;
        t.i[h] = tile_column(g, xi);
        t.j[h] = j;
        t.k[h] = 0;
        t.c[h] = t.i[h] + g.nx * j;
        t.in[h] = mine && l >= tp.ox && l < tp.ox + tp.tw && xi < g.nx;
    }
    const int x0 = x - lane;
    t.inner = j > 0 && j < g.ny - 1 && x0 > 0 && x0 + 63 < g.nx - 1;
    t.rows = false;  // the second cell of an x-face row need not be the first plus 32
    return x + g.nx * j;
}

#if defined(__CUDACC__)
// The new populations of the owned cells to memory, and to v the values as a pull reads them back.
template <int Q, class S>
__device__ __forceinline__ void tile_store(S* out, int n, int at, const Duo& t, f2* v, const PhysF& P,
                                           unsigned long long tick, unsigned kind) {
    S h[2][Q];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
        float y[Q];
#pragma unroll
        for (int a = 0; a < Q; ++a) y[a] = w ? f2_hi(v[a]) : f2_lo(v[a]);
        round_cell<Q>(y, h[w], P.sr != 0, sizeof(S) == 2 ? sr_seed(tick, t.c[w], kind) : 0u);
    }
#pragma unroll
    for (int a = 0; a < Q; ++a) {
        S* p = out + (a * n + at);
        if (t.in[0]) p[0] = h[0][a];
        if (t.in[1]) p[32] = h[1][a];
        v[a] = make_f2(stored_value(h[0][a]), stored_value(h[1][a]));
    }
}
__device__ __forceinline__ void tile_put(float* p, int at, const Duo& t, f2 v) {
    if (t.in[0]) p[at] = f2_lo(v);
    if (t.in[1]) p[at + 32] = f2_hi(v);
}

// The step of tile `tile` (a whole block of W warps).  sf: eight directions of 64 * W values.
template <class S, int W>
__device__ __forceinline__ void tile_step(const Geo& g, const PhysF& P, const TilePlan& tp, const FastArgs<S>& Af,
                                          const FastArgs<S>& At, const S* fin, const S* gin, S* fout, S* gout, int tile,
                                          unsigned long long tick, float* sf) {
    constexpr int CAP = 64 * W;
    const int row = (int)(threadIdx.x >> 5), lane = (int)(threadIdx.x & 31u), n = (int)g.ncell;
    Duo t;
    const int at = tile_cells(g, tp, tile, row, lane, t);
    float* s = sf + row * 64 + lane;
    f2 d[9], e[5], ts = make_f2(0.0f, 0.0f);
    duo_pull<9, 5, S>(g, fin, gin, t, d, e);
    const f2 lag = steady_lag<2>(duo_load(Af.lag_in, t), P);
    f2 B[3] = {duo_load(At.Bin0, t), duo_load(At.Bin1, t), make_f2(0.0f, 0.0f)};
#pragma unroll
    for (int a = 0; a < 5; ++a) ts = vadd(ts, e[a]);
    const f2 Fy = steady_flow<2>(d, lag, ts, P);
    tile_put(Af.lag_out, at, t, Fy);
    tile_store<9>(fout, n, at, t, d, P, tick, 0);
#pragma unroll
    for (int a = 1; a < 9; ++a) {
        s[(a - 1) * CAP] = f2_lo(d[a]);
        s[(a - 1) * CAP + 32] = f2_hi(d[a]);
    }
    __syncthreads();
    if (!t.in[0] && !t.in[1]) return;
    if (t.inner) {
#pragma unroll
        for (int a = 1; a < 9; ++a) {
            const float* q = s + ((a - 1) * CAP - Lat<9>::ex(a) - 64 * Lat<9>::ey(a));
            d[a] = make_f2(q[0], q[32]);
        }
    } else {
        const PullRule r = pull_rule<false>(g);
#pragma unroll
        for (int a = 1; a < 9; ++a) {
            float v[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                bool back;
                const int p = row * 64 + lane + 32 * h, from = tile_pull<9, 64>(g, r, a, t.i[h], t.j[h], p, back);
                v[h] = sf[(back ? Lat<9>::opp(a) - 1 : a - 1) * CAP + (t.in[h] ? from : p)];
            }
            d[a] = make_f2(v[0], v[1]);
        }
    }
    steady_thermal<2>(d, e, Fy, B, P);
    tile_put(At.Bout0, at, t, B[0]);
    tile_put(At.Bout1, at, t, B[1]);
    tile_store<5>(gout, n, at, t, e, P, tick, 1);
}

// End of a lattice's step of `blocks` blocks, whose last one to arrive advances the step counter:
// by then every block has read it (FP16).  ticks[2] counts the arrivals.
template <class S>
__device__ __forceinline__ void tile_tick(unsigned long long* ticks, unsigned blocks, bool one) {
    if (sizeof(S) != 2) {
        if (one) ticks[0] += 1ULL;
        return;
    }
    __syncthreads();
    if (threadIdx.x == 0 && atomicInc(reinterpret_cast<unsigned*>(ticks + 2), blocks - 1) == blocks - 1) ticks[0] += 1ULL;
}
#endif

}  // namespace lbm

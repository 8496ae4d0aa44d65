// lbm_tile2d.h - tiles of the one-launch steps of a 2D lattice (lbm_fast_tile.cuh, lbm_fixed.cu): a
// block runs the flow collisions of its tile and of the ring of cells around it, then the thermal
// collisions of the tile from shared memory.
#pragma once

#include "lbm_device.cuh"

namespace lbm {

// ntx x nty blocks of `width` x `rows` cells, each owning up to tw x th of them that begin at
// (ox, oy).  An axis that one block covers has no ring, unless it is periodic (the y faces are
// walls).
struct TilePlan {
    int tw, th, ntx, nty, ox, oy;
};
__host__ __device__ __forceinline__ bool tile_wraps(const Geo& g) {
    return g.bcf[0] == LBM_BC_PERIODIC || g.bct[0] == LBM_BCT_PERIODIC;
}
inline TilePlan tile_plan(const Geo& g, int width, int rows) {
    TilePlan t;
    t.ox = g.nx > width || tile_wraps(g) ? 1 : 0;
    t.oy = g.ny > rows ? 1 : 0;
    t.tw = width - 2 * t.ox;
    t.th = rows - 2 * t.oy;
    t.ntx = (g.nx + t.tw - 1) / t.tw;
    t.nty = (g.ny + t.th - 1) / t.th;
    return t;
}

// Lattice column of a block's column x and row of its row y: beyond the lattice the nearest one, or
// the wrapped one across a periodic x face.
__host__ __device__ __forceinline__ int tile_column(const Geo& g, int x) {
    if (x < 0) return tile_wraps(g) ? g.nx - 1 : 0;
    return x < g.nx ? x : (tile_wraps(g) && x == g.nx ? 0 : g.nx - 1);
}
__host__ __device__ __forceinline__ int tile_line(const Geo& g, int y) { return y < 0 ? 0 : (y < g.ny ? y : g.ny - 1); }

// Where an owned cell (i, j) at p of the block's cells pulls direction a from: pull_index's rule,
// back standing for its own value of the opposite direction.
template <int Q, int WIDTH>
__host__ __device__ __forceinline__ int tile_pull(const Geo& g, const PullRule& r, int a, int i, int j, int p, bool& back) {
    const int ex = Lat<Q>::ex(a), ey = Lat<Q>::ey(a);
    const bool xout = ex != 0 && (ex > 0 ? i == 0 : i == g.nx - 1);
    const bool yout = ey != 0 && (ey > 0 ? j == 0 : j == g.ny - 1);
    back = yout || (xout && r.wx);
    return back ? p : (xout ? p - ex : p - ex - WIDTH * ey);
}

}  // namespace lbm

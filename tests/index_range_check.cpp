// The 32-bit cell indices of the step kernels on the largest lattices that take them (narrow_index,
// csrc/lbm_device.cuh), compiled with the undefined-behaviour sanitizer for test_cpu_index_range.py:
// pull_index, push_index and the tiles' own indices at every kind of cell, against the 64-bit rule.
#include "host_device.h"
#define __CUDACC__ 1  // the tile's index functions
#include "lbm_fast_aa_duo.cuh"
#undef __CUDACC__
#include "lbm_fast_tile.cuh"

#include <cstdio>
#include <cstdlib>
#include <vector>

using namespace lbm;

static long long checked = 0;
static void same(long long got, long long want, const char* what) {
    ++checked;
    if (got != want) {
        std::printf("FAIL %s %lld %lld\n", what, got, want);
        std::exit(1);
    }
}

template <int Q, bool TH>
static void cells(const Geo& g) {
    const PullRule r = pull_rule<TH>(g);
    const int n = (int)g.ncell;
    auto picks = [](int m) { return m > 2 ? std::vector<int>{0, 1, m - 2, m - 1} : (m > 1 ? std::vector<int>{0, 1} : std::vector<int>{0}); };
    for (int k : picks(g.nz))
        for (int j : picks(g.ny))
            for (int i : picks(g.nx)) {
                const int c = (int)cell_index(g, i, j, k);
                for (int a = 0; a < Q; ++a) {
                    auto at = [&](int b, long long cc) { return b * (long long)n + cc; };
                    auto swapped = [&](int b, long long cc) { return Lat<Q>::opp(b) * (long long)n + cc; };
                    const long long want = pull_flow<Q, long long>(g, a, i, j, k, c, at);
                    same(pull_index<Q, true>(g, n, r, a, i, j, k, c), want, "pull");
                    same(pull_index<Q, true, true>(g, n, r, a, i, j, k, c),
                         pull_flow<Q, long long>(g, a, i, j, k, c, swapped), "swapped pull");
                    if (row_off_faces(g, j, k)) same(pull_index<Q, false>(g, n, r, a, i, j, k, c), want, "row pull");
                    if (g.bcf[0] != LBM_BC_PERIODIC && g.bcf[2] != LBM_BC_PERIODIC)
                        same(push_index<Q, kFaces>(g, n, a, i, j, k, c),
                             pull_flow<Q, long long>(g, Lat<Q>::opp(a), i, j, k, c,
                                                     [&](int b, long long cc) { return (b == Lat<Q>::opp(a) ? a : Lat<Q>::opp(a)) * (long long)n + cc; }),
                             "push");
                }
            }
}

template <int D>
static void lattice(int nx, int ny, int nz, bool periodic) {
    constexpr int Q = D == 3 ? 19 : 9, QT = D == 3 ? 7 : 5;
    Geo g{};
    g.nx = nx, g.ny = ny, g.nz = nz;
    g.ncell = (long long)nx * ny * nz;
    for (int x = 0; x < 3; ++x) g.bcf[x] = LBM_BC_NOSLIP, g.bct[x] = LBM_BCT_ADIABATIC;
    if (periodic) {
        g.bcf[0] = LBM_BC_PERIODIC, g.bct[0] = LBM_BCT_PERIODIC;
        if (D == 3) g.bcf[2] = LBM_BC_PERIODIC, g.bct[2] = LBM_BCT_PERIODIC;
    }
    if (!narrow_index(g, Q)) return;
    cells<Q, false>(g);
    cells<QT, true>(g);
    if (D == 2) {
        for (int rows : {4, 8}) {
            const TilePlan tp = tile_plan(g, 64, rows);
            const int n = (int)g.ncell;
            for (int tile : {0, tp.ntx * tp.nty - 1})
                for (int row = 0; row < rows; ++row)
                    for (int lane = 0; lane < 32; ++lane) {
                        Duo t;
                        const int at = tile_cells(g, tp, tile, row, lane, t);
                        same(8 * n + at + 32, 8LL * n + at + 32, "tile");
                    }
        }
    }
}

int main() {
    // for rows and planes of many sizes, the extents around the last one that is taken
    for (int periodic = 0; periodic < 2; ++periodic) {
        for (long long nx : {5LL, 64LL, 1000LL, 4099LL, 100003LL, 9000000LL}) {
            const long long most = (1LL << 31) / 9 / nx;
            for (long long ny = most + 1; ny > most - 80 && ny >= 5; --ny) lattice<2>((int)nx, (int)ny, 1, periodic);
            for (long long ny : {5LL, 70LL, 999LL, 5000LL}) {
                const long long mz = (1LL << 31) / 19 / nx / ny;
                for (long long nz = mz + 1; nz > mz - 4 && nz >= 2; --nz) lattice<3>((int)nx, (int)ny, (int)nz, periodic);
            }
        }
    }
    std::printf("ok %lld\n", checked);
    return 0;
}

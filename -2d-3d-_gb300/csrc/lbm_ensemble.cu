// lbm_ensemble.cu - one flow launch and one thermal launch per time step (most FP32 in 2D: one launch) for
// any number of FP32/FP16 lattices of uneven sizes and parameters (the batched form).
//
// A grid of about SMs x grid_mul persistent blocks walks a packed tile table: tile t is
// (member m, first cell c0) and covers tile_cells consecutive cells of member m.  Each
// block reads the member's descriptor (geometry, relaxation rates, buffer pointers and
// parity), then runs the same per-cell bodies as the single-lattice two-kernel step
// (lbm_fast_duo.cuh, or lbm_fast_cells.cuh for members beyond 32-bit indices) on its cells.  Small
// lattices therefore fill the GPU together instead of one launch each.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <vector>

#include "lbm_ensemble.h"
#include "lbm_fast_duo.cuh"
#include "lbm_fast_tile.cuh"
#include "lbm_launch.cuh"

namespace lbm {

template <class S>
struct EnsMember {
    Geo g;      // wall terms in deviation form
    PhysF P;
    S* f[2];
    S* gp[2];
    float* B[2][3];
    float* L[2];
    unsigned long long* tick;  // the member's step counter (stochastic rounding of FP16)
    int cur;    // buffer parity when the table was built
    TilePlan tp;  // 2D: its tiles of the one-launch step
};

// Resident blocks per SM: of 128 threads with two cells each, or of 256 with one (wide: 64-bit
// indices).  GB300, us per step of 30 members with 5 / 6 / 7 / 8 blocks: 2D FP16 93.5 / 91.9 / 91.4 /
// 85.8 (10: 94.4), 3D FP32 2492 / 2553 / 2627 / 2778, 3D FP16 2000 / 2049 / 2051 / 2163 (4: 2121).
constexpr int ens_blocks(int dim, bool wide) { return wide ? 3 : (dim == 2 ? 8 : 5); }

// Cell coordinates of a thread's cells in a tile, stepped instead of divided: one division
// at the thread's first cell, then (i, j, k) advance by `stride` cells with carries (i by
// less than a row; j may wrap several planes on narrow lattices).
struct CellWalk {
    long long c;
    int i, j, k, di, dj, stride;
    __device__ __forceinline__ CellWalk(const Geo& g, long long c0, int stride_) : c(c0), stride(stride_) {
        cell_coords(g, c0, i, j, k);
        di = (int)((unsigned)stride % (unsigned)g.nx);
        dj = (int)((unsigned)stride / (unsigned)g.nx);
    }
    __device__ __forceinline__ void next(const Geo& g) {
        c += stride;
        i += di;
        j += dj;
        if (i >= g.nx) {
            i -= g.nx;
            j += 1;
        }
        while (j >= g.ny) {
            j -= g.ny;
            k += 1;
        }
    }
};

// The member descriptor of a block's current tile and the buffer arguments of this step,
// staged in shared memory: the cell bodies read geometry, constants and buffer pointers
// from there as the single-lattice kernels read them from the kernel parameters, instead of
// holding register copies across the cell loop.  `args` (thread 0) fills the arguments from
// the descriptor in global memory.
template <class S>
struct EnsStage {
    EnsMember<S> m;
    FastArgs<S> A;
};

template <class S, class ARGS>
__device__ __forceinline__ const EnsStage<S>& stage_member(const EnsMember<S>* __restrict__ mem, int idx,
                                                           unsigned* __restrict__ sh, ARGS args) {
    static_assert(sizeof(EnsMember<S>) % 4 == 0, "descriptor copied in 32-bit words");
    EnsStage<S>& st = *reinterpret_cast<EnsStage<S>*>(sh);
    const unsigned* src = reinterpret_cast<const unsigned*>(mem + idx);
    __syncthreads();  // the block's previous tile is done with the staged copy
    for (int w = threadIdx.x; w < (int)(sizeof(EnsMember<S>) / 4); w += blockDim.x) sh[w] = __ldg(src + w);
    if (threadIdx.x == 0) {
        FastArgs<S> A{};
        args(mem[idx], A);
        st.A = A;
    }
    __syncthreads();
    return st;
}

// WIDE: one cell per thread with 64-bit indices (members too large for 32-bit ones); otherwise two
// cells per thread (lbm_fast_duo.cuh), a block taking 2 * blockDim.x cells of its tile at a time.
template <int D, class S, bool WIDE>
__global__ void __launch_bounds__(WIDE ? 256 : 128, ens_blocks(D, WIDE))
    k_ens_flow(const EnsMember<S>* __restrict__ mem, const int2* __restrict__ tiles, int ntiles, int tile_cells, int flip) {
    __shared__ __align__(16) unsigned sh[(sizeof(EnsStage<S>) + 3) / 4];
    wait_for_previous();
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int2 tt = tiles[t];
        const EnsStage<S>& st = stage_member<S>(mem, tt.x, sh, [flip](const EnsMember<S>& gm, FastArgs<S>& A) {
            const int c = gm.cur ^ flip;
            A.lag_in = gm.L[c];
            A.lag_out = gm.L[c ^ 1];
            A.tick = gm.tick;
            A.ticks = gm.tick;
        });
        const EnsMember<S>& m = st.m;
        const FastArgs<S>& A = st.A;
        const Geo& g = m.g;
        const PhysF& P = m.P;
        const int cur = m.cur ^ flip, nxt = cur ^ 1;
        const long long c0 = (long long)tt.y * tile_cells;
        const long long ce = min(c0 + tile_cells, g.ncell);
        const bool one = tt.y == 0 && threadIdx.x == 0;
        const unsigned long long tick = sizeof(S) == 2 || one ? flow_tick(A.ticks, one) : 0ULL;
        if constexpr (WIDE) {
            for (CellWalk w(g, c0 + (long long)threadIdx.x, (int)blockDim.x); w.c < ce; w.next(g))
                flow_cell_2k<D, false, S>(g, P, A, m.f[cur], m.gp[cur], m.f[nxt], w.c, w.i, w.j, w.k);
        } else {
            for (int c = (int)c0 + 2 * (int)(threadIdx.x & ~31u); c < (int)ce; c += 2 * (int)blockDim.x)
                flow_duo_2k<D, S>(g, P, A, m.f[cur], m.gp[cur], m.f[nxt], duo_at(g, c + (int)(threadIdx.x & 31u), (int)ce),
                                  tick);
        }
    }
    start_next();
}

template <int D, class S, bool WIDE>
__global__ void __launch_bounds__(WIDE ? 256 : 128, ens_blocks(D, WIDE))
    k_ens_thermal(const EnsMember<S>* __restrict__ mem, const int2* __restrict__ tiles, int ntiles, int tile_cells,
                  int flip) {
    __shared__ __align__(16) unsigned sh[(sizeof(EnsStage<S>) + 3) / 4];
    wait_for_previous();
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int2 tt = tiles[ntiles - 1 - t];  // last tile first (last_first)
        const EnsStage<S>& st = stage_member<S>(mem, tt.x, sh, [flip](const EnsMember<S>& gm, FastArgs<S>& A) {
            const int c = gm.cur ^ flip, n = c ^ 1;
            A.Bin0 = gm.B[c][0]; A.Bin1 = gm.B[c][1]; A.Bin2 = gm.B[c][2];
            A.Bout0 = gm.B[n][0]; A.Bout1 = gm.B[n][1]; A.Bout2 = gm.B[n][2];
            A.lag_in = gm.L[n];
            A.lag_out = gm.L[n];
            A.tick = gm.tick + 1;  // the copy the flow kernel left
            A.ticks = gm.tick;
        });
        const EnsMember<S>& m = st.m;
        const FastArgs<S>& A = st.A;
        const Geo& g = m.g;
        const PhysF& P = m.P;
        const int cur = m.cur ^ flip, nxt = cur ^ 1;
        const long long c0 = (long long)tt.y * tile_cells;
        const long long ce = min(c0 + tile_cells, g.ncell);
        const bool one = tt.y == 0 && threadIdx.x == 0;
        const unsigned long long tick = sizeof(S) == 2 || one ? thermal_tick(A.ticks, one) : 0ULL;
        if constexpr (WIDE) {
            for (CellWalk w(g, c0 + (long long)threadIdx.x, (int)blockDim.x); w.c < ce; w.next(g))
                thermal_cell_2k<D, false, S>(g, P, A, m.f[nxt], m.gp[cur], m.gp[nxt], w.c, w.i, w.j, w.k);
        } else {
            for (int c = (int)c0 + 2 * (int)(threadIdx.x & ~31u); c < (int)ce; c += 2 * (int)blockDim.x)
                thermal_duo_2k<D, S>(g, P, A, m.f[nxt], m.gp[cur], m.gp[nxt],
                                     duo_at(g, c + (int)(threadIdx.x & 31u), (int)ce), tick);
        }
    }
    start_next();
}

// Rows of a block of the one-launch 2D step.
constexpr int kEnsRows = 8;

// The step of 2D members in one launch (lbm_fast_tile.cuh), those that TileRule picks.  FP32 only: as
// for one lattice, half storage saves too little traffic to pay for the cells that are collided
// twice.  GB300, 60 members of up to 1024x512: 179 us a step; 200 steps and the read-out 44.7 ms
// against 49.5 of two kernels.
__global__ void __launch_bounds__(32 * kEnsRows, 32 / kEnsRows)
    k_ens_tile(const EnsMember<float>* __restrict__ mem, const int2* __restrict__ tiles, int ntiles, int flip) {
    using S = float;
    __shared__ __align__(16) unsigned sh[(sizeof(EnsStage<S>) + 3) / 4];
    __shared__ float sf[8 * 64 * kEnsRows];
    wait_for_previous();
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int2 tt = tiles[flip ? ntiles - 1 - t : t];  // every other step last tile first, as k_fast_tile
        const EnsStage<S>& st = stage_member<S>(mem, tt.x, sh, [flip](const EnsMember<S>& gm, FastArgs<S>& A) {
            const int c = gm.cur ^ flip, n = c ^ 1;
            A.Bin0 = gm.B[c][0]; A.Bin1 = gm.B[c][1];
            A.Bout0 = gm.B[n][0]; A.Bout1 = gm.B[n][1];
            A.lag_in = gm.L[c];
            A.lag_out = gm.L[n];
            A.ticks = gm.tick;
        });
        const EnsMember<S>& m = st.m;
        const int cur = m.cur ^ flip, nxt = cur ^ 1;
        tile_step<S, kEnsRows>(m.g, m.P, m.tp, st.A, st.A, m.f[cur], m.gp[cur], m.f[nxt], m.gp[nxt], tt.y, 0ULL, sf);
        tile_tick<S>(st.A.ticks, (unsigned)(m.tp.ntx * m.tp.nty), tt.y == 0 && threadIdx.x == 0);
    }
    start_next();
}

// Which 2D FP32 members take the one-launch step: those whose blocks own two fifths of the cells they
// hold (72% of a wide and tall member's; a member narrower than a block leaves columns idle, one a little
// wider than a block nearly a whole one), and the others as long as their blocks run in about two
// waves (four per SM), where the launch that is saved is most of the step.  GB300, us per step of one
// launch / two, with the share owned: 50 of 124x300 (73%) 49.9 / 59.2, 64 of 48x400 (56%) 38.6 /
// 39.9, 50 of 66x500 (38%) 66.4 / 54.8, 50 of 33x300 (39%) 21.2 / 16.9, 50 of 8x2000 (9%) 117.6 / 25.3;
// few blocks: 100 of 70x20 (34%) 8.2 / 12.9, 200 of 10x10 (10%) 4.8 / 6.1.
struct TileRule {
    bool sparse = false;  // members that own less take it as well
    static bool narrow(const EnsMemberHost& mh) { return !mh.F->wide && narrow_index(mh.geo, mh.dim == 3 ? 19 : 9); }
    static bool takes_tiles(const EnsMemberHost& mh, int precision) {
        return mh.dim == 2 && precision == LBM_FP32 && narrow(mh);
    }
    static long long blocks(const EnsMemberHost& mh) {
        const TilePlan tp = tile_plan(mh.geo, 64, kEnsRows);
        return (long long)tp.ntx * tp.nty;
    }
    static bool owns_enough(const EnsMemberHost& mh) { return 5 * mh.geo.ncell >= 2 * 64 * kEnsRows * blocks(mh); }
    TileRule(const std::vector<EnsMemberHost>& members, int precision, int sms) {
        long long n = 0;
        for (const EnsMemberHost& mh : members)
            if (takes_tiles(mh, precision) && !owns_enough(mh)) n += blocks(mh);
        sparse = n <= 8LL * sms;
    }
    int list_of(const EnsMemberHost& mh, int precision) const {
        if (takes_tiles(mh, precision) && (sparse || owns_enough(mh))) return kEnsTiles;
        return (mh.dim == 3 ? 1 : 0) + (narrow(mh) ? 0 : 2);
    }
};

template <class S>
static cudaError_t build_typed(EnsPlan& plan, const std::vector<EnsMemberHost>& members) {
    const TileRule rule(members, plan.precision, plan.sms);
    for (int li = 0; li < kEnsLists; ++li) {
        std::vector<EnsMember<S>> hm;
        std::vector<int2> tiles;
        for (const EnsMemberHost& mh : members) {
            if (rule.list_of(mh, plan.precision) != li) continue;
            EnsMember<S> m{};
            m.g = dev_geo(mh.geo, mh.phys);
            m.P = fast_physf(*mh.F, mh.phys);
            m.tick = mh.F->tick;
            for (int b = 0; b < 2; ++b) {
                m.f[b] = (S*)mh.F->fbuf[b];
                m.gp[b] = (S*)mh.F->gbuf[b];
                for (int c = 0; c < 3; ++c) m.B[b][c] = mh.F->B[b][c];
                m.L[b] = mh.F->L[b];
            }
            m.cur = mh.F->cur;
            const int idx = (int)hm.size();
            m.tp = tile_plan(m.g, 64, kEnsRows);
            const long long nt = li == kEnsTiles ? (long long)m.tp.ntx * m.tp.nty
                                                      : (m.g.ncell + plan.cfg.tile_cells - 1) / plan.cfg.tile_cells;
            for (long long t = 0; t < nt; ++t) tiles.push_back(make_int2(idx, (int)t));
            plan.cells += m.g.ncell;
            hm.push_back(m);
        }
        plan.nmembers[li] = (int)hm.size();
        plan.ntiles[li] = (int)tiles.size();
        if (hm.empty()) continue;
        cudaError_t e = cudaMalloc(&plan.d_members[li], hm.size() * sizeof(EnsMember<S>));
        if (e != cudaSuccess) return e;
        e = cudaMalloc((void**)&plan.d_tiles[li], tiles.size() * sizeof(int2));
        if (e != cudaSuccess) return e;
        e = cudaMemcpy(plan.d_members[li], hm.data(), hm.size() * sizeof(EnsMember<S>), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) return e;
        e = cudaMemcpy(plan.d_tiles[li], tiles.data(), tiles.size() * sizeof(int2), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

void ens_free(EnsPlan& plan) {
    for (int li = 0; li < kEnsLists; ++li) {
        if (plan.d_members[li]) cudaFree(plan.d_members[li]);
        if (plan.d_tiles[li]) cudaFree(plan.d_tiles[li]);
        plan.d_members[li] = nullptr;
        plan.d_tiles[li] = nullptr;
        plan.nmembers[li] = plan.ntiles[li] = 0;
    }
    plan.cells = 0;
}

cudaError_t ens_build(EnsPlan& plan, const std::vector<EnsMemberHost>& members, const EnsLaunchCfg& cfg, int sms) {
    ens_free(plan);
    plan.cfg = cfg;
    plan.sms = sms > 0 ? sms : 152;
    plan.precision = members.empty() ? LBM_FP32 : members[0].F->precision;
    return plan.precision == LBM_FP16 ? build_typed<__half>(plan, members) : build_typed<float>(plan, members);
}

template <int D, class S, bool WIDE>
static void launch_list(const EnsPlan& plan, int li, int stage, int flip, cudaStream_t s) {
    // a duo block of 128 threads takes the cells that a one-cell block of 256 takes
    const unsigned block = WIDE ? (unsigned)plan.cfg.block : 128u;
    const unsigned grid = (unsigned)min(plan.ntiles[li], plan.sms * plan.cfg.grid_mul);
    const EnsMember<S>* mem = (const EnsMember<S>*)plan.d_members[li];
    if (WIDE) {  // its cell bodies take read-only loads: no start before the last kernel's end
        if (stage == 0)
            k_ens_flow<D, S, WIDE><<<grid, block, 0, s>>>(mem, plan.d_tiles[li], plan.ntiles[li], plan.cfg.tile_cells, flip);
        else
            k_ens_thermal<D, S, WIDE><<<grid, block, 0, s>>>(mem, plan.d_tiles[li], plan.ntiles[li], plan.cfg.tile_cells, flip);
        return;
    }
    if (stage == 0)
        launch_after(k_ens_flow<D, S, WIDE>, grid, block, s, mem, plan.d_tiles[li], plan.ntiles[li], plan.cfg.tile_cells,
                     flip);
    else
        launch_after(k_ens_thermal<D, S, WIDE>, grid, block, s, mem, plan.d_tiles[li], plan.ntiles[li],
                     plan.cfg.tile_cells, flip);
}

template <class S>
static void step_typed(const EnsPlan& plan, int flip, cudaStream_t s) {
    for (int stage = 0; stage < 2; ++stage) {
        for (int li = 0; li < kEnsLists; ++li) {
            if (plan.ntiles[li] == 0) continue;
            if (li == kEnsTiles) {
                if (stage == 1) continue;
                const unsigned grid = (unsigned)min(plan.ntiles[li], plan.sms * plan.cfg.grid_mul);
                launch_after(k_ens_tile, grid, 32 * kEnsRows, s, (const EnsMember<float>*)plan.d_members[li],
                             plan.d_tiles[li], plan.ntiles[li], flip);
                continue;
            }
            switch (li) {
                case 0: launch_list<2, S, false>(plan, li, stage, flip, s); break;
                case 1: launch_list<3, S, false>(plan, li, stage, flip, s); break;
                case 2: launch_list<2, S, true>(plan, li, stage, flip, s); break;
                default: launch_list<3, S, true>(plan, li, stage, flip, s); break;
            }
        }
    }
}

void ens_step(const EnsPlan& plan, int flip, cudaStream_t s) {
    if (plan.precision == LBM_FP16) step_typed<__half>(plan, flip, s);
    else step_typed<float>(plan, flip, s);
}

}  // namespace lbm

// 1/rho of the fixed arithmetic (recip, csrc/lbm_fixed_cell.cuh) against long double over its range
// (1/2, 4), for test_cpu_fixed_recip.py.  Prints the largest relative error found just
// above 1/2, just below 4 and in between.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <random>

#include "lbm_fixed_cell.cuh"

using namespace lbm::fxa;

static long double err(long long rho) {
    const long double want = 1152921504606846976.0L * (1152921504606846976.0L / (long double)rho);
    return fabsl((long double)recip(Qb(rho)).s() - want) / want;
}

int main() {
    std::mt19937_64 rng(7);
    const long long lo = kOne / 2, hi = 4 * kOne;
    long double e[3] = {0, 0, 0};
    for (int b = 0; b < 59; ++b)  // distances 1, 2, 4 ... from both ends, with random low bits
        for (int r = 0; r < 2000; ++r) {
            const long long d = (1LL << b) + (long long)(rng() & ((1ULL << b) - 1));
            if (lo + d < hi) e[0] = std::max(e[0], err(lo + d));
            if (hi - d > lo) e[1] = std::max(e[1], err(hi - d));
        }
    for (int r = 0; r < 2000000; ++r) e[2] = std::max(e[2], err(lo + 1 + (long long)(rng() % (unsigned long long)(hi - lo - 1))));
    std::printf("%.3Le %.3Le %.3Le\n", e[0], e[1], e[2]);
    return 0;
}

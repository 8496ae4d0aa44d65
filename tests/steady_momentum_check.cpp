// Momentum through one steady-state FP32 flow collision (steady_flow, csrc/lbm_fast_math.cuh) over
// random states, for test_cpu_steady_momentum.py: the mean over all states of the relative gain of
// sum e d' along j + F against j + F itself (F the collision's force), and of the mass against its
// own.  Prints per dimension, relaxation time and force: mean momentum gain, mean mass gain.
#include "host_device.h"
#include "lbm_fast_math.cuh"

#include <cstdio>
#include <random>

using namespace lbm;

template <int D>
static void run(double tau, double force) {
    constexpr int Q = D == 3 ? 19 : 9;
    PhysC C{};
    C.Snu = 1.0 / tau;
    C.Sq = 8.0 * (2.0 * tau - 1.0) / (8.0 * tau - 1.0);
    PhysF P{};
    P.gBeta = (float)force;
    steady_constants(C, D, P);
    std::mt19937_64 rng(11);
    std::normal_distribution<double> N(0.0, 1.0);
    const int n = 400000;
    double gain = 0.0, mass = 0.0;
    for (int s = 0; s < n; ++s) {
        // a flow of speed about 0.05 with a density and a non-equilibrium part of its scale
        const double u[3] = {0.05 * N(rng), 0.05 * N(rng), D == 3 ? 0.05 * N(rng) : 0.0}, dr = 0.01 * N(rng);
        const double uu = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
        float d[Q];
        for (int a = 0; a < Q; ++a) {
            const int ex = Lat<Q>::ex(a), ey = Lat<Q>::ey(a), ez = Lat<Q>::ez(a), e2 = ex * ex + ey * ey + ez * ez;
            const double w = D == 3 ? (e2 == 0 ? 1.0 / 3 : e2 == 1 ? 1.0 / 18 : 1.0 / 36)
                                    : (e2 == 0 ? 4.0 / 9 : e2 == 1 ? 1.0 / 9 : 1.0 / 36);
            const double eu = ex * u[0] + ey * u[1] + ez * u[2];
            d[a] = (float)(w * ((1.0 + dr) * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * uu) - 1.0) + 1e-4 * w * N(rng));
        }
        double want[4] = {0, 0, 0, 0}, got[4] = {0, 0, 0, 0};
        auto moments = [&](double* m) {
            for (int a = 0; a < Q; ++a) {
                m[0] += Lat<Q>::ex(a) * (double)d[a];
                m[1] += Lat<Q>::ey(a) * (double)d[a];
                m[2] += Lat<Q>::ez(a) * (double)d[a];
                m[3] += (double)d[a];
            }
        };
        moments(want);
        want[1] += (double)steady_flow<D, float>(d, 0.0f, (float)(0.3 * N(rng)), P);
        moments(got);
        const double jj = want[0] * want[0] + want[1] * want[1] + want[2] * want[2];
        gain += (got[0] * want[0] + got[1] * want[1] + got[2] * want[2]) / jj - 1.0;
        mass += got[3] - want[3];
    }
    std::printf("%d %.2f %g %.3e %.3e\n", D, tau, force, gain / n, mass / n);
}

int main() {
    for (double tau : {0.51, 0.55, 0.7, 1.0})
        for (double force : {0.0, 1e-3}) {
            run<2>(tau, force);
            run<3>(tau, force);
        }
    return 0;
}

// Momentum through one FP32 flow collision over random states, for test_cpu_steady_momentum.py: the
// steady-state form (steady_flow, csrc/lbm_fast_math.cuh) beside the moment-space form that the first
// step takes (fcollide_2d, fcollide_3d).  Prints per dimension and relaxation time the mean relative gain
// of sum e d' along j against j itself of either form, and the mean mass gain of the steady-state form.
#include "host_device.h"
#include "lbm_fast_math.cuh"

#include <cstdio>
#include <random>

using namespace lbm;

template <int D>
static void run(double tau) {
    constexpr int Q = D == 3 ? 19 : 9;
    PhysC C{};
    C.Snu = C.Se = C.Seps = C.Spi = 1.0 / tau;
    C.Sq = C.Sm = 8.0 * (2.0 * tau - 1.0) / (8.0 * tau - 1.0);
    PhysF P = to_physf(C);
    steady_constants(C, D, P);
    std::mt19937_64 rng(11);
    std::normal_distribution<double> N(0.0, 1.0);
    const int n = 400000;
    double gain[2] = {0.0, 0.0}, mass = 0.0;
    for (int s = 0; s < n; ++s) {
        // a flow of speed about 0.05 with a density and a non-equilibrium part of its scale
        const double u[3] = {0.05 * N(rng), 0.05 * N(rng), D == 3 ? 0.05 * N(rng) : 0.0}, dr = 0.01 * N(rng);
        const double uu = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
        float d[Q], dp[Q];
        for (int a = 0; a < Q; ++a) {
            const int ex = Lat<Q>::ex(a), ey = Lat<Q>::ey(a), ez = Lat<Q>::ez(a), e2 = ex * ex + ey * ey + ez * ez;
            const double w = D == 3 ? (e2 == 0 ? 1.0 / 3 : e2 == 1 ? 1.0 / 18 : 1.0 / 36)
                                    : (e2 == 0 ? 4.0 / 9 : e2 == 1 ? 1.0 / 9 : 1.0 / 36);
            const double eu = ex * u[0] + ey * u[1] + ez * u[2];
            d[a] = (float)(w * ((1.0 + dr) * (1.0 + 3.0 * eu + 4.5 * eu * eu - 1.5 * uu) - 1.0) + 1e-4 * w * N(rng));
        }
        struct Moments {
            double m[4] = {0, 0, 0, 0};
            explicit Moments(const float* x) {
                for (int a = 0; a < Q; ++a) {
                    m[0] += Lat<Q>::ex(a) * (double)x[a];
                    m[1] += Lat<Q>::ey(a) * (double)x[a];
                    m[2] += Lat<Q>::ez(a) * (double)x[a];
                    m[3] += (double)x[a];
                }
            }
            double along(const Moments& o) const {
                return (m[0] * o.m[0] + m[1] * o.m[1] + m[2] * o.m[2]) / (o.m[0] * o.m[0] + o.m[1] * o.m[1] + o.m[2] * o.m[2]);
            }
        };
        const Moments want(d);
        float r, rho, v[3], Fy;
        fmacro<D>(d, 0.0f, P, r, rho, v[0], v[1], v[2], Fy);
        if (D == 2) fcollide_2d(d, r, rho, v[0], v[1], 0.0f, P, dp);
        else fcollide_3d(d, r, rho, v[0], v[1], v[2], 0.0f, P, dp);
        gain[0] += Moments(dp).along(want) - 1.0;
        steady_flow<D, float>(d, 0.0f, 0.0f, P);
        gain[1] += Moments(d).along(want) - 1.0;
        mass += Moments(d).m[3] - want.m[3];
    }
    std::printf("%d %.2f %.4e %.4e %.3e\n", D, tau, gain[0] / n, gain[1] / n, mass / n);
}

int main() {
    for (double tau : {0.51, 0.55, 0.7, 1.0}) {
        run<2>(tau);
        run<3>(tau);
    }
    return 0;
}

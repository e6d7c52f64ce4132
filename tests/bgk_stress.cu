// Host program of test_cells_host.py: the stress that the packed BGK kernel takes its Smagorinsky tau from, against FP64.
//
// Nodes near equilibrium, density and velocity rounded as the kernel has them. Bound: the error, on the same nodes, of the
// form that the one-node kernels use, the sum over the pairs of c c (f_q + f_opp - 2 f_eq,even).
#include <cmath>
#include <cstdio>
#include <random>

#include "pairs2.cuh"

using namespace wk;

template <int Q>
int check() {
    using L = Lat<Q>;
    std::mt19937 rng(7);
    std::normal_distribution<double> n01;
    double err[2][2] = {};  // [packed, pair sums][diagonal, off-diagonal]
    const int nodes = 100000, ax[6] = {0, 1, 2, 0, 1, 0}, bx[6] = {0, 1, 2, 1, 2, 2};
    for (int i = 0; i < nodes; ++i) {
        const double rho = 1.0 + 0.01 * n01(rng), u[3] = {0.04 * n01(rng), 0.04 * n01(rng), 0.04 * n01(rng)};
        float2 f[Q];
        double F = 0.0, J[3] = {}, M[6] = {};
        for (int q = 0; q < Q; ++q) {
            const double c[3] = {double(L::cx(q)), double(L::cy(q)), double(L::cz(q))};
            const double cu = c[0] * u[0] + c[1] * u[1] + c[2] * u[2], u2 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2];
            const double feq = L::w(q) * rho * (1.0 + 3.0 * cu + 4.5 * cu * cu - 1.5 * u2);
            f[q] = bc2(static_cast<float>(feq + 1e-3 * L::w(q) * n01(rng)));
            F += f[q].x;
            for (int a = 0; a < 3; ++a) J[a] += c[a] * f[q].x;
            for (int k = 0; k < 6; ++k) M[k] += c[ax[k]] * c[bx[k]] * f[q].x;
        }
        float2 r, j[3], dev, p[6], v[3];
        bgk_sums2<Q, true>(f, r, j, dev, p);
        const float inv = 1.0f / r.x;
        for (int a = 0; a < 3; ++a) v[a] = mul2(j[a], bc2(inv));
        bgk_stress2(r, v, dev, p);
        float pair[6] = {};
        const float a0 = 1.0f - 1.5f * (v[0].x * v[0].x + v[1].x * v[1].x + v[2].x * v[2].x);
        for (int q = 1; q < Q; ++q) {
            const int o = L::opp(q), c[3] = {L::cx(q), L::cy(q), L::cz(q)};
            if (o < q) continue;
            const float cu = float(c[0]) * v[0].x + float(c[1]) * v[1].x + float(c[2]) * v[2].x;
            const float fn = (f[q].x + f[o].x) - 2.0f * (L::w(q) * r.x * (a0 + 4.5f * cu * cu));
            for (int k = 0; k < 6; ++k) pair[k] += float(c[ax[k]] * c[bx[k]]) * fn;
        }
        for (int k = 0; k < 6; ++k) {
            const double want = M[k] - (k < 3 ? F / 3.0 : 0.0) - J[ax[k]] * J[bx[k]] / F;
            err[0][k / 3] += (p[k].x - want) * (p[k].x - want);
            err[1][k / 3] += (pair[k] - want) * (pair[k] - want);
        }
    }
    int bad = 0;
    for (int k = 0; k < 2; ++k) {
        const double a = std::sqrt(err[0][k] / (3.0 * nodes)), b = std::sqrt(err[1][k] / (3.0 * nodes));
        std::printf("D3Q%d %s: %.2e, pair sums %.2e\n", Q, k ? "off-diagonal" : "diagonal", a, b);
        bad += !(a <= b);
    }
    return bad;
}

int main() { return check<19>() + check<27>(); }

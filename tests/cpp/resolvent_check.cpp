// Host-only check of tridiag_resolvent: T of plain Lanczos runs (FP64, no
// reorthogonalisation) on diagonal matrices, the start vector orthogonal to the
// lowest level but for 1e-11 of it; against the sum over the other levels.  Runs
// past the point where the level comes back; small gaps; and a level of real
// weight on z, which is not left out.
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "ed_tridiag.hpp"

using namespace ed;

static long double fraction(int n, const double* a, const double* off, double z) {
    long double g = 1.0L / ((long double)z - a[n - 1]);
    for (int k = n - 2; k >= 0; --k) g = 1.0L / ((long double)z - a[k] - g * (long double)off[k] * off[k]);
    return g;
}

int main() {
    const int dim = 600;
    int fails = 0, plain_bad = 0, runs = 0;
    double worst = 0.0, worst_plain = 0.0;
    for (int seed = 0; seed < 40; ++seed)
        for (double gap : {0.5, 0.05}) {
            std::mt19937_64 rng(seed);
            std::uniform_real_distribution<double> u(-1.0, 1.0);
            std::vector<double> d(dim), b(dim);
            d[0] = -5.0;
            d[1] = -5.0 + gap;
            for (int i = 2; i < dim; ++i) d[i] = 5.5 + 9.5 * u(rng);
            long double exact = 0.0L;
            double nn = 0.0;
            for (int i = 0; i < dim; ++i) b[i] = i ? u(rng) : 0.0, nn += b[i] * b[i];
            for (int i = 0; i < dim; ++i) b[i] /= std::sqrt(nn);
            for (int i = 1; i < dim; ++i) exact += (long double)b[i] * b[i] / ((long double)d[0] - d[i]);
            b[0] = 1e-11;
            for (int steps : {60, 100, 150, 200, 250}) {
                std::vector<double> a, off(1, 0.0), q = b, p(dim, 0.0);
                for (int k = 0; k < steps; ++k) {
                    std::vector<double> w(dim);
                    double al = 0.0, bn = 0.0;
                    for (int i = 0; i < dim; ++i) w[i] = d[i] * q[i] - off[k] * p[i], al += w[i] * q[i];
                    for (int i = 0; i < dim; ++i) w[i] -= al * q[i], bn += w[i] * w[i];
                    bn = std::sqrt(bn);
                    a.push_back(al);
                    off.push_back(bn);
                    p = q;
                    for (int i = 0; i < dim; ++i) q[i] = w[i] / bn;
                }
                const double e = std::fabs((double)(tridiag_resolvent(steps, a.data(), off.data() + 1, d[0]) / exact - 1.0L));
                const double f = std::fabs((double)(fraction(steps, a.data(), off.data() + 1, d[0]) / exact - 1.0L));
                ++runs;
                plain_bad += f > 1e-9;
                worst = std::max(worst, e);
                worst_plain = std::max(worst_plain, f);
                if (steps >= 100 && !(e < 1e-9)) {
                    std::printf("seed %d gap %g steps %d: error %g (fraction %g)\n", seed, gap, steps, e, f);
                    ++fails;
                }
            }
        }
    // 2 x 2 and 1 x 1; a pole of weight 1/2 at 1e-13 from z stays
    const double a1[1] = {2.0}, a2[2] = {1.0, 1.0 + 2e-13}, o2[1] = {1e-13};
    if (std::fabs((double)tridiag_resolvent(1, a1, nullptr, 0.5) + 1.0 / 1.5) > 1e-15) ++fails;
    const double near = (double)fraction(2, a2, o2, 1.0 + 5e-13);
    if (!((double)tridiag_resolvent(2, a2, o2, 1.0 + 5e-13) == near) || std::fabs(near) < 1e11) ++fails;
    std::printf("%d runs, worst %g (fraction alone %g, %d beyond 1e-9), %d fail%s\n", runs, worst, worst_plain, plain_bad,
                fails, fails ? "" : " ok");
    return fails || plain_bad == 0 ? 1 : 0;
}

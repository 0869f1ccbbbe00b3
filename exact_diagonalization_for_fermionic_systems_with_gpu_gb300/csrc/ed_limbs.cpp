// ed_limbs.cpp — see ed_limbs.hpp.
#include "ed_limbs.hpp"

#include <algorithm>
#include <climits>
#include <cmath>

namespace ed {
namespace {

// Fraction bits that keep coefficients of largest magnitude mx and magnitude
// sum `sum` within the limits (one bit below: the roundings of sum and of c_k).
int limb_frac(double mx, double sum) {
    int ka, kb;
    std::frexp(mx, &ka);
    std::frexp(sum, &kb);
    return std::min(56 - ka, 60 - kb);
}

void limb_store(double r, int F, int32_t* hl) {
    const int64_t c = (int64_t)std::llrint(std::ldexp(r, F));
    hl[1] = (int32_t)(c & ((1 << kLimbBits) - 1));
    hl[0] = (int32_t)(c >> kLimbBits);
}

}  // namespace

int limb_coefs(const double* r, int n, int32_t* hl) {
    double mx = 0.0, sum = 0.0;
    for (int k = 0; k < n; ++k) {
        mx = std::max(mx, std::fabs(r[k]));
        sum += std::fabs(r[k]);
    }
    const int F = mx > 0.0 ? limb_frac(mx, sum) : 0;
    for (int k = 0; k < n; ++k) limb_store(r[k], F, hl + 2 * k);
    return F;
}

RitzCoefs ritz_coefs(const double* r, const double* norm, int n, int batch) {
    RitzCoefs out;
    out.hl.resize(2 * (size_t)n);
    const double tol = kRitzTol / std::sqrt((double)std::max(n, 1));
    // fraction bits coefficient k asks for: r_k's last bit, or a rounding error
    // 2^-(F+1) |q_k| within tol
    auto need = [&](int k) {
        if (r[k] == 0.0) return INT_MIN;
        int kr, kt;
        std::frexp(r[k], &kr);
        std::frexp(tol / norm[k], &kt);
        return std::min(53 - kr, -kt);
    };
    struct Run {
        double mx = 0.0, sum = 0.0;
        int need = INT_MIN;
    };
    auto add = [&](Run a, int k0, int k1) {
        for (int k = k0; k < k1; ++k) {
            a.mx = std::max(a.mx, std::fabs(r[k]));
            a.sum += std::fabs(r[k]);
            a.need = std::max(a.need, need(k));
        }
        return a;
    };
    auto fits = [](const Run& a) { return a.mx == 0.0 || limb_frac(a.mx, a.sum) >= a.need; };
    std::vector<int> F;
    for (int k0 = 0; k0 < n;) {
        Run a;
        int k = k0;
        // whole batches; else fours, else one by one (a single one always fits)
        for (int step : {batch, 4, 1}) {
            while (k < n) {
                const int k1 = std::min(n, k + step);
                const Run b = add(a, k, k1);
                if (!fits(b) && !(step == 1 && k == k0)) break;
                a = b;
                k = k1;
            }
            if (k > k0) break;
        }
        F.push_back(a.mx > 0.0 ? limb_frac(a.mx, a.sum) : INT_MAX);
        if (a.mx > 0.0)
            for (int t = k0; t < k; ++t) limb_store(r[t], F.back(), out.hl.data() + 2 * t);
        out.segs.push_back({k, 0});
        k0 = k;
    }
    // the total's F: the segments' smallest, less the guard bits of their sum
    int Fmin = INT_MAX, guard = 0;
    for (int f : F) Fmin = std::min(Fmin, f);
    if (Fmin == INT_MAX) return out;
    while ((1LL << guard) < (long long)F.size()) ++guard;
    out.F = Fmin - guard;
    for (size_t s = 0; s < F.size(); ++s)
        out.segs[s].shift = F[s] == INT_MAX ? 0 : (int32_t)std::min<long long>((long long)F[s] - out.F, 126);
    return out;
}

}  // namespace ed

// Host-only check of the Ritz sum's integer coefficients (ed_limbs.cpp): the
// limbs put together are r_k 2^F to its last bit, or to an error of at most
// kRitzTol / sqrt(n) in the sum's norm; the limits the device sums rely on; the
// segments and their shifts.  The common F of limb_coefs does not keep those bits
// where the vectors' norms are far apart.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <string>
#include <vector>

#include "ed_limbs.hpp"

using namespace ed;

struct Profile {
    std::vector<double> r, norm;
};

static double uni() { return (std::rand() + 0.5) / ((double)RAND_MAX + 1.0); }

// weights z_k, |q_k| between 2^53 (one large element) and spread over rows
static Profile make(const std::string& kind, int n) {
    Profile p;
    for (int k = 0; k < n; ++k) {
        double z = (2.0 * uni() - 1.0) / std::sqrt((double)n), norm = std::ldexp(1.0 + uni(), 53);
        if (kind == "lanczos14") norm *= 1.0 + 2000.0 * std::exp(-k / 6.0), z *= std::exp(-0.02 * (n - k));
        if (kind == "decay") z = std::exp(-2.0 * k) * (1.0 - 0.5 * uni());
        if (kind == "grow") z = std::exp(-2.5 * (n - 1 - k));
        if (kind == "wild") norm *= std::ldexp(1.0, std::rand() % 40), z *= std::ldexp(1.0, -(std::rand() % 50));
        if (kind == "zeros" && k % 3) z = 0.0;
        if (kind == "all_zero") z = 0.0;
        if (kind == "scaled") z *= 1e-200, norm *= 1e200;
        p.r.push_back(z / norm);
        p.norm.push_back(norm);
    }
    return p;
}

// the largest error of a term against what it may be (1: at the limit)
static double worst(const Profile& p, const std::vector<int32_t>& hl, const std::vector<int>& F) {
    const int n = (int)p.r.size();
    double w = 0.0;
    for (int k = 0; k < n; ++k) {
        const long double c = (long double)hl[2 * k] * (1 << kLimbBits) + hl[2 * k + 1];
        const double err = (double)fabsl(ldexpl(c, -F[k]) - (long double)p.r[k]);
        w = std::max(w, err * p.norm[k] / (kRitzTol / std::sqrt((double)n)));
    }
    return w;
}

static int check(const std::string& kind, int n, int batch) {
    std::srand(17 + n);
    const Profile p = make(kind, n);
    const RitzCoefs rc = ritz_coefs(p.r.data(), p.norm.data(), n, batch);
    std::vector<int> F(n, 0);
    int k = 0, odd = 0;
    long double total = 0.0L;  // the largest the total can get, in units of 2^-F
    for (const RitzSeg& s : rc.segs) {
        if (s.end <= k || s.end > n || s.shift < 0 || s.shift > 126) return std::printf("%s %d: segment\n", kind.c_str(), n), 1;
        odd += s.end < n && (s.end - k) % batch != 0;
        long double sum = 0.0L;
        for (; k < s.end; ++k) {
            F[k] = rc.F + s.shift;
            const long long c = (long long)rc.hl[2 * k] * (1 << kLimbBits) + rc.hl[2 * k + 1];
            if (std::llabs(c) >= 1LL << 57 || rc.hl[2 * k + 1] < 0 || rc.hl[2 * k + 1] >= 1 << kLimbBits)
                return std::printf("%s %d: coefficient %d\n", kind.c_str(), n, k), 1;
            sum += std::llabs(c);
        }
        if (sum >= ldexpl(1.0L, 61)) return std::printf("%s %d: sum\n", kind.c_str(), n), 1;
        total += ldexpl(sum, 54 - s.shift);
    }
    if (k != n || total >= ldexpl(1.0L, 126)) return std::printf("%s %d: total\n", kind.c_str(), n), 1;
    const double w = worst(p, rc.hl, F);
    std::vector<int32_t> hl(2 * (size_t)n);
    const double w1 = worst(p, hl, std::vector<int>(n, limb_coefs(p.r.data(), n, hl.data())));
    if (!(w <= 1.0)) return std::printf("%s %d: error %g\n", kind.c_str(), n, w), 1;
    if (kind == "lanczos14" && n >= 100 && !(w1 > 1.0)) return std::printf("%s %d: one F would do\n", kind.c_str(), n), 1;
    std::printf("%s %d: %zu segments (%d inside a batch), error %.3f of the limit (one F: %.3g) ok\n", kind.c_str(), n,
                rc.segs.size(), odd, w, w1);
    return 0;
}

int main() {
    int fails = 0;
    for (const char* kind : {"flat", "lanczos14", "decay", "grow", "wild", "zeros", "all_zero", "scaled"})
        for (int n : {1, 15, 16, 17, 100, 128, 129, 300, 1000}) fails += check(kind, n, 16);
    return fails ? 1 : 0;
}

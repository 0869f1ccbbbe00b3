// Host-only check of the complex row engine's class schedule
// (build_class_schedule): every entry of a column is read exactly once, in the
// steps of its class and with its sign; every other step reads the zero slot;
// negative counts per class.
#include <cstdio>
#include <map>
#include <string>
#include <vector>

#include "ed_tables.hpp"

using namespace ed;

static int check(const char* name, int n, int q, const std::vector<ed_term>& terms, bool takes = true) {
    SpinBasis b;
    b.build(n, q);
    SpinTable t;
    std::string err;
    if (build_spin(b, terms.data(), (int)terms.size(), true, &t, nullptr, &err) != ED_OK) {
        std::printf("%s: table failed: %s\n", name, err.c_str());
        return 1;
    }
    ClassSchedule g;
    if (build_class_schedule(t, &g, &err) != takes) {
        std::printf("%s: %s\n", name, err.c_str());
        return 1;
    }
    for (int64_t d = 0; takes && d < g.cpad; ++d) {
        int s = 0;
        for (int c = 0; c < 4; ++c) {
            std::map<int64_t, int> want, got;
            int neg = 0;
            if (d < t.count)
                for (int k = 0; k < t.len[d]; ++k) {
                    const uint32_t e = t.ent[(size_t)k * t.count + d];
                    if ((int)((e >> kClassShift) & kClassMask) != c) continue;
                    const bool m = e & kSignBit;
                    neg += m;
                    const int64_t tc = (int64_t)(e & kColMask) + 1;
                    ++want[m ? -tc : tc];
                }
            const int ns = (g.steps4[d / 32] >> (8 * c)) & 0xFF;
            for (int k = 0; k < ns; ++k, ++s) {
                const uint32_t w = g.words[(size_t)s * g.cpad + d], col = w & 0x7FFFu;
                if (col == (uint64_t)t.count && !(w & 0x8000u)) continue;
                ++got[w & 0x8000u ? -((int64_t)col + 1) : (int64_t)col + 1];
            }
            if (want != got || (int)((g.negcnt[d] >> (8 * c)) & 0xFF) != neg) {
                std::printf("%s: column %lld class %d\n", name, (long long)d, c);
                return 1;
            }
        }
        if (s > g.steps) {
            std::printf("%s: steps\n", name);
            return 1;
        }
    }
    std::printf("%s classes %zu steps %d ok\n", name, t.coef.size(), g.steps);
    return 0;
}

int main() {
    auto ring = [](int n, double phase, bool two) {
        std::vector<ed_term> v;
        for (int i = 0; i < n; ++i) v.push_back({ED_TERM_PEIERLS, i, (i + 1) % n, 0, -1.0, phase});
        for (int i = 0; two && i < n; ++i) v.push_back({ED_TERM_PEIERLS, i, (i + 2) % n, 0, -0.5, 2 * phase});
        return v;
    };
    int fails = 0;
    fails += check("ring10_flux", 10, 5, ring(10, 0.3, false));
    fails += check("ring12_two_ranges", 12, 6, ring(12, 0.2, true));
    fails += check("ring9_odd", 9, 4, ring(9, 0.7, true));
    fails += check("ring6_imaginary", 6, 3, ring(6, 1.5707963267948966, false));
    fails += check("dimer", 2, 1, {{ED_TERM_PEIERLS, 0, 1, 0, 1.0, 0.4}});
    fails += check("no_hops", 6, 6, ring(6, 0.3, true));
    std::vector<ed_term> many;
    for (int i = 0; i < 8; ++i) many.push_back({ED_TERM_PEIERLS, i, (i + 1) % 8, 0, -1.0 - i, 0.3});
    fails += check("too_many_classes", 8, 4, many, false);
    return fails ? 1 : 0;
}

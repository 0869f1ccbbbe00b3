// Host-only check of the row-pair matvec's schedule (build_pair_schedule): for
// tables of several shapes and both column assignments, every entry of a
// column is read exactly once with its sign, every other step reads a zero
// slot, the slots of a quarter warp's step are on different bank groups, and
// pair_slot is a bijection below zbase.
#include <cstdio>
#include <map>
#include <set>
#include <string>
#include <vector>

#include "ed_tables.hpp"

using namespace ed;

static int check(const char* name, int n, int q, const std::vector<ed_term>& terms) {
    SpinBasis b;
    b.build(n, q);
    SpinTable t;
    std::string err;
    if (build_spin(b, terms.data(), (int)terms.size(), false, &t, nullptr, &err) != ED_OK) {
        std::printf("%s: table failed: %s\n", name, err.c_str());
        return 1;
    }
    for (int adjacent = 0; adjacent < 2; ++adjacent) {
        PairSchedule g;
        if (!build_pair_schedule(t, adjacent != 0, &g, &err)) {
            std::printf("%s: %s\n", name, err.c_str());
            return 1;
        }
        std::map<uint32_t, uint32_t> column;  // slot -> column
        for (uint32_t c = 0; c < (uint32_t)t.count; ++c) {
            if (pair_slot(c) >= (uint64_t)g.zbase || !column.emplace(pair_slot(c), c).second) {
                std::printf("%s: slot of column %u\n", name, c);
                return 1;
            }
        }
        bool neg = false, pos = false;
        for (int64_t c = 0; c < t.count; ++c)
            for (int k = 0; k < t.len[c]; ++k) (t.ent[(size_t)k * t.count + c] & kSignBit ? neg : pos) = true;
        if (g.sign != (neg && pos ? 0 : (neg ? -1 : 1))) {
            std::printf("%s: sign %d\n", name, g.sign);
            return 1;
        }
        std::set<int64_t> seen;
        for (int64_t hb = 0; hb < 2 * g.blocks; ++hb)
            for (int lane = 0; lane < 32; ++lane) {
                const int64_t c = (hb / 2) * 64 + (adjacent ? 2 * lane + (hb & 1) : lane + 32 * (hb & 1));
                std::map<int64_t, int> want, got;
                int negs = 0;
                if (c < t.count) {
                    seen.insert(c);
                    for (int k = 0; k < t.len[c]; ++k) {
                        const uint32_t e = t.ent[(size_t)k * t.count + c];
                        const bool m = g.sign == 0 && (e & kSignBit);
                        negs += m;
                        const int64_t tc = (int64_t)(e & kColMask) + 1;
                        ++want[m ? -tc : tc];
                    }
                    if (g.negcnt[c] != negs) {
                        std::printf("%s: negative count of column %lld\n", name, (long long)c);
                        return 1;
                    }
                }
                for (int s = 0; s < 8 * g.groups; ++s) {
                    const uint32_t w = g.words[(((size_t)hb * g.groups + s / 8) * 32 + lane) * 8 + s % 8];
                    const uint32_t slot = w & 0x7FFFu;
                    if (slot >= (uint64_t)g.zbase) {
                        if (slot >= (uint64_t)g.zbase + 8 || (w & 0x8000u)) {
                            std::printf("%s: zero slot %u\n", name, w);
                            return 1;
                        }
                        continue;
                    }
                    if (s >= g.steps[hb] || !column.count(slot)) {
                        std::printf("%s: entry past the steps or outside the row\n", name);
                        return 1;
                    }
                    const int64_t tc = (int64_t)column[slot] + 1;
                    ++got[w & 0x8000u ? -tc : tc];
                }
                if (want != got) {
                    std::printf("%s: column %lld differs from the table\n", name, (long long)c);
                    return 1;
                }
            }
        if ((int64_t)seen.size() != t.count) {
            std::printf("%s: columns missing\n", name);
            return 1;
        }
        for (int64_t hb = 0; hb < 2 * g.blocks; ++hb)
            for (int qw = 0; qw < 4; ++qw)
                for (int s = 0; s < g.steps[hb]; ++s) {
                    std::map<uint32_t, uint32_t> bank;  // bank group -> slot
                    for (int l = 0; l < 8; ++l) {
                        const uint32_t slot = g.words[(((size_t)hb * g.groups + s / 8) * 32 + 8 * qw + l) * 8 + s % 8] & 0x7FFFu;
                        const auto it = bank.emplace(slot & 7u, slot).first;
                        // past a quarter's own steps the lanes share one zero slot
                        if (it->second != slot) {
                            std::printf("%s: two slots of one bank group in a step\n", name);
                            return 1;
                        }
                    }
                }
        std::printf("%s adjacent %d count %lld groups %d sign %d ok\n", name, adjacent, (long long)t.count, g.groups, g.sign);
    }
    return 0;
}

int main() {
    auto ring = [](int n, bool closed, double t) {
        std::vector<ed_term> v;
        for (int i = 0; i + 1 < n + (closed ? 1 : 0); ++i) v.push_back({ED_TERM_HOP, i, (i + 1) % n, 0, t, 0.0});
        return v;
    };
    auto two = ring(12, true, -1.0);
    for (int i = 0; i < 12; ++i) two.push_back({ED_TERM_HOP, i, (i + 2) % 12, 0, -1.0, 0.0});
    int fails = 0;
    fails += check("chain13_q6", 13, 6, ring(13, false, -1.0));
    fails += check("chain9_q4_plus", 9, 4, ring(9, false, 1.0));
    fails += check("ring10_q5", 10, 5, ring(10, true, -1.0));
    fails += check("ring12_nnn_q7", 12, 7, two);
    fails += check("ring12_nnn_q1", 12, 1, two);
    fails += check("dimer_q1", 2, 1, ring(2, false, -1.0));
    fails += check("full_q6", 6, 6, ring(6, true, -1.0));
    return fails ? 1 : 0;
}

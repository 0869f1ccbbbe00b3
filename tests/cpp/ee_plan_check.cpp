// Host-only check of the entanglement blocks' plan (ed_ee_plan.hpp): every block
// whose rows, dealt evenly to 16 CTAs, fit shared memory beside five column vectors
// and a row vector takes a cluster, whatever its share of the work; the cuts of
// half-filled 14- to 16-site chains that are near that limit among them.
#include <cstdio>
#include <initializer_list>

#include "ed_ee_plan.hpp"

using namespace ed;

int main() {
    const size_t cap = 232448 / sizeof(double);  // 227 KB
    int fails = 0, blocks = 0;
    for (int n = 1; n <= 700; ++n)
        for (int m = n; m <= 30000; ++m) {
            const size_t R = (m + 15) / 16;
            if (R * n + 5 * (size_t)n + R + 4 > cap) break;
            ++blocks;
            for (double share : {1.0, 1e-6})
                for (int top : {1, 4, 16}) {
                    const int g = bd_cluster(m, n, share, top, cap);
                    if (g >= kBdSizes || bd_smem_doubles(m, n, kBdGroups >> g) > cap) ++fails;
                }
        }
    const int cuts[][2] = {{735, 560}, {1960, 225}, {1960, 224}, {3024, 147}, {924, 448}};
    for (const auto& c : cuts)
        if (bd_cluster(c[0], c[1], 1.0, 16, cap) != kBdSizes - 1) {
            std::printf("%d x %d\n", c[0], c[1]);
            ++fails;
        }
    std::printf("%d blocks, %d fail%s\n", blocks, fails, fails ? "" : " ok");
    return fails ? 1 : 0;
}

// ed_ee_plan.hpp — row groups, shared memory and cluster size of the entanglement
// blocks' bidiagonalisation (ed_ee_bidiag.cu).
#pragma once

#include <cstddef>

namespace ed {

// Rows are summed in kBdGroups fixed groups combined in a binary tree, whatever
// the cluster size, so that a block's result does not depend on how many CTAs
// it got (and a state's not on the batch it came in).
constexpr int kBdGroups = 32;

constexpr int bd_group_rows(int m) { return (m + kBdGroups - 1) / kBdGroups; }

// Dynamic shared memory (doubles) of a CTA holding G groups of an m x n block: its
// rows, the groups' column sums (which double as the sums' total and the two
// reflectors' local copies), row k, the right reflector with its tau, a vector over
// the rows, two scalars.  On 16 CTAs (G = 2) four column vectors; with one for each
// of those purposes it was seven, and 1960 x 225 (14 sites, six in A) and 735 x 560
// (15 sites, seven in A) were left to gesvd: the entropies of a 14-site 6+6 state
// 201 -> 169 ms.
constexpr size_t bd_smem_doubles(int m, int n, int G) {
    const size_t R = (size_t)bd_group_rows(m) * G;
    return R * n + (size_t)(G + 2) * n + 1 + R + 2;
}

// Cluster size (log2) of an m x n block that is `share` times the largest one's
// work when that gets `top` CTAs: in proportion to the work, and large enough
// for the rows to fit the CTAs' shared memory (kBdSizes: it fits none).
constexpr int kBdSizes = 5;  // cluster sizes 1, 2, 4, 8, 16

inline int bd_cluster(int m, int n, double share, int top, size_t cap) {
    int g = 0;
    while (g < kBdSizes - 1 && (double)(1 << g) < top * share) ++g;
    while (g < kBdSizes && bd_smem_doubles(m, n, kBdGroups >> g) > cap) ++g;
    return g;
}

// Time of a block on 2^g CTAs: 7.5 us of barriers and scalar code a step and
// 2.4e9 multiply-adds/s a CTA (300 x 300 on 16, 8 and 4 CTAs: 3.32, 3.98, 5.83 ms).
inline double bd_seconds(int m, int n, int g) {
    const double fma = 2.0 * n * n * ((double)m - n / 3.0);
    return 7.5e-6 * n + fma / (2.4e9 * (1 << g));
}

}  // namespace ed

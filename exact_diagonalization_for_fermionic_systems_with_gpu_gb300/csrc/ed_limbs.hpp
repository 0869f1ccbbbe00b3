// ed_limbs.hpp — integer coefficients of the exact sums over basis vectors
// (dev::limb_mac in ed_device.cuh): sum_k r_k q_k with 54-bit integers q_k.
#pragma once

#include <cstdint>
#include <vector>

namespace ed {

constexpr int kLimbBits = 27;

// The real r[0..n) scaled to c_k = round(r_k 2^F), |c_k| < 2^57 and sum |c_k| <
// 2^61, each split at 27 bits into (high, low); returns F.
int limb_coefs(const double* r, int n, int32_t* hl);

// The same with an F for each run of coefficients, where one F would round the
// small coefficients of a run to fewer bits than they have: the vectors of a
// Lanczos run are scaled by their largest element, so the coefficient of a spread
// vector is far below that of a localised one of the same weight (14-site chain,
// 100 steps: |q_0| = 2^65, |q_10| = 2^55.4; against a sum whose coefficients keep 62
// bits each, the vector under the common F was off by 1.3e-15 in norm, 13-site
// 6+6 3.3e-15; in segments 7e-17, the rounding of the normalised elements).  A
// coefficient keeps the 53 bits of r_k, or, where its whole term is small, an
// error of at most kRitzTol / sqrt(n) in the sum's norm; norm[k] = |q_k|.
struct RitzSeg {
    int32_t end;    // vectors of this segment: from the end of the one before
    int32_t shift;  // its sum's fraction bits beyond the total's
};
constexpr double kRitzTol = 1.0 / (1LL << 55);

struct RitzCoefs {
    std::vector<int32_t> hl;    // 2 n
    std::vector<RitzSeg> segs;  // ends on multiples of `batch` from the segment's start where the bits allow
    int F = 0;                  // fraction bits of the total
};

RitzCoefs ritz_coefs(const double* r, const double* norm, int n, int batch);

}  // namespace ed

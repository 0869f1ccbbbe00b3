// ed_lanczos_dev.cuh — scalar bookkeeping of the FX Lanczos recurrence,
// run by one thread of the last block of each grid reduction.
//
// Recurrence (HubMatrix_GPU.cuh:573-582 restated on unnormalised vectors):
//   v_j = w_j / beta_j,  u = H w_j (exact integer accumulation, then >> s_u)
//   alpha_j   = <w_j, u> / beta_j^2
//   w_{j+1}   = u/beta_j - (alpha_j/beta_j) w_j - (beta_j/beta_{j-1}) w_{j-1}
//   beta_{j+1} = |w_{j+1}|
// Every vector is int64 with its own exponent; the three real multipliers of
// the axpy become int64 coefficients at[k] with per-term fractional bits so
// that |w_{j+1} q| < 2^54 by construction (room for the matvec's sums).
#pragma once

#include "ed_device.cuh"
#include "ed_lanczos.hpp"

namespace ed {
namespace dev {

// x * 2^k, exact: an add to the exponent field when x and the result are
// normal numbers, ldexp otherwise.
__device__ __forceinline__ double scale2(double x, int k) {
    const long long b = __double_as_longlong(x);
    const int ex = (int)((b >> 52) & 0x7FF);
    if (ex == 0 || ex + k <= 0 || ex + k >= 0x7FF) return ldexp(x, k);
    return __longlong_as_double(b + ((long long)k << 52));
}

// The exponent frexp returns for x != 0 (|x| in [2^(e-1), 2^e)).
__device__ __forceinline__ int frexp_exp(double x) {
    const int ex = (int)((__double_as_longlong(x) >> 52) & 0x7FF);
    if (ex == 0 || ex == 0x7FF) {
        int e = 0;
        frexp(x, &e);
        return e;
    }
    return ex - 1022;
}

// Scalars of one step after the matvec reduction.
struct LzCoefs {
    double alpha;
    int64_t at[3];
    int Fa;
    int e_w;
};

// alpha_j and the integer axpy coefficients of step j from the exact
// <w_j, u> (alpha_raw), slot j (eX, mX, bj and ib = 1 / bj, computed when
// slot j was completed) and slot j-1 (eP, mP and ibP = 1 / beta_{j-1}).
__device__ inline LzCoefs lz_coefs(int j, i128 alpha_raw, int e_u, uint64_t m_u, int eX, uint64_t mX, double bj,
                                   double ib, int eP, uint64_t mP, double ibP, int status) {
    LzCoefs c;
    if (!(bj > 0.0) || status != 0) {
        // after a breakdown (or a bad start) the recurrence only carries zeros
        c.alpha = 0.0;
        for (int k = 0; k < 3; ++k) c.at[k] = 0;
        c.Fa = 0;
        c.e_w = eX;
        return c;
    }
    const double anum = i128_to_f64(alpha_raw, eX + e_u + 24);
    const double aj = (anum * ib) * ib;
    c.alpha = aj;

    double a[3];
    uint64_t mm[3];
    a[0] = scale2(ib, e_u);
    mm[0] = m_u;
    a[1] = -aj * scale2(ib, eX);
    mm[1] = mX;
    if (j > 0) {
        a[2] = -bj * scale2(ibP, eP);
        mm[2] = mP;
    } else {
        a[2] = 0.0;
        mm[2] = 0;
    }
    double B = 0.0;
    for (int k = 0; k < 3; ++k) B = fma(fabs(a[k]), (double)mm[k], B);
    B *= (1.0 + 1e-9);
    const int kB = B > 0.0 ? frexp_exp(B) : 0;  // B < 2^kB
    const int e_w = kB - 54;
    // One common number of fractional bits for the three integer
    // coefficients: the largest |a_k| 2^-e_w sets it so every |at_k| < 2^62
    // (scaling by 2^-e_w is exact, so its frexp exponent is the largest
    // exponent of the a_k minus e_w).
    int ka = 0;
    bool any = false;
    for (int k = 0; k < 3; ++k)
        if (mm[k] != 0 && a[k] != 0.0) {
            const int ek = frexp_exp(a[k]) - e_w;
            ka = any ? max(ka, ek) : ek;
            any = true;
        }
    const int Fmin = 62 - ka;
    for (int k = 0; k < 3; ++k) c.at[k] = (mm[k] != 0 && a[k] != 0.0) ? llrint(scale2(a[k], Fmin - e_w)) : 0;
    c.Fa = Fmin;
    c.e_w = e_w;
    return c;
}

// lz_coefs by a whole warp (all 32 lanes, the same arguments; result in every
// lane): lane k works out coefficient k, the same operations on the same
// numbers.  The persistent kernels run it once a step in cold code, where the
// instructions fetched count: a third of them, 2.2 -> 1.7 us.
__device__ inline LzCoefs lz_coefs_warp(int j, i128 alpha_raw, int e_u, uint64_t m_u, int eX, uint64_t mX, double bj,
                                        double ib, int eP, uint64_t mP, double ibP, int status) {
    constexpr unsigned kAll = 0xffffffffu;
    const int k = threadIdx.x & 31;
    LzCoefs c;
    if (!(bj > 0.0) || status != 0) {
        c.alpha = 0.0;
        c.at[0] = c.at[1] = c.at[2] = 0;
        c.Fa = 0;
        c.e_w = eX;
        return c;
    }
    const double anum = i128_to_f64(alpha_raw, eX + e_u + 24);
    const double aj = (anum * ib) * ib;
    c.alpha = aj;
    const bool on = k < 2 || (k == 2 && j > 0);
    const double f = k == 0 ? 1.0 : (k == 1 ? -aj : -bj);
    const double a = on ? f * scale2(k == 2 ? ibP : ib, k == 0 ? e_u : (k == 1 ? eX : eP)) : 0.0;
    const uint64_t mm = on ? (k == 0 ? m_u : (k == 1 ? mX : mP)) : 0;
    const double fa = fabs(a), fm = (double)mm;
    double B = 0.0;
#pragma unroll
    for (int t = 0; t < 3; ++t) B = fma(__shfl_sync(kAll, fa, t), __shfl_sync(kAll, fm, t), B);
    B *= (1.0 + 1e-9);
    const int kB = B > 0.0 ? frexp_exp(B) : 0;
    const int e_w = kB - 54;
    const bool nz = mm != 0 && a != 0.0;
    const int ka = __reduce_max_sync(kAll, nz ? frexp_exp(a) - e_w : INT_MIN);
    const int Fmin = 62 - (ka == INT_MIN ? 0 : ka);
    const long long at = nz ? llrint(scale2(a, Fmin - e_w)) : 0;
#pragma unroll
    for (int t = 0; t < 3; ++t) c.at[t] = __shfl_sync(kAll, at, t);
    c.Fa = Fmin;
    c.e_w = e_w;
    return c;
}

// 1 / beta for the w_{j-1} coefficient (beta > 0 on every step that uses it;
// 0 keeps a breakdown's zeros finite).
__device__ inline double lz_inv(double b) { return b > 0.0 ? 1.0 / b : 0.0; }

// |w_{j+1}| from the exact sum of (q q) >> 16 at exponent e_w.
__device__ inline double lz_beta(i128 sumsq, int e_w) { return sqrt(i128_to_f64(sumsq, 2 * e_w + 16)); }

// Coefficient on q_k of one Gram-Schmidt pass from the exact dot acc = sum
// (q_k q_w) >> 24: <w_k, w> / beta_k^2 in units of w's exponent ew (the total
// rounded once, as a host conversion of it would be; IEEE divide and exact
// scalings).
__device__ inline double reorth_r(i128 acc, int ek, double bk, int ew) {
    const double dotv = i128_to_f64(acc, ek + ew + 24);
    return scale2(dotv / (bk * bk), ek - ew);
}

// Guard bits of a sum of nk terms in a Gram-Schmidt pass.
__device__ inline int reorth_guard(int nk) {
    int extra = 0;
    while ((1 << (10 + extra)) < nk) ++extra;
    return extra;
}

// Fraction bits that keep r within 62 - extra bits (r != 0).
__device__ inline int reorth_bits(double r, int extra) {
    return 62 - frexp_exp(r) - extra;
}

// The integer coefficient t of r and its right shift sh to the pass's common
// F (the smallest reorth_bits of the nonzero r).
__device__ inline void reorth_fix(double r, int extra, int F, int64_t* t, int* sh) {
    *t = 0;
    *sh = 0;
    if (r == 0.0) return;
    const int f = reorth_bits(r, extra);
    if (f - F < 120) {
        *t = (int64_t)llrint(scale2(r, f));
        *sh = f - F;
    }
}

// Step j's coefficients into the run's state.
__device__ inline void lz_store_coefs(LzState* lz, int j, const LzCoefs& c) {
    lz->alpha[j] = c.alpha;
    for (int k = 0; k < 3; ++k) {
        lz->at[k] = lz->at_hist[3 * j + k] = c.at[k];
        lz->sh[k] = 0;
    }
    lz->Fa = lz->Fa_hist[j] = c.Fa;
    lz->e_w = c.e_w;
}

__device__ inline void lz_after_matvec(LzState* lz, int j, i128 alpha_raw, uint64_t m_u, int s_u, int Fc) {
    const int eX = lz->e[j];
    const int e_u = eX - Fc + s_u;
    lz->s_u = s_u;
    lz->e_u = e_u;
    lz->m_u = m_u;
    const LzCoefs c = lz_coefs(j, alpha_raw, e_u, m_u, eX, lz->m[j], lz->beta[j], lz_inv(lz->beta[j]),
                               j > 0 ? lz->e[j - 1] : 0,
                               j > 0 ? lz->m[j - 1] : 0, j > 0 ? lz_inv(lz->beta[j - 1]) : 0.0, lz->status);
    lz_store_coefs(lz, j, c);
}

__device__ inline void lz_after_axpy(LzState* lz, int j, i128 sumsq, uint64_t m_w) {
    const int e_w = lz->e_w;
    lz->e[j + 1] = e_w;
    lz->m[j + 1] = m_w;
    lz->beta[j + 1] = lz_beta(sumsq, e_w);
    const int bits = bitlen_u64(m_w);
    if (bits < lz->min_bits) lz->min_bits = bits;
    if (m_w == 0 && lz->status == 0) lz->status = 7;  // breakdown
    lz->steps_done = j + 1;
}

struct SlotScalars {
    int e;
    uint64_t m;
    double beta;
    double ib;  // 1 / beta (0 when beta is 0)
};

// Thread 0: slot k (= w_k) is complete with exponent e, exact sum of
// (q q) >> 16 and max |q|: beta_k, breakdown and precision bookkeeping
// (lz_after_axpy's), shift the slot scalars, block 0 stores them.
__device__ __forceinline__ void slot_done(LzState* lz, int k, int e, i128 ss, uint64_t m, SlotScalars& sX,
                                          SlotScalars& sP, int& status, int& min_bits, bool store) {
    const double beta = lz_beta(ss, e);
    const int bits = bitlen_u64(m);
    if (bits < min_bits) min_bits = bits;
    if (m == 0 && status == 0) status = 7;  // breakdown
    if (store) {
        lz->e[k] = e;
        lz->m[k] = m;
        lz->beta[k] = beta;
        lz->min_bits = min_bits;
        lz->status = status;
        lz->steps_done = k;
    }
    sP = sX;
    sX = {e, m, beta, lz_inv(beta)};
}

}  // namespace dev
}  // namespace ed

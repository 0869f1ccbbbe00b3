// ed_lanczos_reorth.cu — a fully reorthogonalised run of FX Lanczos steps in
// one cooperative launch (the recurrence of Lanczos::eigen,
// HubMatrix_GPU.cuh:561-590, with every new vector orthogonalised twice
// against the whole basis).
//
// Small sectors spend a reorthogonalised step on latency: launched one by
// one, its nine kernels (matvec, axpy, twice dots / coefficients / update,
// norm) take 65 us a step at 4,900 rows for a few microseconds of work.  Here
// one grid of resident CTAs runs all steps.  A CTA owns a contiguous range of
// elements: its part of u, of w_{j+1} and, where it fits, of every basis
// vector stays in its shared memory, so that only four things cross CTAs:
//   matvec of the own rows, <w_j, u>, max|u|             -> grid barrier
//   axpy, |w|^2, max|w|, own partials of <w_k, w_{j+1}>  -> grid barrier
//   coefficients, update, second partials                -> grid barrier
//   coefficients, update, new norm and max, w_{j+1} out  -> grid barrier
// Partial dots go to three 42-bit limb words per k by integer atomics.  Every
// CTA forms the coefficients itself.  All sums are exact integers and the
// scalar code is that of the per-step kernels, so alpha, beta and the vectors
// equal theirs bit for bit.  What is left is the barriers (1.9 to 4.5 us
// each with the reductions before them) and FP64 scalar code (1.7 us for the
// axpy coefficients, 1.8 us for those of a pass).  Us a step of
// 100, per-step kernels and this one: 400 rows 62 / 23, 4,900 rows 69 / 25, 63,504
// rows 102 / 49, 213,444 rows 188 / 127, 853,776 rows 466 / 393; longer runs of
// large sectors go over to the per-step kernels (reorth_launch_steps).
// Vectors written in the launch are read through L2; barriers
// are bounded (grid_sync).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "ed_device.cuh"
#include "ed_grid.cuh"
#include "ed_internal.hpp"
#include "ed_lanczos.hpp"
#include "ed_lanczos_dev.cuh"
#include "ed_matvec_common.cuh"

namespace ed {
using namespace dev;

namespace {

constexpr int kRoThreads = 512;
constexpr int kRoWarps = kRoThreads / 32;
constexpr int kRoMinRange = 64;

template <bool CPLX>
__device__ __forceinline__ void load_l2(const int64_t* xq, uint32_t idx, int64_t& r, int64_t& i) {
    if (CPLX) {
        const longlong2 v = __ldcg(reinterpret_cast<const longlong2*>(xq) + idx);
        r = v.x;
        i = v.y;
    } else {
        r = __ldcg(xq + idx);
        i = 0;
    }
}

// Row (u, d) of H x as exact 128-bit sums.  Entries are ordered by class, and
// within a single class positive first.
template <bool CPLX, bool FAST>
__device__ __forceinline__ void mv_element(const MvArgs& a, const int64_t* xq, uint32_t u, uint32_t d, int64_t xr,
                                           int64_t xi, i128& ar, i128& ai) {
    const uint32_t dimDN = (uint32_t)a.dimDN;
    const uint32_t* ue = a.upEntC + __ldg(a.upPtr + u);
    const int lenU = a.upLen[u], lenD = a.dnLen[d];
    const uint32_t* de = a.dnEnt + d;
    const bool unitU = a.unitUP != 0 && a.nclsUP == 1, unitD = a.unitDN != 0 && a.nclsDN == 1;
    auto up = [&](int k, uint32_t& e, int64_t& r, int64_t& i) {
        e = __ldg(ue + k);
        load_l2<CPLX>(xq, (e & kColMask) * dimDN + d, r, i);
    };
    auto dn = [&](int k, uint32_t& e, int64_t& r, int64_t& i) {
        e = __ldg(de + (size_t)k * dimDN);
        load_l2<CPLX>(xq, u * dimDN + (e & kColMask), r, i);
    };
    ar = ai = 0;
    if (FAST) {
        int64_t sur = 0, sui = 0, sdr = 0, sdi = 0;
#pragma unroll 4
        for (int k = 0; k < lenU; ++k) {
            uint32_t e;
            int64_t r, i;
            up(k, e, r, i);
            sur += apply_sign(r, e);
            if (CPLX) sui += apply_sign(i, e);
        }
#pragma unroll 4
        for (int k = 0; k < lenD; ++k) {
            uint32_t e;
            int64_t r, i;
            dn(k, e, r, i);
            sdr += apply_sign(r, e);
            if (CPLX) sdi += apply_sign(i, e);
        }
        if (lenU) apply_class<CPLX>(ar, ai, sur, sui, a.coefUP, 0, unitU, a.Fc);
        if (lenD) apply_class<CPLX>(ar, ai, sdr, sdi, a.coefDN, 0, unitD, a.Fc);
    } else {
        for (int side = 0; side < 2; ++side) {
            const int len = side ? lenD : lenU;
            const int64_t* coef = side ? a.coefDN : a.coefUP;
            const bool unit = side ? unitD : unitU;
            int cur = -1;
            int64_t sr = 0, si = 0;
            for (int k = 0; k < len; ++k) {
                uint32_t e;
                int64_t r, i;
                if (side) dn(k, e, r, i);
                else up(k, e, r, i);
                const int c = (int)((e >> kClassShift) & kClassMask);
                if (c != cur) {
                    if (cur >= 0) apply_class<CPLX>(ar, ai, sr, si, coef, cur, unit, a.Fc);
                    sr = si = 0;
                    cur = c;
                }
                sr += apply_sign(r, e);
                if (CPLX) si += apply_sign(i, e);
            }
            if (cur >= 0) apply_class<CPLX>(ar, ai, sr, si, coef, cur, unit, a.Fc);
        }
    }
    const int64_t dq = __ldg(a.dUPq + u) + __ldg(a.dDNq + d) +
                       a.Uq * (int64_t)__popcll(__ldg(a.stUP + u) & __ldg(a.stDN + d) & a.mask);
    ar += mul_wide(dq, xr);
    if (CPLX) ai += mul_wide(dq, xi);
}

// Sum over groups of `lanes` adjacent lanes (a power of two); every lane gets it.
__device__ __forceinline__ i128 group_sum_i128(i128 v, int lanes) {
    for (int o = 1; o < lanes; o <<= 1) {
        const uint64_t lo = __shfl_xor_sync(0xffffffffu, (uint64_t)v, o);
        const uint64_t hi = __shfl_xor_sync(0xffffffffu, (uint64_t)((u128)v >> 64), o);
        v += (i128)(((u128)hi << 64) | lo);
    }
    return v;
}

__device__ __forceinline__ int pow2_floor(int v) { return 1 << (31 - __clz(v)); }

}  // namespace

// Dynamic shared memory: u and w of the own range, then the own part of every
// basis vector (cached != 0), then with `lists` the gather offsets of each
// thread's element (sign in bit 31).
template <bool CPLX, bool FAST>
__global__ void __launch_bounds__(kRoThreads, 1) k_lz_reorth_run(const MvArgs a, const LzReorthArgs f, const int R,
                                                                 const int cached, const int lists) {
    extern __shared__ __align__(16) unsigned char ro_smem[];
    __shared__ i128 s128[32];
    __shared__ uint64_t s64[32];
    __shared__ int give_up, s_F[kRoWarps], s_Fmin;
    __shared__ int s_e[2], s_status, s_min_bits;  // slots j, j-1
    __shared__ uint64_t s_m[2];
    __shared__ double s_beta[2], s_ib[2];
    __shared__ i128 s_ss;  // exact norm sum of slot j, while its beta is pending
    __shared__ LzCoefs s_coef;
    __shared__ int64_t s_rt[kReorthMaxSteps];
    __shared__ uint8_t s_rs[kReorthMaxSteps];
    constexpr int W = CPLX ? 2 : 1;
    const int tid = threadIdx.x;
    const uint32_t dimDN = (uint32_t)a.dimDN;
    const int64_t lo = (int64_t)blockIdx.x * R;
    const int nr = (int)max((int64_t)0, min((int64_t)R, f.n - lo));  // own elements
    int64_t* su = reinterpret_cast<int64_t*>(ro_smem);
    int64_t* sw = su + R;
    int64_t* slab = sw + R;
    uint32_t* list = reinterpret_cast<uint32_t*>(slab + (cached ? (size_t)R * (f.max_steps + 1) : 0));
    // own part of slot k: element i at own[k * ostride + i]
    int64_t* const own = cached ? slab : f.basis + lo;
    const int64_t ostride = cached ? R : f.stride;
    LzState* lz = f.lz;
    const bool store = blockIdx.x == 0 && tid == 0;
    if (tid == 0) {
        give_up = 0;
        const int j = f.j0;
        s_e[0] = lz->e[j];
        s_m[0] = lz->m[j];
        s_beta[0] = lz->beta[j];
        s_ib[0] = lz_inv(s_beta[0]);
        s_e[1] = j > 0 ? lz->e[j - 1] : 0;
        s_m[1] = j > 0 ? lz->m[j - 1] : 0;
        s_ib[1] = j > 0 ? lz_inv(lz->beta[j - 1]) : 0.0;
        s_status = lz->status;
        s_min_bits = lz->min_bits;
    }
    if (cached)
        for (int k = 0; k <= f.j0; ++k)
            for (int i = tid; i < nr; i += kRoThreads) slab[(size_t)k * R + i] = __ldcg(f.basis + (size_t)k * f.stride + lo + i);
    // this thread's element with its gather list (one element a thread)
    int lenU = 0, lenD = 0;
    int64_t diag = 0;
    if (lists && tid * W < nr) {
        const uint32_t i = (uint32_t)(lo / W) + tid, u = i / dimDN, d = i - u * dimDN;
        const uint32_t* ue = a.upEntC + a.upPtr[u];
        lenU = a.upLen[u];
        lenD = a.dnLen[d];
        for (int k = 0; k < lenU; ++k)
            list[k * kRoThreads + tid] = ((ue[k] & kColMask) * dimDN + d) | (ue[k] & kSignBit);
        for (int k = 0; k < lenD; ++k) {
            const uint32_t e = a.dnEnt[(size_t)k * dimDN + d];
            list[(lenU + k) * kRoThreads + tid] = (u * dimDN + (e & kColMask)) | (e & kSignBit);
        }
        diag = a.dUPq[u] + a.dDNq[d] + a.Uq * (int64_t)__popcll(a.stUP[u] & a.stDN[d] & a.mask);
    }
    __syncthreads();
    unsigned int target = 0;
    for (int j = f.j0; j < f.j1; ++j) {
        const int64_t* xq = f.basis + (size_t)j * f.stride;
        const int64_t* ox = own + (size_t)j * ostride;
        const int64_t* op = j > 0 ? ox - ostride : ox;
        LzRedSet* red = f.red + 3 * (j & 1);
        const int nk = j + 1;
        unsigned long long* acc0 = f.acc;
        unsigned long long* acc1 = f.acc + 3 * (int64_t)f.max_steps;
        // ---- u = H w_j on the own range; the second pass's dot words of the
        // previous step were read before the last barrier
        for (int k = blockIdx.x * kRoThreads + tid; k < 3 * j; k += gridDim.x * kRoThreads) acc1[k] = 0;
        const int sb = a.bq_bits + bitlen_u64(s_m[0]) - 62;
        const int s_u = sb > 0 ? sb : 0;
        if (tid == kRoThreads - 32 && j > f.j0) {
            // beta_j and its inverse, wanted after the next barrier: by a
            // thread of the last warp, which has the least of a short matvec
            s_ib[1] = s_ib[0];
            s_beta[0] = lz_beta(s_ss, s_e[0]);
            s_ib[0] = lz_inv(s_beta[0]);
            if (blockIdx.x == 0) lz->beta[j] = s_beta[0];
        }
        {
            i128 dot = 0;
            uint64_t mx = 0;
            for (int t = tid; t * W < nr; t += kRoThreads) {
                const int64_t xr = ox[t * W], xi = CPLX ? ox[t * W + 1] : 0;
                i128 ar = 0, ai = 0;
                if (FAST && lists) {
                    int64_t sr[2] = {0, 0}, si[2] = {0, 0};
                    const int len = lenU + lenD;
#pragma unroll 8
                    for (int k = 0; k < len; ++k) {
                        const uint32_t e = list[k * kRoThreads + tid];
                        int64_t r, i;
                        load_l2<CPLX>(xq, e & ~kSignBit, r, i);
                        r = apply_sign(r, e);
                        i = CPLX ? apply_sign(i, e) : 0;
                        sr[0] += k < lenU ? r : 0;
                        sr[1] += k < lenU ? 0 : r;
                        if (CPLX) {
                            si[0] += k < lenU ? i : 0;
                            si[1] += k < lenU ? 0 : i;
                        }
                    }
                    if (lenU) apply_class<CPLX>(ar, ai, sr[0], si[0], a.coefUP, 0, a.unitUP != 0, a.Fc);
                    if (lenD) apply_class<CPLX>(ar, ai, sr[1], si[1], a.coefDN, 0, a.unitDN != 0, a.Fc);
                    ar += mul_wide(diag, xr);
                    if (CPLX) ai += mul_wide(diag, xi);
                } else {
                    const uint32_t i = (uint32_t)(lo / W) + t, u = i / dimDN, d = i - u * dimDN;
                    mv_element<CPLX, FAST>(a, xq, u, d, xr, xi, ar, ai);
                }
                const int64_t qr = shr_round_i64(ar, s_u);
                su[t * W] = qr;
                dot += mul_wide(xr, qr) >> 24;
                uint64_t aq = (uint64_t)(qr < 0 ? -qr : qr);
                mx = aq > mx ? aq : mx;
                if (CPLX) {
                    const int64_t qi = shr_round_i64(ai, s_u);
                    su[t * W + 1] = qi;
                    dot += mul_wide(xi, qi) >> 24;
                    aq = (uint64_t)(qi < 0 ? -qi : qi);
                    mx = aq > mx ? aq : mx;
                }
            }
            block_sum_max(dot, mx, s128, s64);
            if (tid == 0) red_push(&red[0], dot, mx);
        }
        if (!grid_sync(f.gbar, target, &give_up, a.err, f.wait)) return;
        if (tid < 32) {
            i128 s;
            uint64_t m;
            red_pull(&red[0], s, m);
            const int e_u = s_e[0] - a.Fc + s_u;
            const LzCoefs c = lz_coefs_warp(j, s, e_u, m, s_e[0], s_m[0], s_beta[0], s_ib[0], s_e[1], s_m[1], s_ib[1], s_status);
            if (tid == 0) {
                s_coef = c;
                // the other parity's sets were last read before this barrier
                if (blockIdx.x == 0)
                    for (int r = 0; r < 3; ++r) f.red[3 * ((j + 1) & 1) + r] = LzRedSet{0, 0, 0, 0};
                if (store) {
                    lz->s_u = s_u;
                    lz->e_u = e_u;
                    lz->m_u = m;
                    lz_store_coefs(lz, j, c);
                    lz->e[j + 1] = c.e_w;
                }
            }
        }
        __syncthreads();
        // ---- w_{j+1} on the own range
        {
            i128 ss = 0;
            uint64_t mw = 0;
            for (int i = tid; i < nr; i += kRoThreads) {
                const int64_t w = shr_round_i64(mul_wide(s_coef.at[0], su[i]) + mul_wide(s_coef.at[1], ox[i]) +
                                                    mul_wide(s_coef.at[2], op[i]),
                                                s_coef.Fa);
                sw[i] = w;
                ss += mul_wide(w, w) >> 16;
                const uint64_t aw = (uint64_t)(w < 0 ? -w : w);
                mw = aw > mw ? aw : mw;
            }
            block_sum_max(ss, mw, s128, s64);
            if (tid == 0) red_push(&red[1], ss, mw);
        }
        __syncthreads();
        const int ew = s_coef.e_w;
        // ---- classical Gram-Schmidt, twice, against w_0 .. w_j
        const int lk = max(1, min(32, pow2_floor(max(1, kRoThreads / nk))));  // lanes per dot
        const int le = max(1, min(32, pow2_floor(max(1, kRoThreads / max(nr, 1)))));  // lanes per updated element
        for (int pass = 0; pass < 2; ++pass) {
            unsigned long long* acc = pass ? acc1 : acc0;
            for (int k0 = 0; k0 < nk; k0 += kRoThreads / lk) {
                const int k = k0 + tid / lk;
                i128 v = 0;
                if (k < nk) {
                    const int64_t* q = own + (size_t)k * ostride;
#pragma unroll 4
                    for (int i = tid & (lk - 1); i < nr; i += lk) v += mul_wide(q[i], sw[i]) >> 24;
                }
                v = group_sum_i128(v, lk);
                if (k < nk && (tid & (lk - 1)) == 0) {
                    atomicAdd(acc + 3 * k, (unsigned long long)((u128)v & kLimb));
                    atomicAdd(acc + 3 * k + 1, (unsigned long long)(((u128)v >> 42) & kLimb));
                    atomicAdd(acc + 3 * k + 2, (unsigned long long)(int64_t)(v >> 84));
                }
            }
            if (!grid_sync(f.gbar, target, &give_up, a.err, f.wait)) return;
            if (pass == 0) {
                if (tid == 0) {
                    i128 ss;
                    uint64_t mw;
                    red_pull(&red[1], ss, mw);
                    s_min_bits = min(s_min_bits, bitlen_u64(mw));
                    if (mw == 0 && s_status == 0) s_status = 7;  // breakdown
                }
            } else {
                // the first pass's words were read before this barrier
                for (int k = blockIdx.x * kRoThreads + tid; k < 3 * nk; k += gridDim.x * kRoThreads) acc0[k] = 0;
            }
            // the coefficients (the same integers and code in every CTA)
            const int extra = reorth_guard(nk);
            int fmin = 1 << 20;
            for (int k = tid; k < nk; k += kRoThreads) {
                const i128 v = (i128)((u128)__ldcg(acc + 3 * k) + ((u128)__ldcg(acc + 3 * k + 1) << 42) +
                                      ((u128)(i128)(int64_t)__ldcg(acc + 3 * k + 2) << 84));
                const double r = reorth_r(v, __ldcg(lz->e + k), __ldcg(lz->beta + k), ew);
                s_rt[k] = __double_as_longlong(r);
                if (r != 0.0) fmin = min(fmin, reorth_bits(r, extra));
            }
            fmin = __reduce_min_sync(0xffffffffu, fmin);
            if ((tid & 31) == 0) s_F[tid >> 5] = fmin;
            __syncthreads();
            if (tid == 0) {
                int m = 1 << 20;
                for (int w = 0; w < kRoWarps; ++w) m = min(m, s_F[w]);
                s_Fmin = m == (1 << 20) ? 0 : m;
            }
            __syncthreads();
            const int F = s_Fmin;
            for (int k = tid; k < nk; k += kRoThreads) {
                int64_t t;
                int sh;
                reorth_fix(__longlong_as_double(s_rt[k]), extra, F, &t, &sh);
                s_rt[k] = t;
                s_rs[k] = (uint8_t)sh;
            }
            __syncthreads();
            i128 ss = 0;
            uint64_t mw = 0;
            const int r0 = tid & (le - 1);
            for (int i0 = 0; i0 < nr; i0 += kRoThreads / le) {  // the same iterations for every lane (shuffles)
                const int i = i0 + tid / le;
                i128 sum = 0;
                if (i < nr) {
#pragma unroll 4
                    for (int k = r0; k < nk; k += le) sum += mul_wide(s_rt[k], own[(size_t)k * ostride + i]) >> s_rs[k];
                }
                sum = group_sum_i128(sum, le);
                if (i < nr && r0 == 0) {
                    const int64_t w = sw[i] - (int64_t)shr_round(sum, F);
                    sw[i] = w;
                    if (pass == 1) {
                        f.basis[(size_t)(j + 1) * f.stride + lo + i] = w;
                        if (cached) slab[(size_t)(j + 1) * R + i] = w;
                        ss += mul_wide(w, w) >> 16;
                        const uint64_t aw = (uint64_t)(w < 0 ? -w : w);
                        mw = aw > mw ? aw : mw;
                    }
                }
            }
            if (pass == 1) {
                block_sum_max(ss, mw, s128, s64);
                if (tid == 0) red_push(&red[2], ss, mw);
            }
            __syncthreads();
        }
        if (!grid_sync(f.gbar, target, &give_up, a.err, f.wait)) return;
        if (tid == 0) {
            i128 ss;
            uint64_t mw;
            red_pull(&red[2], ss, mw);
            s_min_bits = min(s_min_bits, bitlen_u64(mw));
            if (mw == 0 && s_status == 0) s_status = 7;
            s_e[1] = s_e[0];
            s_m[1] = s_m[0];
            s_e[0] = ew;
            s_m[0] = mw;
            s_ss = ss;
            if (store) {
                lz->m[j + 1] = mw;
                if (j + 1 == f.j1) lz->beta[j + 1] = lz_beta(ss, ew);  // the last slot of this launch
                lz->min_bits = s_min_bits;
                lz->status = s_status;
                lz->steps_done = j + 1;
            }
        }
        __syncthreads();
    }
}

// cudaErrorNotSupported when the device cannot hold the grid; f.gbar, f.red
// and f.acc must be zero.
cudaError_t launch_lz_reorth(const ed_op* op, const LzReorthArgs& f, cudaStream_t s) {
    const void* fn = op->cplx ? (op->mv_fast ? (const void*)k_lz_reorth_run<true, true> : (const void*)k_lz_reorth_run<true, false>)
                              : (op->mv_fast ? (const void*)k_lz_reorth_run<false, true> : (const void*)k_lz_reorth_run<false, false>);
    int sms = 0, coop = 0;
    cudaError_t e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, op->device)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, op->device)) != cudaSuccess) return e;
    if (!coop) return cudaErrorNotSupported;
    const int W = op->cplx ? 2 : 1;
    // every SM, but at least kRoMinRange elements a CTA (more CTAs add to each
    // dot word than they save in the sums: 4,900 rows 27.8, 26.7, 29.7, 40.9 us
    // a step at 32, 64, 128, 256); whole complex pairs
    const int g = (int)std::min<int64_t>(sms, std::max<int64_t>(1, f.n / kRoMinRange));
    int R = (int)((f.n / W + g - 1) / g) * W;
    // the shared memory: u, w, then the gather lists, then the own part of the
    // basis while both fit
    const size_t cap = 200 * 1024;
    size_t smem = sizeof(int64_t) * 2 * (size_t)R;
    const int64_t len = op->tup.max_len + op->tdn.max_len;
    const size_t list_bytes = sizeof(uint32_t) * kRoThreads * (size_t)len;
    int lists = op->mv_fast && R / W <= kRoThreads && smem + list_bytes <= cap / 2 ? 1 : 0;
    if (lists) smem += list_bytes;
    const size_t slab = sizeof(int64_t) * (size_t)R * (size_t)(f.max_steps + 1);
    int cached = smem + slab <= cap ? 1 : 0;
    if (cached) smem += slab;
    if (smem > cap) return cudaErrorNotSupported;
    if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)) != cudaSuccess) return e;
    int per_sm = 0;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kRoThreads, smem)) != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorNotSupported;
    MvArgs av = op->mv;
    LzReorthArgs fv = f;
    void* args[] = {&av, &fv, &R, &cached, &lists};
    return cudaLaunchCooperativeKernel(fn, dim3((unsigned)g), dim3(kRoThreads), args, smem, s);
}

}  // namespace ed

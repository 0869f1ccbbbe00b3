// ed_matvec_tma.cuh — the shared-memory row engine of the matvec, used by the
// one-launch matvec (ed_matvec_tma.cu) and by the persistent Lanczos kernel
// (ed_lanczos_fused.cu).
//
// A CTA of kTmaThreads threads
//  * holds the whole down-spin operator (CSR entries, row pointers, npos,
//    folded diagonal, bitstrings) in shared memory, moved there by TMA bulk
//    copies (cp.async.bulk global->shared, completion counted on an mbarrier);
//  * walks the up-rows u = blockIdx.x, + gridDim.x, ... with x[u, :] double
//    buffered by bulk copies: row u+gridDim.x streams in while row u is
//    computed;
//  * computes the down term entirely from shared memory and the up term with
//    coalesced L2 loads, two output columns per thread so at least eight
//    up-term loads are in flight per thread.
// Every mbarrier wait is bounded: after kMaxSpin polls the CTA records an
// error in *err, waits (bounded) for its copies in flight and stops.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "ed_device.cuh"
#include "ed_internal.hpp"
#include "ed_matvec_common.cuh"

namespace ed {
using namespace dev;

constexpr int kTmaThreads = 512;
constexpr int kTmaUpStage = 256;  // longest up-row held in the static offset arrays
constexpr long long kMaxSpin = 1LL << 22;

namespace tma {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

// generic-proxy accesses of shared memory before async-proxy writes into it
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// generic-proxy writes of global memory (observed by this thread) before
// async-proxy reads of it
__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

__device__ __forceinline__ void expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// dst, src 16-byte aligned; bytes a multiple of 16
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// Bounded wait for the phase with the given parity; false when it gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    const uint32_t addr = smem_u32(bar);
    for (long long it = 0; it < kMaxSpin; ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__host__ __device__ constexpr uint32_t round16(uint32_t b) { return (b + 15u) / 16u * 16u; }

}  // namespace tma

// Shared-memory views: the dynamic area follows the byte offsets in MvArgs
// (barriers at 0: [0], [1] row buffers, [2] down tables); the up-row offsets
// and the give-up word are static arrays of the kernel.
struct TmaSmem {
    uint64_t* bar;
    int64_t* row0;
    int64_t* row1;
    uint32_t* dptr;
    uint32_t* dent;
    uint8_t* dnpos;
    int64_t* ddq;
    uint64_t* dst;
    uint16_t* sched;  // gather schedule (a.dnSched) or class schedule (a.clsSched, its
    uint8_t* steps;   // step words here, its negative counts at dnpos)
    uint32_t* uoff;
    uint32_t* uent;
    int* give_up;
    const int64_t* cup;  // coefficient classes in shared memory (a.perEntry)
    const int64_t* cdn;
};

// General (neither single-class nor segmented) kernels: the coefficient
// classes in shared memory, where lanes may read different ones at a time.
// Valid after the next block barrier.
template <bool GEN>
__device__ __forceinline__ void tma_stage_classes(const MvArgs& a, int64_t* s_cls, TmaSmem& S) {
    if constexpr (GEN) {
        for (int t = threadIdx.x; t < 2 * kMaxCls; t += blockDim.x) {
            s_cls[t] = a.coefUP[t];
            s_cls[2 * kMaxCls + t] = a.coefDN[t];
        }
        S.cup = s_cls;
        S.cdn = s_cls + 2 * kMaxCls;
    }
}

__device__ __forceinline__ TmaSmem tma_view(const MvArgs& a, unsigned char* sm, uint32_t* uoff, uint32_t* uent,
                                            int* give_up) {
    TmaSmem S;
    S.bar = reinterpret_cast<uint64_t*>(sm);
    S.row0 = reinterpret_cast<int64_t*>(sm + a.sm_row0);
    S.row1 = reinterpret_cast<int64_t*>(sm + a.sm_row1);
    S.dptr = reinterpret_cast<uint32_t*>(sm + a.sm_dnptr);
    S.dent = reinterpret_cast<uint32_t*>(sm + a.sm_dnent);
    S.dnpos = sm + a.sm_dnnpos;
    S.ddq = reinterpret_cast<int64_t*>(sm + a.sm_ddnq);
    S.dst = reinterpret_cast<uint64_t*>(sm + a.sm_stdn);
    S.sched = reinterpret_cast<uint16_t*>(sm + a.sm_sched);
    S.steps = sm + a.sm_steps;
    S.uoff = uoff;
    S.uent = uent;
    S.give_up = give_up;
    S.cup = S.cdn = nullptr;
    return S;
}

// Thread 0: initialise the three barriers.
__device__ __forceinline__ void tma_init(const TmaSmem& S) {
    for (int k = 0; k < 3; ++k) tma::mbar_init(&S.bar[k], 1);
    tma::fence_mbar_init();
    *S.give_up = 0;
}

// Thread 0: start the copies of the down-spin tables (completion on bar[2]).
// The device tables are allocated in multiples of 16 bytes and the shared
// regions in multiples of 128, so every copy is rounded up to 16 bytes.
__device__ __forceinline__ void tma_issue_tables(const MvArgs& a, const TmaSmem& S) {
    const uint32_t dimDN = (uint32_t)a.dimDN;
    if (a.dnSched) {
        const uint32_t b_sc = tma::round16((uint32_t)a.schedSteps * (uint32_t)a.dimDNp * 2u),
                       b_stp = tma::round16((uint32_t)a.dimDNp / 32u), b_dq = tma::round16(dimDN * 8u);
        tma::expect_tx(&S.bar[2], b_sc + b_stp + 2 * b_dq);
        if (b_sc) tma::bulk_g2s(S.sched, a.dnSched, b_sc, &S.bar[2]);
        tma::bulk_g2s(S.steps, a.dnSteps, b_stp, &S.bar[2]);
        tma::bulk_g2s(S.ddq, a.dDNq, b_dq, &S.bar[2]);
        tma::bulk_g2s(S.dst, a.stDN, b_dq, &S.bar[2]);
        return;
    }
    if (a.clsSched) {
        const uint32_t b_sc = tma::round16((uint32_t)a.schedSteps * (uint32_t)a.dimDNp * 2u),
                       b_stp = tma::round16((uint32_t)a.dimDNp / 32u * 4u), b_neg = tma::round16((uint32_t)a.dimDNp * 4u),
                       b_dq = tma::round16(dimDN * 8u);
        tma::expect_tx(&S.bar[2], b_sc + b_stp + b_neg + 2 * b_dq);
        tma::bulk_g2s(S.sched, a.clsSched, b_sc, &S.bar[2]);
        tma::bulk_g2s(S.steps, a.clsSteps, b_stp, &S.bar[2]);
        tma::bulk_g2s(S.dnpos, a.clsNeg, b_neg, &S.bar[2]);
        tma::bulk_g2s(S.ddq, a.dDNq, b_dq, &S.bar[2]);
        tma::bulk_g2s(S.dst, a.stDN, b_dq, &S.bar[2]);
        return;
    }
    const uint32_t b_ptr = tma::round16((dimDN + 1) * 4u), b_ent = tma::round16(a.dnNnz * 4u),
                   b_pos = tma::round16(dimDN), b_dq = tma::round16(dimDN * 8u), b_st = b_dq;
    tma::expect_tx(&S.bar[2], b_ptr + b_ent + b_pos + b_dq + b_st);
    tma::bulk_g2s(S.dptr, a.dnPtr, b_ptr, &S.bar[2]);
    if (b_ent) tma::bulk_g2s(S.dent, a.dnEntC, b_ent, &S.bar[2]);  // no down hops: nothing to copy
    tma::bulk_g2s(S.dnpos, a.dnNpos, b_pos, &S.bar[2]);
    tma::bulk_g2s(S.ddq, a.dDNq, b_dq, &S.bar[2]);
    tma::bulk_g2s(S.dst, a.stDN, b_st, &S.bar[2]);
}

// The 16 zeros of both row buffers that idle lanes of the gather schedule
// read (the bulk copies only ever write [0, dimDN)), or the zero slot after a
// complex row.
__device__ __forceinline__ void tma_zero_slots(const MvArgs& a, const TmaSmem& S) {
    if (a.clsSched) {
        if (threadIdx.x < 2) {
            S.row0[2 * a.dimDN + threadIdx.x] = 0;
            S.row1[2 * a.dimDN + threadIdx.x] = 0;
        }
        return;
    }
    if (threadIdx.x < 17) {  // 16 zeros after [x | -x] at either row offset
        S.row0[2 * a.schedNeg + threadIdx.x] = 0;
        S.row1[2 * a.schedNeg + threadIdx.x] = 0;
    }
}

// Offset (0 or 1 element) of row u inside its row buffer: a bulk copy starts
// on a 16-byte boundary, so with an odd dim_dn (real vectors) every other
// row is copied from the element before it.
template <bool CPLX>
__device__ __forceinline__ uint32_t tma_row_off(const MvArgs& a, uint32_t u) {
    return CPLX ? 0u : (uint32_t)(((uint64_t)u * (uint64_t)a.dimDN) & 1u);
}

// Thread 0: start the copy of row u of x into row buffer `buf`: the
// 16-byte-aligned run of whole 16-byte words around the row (one element
// before it when it starts at an odd index, one after it to round up; the
// vectors carry two elements of padding), the row at tma_row_off.
template <bool CPLX>
__device__ __forceinline__ void tma_issue_row(const MvArgs& a, const TmaSmem& S, const int64_t* xq, uint32_t u,
                                              int buf) {
    constexpr int W = CPLX ? 2 : 1;
    const uint32_t off = tma_row_off<CPLX>(a, u);
    const uint32_t n = CPLX ? (uint32_t)a.dimDN * 2u : (((uint32_t)a.dimDN + off + 1u) & ~1u);
    const uint32_t bytes = n * 8u;
    tma::expect_tx(&S.bar[buf], bytes);
    tma::bulk_g2s(buf ? S.row1 : S.row0, xq + (size_t)u * a.dimDN * W - off, bytes, &S.bar[buf]);
}

// Up-term element load: read-only path for a one-launch matvec, L2
// (coherent) loads when x was written earlier in the same launch.
template <bool CPLX, bool COH>
__device__ __forceinline__ void up_load(const int64_t* __restrict__ xq, uint32_t idx, int64_t& r, int64_t& i) {
    if (CPLX) {
        const longlong2* p = reinterpret_cast<const longlong2*>(xq) + idx;
        const longlong2 v = COH ? __ldcg(p) : __ldg(p);
        r = v.x;
        i = v.y;
    } else {
        r = COH ? __ldcg(xq + idx) : __ldg(xq + idx);
        i = 0;
    }
}

template <bool CPLX, bool COH>
__device__ __forceinline__ void acc_up(const int64_t* __restrict__ xq, uint32_t idx, int64_t& r, int64_t& i) {
    int64_t vr, vi;
    up_load<CPLX, COH>(xq, idx, vr, vi);
    r += vr;
    if (CPLX) i += vi;
}

// Element col of a staged row: one 16-byte shared load for a complex
// element (row buffers are 16-byte aligned and complex rows start at
// offset 0), one 8-byte load for a real one.
template <bool CPLX>
__device__ __forceinline__ void row_elem(const int64_t* xrow, uint32_t col, int64_t& r, int64_t& i) {
    if (CPLX) {
        const longlong2 v = *reinterpret_cast<const longlong2*>(xrow + col);
        r = v.x;
        i = v.y;
    } else {
        r = xrow[col];
        i = 0;
    }
}

// The classes' complex sums (sr, si) times their coefficients, added to
// (ar, ai).  A class and the one with the conjugate coefficient share four
// products where each alone takes four: with c, S1 and c*, S2,
//   Re = Re c Re(S1 + S2) - Im c Im(S1 - S2), Im = Re c Im(S1 + S2) + Im c Re(S1 - S2)
struct ClassSum {
    int64_t r, i;
};

__device__ __forceinline__ void class_products(i128& ar, i128& ai, const ClassSum s0, const ClassSum s1,
                                               const ClassSum s2, const ClassSum s3, const int64_t* __restrict__ coef,
                                               const int8_t* __restrict__ part, int n) {
    auto four = [&](ClassSum p, ClassSum q, int c) {
        const int64_t cr = coef[2 * c], ci = coef[2 * c + 1];
        mac_wide(ar, p.r, cr);
        mac_wide(ai, p.i, cr);
        if (ci != 0) {
            mac_wide(ar, -q.i, ci);
            mac_wide(ai, q.r, ci);
        }
    };
    auto one = [&](const ClassSum& s, int c) {
        if (c < n && part[c] == c) four(s, s, c);
    };
    auto two = [&](const ClassSum& s, const ClassSum& t, int c, int q) {
        if (c < n && part[c] == q) four({s.r + t.r, s.i + t.i}, {s.r - t.r, s.i - t.i}, c);
    };
    one(s0, 0);
    two(s0, s1, 0, 1);
    two(s0, s2, 0, 2);
    two(s0, s3, 0, 3);
    one(s1, 1);
    two(s1, s2, 1, 2);
    two(s1, s3, 1, 3);
    one(s2, 2);
    two(s2, s3, 2, 3);
    one(s3, 3);
}

// Up offsets of row u into uo: thread i of n.
__device__ __forceinline__ void tma_stage_up(const MvArgs& a, uint32_t u, uint32_t* uo, uint32_t i, uint32_t n) {
    const uint32_t p0 = __ldg(a.upPtr + u), len = __ldg(a.upPtr + u + 1) - p0, dimDN = (uint32_t)a.dimDN;
    for (uint32_t k = i; k < len; k += n) uo[k] = (__ldg(a.upEntC + p0 + k) & kColMask) * dimDN;
}

// First row of this CTA (rowList[rowStart[b]]); false when it has none.
__device__ __forceinline__ bool tma_first_row(const MvArgs& a, uint32_t* u) {
    const uint32_t r0 = __ldg(a.rowStart + blockIdx.x);
    if (r0 >= __ldg(a.rowStart + blockIdx.x + 1)) return false;
    *u = __ldg(a.rowList + r0);
    return true;
}

// The rows of this CTA: u = H x (OUT 0: FP64 y with exponent E_out; OUT 1:
// FX uq >> s_u with the <x,u> and max|u| partials in dot, mx).
// On entry thread 0 has issued the copy of the CTA's first row into buffer
// rc & 1 (when it has rows) and the tables are in shared memory; rc counts
// the rows this CTA has streamed so far (it fixes buffer and barrier phase)
// and is advanced past the rows done.  On a give-up *S.give_up is set, the
// copy in flight has been waited for and the function returns early.
// Rows of the CTA.  Static: the host plan rowList[rowStart[b] ..).  Dynamic
// (taken != null): CTA b starts at rowQueue[b] and takes each further row as
// rowQueue[gridDim.x + atomicAdd(taken, 1)] while it computes the current
// one, so CTAs that finish early take more rows (the queue is in decreasing
// order of cost).  *snext is a shared word for the index taken.
// SPLIT: the unit queue (a.unitQueue), whose last entries are column ranges
// of rows (low 24 bits: the row).
template <bool SPLIT = false>
__device__ __forceinline__ bool tma_first_row_dyn(const MvArgs& a, uint32_t* u) {
    if (blockIdx.x >= (SPLIT ? a.nunits : (uint32_t)a.dimUP)) return false;
    *u = SPLIT ? (__ldg(a.unitQueue + blockIdx.x) & 0xFFFFFFu) : __ldg(a.rowQueue + blockIdx.x);
    return true;
}

// GDIAG: the folded down diagonal is read from a.dDNq in global memory
// instead of the staged copy (instances that share staged tables but not
// their on-site terms, k_lz_multi).
// PRE: the caller has staged the first row's up offsets in S.uoff (FAST).
template <bool CPLX, int OUT, bool FAST, bool COH, bool SCHED, bool DYN, bool SEG = false, bool GDIAG = false,
          bool SPLIT = false, bool PRE = false>
__device__ __forceinline__ void tma_rows(const MvArgs& a, const TmaSmem& S, const int64_t* __restrict__ xq,
                                         int64_t* __restrict__ uq, double* __restrict__ y, uint32_t& rc, int E_out,
                                         int s_u, i128& dot, uint64_t& mx, unsigned int* taken = nullptr,
                                         uint32_t* snext = nullptr) {
    constexpr int W = CPLX ? 2 : 1;
    const uint32_t dimDN = (uint32_t)a.dimDN;
    const int tid = threadIdx.x, T = blockDim.x;
    const bool merge = a.mergeUD != 0;
    const bool unitU = a.unitUP != 0 && a.nclsUP == 1;
    const bool unitD = a.unitDN != 0 && a.nclsDN == 1;
    const uint32_t nq = SPLIT ? a.nunits : (uint32_t)a.dimUP;
    const uint32_t* const queue = SPLIT ? a.unitQueue : a.rowQueue;

    // The next row is taken and its copy issued by the last thread (with
    // rows shorter than 2T it has the fewest columns) after the barrier below:
    // the queue atomic, issued at the row start, and the row-index lookup
    // then keep no thread from that barrier.
    const int qt = T - 1;
    const uint32_t r1 = DYN ? nq : __ldg(a.rowStart + blockIdx.x + 1);
    uint32_t ub = 0;      // FAST: which of uoff, uent holds the row's up offsets
    bool staged = PRE;
    for (uint32_t r = DYN ? blockIdx.x : __ldg(a.rowStart + blockIdx.x); r < r1; ++rc) {
        const uint32_t qe = DYN ? __ldg(queue + r) : __ldg(a.rowList + r);
        const uint32_t u = SPLIT ? (qe & 0xFFFFFFu) : qe;
        // the unit's columns: the whole row, or a range of a multiple of 32
        // columns (the lanes keep their columns mod 32)
        uint32_t lo = 0, hi = dimDN;
        if (SPLIT && (qe >> 24)) {
            const uint32_t P = 1u << (qe >> 28), ch = ((dimDN + P - 1) / P + 31u) & ~31u;
            lo = ((qe >> 24) & 0xFu) * ch;
            hi = min(dimDN, lo + ch);
        }
        const int buf = rc & 1;
        const uint32_t parity = (rc >> 1) & 1;
        uint32_t taken_at = 0;
        if (DYN && tid == qt) taken_at = atomicAdd(taken, 1u);  // consumed after the barrier
        const uint32_t p0 = __ldg(a.upPtr + u), lenU = __ldg(a.upPtr + u + 1) - p0;
        const int nposU = FAST ? (int)__ldg(a.upNpos + u) : 0;
        uint32_t* const uo = FAST && ub ? S.uent : S.uoff;
        if (!staged) {
            for (uint32_t k = tid; k < lenU; k += T) {
                const uint32_t e = __ldg(a.upEntC + p0 + k);
                uo[k] = (e & kColMask) * dimDN;
                if (!FAST) S.uent[k] = e;
            }
        }
        if (!tma::mbar_wait(&S.bar[buf], parity)) {
            if (tid == 0) atomicExch(a.err, 1);
            *S.give_up = 1;
        } else if (SCHED) {
            // -x beside x, so that a schedule index carries the sign
            int64_t* xb = (buf ? S.row1 : S.row0) + tma_row_off<CPLX>(a, u);
            for (uint32_t i = tid; i < dimDN; i += T) xb[a.schedNeg + i] = -xb[i];
        }
        __syncthreads();
        if (*S.give_up) {
            // the current row's copy (the wait that gave up) is the only one
            // counted on a barrier: it must land before the CTA leaves and its
            // shared memory is reassigned (bounded; if it gives up again the
            // rows are undefined)
            if (tid == 0) tma::mbar_wait(&S.bar[buf], parity);
            return;
        }
        // prefetch the next row into the other buffer (its readers finished
        // at the barrier that closed the previous iteration); in the
        // single-class kernel the same warp stages that row's up offsets, two
        // dependent L2 reads that kept every thread from the next row's sums
        // (Kagome12 6+6 step 32.8 -> 32.2 us)
        if (tid >= qt - 31) {
            const uint32_t rn = DYN ? gridDim.x + __shfl_sync(0xffffffffu, taken_at, 31) : r + 1;
            if (DYN && tid == qt) *snext = rn;
            if (rn < r1) {
                const uint32_t un = DYN ? (__ldg(queue + rn) & (SPLIT ? 0xFFFFFFu : 0xFFFFFFFFu)) : __ldg(a.rowList + rn);
                if (tid == qt) {
                    tma::fence_proxy_async_smem();
                    tma_issue_row<CPLX>(a, S, xq, un, buf ^ 1);
                }
                if (FAST) tma_stage_up(a, un, ub ? S.uoff : S.uent, tid & 31, 32);
            }
        }
        const int64_t* xrow = (buf ? S.row1 : S.row0) + tma_row_off<CPLX>(a, u);
        const uint32_t ubase = u * dimDN;

        // two columns (d0, d0 + T) per iteration; one in the class-segmented
        // path, which takes its columns one after the other anyway (fewer
        // live 128-bit accumulators)
        for (uint32_t d0 = lo + tid; d0 < hi; d0 += (SEG ? 1u : 2u) * T) {
            const uint32_t d1 = d0 + T;
            const bool v1 = !SEG && d1 < hi;
            const uint32_t d1c = v1 ? d1 : d0;  // clamp: the second column repeats d0 and is not stored
            i128 ar0 = 0, ai0 = 0, ar1 = 0, ai1 = 0;
            if (FAST) {
                int64_t upr0 = 0, upi0 = 0, unr0 = 0, uni0 = 0, upr1 = 0, upi1 = 0, unr1 = 0, uni1 = 0;
                int k = 0;
                if (v1) {
#pragma unroll 4
                    for (; k < nposU; ++k) {
                        const uint32_t o = uo[k];
                        acc_up<CPLX, COH>(xq, o + d0, upr0, upi0);
                        acc_up<CPLX, COH>(xq, o + d1, upr1, upi1);
                    }
#pragma unroll 4
                    for (; k < (int)lenU; ++k) {
                        const uint32_t o = uo[k];
                        acc_up<CPLX, COH>(xq, o + d0, unr0, uni0);
                        acc_up<CPLX, COH>(xq, o + d1, unr1, uni1);
                    }
                } else {
#pragma unroll 4
                    for (; k < nposU; ++k) acc_up<CPLX, COH>(xq, uo[k] + d0, upr0, upi0);
#pragma unroll 4
                    for (; k < (int)lenU; ++k) acc_up<CPLX, COH>(xq, uo[k] + d0, unr0, uni0);
                }
                int64_t dr0 = 0, di0 = 0, dr1 = 0, di1 = 0;
                if (SCHED) {
                    // conflict-free schedule: in every step the 16 lanes of a
                    // half warp read 16 different bank pairs of [x | -x | 0]
                    const uint32_t dp = (uint32_t)a.dimDNp;
                    const uint16_t* sc0 = S.sched + d0;
                    const int n0 = S.steps[d0 >> 5];
#pragma unroll 4
                    for (int s = 0; s < n0; ++s) dr0 += xrow[sc0[s * dp]];
                    if (v1) {
                        const uint16_t* sc1 = S.sched + d1;
                        const int n1 = S.steps[d1 >> 5];
#pragma unroll 4
                        for (int s = 0; s < n1; ++s) dr1 += xrow[sc1[s * dp]];
                    }
                } else {
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const uint32_t d = c ? d1c : d0;
                    const uint32_t q0 = S.dptr[d], q1 = S.dptr[d + 1], qp = q0 + S.dnpos[d];
                    int64_t pr = 0, pi = 0, nr = 0, ni = 0;
                    for (uint32_t q = q0; q < qp; ++q) {
                        const uint32_t col = (S.dent[q] & kColMask) * W;
                        int64_t vr, vi;
                        row_elem<CPLX>(xrow, col, vr, vi);
                        pr += vr;
                        if (CPLX) pi += vi;
                    }
                    for (uint32_t q = qp; q < q1; ++q) {
                        const uint32_t col = (S.dent[q] & kColMask) * W;
                        int64_t vr, vi;
                        row_elem<CPLX>(xrow, col, vr, vi);
                        nr += vr;
                        if (CPLX) ni += vi;
                    }
                    if (c) {
                        dr1 = pr - nr;
                        di1 = pi - ni;
                    } else {
                        dr0 = pr - nr;
                        di0 = pi - ni;
                    }
                }
                }
                if (merge) {
                    apply_class<CPLX>(ar0, ai0, (upr0 - unr0) + dr0, (upi0 - uni0) + di0, a.coefUP, 0, unitU, a.Fc);
                    apply_class<CPLX>(ar1, ai1, (upr1 - unr1) + dr1, (upi1 - uni1) + di1, a.coefUP, 0, unitU, a.Fc);
                } else {
                    if (lenU) {
                        apply_class<CPLX>(ar0, ai0, upr0 - unr0, upi0 - uni0, a.coefUP, 0, unitU, a.Fc);
                        apply_class<CPLX>(ar1, ai1, upr1 - unr1, upi1 - uni1, a.coefUP, 0, unitU, a.Fc);
                    }
                    if (a.nclsDN) {
                        apply_class<CPLX>(ar0, ai0, dr0, di0, a.coefDN, 0, unitD, a.Fc);
                        apply_class<CPLX>(ar1, ai1, dr1, di1, a.coefDN, 0, unitD, a.Fc);
                    }
                }
            } else if constexpr (SEG && CPLX) {
                // at most kSegCls classes, one sum for each, products at the end.
                // Up entries (the same for every lane) are loaded four at a time
                // and added by class; the down schedule's steps go class by
                // class.  Against a loop per signed class segment, whose trip
                // counts follow the warp's longest lane (25 steps for 13 hops;
                // 18.5 here) and put each load behind the last: complex
                // Kagome12 apply 84 -> 74 us, persistent step 89 -> 75 us.
                const uint32_t d = d0;
                // (named sums: an array would be indexed by the class, in local
                // memory)
                ClassSum s0{0, 0}, s1{0, 0}, s2{0, 0}, s3{0, 0};
                for (uint32_t k = 0; k < lenU; k += 4) {
                    int64_t vr[4], vi[4];
#pragma unroll
                    for (int t = 0; t < 4; ++t) up_load<CPLX, COH>(xq, S.uoff[min(k + t, lenU - 1)] + d, vr[t], vi[t]);
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        if (k + t >= lenU) break;
                        const uint32_t e = S.uent[k + t], cl = (e >> kClassShift) & 3u;
                        const int64_t r = apply_sign(vr[t], e), i = apply_sign(vi[t], e);
                        if (cl & 2u) {
                            if (cl & 1u) { s3.r += r; s3.i += i; } else { s2.r += r; s2.i += i; }
                        } else {
                            if (cl & 1u) { s1.r += r; s1.i += i; } else { s0.r += r; s0.i += i; }
                        }
                    }
                }
                if (!a.mergeMC) {
                    class_products(ar0, ai0, s0, s1, s2, s3, a.coefUP, a.partUP, a.nclsUP);
                    s0 = s1 = s2 = s3 = ClassSum{0, 0};
                }
                const uint32_t dp = (uint32_t)a.dimDNp;
                const uint32_t ns = reinterpret_cast<const uint32_t*>(S.steps)[d >> 5];
                const uint32_t ng = reinterpret_cast<const uint32_t*>(S.dnpos)[d];
                const uint16_t* sc = S.sched + d;
                // v ^ m with m = 0 or -1; the -m parts, the class's negative
                // entries of the column, are added once
                auto steps = [&](ClassSum& sum, int n, int neg) {
                    int64_t r = neg, i = neg;
#pragma unroll 2
                    for (int t = 0; t < n; ++t, sc += dp) {
                        const uint32_t w = *sc;
                        const longlong2 v = *reinterpret_cast<const longlong2*>(xrow + 2 * (w & 0x7FFFu));
                        const int64_t m = -(int64_t)(w >> 15);
                        r += v.x ^ m;
                        i += v.y ^ m;
                    }
                    sum.r += r;
                    sum.i += i;
                };
                steps(s0, ns & 0xFFu, ng & 0xFFu);
                steps(s1, (ns >> 8) & 0xFFu, (ng >> 8) & 0xFFu);
                steps(s2, (ns >> 16) & 0xFFu, (ng >> 16) & 0xFFu);
                steps(s3, ns >> 24, ng >> 24);
                class_products(ar0, ai0, s0, s1, s2, s3, a.coefDN, a.partDN, a.nclsDN);
            } else if constexpr (SEG) {
                // at most kSegCls classes: class by class over segments taken
                // from the rows' class-end bytes (+ entries first), the same
                // loop bounds for every lane in the up row; with equal class
                // lists the up and down sums of a class share one product.
                const uint32_t se_u = __ldg(a.upSegE + u), sp_u = __ldg(a.upSegP + u);
                const uint32_t se = __ldg(a.dnSegE + d0), sp = __ldg(a.dnSegP + d0);
                const uint32_t q0 = S.dptr[d0];
                const int ncl = max(a.nclsUP, a.nclsDN);
                uint32_t ub = 0, b = 0;
                for (int c = 0; c < ncl; ++c) {
                    int64_t r = 0, none = 0;
                    if (c < a.nclsUP) {
                        const uint32_t up = (sp_u >> (8 * c)) & 0xFFu, ue = (se_u >> (8 * c)) & 0xFFu;
                        for (uint32_t k = ub; k < up; ++k) acc_up<false, COH>(xq, S.uoff[k] + d0, r, none);
                        for (uint32_t k = up; k < ue; ++k) {
                            int64_t vr;
                            up_load<false, COH>(xq, S.uoff[k] + d0, vr, none);
                            r -= vr;
                        }
                        ub = ue;
                        if (!a.mergeMC) {
                            apply_class<false>(ar0, ai0, r, 0, a.coefUP, c, unitU, a.Fc);
                            r = 0;
                        }
                    }
                    if (c < a.nclsDN) {
                        const uint32_t pc = (sp >> (8 * c)) & 0xFFu, ec = (se >> (8 * c)) & 0xFFu;
                        for (uint32_t q = q0 + b; q < q0 + pc; ++q) r += xrow[S.dent[q] & kColMask];
                        for (uint32_t q = q0 + pc; q < q0 + ec; ++q) r -= xrow[S.dent[q] & kColMask];
                        b = ec;
                        apply_class<false>(ar0, ai0, r, 0, a.coefDN, c, unitD, a.Fc);
                    } else if (a.mergeMC) {
                        apply_class<false>(ar0, ai0, r, 0, a.coefUP, c, unitU, a.Fc);
                    }
                }
            } else if (a.perEntry) {
                // A row of a table with a coefficient per bond holds about one
                // entry of each class, so a running class sum saves no products
                // and its branches put every load behind the last one's use.
                // Here kN entries of the row are loaded at a time and multiplied
                // one by one (the same exact total): random-hopping Kagome12 6+6
                // 88 -> 69 us a persistent step, Lieb12 6+6 70 -> 56 us.
                constexpr int kN = CPLX ? 2 : 4;
                auto mac = [&](i128& ar, i128& ai, int64_t r, int64_t i, uint32_t e, const int64_t* coef) {
                    const uint32_t cl = (e >> kClassShift) & kClassMask;
                    r = apply_sign(r, e);
                    const int64_t cr = coef[2 * cl];
                    mac_wide(ar, r, cr);
                    if (CPLX) {
                        i = apply_sign(i, e);
                        const int64_t ci = coef[2 * cl + 1];
                        mac_wide(ai, i, cr);
                        mac_wide(ar, -i, ci);
                        mac_wide(ai, r, ci);
                    }
                };
                for (uint32_t k = 0; k < lenU; k += kN) {
                    int64_t r0[kN], i0[kN], r1[kN], i1[kN];
#pragma unroll
                    for (int t = 0; t < kN; ++t) {
                        const uint32_t o = S.uoff[min(k + t, lenU - 1)];  // past the end: a load that is not used
                        up_load<CPLX, COH>(xq, o + d0, r0[t], i0[t]);
                        up_load<CPLX, COH>(xq, o + d1c, r1[t], i1[t]);
                    }
#pragma unroll
                    for (int t = 0; t < kN; ++t) {
                        if (k + t >= lenU) break;
                        const uint32_t e = S.uent[k + t];
                        mac(ar0, ai0, r0[t], i0[t], e, S.cup);
                        mac(ar1, ai1, r1[t], i1[t], e, S.cup);
                    }
                }
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const uint32_t d = c ? d1c : d0;
                    const uint32_t q1 = S.dptr[d + 1];
#pragma unroll 2
                    for (uint32_t q = S.dptr[d]; q < q1; ++q) {
                        const uint32_t e = S.dent[q];
                        int64_t vr, vi;
                        row_elem<CPLX>(xrow, (e & kColMask) * W, vr, vi);
                        mac(c ? ar1 : ar0, c ? ai1 : ai0, vr, vi, e, S.cdn);
                    }
                }
            } else {
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const uint32_t d = c ? d1c : d0;
                    i128& ar = c ? ar1 : ar0;
                    i128& ai = c ? ai1 : ai0;
                    {
                        int cur = -1;
                        int64_t sr = 0, si = 0;
                        for (uint32_t k = 0; k < lenU; ++k) {
                            const uint32_t e = S.uent[k];
                            const int cl = (int)((e >> kClassShift) & kClassMask);
                            if (cl != cur) {
                                if (cur >= 0) apply_class<CPLX>(ar, ai, sr, si, a.coefUP, cur, unitU, a.Fc);
                                sr = 0;
                                si = 0;
                                cur = cl;
                            }
                            int64_t r, i;
                            up_load<CPLX, COH>(xq, S.uoff[k] + d, r, i);
                            sr += apply_sign(r, e);
                            if (CPLX) si += apply_sign(i, e);
                        }
                        if (cur >= 0) apply_class<CPLX>(ar, ai, sr, si, a.coefUP, cur, unitU, a.Fc);
                    }
                    {
                        int cur = -1;
                        int64_t sr = 0, si = 0;
                        for (uint32_t q = S.dptr[d]; q < S.dptr[d + 1]; ++q) {
                            const uint32_t e = S.dent[q];
                            const int cl = (int)((e >> kClassShift) & kClassMask);
                            if (cl != cur) {
                                if (cur >= 0) apply_class<CPLX>(ar, ai, sr, si, a.coefDN, cur, unitD, a.Fc);
                                sr = 0;
                                si = 0;
                                cur = cl;
                            }
                            const uint32_t col = (e & kColMask) * W;
                            int64_t vr, vi;
                            row_elem<CPLX>(xrow, col, vr, vi);
                            sr += apply_sign(vr, e);
                            if (CPLX) si += apply_sign(vi, e);
                        }
                        if (cur >= 0) apply_class<CPLX>(ar, ai, sr, si, a.coefDN, cur, unitD, a.Fc);
                    }
                }
            }
            // the row's diagonal terms, read here rather than held across the sums
            const uint64_t stu = __ldg(a.stUP + u);
            const int64_t du = __ldg(a.dUPq + u);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                if (c == 1 && !v1) break;
                const uint32_t d = c ? d1 : d0;
                i128& ar = c ? ar1 : ar0;
                i128& ai = c ? ai1 : ai0;
                int64_t xr, xi;
                row_elem<CPLX>(xrow, d * W, xr, xi);
                const int64_t ddn = GDIAG ? __ldg(a.dDNq + d) : S.ddq[d];
                const int64_t dq = du + ddn + a.Uq * (int64_t)__popcll(stu & S.dst[d] & a.mask);
                ar += mul_wide(dq, xr);
                if (CPLX) ai += mul_wide(dq, xi);
                const size_t o = (size_t)(ubase + d) * W;
                if (OUT == 0) {
                    y[o] = i128_to_f64(ar, E_out);
                    if (CPLX) y[o + 1] = i128_to_f64(ai, E_out);
                } else {
                    const int64_t qr = shr_round_i64(ar, s_u);
                    uq[o] = qr;
                    dot += mul_wide(xr, qr) >> 24;
                    uint64_t aq = (uint64_t)(qr < 0 ? -qr : qr);
                    mx = aq > mx ? aq : mx;
                    if (CPLX) {
                        const int64_t qi = shr_round_i64(ai, s_u);
                        uq[o + 1] = qi;
                        dot += mul_wide(xi, qi) >> 24;
                        aq = (uint64_t)(qi < 0 ? -qi : qi);
                        mx = aq > mx ? aq : mx;
                    }
                }
            }
        }
        __syncthreads();  // row buffer and uoff are free for the next iteration; *snext is written
        r = DYN ? *snext : r + 1;
        if (FAST) {
            ub ^= 1;
            staged = true;
        }
    }
}

}  // namespace ed

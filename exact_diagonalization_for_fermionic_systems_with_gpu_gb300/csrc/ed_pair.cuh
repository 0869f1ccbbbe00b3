// ed_pair.cuh — row-pair sums: two up rows of x interleaved in shared memory,
// used by the one-launch matvec (ed_matvec_pair.cu, which has the layout) and by
// the batched persistent Lanczos kernel.
#pragma once

#include "ed_device.cuh"
#include "ed_internal.hpp"
#include "ed_matvec_common.cuh"
#include "ed_matvec_tma.cuh"

namespace ed {
using namespace dev;


struct Two {
    int64_t a, b;  // rows u, u + 1
};

// 16 bytes of shared memory at a 32-bit address (volatile: ordered with the
// barriers around the staged rows)
__device__ __forceinline__ void lds2(uint32_t addr, int64_t& x, int64_t& y) {
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "r"(addr));
}

__device__ __forceinline__ void cp_async8(uint32_t dst, const int64_t* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tma::smem_u32(bar)) : "memory");
}

// Arrives on bar when this thread's copies so far have landed.
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tma::smem_u32(bar)) : "memory");
}

// One step of both rows: slot word w (low 15 bits; sign in bit 15).
template <bool SIGN>
__device__ __forceinline__ void pair_step(uint32_t addr, uint32_t m, Two& acc) {
    int64_t x, y;
    lds2(addr, x, y);
    if (SIGN) {
        uint64_t mm;
        asm("mov.b64 %0, {%1, %1};" : "=l"(mm) : "r"(m));
        x ^= (int64_t)mm;
        y ^= (int64_t)mm;
    }
    acc.a += x;
    acc.b += y;
}

template <bool SIGN>
__device__ __forceinline__ void pair_lo(uint32_t xs, uint32_t w, Two& acc) {
    uint32_t m = 0;
    if (SIGN) asm("prmt.b32 %0, %1, 0, 0x9999;" : "=r"(m) : "r"(w));  // bit 15 replicated
    pair_step<SIGN>(xs + ((w & 0x7FFFu) << 4), m, acc);
}

template <bool SIGN>
__device__ __forceinline__ void pair_hi(uint32_t xs, uint32_t w, Two& acc) {
    pair_step<SIGN>(xs + ((w >> 12) & 0x7FFF0u), (uint32_t)((int32_t)w >> 31), acc);
}

// n (0..8, the same for the warp) steps of a schedule word
template <bool SIGN>
__device__ __forceinline__ void pair_group(uint32_t xs, const uint4 w, int n, Two& acc) {
    switch (n) {
        case 8: pair_hi<SIGN>(xs, w.w, acc); [[fallthrough]];
        case 7: pair_lo<SIGN>(xs, w.w, acc); [[fallthrough]];
        case 6: pair_hi<SIGN>(xs, w.z, acc); [[fallthrough]];
        case 5: pair_lo<SIGN>(xs, w.z, acc); [[fallthrough]];
        case 4: pair_hi<SIGN>(xs, w.y, acc); [[fallthrough]];
        case 3: pair_lo<SIGN>(xs, w.y, acc); [[fallthrough]];
        case 2: pair_hi<SIGN>(xs, w.x, acc); [[fallthrough]];
        case 1: pair_lo<SIGN>(xs, w.x, acc); [[fallthrough]];
        default: break;
    }
}

// What a unit needs of one staged row.
struct PairRow {
    uint64_t st;
    int64_t du;
    int len, npos;
};

// Buffer k of a CTA's dynamic shared memory: the interleaved rows with eight zero
// slots, the up offsets of both rows, their PairRows.
struct PairBuf {
    uint32_t x32;             // shared address of the rows
    uint32_t (*uoff)[kPairUp];
    PairRow* rows;
    __device__ __forceinline__ PairBuf(unsigned char* xs, const PairArgs& g, int k) {
        unsigned char* p = xs + (size_t)k * pair_buf_bytes(g.zbase);
        x32 = (uint32_t)__cvta_generic_to_shared(p);
        uoff = reinterpret_cast<uint32_t(*)[kPairUp]>(p + (g.zbase + 8) * 16);
        rows = reinterpret_cast<PairRow*>(p + (g.zbase + 8) * 16 + sizeof(uint32_t) * 2 * kPairUp);
    }
};

// Zero slots and barriers of nbuf buffers (all threads; a __syncthreads follows).
__device__ __forceinline__ void pair_init(unsigned char* xs, const PairArgs& g, int nbuf, int nc, uint64_t* full,
                                          uint64_t* empty) {
    const int tid = threadIdx.x;
    if (tid < 8 * nbuf)
        *reinterpret_cast<longlong2*>(xs + (size_t)(tid >> 3) * pair_buf_bytes(g.zbase) + (g.zbase + (tid & 7)) * 16) =
            make_longlong2(0, 0);
    if (tid == 0) {
        for (int k = 0; k < nbuf; ++k) {
            tma::mbar_init(&full[k], 64);
            tma::mbar_init(&empty[k], nc);
        }
        tma::fence_mbar_init();
    }
}

// Rows u0 and u0 + 1 (an odd count ends on a pair of one row) into a buffer:
// thread i0 of n.  dUPq: the folded up diagonal.  The copies go through L1: xq was
// written before the launch, or lies where nothing has been read since it began.
__device__ __forceinline__ void pair_stage(const MvArgs& a, const int64_t* xq, const int64_t* dUPq, uint32_t u0,
                                           const PairBuf& B, uint32_t i0, uint32_t n) {
    const uint32_t dimDN = (uint32_t)a.dimDN;
    const int nrow = u0 + 1 < (uint32_t)a.dimUP ? 2 : 1;
    const int64_t* const r0 = xq + (size_t)u0 * dimDN;
    const int64_t* const r1 = nrow == 2 ? r0 + dimDN : r0;
#pragma unroll 4
    for (uint32_t c = i0; c < dimDN; c += n) {
        const uint32_t d = B.x32 + pair_slot(c) * 16u;
        cp_async8(d, r0 + c);
        cp_async8(d + 8, r1 + c);
    }
    // two dependent reads, while the copies are under way
    for (int r = 0; r < nrow; ++r) {
        const uint32_t u = u0 + r, q0 = __ldg(a.upPtr + u), len = __ldg(a.upPtr + u + 1) - q0;
        for (uint32_t i = i0; i < len; i += n) B.uoff[r][i] = (__ldg(a.upEntC + q0 + i) & kColMask) * dimDN;
        if (i0 == r) B.rows[r] = {__ldg(a.stUP + u), __ldg(dUPq + u), (int)len, (int)__ldg(a.upNpos + u)};
    }
}

// Sums of columns c0, c1 of a staged pair, lane by lane: down hops from shared
// memory into dn, up hops into up (MERGE: added to dn's values there).
template <bool VEC, bool SIGN, bool MERGE>
__device__ __forceinline__ void pair_sums(const PairArgs& g, const int64_t* xq, const PairBuf& B, bool has1, int b,
                                          int lane, uint32_t c0, uint32_t c1, bool v1, Two (&dn)[2], Two (&up)[2]) {
    const uint4* __restrict__ words = reinterpret_cast<const uint4*>(g.words);
    const int64_t* const xc = xq + c0;
    auto get = [&](uint32_t off, int64_t& w0, int64_t& w1) {
        if (VEC) {
            const longlong2 v = __ldcg(reinterpret_cast<const longlong2*>(xc + off));
            w0 = v.x;
            w1 = v.y;
        } else {
            w0 = __ldcg(xc + off);
            w1 = v1 ? __ldcg(xc + off + 32) : 0;
        }
    };
    // down sums of columns c0, c1 in both rows
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint4* sp = words + ((size_t)(2 * b + h) * g.groups) * 32 + lane;
        int n = __ldg(g.steps + 2 * b + h);
        const int64_t neg = SIGN && (h == 0 || v1) ? __ldg(g.negcnt + (h ? c1 : c0)) : 0;
        dn[h] = Two{neg, neg};
        for (; n > 8; n -= 8, sp += 32) pair_group<SIGN>(B.x32, __ldg(sp), 8, dn[h]);
        pair_group<SIGN>(B.x32, __ldg(sp), n, dn[h]);
        if (!SIGN && g.sign < 0) dn[h] = Two{-dn[h].a, -dn[h].b};
    }
    // up sums (added to the down sums where one product serves both)
    if (MERGE) {
        up[0] = dn[0];
        up[1] = dn[1];
    } else {
        up[0] = up[1] = Two{0, 0};
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        if (r == 1 && !has1) break;
        const int len = B.rows[r].len, npos = B.rows[r].npos;
        int64_t s0 = 0, s1 = 0;
        int k = 0;
#pragma unroll 4
        for (; k < npos; ++k) {
            int64_t w0, w1;
            get(B.uoff[r][k], w0, w1);
            s0 += w0;
            s1 += w1;
        }
#pragma unroll 4
        for (; k < len; ++k) {
            int64_t w0, w1;
            get(B.uoff[r][k], w0, w1);
            s0 -= w0;
            s1 -= w1;
        }
        (r ? up[0].b : up[0].a) += s0;
        (r ? up[1].b : up[1].a) += s1;
    }
}

}  // namespace ed

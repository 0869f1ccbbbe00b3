// ed_matvec_pair.cu — one-launch matvec over pairs of up rows, for real
// operators with one coefficient class per spin whose down rows are too long
// for the table-resident row engine (14- to 16-site sectors: 3,000 to 14,000
// down states), or whose vectors are large (prefer_pair has the sizes).
//
// A CTA stages rows u and u + 1 of x interleaved in shared memory, 16 bytes a
// column, so that one 16-byte load of a down hop serves both rows and one
// decoded schedule entry four additions.  The schedule (ed::PairSchedule, read
// from L1 / L2, eight steps in a 16-byte word) gives the eight lanes of every
// quarter warp different bank groups in each step.  A lane computes two columns
// of both rows: down sums from shared memory, then the up neighbours of each
// row with 16-byte loads of its column pair (dim_dn even; two 8-byte loads
// otherwise), the diagonal, one rounding, and the Lanczos partials.
// Where two or more pairs fit in shared memory the last warp stages the next ones
// with 8-byte asynchronous copies (each row is contiguous, the pair is not) while the
// other 31 compute, with a full and an empty barrier a buffer (as many buffers as
// give every warp two units: 16-site 8+3, nine units a pair, 205 -> 157 us with seven
// for two): units of 64 columns
// go round the computing warps across pairs, so that no warp waits at the end of
// a pair for the slowest (54 units on 16 warps: four rounds for 3.4).  Longer rows
// are staged by all threads between two barriers; the next pair is prefetched into
// L2 meanwhile.
//
// Measured against the one-thread-per-element kernel it replaces there (Lanczos
// matvec): 14-site chain 7+7 230 -> 142 us, 14-site 7+6 237 -> 134 us, 15-site
// 7+8 1,470 -> 516 us, 16-site 8+8 6,300 -> 2,515 us (with one pair a CTA, two CTAs
// of 512 threads and barriers around each pair: 160, 144, 606 and 2,530 us).
// About 240 instructions an output at half of the issue slots (16 sites: 40 %):
// bound by the latency of the up loads and the schedule words (32 warps an SM at
// 64 registers).  Loading the words and the first up loads ahead of the sums (74 to
// 90 registers, 24 or 20 warps), prefetching the up neighbours of a warp's next
// unit into L2 (16-site 2,530 -> 2,650 us) and batching the up loads' remainders
// were slower or the same.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "ed_pair.cuh"

namespace ed {
using namespace dev;

// OUT = 0: FP64 y; OUT = 1: FX u with the Lanczos epilogue.  VEC: dim_dn even,
// lane l has columns 2l, 2l + 1 of a 64-column block; otherwise l, l + 32.
// MERGE: equal hopping coefficients, one product for the up and down sums.
// nbuf: row pairs in shared memory (several: the last warp stages, one: all do).
template <int OUT, bool VEC, bool SIGN, bool MERGE>
__global__ void __launch_bounds__(1024, 1) k_mv_pair(const MvArgs a, const PairArgs g, const int nbuf) {
    extern __shared__ __align__(128) unsigned char xs[];
    __shared__ uint64_t full[kPairBufs], empty[kPairBufs];
    const uint32_t dimUP = (uint32_t)a.dimUP, dimDN = (uint32_t)a.dimDN;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const int nc = nbuf == 1 ? nwarps : nwarps - 1;  // computing warps
    const int64_t* __restrict__ xq = a.xq;
    int E_out = 0, s_u = 0;
    if (OUT == 0) {
        E_out = fx_exp_from_emax(*a.p_emax) - a.Fc;
    } else {
        const int b = a.bq_bits + bitlen_u64(*a.p_mx) - 62;
        s_u = b > 0 ? b : 0;
    }
    const bool unitU = a.unitUP != 0 && a.nclsUP == 1, unitD = a.unitDN != 0 && a.nclsDN == 1;
    const bool fold = OUT == 1 && MERGE && unitU && s_u > 0 && a.Fc >= s_u;
    const bool y16 = OUT == 1 || (reinterpret_cast<uintptr_t>(a.y) & 15) == 0;  // y may start on any double
    i128 dot = 0;
    uint64_t mx = 0;
    pair_init(xs, g, nbuf, nc, full, empty);
    __syncthreads();
    const uint32_t npairs = (dimUP + 1) / 2;
    int buf = 0;
    uint32_t parity = 0;  // of the buffer's current use
    if (warp == nc) {
        for (uint32_t it = blockIdx.x; it < npairs; it += gridDim.x) {
            if (!tma::mbar_wait(&empty[buf], parity ^ 1)) {  // at once in the buffer's first use
                if (lane == 0) atomicExch(a.err, 1);
                break;
            }
            pair_stage(a, xq, a.dUPq, 2 * it, PairBuf(xs, g, buf), lane, 32);
            cp_async_arrive(&full[buf]);
            mbar_arrive(&full[buf]);
            if (++buf == nbuf) {
                buf = 0;
                parity ^= 1;
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    uint32_t b0 = warp;  // this warp's first unit of the item: units go round the computing warps across items
    for (uint32_t it = warp == nc ? npairs : blockIdx.x; it < npairs; it += gridDim.x) {
        const uint32_t u0 = 2 * it;
        const bool has1 = u0 + 1 < dimUP;
        const PairBuf B(xs, g, buf);
        if (nbuf == 1) {
            __syncthreads();  // the previous rows are no longer read
            pair_stage(a, xq, a.dUPq, 2 * it, B, tid, blockDim.x);
            if (tid == 0 && it + gridDim.x < npairs) {
                // an even row starts on a 16-byte boundary
                const uint32_t un = 2 * (it + gridDim.x);
                const uint32_t bytes = (dimDN * (un + 1 < dimUP ? 2u : 1u) * 8u) & ~15u;
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(xq + (size_t)un * dimDN), "r"(bytes)
                             : "memory");
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
        } else if (!tma::mbar_wait(&full[buf], parity)) {
            if (lane == 0) atomicExch(a.err, 1);
            break;
        }
        int b = b0;
        for (; b < g.blocks; b += nc) {
            const uint32_t c0 = 64u * b + (VEC ? 2u * lane : (uint32_t)lane), c1 = VEC ? c0 + 1 : c0 + 32;
            if (c0 >= dimDN) continue;
            const bool v1 = VEC || c1 < dimDN;  // the second column exists
            Two dn[2], up[2];
            pair_sums<VEC, SIGN, MERGE>(g, xq, B, has1, b, lane, c0, c1, v1, dn, up);
            int64_t qo[2][2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                if (h == 1 && !v1) break;
                const uint32_t c = h ? c1 : c0;
                int64_t xr[2];
                lds2(B.x32 + pair_slot(c) * 16u, xr[0], xr[1]);
                const int64_t ddn = __ldg(a.dDNq + c);
                const uint64_t std_ = __ldg(a.stDN + c) & a.mask;
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const PairRow& R = B.rows[has1 ? r : 0];
                    const int64_t x = xr[r], us = r ? up[h].b : up[h].a, ds = r ? dn[h].b : dn[h].a;
                    const int64_t dq = R.du + ddn + a.Uq * (int64_t)__popcll(R.st & std_);
                    if (OUT == 1 && fold) {
                        qo[r][h] = fold_round(us, mul_wide(dq, x), a.Fc, s_u);
                    } else {
                        i128 ar = 0, ai = 0;
                        if (MERGE) {
                            apply_class<false>(ar, ai, us, 0, a.coefUP, 0, unitU, a.Fc);
                        } else {
                            if (R.len) apply_class<false>(ar, ai, us, 0, a.coefUP, 0, unitU, a.Fc);
                            if (a.nclsDN) apply_class<false>(ar, ai, ds, 0, a.coefDN, 0, unitD, a.Fc);
                        }
                        ar += mul_wide(dq, x);
                        qo[r][h] = OUT == 0 ? __double_as_longlong(i128_to_f64(ar, E_out)) : shr_round_i64(ar, s_u);
                    }
                    if (OUT == 1 && (r == 0 || has1)) {
                        const int64_t q = qo[r][h];
                        dot += mul_wide(x, q) >> 24;
                        const uint64_t aq = (uint64_t)(q < 0 ? -q : q);
                        mx = aq > mx ? aq : mx;
                    }
                }
            }
            int64_t* out = OUT == 0 ? reinterpret_cast<int64_t*>(a.y) : a.uq;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                if (r == 1 && !has1) break;
                int64_t* o = out + (size_t)(u0 + r) * dimDN + c0;
                if (VEC && y16) {
                    __stcs(reinterpret_cast<longlong2*>(o), make_longlong2(qo[r][0], qo[r][1]));
                } else {
                    o[0] = qo[r][0];
                    if (v1) o[c1 - c0] = qo[r][1];
                }
            }
        }
        if (nbuf > 1) {
            b0 = b - g.blocks;
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[buf]);
            if (++buf == nbuf) {
                buf = 0;
                parity ^= 1;
            }
        }
    }
    if (OUT == 1) mv_lanczos_epilogue(a, dot, mx, s_u);
}

int pair_smem_bytes(int64_t zbase) {
    const int64_t bytes = (zbase + 8) * 16;
    return bytes <= kPairMaxSmem ? (int)bytes : 0;
}

// Buffers of a CTA: units for all the computing warps twice over (a buffer is free
// when its last unit is done), two where a pair has as many units itself.  More
// would take the schedule words' L1.
int pair_buffers(int zbase, int64_t blocks) {
    const int64_t fit = kPairMaxDyn / pair_buf_bytes(zbase);
    const int64_t want = blocks >= 31 ? 2 : (62 + blocks - 1) / blocks;
    return (int)std::max<int64_t>(1, std::min<int64_t>({fit, want, kPairBufs}));
}

template <int OUT, bool VEC, bool MERGE>
static cudaError_t launch_pair3(const ed_op* op, const MvArgs& a, cudaStream_t s) {
    auto kern = op->pair_args.sign == 0 ? k_mv_pair<OUT, VEC, true, MERGE> : k_mv_pair<OUT, VEC, false, MERGE>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, op->pair_nbuf * pair_buf_bytes(op->pair_args.zbase));
    if (e != cudaSuccess) return e;
    kern<<<op->pair_grid, op->pair_threads, op->pair_nbuf * pair_buf_bytes(op->pair_args.zbase), s>>>(a, op->pair_args, op->pair_nbuf);
    return cudaGetLastError();
}

template <int OUT, bool VEC>
static cudaError_t launch_pair2(const ed_op* op, const MvArgs& a, cudaStream_t s) {
    return a.mergeUD ? launch_pair3<OUT, VEC, true>(op, a, s) : launch_pair3<OUT, VEC, false>(op, a, s);
}

cudaError_t launch_matvec_pair(const ed_op* op, const MvArgs& a, int out, cudaStream_t s) {
    if (op->dimDN % 2 == 0) return out == 0 ? launch_pair2<0, true>(op, a, s) : launch_pair2<1, true>(op, a, s);
    return out == 0 ? launch_pair2<0, false>(op, a, s) : launch_pair2<1, false>(op, a, s);
}

}  // namespace ed

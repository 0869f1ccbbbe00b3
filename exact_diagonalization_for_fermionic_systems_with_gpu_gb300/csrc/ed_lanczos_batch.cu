// ed_lanczos_batch.cu — B Lanczos runs in lockstep in one persistent launch:
// instances of one sector that share their hopping tables (real, one class) and
// differ in their diagonals and scalars (LzInst), stored basis, fixed steps.
//
// The matvec phase runs over (instance, row pair) items, instance-major, a fixed
// stride of them per CTA, with the row-pair kernel's sums (ed_pair.cuh): the last
// warp stages the next item's two rows while 31 compute 64-column units of the
// current one, and units go round the warps across items, so that no warp waits at
// the end of a row.  A warp keeps the instance's <x, u> and max|u| partials in
// registers while its units belong to it and adds them to per-instance shared limb
// sums when the instance changes (and its norm partials after each instance's
// axpy slice).  Barriers, the four rotating reduction sets (B sets each) and the
// scalar update (warp b of every CTA for instance b) are the single-run
// kernel's, so every instance's coefficients are bit-identical to its own run;
// the batch saves the per-step barrier and scalar time of B - 1 runs.
//
// Rows are staged through L1 (pair_stage), which keeps lines of vectors that other
// CTAs write: right only because every step writes a slot that no CTA has read in
// this launch (the whole basis is stored) and slots are whole 256-byte blocks, so
// that no line holds two of them.  Runs that reuse slots cannot go this way.  u,
// written anew in every step, and the axpy's operands are read past L1.
//
// Against the row engine's items (512 threads, two barriers a row) that this
// replaces, an instance's step in batches of eight (200 steps, Ritz sums included):
// 12-site chain 7+5 24.2 -> 17.5 us (20.4 with two buffers, 26 units for 31 warps,
// in place of five), 6+6 28.2 -> 20.5, 11-site 5+5 12.0 -> 7.8, 10-site 5+5 8.7 ->
// 5.1, 8-site 4+4 6.0 -> 3.4.  Bound by issue slots and L2 latency in the sums and by
// HBM in the axpy phase (eight 12-site instances' vectors are larger than L2); 64
// registers a thread leave no room for more loads in flight.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "ed_grid.cuh"
#include "ed_lanczos.hpp"
#include "ed_lanczos_dev.cuh"
#include "ed_pair.cuh"

namespace ed {
using namespace dev;

namespace {
constexpr int kBatchThreads = 1024;
}

template <bool VEC, bool SIGN, bool MERGE>
__global__ void __launch_bounds__(kBatchThreads, 1) k_lz_batch(const MvArgs a, const PairArgs g, const LzBatchArgs f,
                                                               const int nbuf) {
    extern __shared__ __align__(128) unsigned char xs[];
    __shared__ uint64_t full[kPairBufs], empty[kPairBufs];
    __shared__ int give_up;
    __shared__ LzInst s_inst[kLzBatchMax];
    __shared__ SlotScalars sX[kLzBatchMax], sP[kLzBatchMax];
    __shared__ int s_status[kLzBatchMax], s_min_bits[kLzBatchMax], s_ew[kLzBatchMax];
    __shared__ LzCoefs s_coef[kLzBatchMax];
    __shared__ unsigned long long accl[kLzBatchMax][3], accm[kLzBatchMax];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int nc = kBatchThreads / 32 - 1;  // computing warps
    const int B = f.B;
    const uint32_t dimUP = (uint32_t)a.dimUP, dimDN = (uint32_t)a.dimDN, G = gridDim.x;
    const uint32_t npairs = (dimUP + 1) / 2, nitems = (uint32_t)B * npairs;
    if (tid < B) {
        const LzInst& I = f.inst[tid];
        s_inst[tid] = I;
        const LzState* lz = I.lz;
        const int j = f.j0;
        sX[tid] = {lz->e[j], lz->m[j], lz->beta[j], lz_inv(lz->beta[j])};
        if (j > 0) sP[tid] = {lz->e[j - 1], lz->m[j - 1], lz->beta[j - 1], lz_inv(lz->beta[j - 1])};
        else sP[tid] = {0, 0, 0.0, 0.0};
        s_status[tid] = lz->status;
        s_min_bits[tid] = lz->min_bits;
        s_ew[tid] = 0;
        accl[tid][0] = accl[tid][1] = accl[tid][2] = 0;
        accm[tid] = 0;
    }
    if (tid == 0) give_up = 0;
    pair_init(xs, g, nbuf, nc, full, empty);
    __syncthreads();

    int buf = 0;              // buffer of this thread's next item, and the parity of its use
    uint32_t parity = 0;
    unsigned int target = 0;  // grid-barrier arrivals expected so far
    for (int j = f.j0; j < f.j1; ++j) {
        const int rM = 2 * (j - f.j0), rA = rM + 1;
        // ---- phase M: u_b = H_b w_j of every instance, item by item --------
        if (warp == nc) {
            for (uint32_t it = blockIdx.x; it < nitems; it += G) {
                const uint32_t ib = it / npairs, u0 = 2 * (it - ib * npairs);
                const LzInst& I = s_inst[ib];
                if (!tma::mbar_wait(&empty[buf], parity ^ 1)) {  // at once in the buffer's first use
                    if (lane == 0) atomicExch(a.err, 1);
                    give_up = 1;
                    break;
                }
                pair_stage(a, I.basis + (size_t)j * f.stride, I.dUPq, u0, PairBuf(xs, g, buf), lane, 32);
                cp_async_arrive(&full[buf]);
                mbar_arrive(&full[buf]);
                if (++buf == nbuf) {
                    buf = 0;
                    parity ^= 1;
                }
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
        } else {
            if (warp == nc - 1 && lane < B && j > f.j0) {
                // slot j of instance b from the previous step's axpy reduction
                // (read at the scalar update after the next barrier)
                const int b = lane;
                i128 ss;
                uint64_t mw;
                red_pull(&f.red[((rM - 1) % 4) * B + b], ss, mw);
                slot_done(s_inst[b].lz, j, s_ew[b], ss, mw, sX[b], sP[b], s_status[b], s_min_bits[b], blockIdx.x == 0);
            }
            __syncwarp();
            i128 dot = 0;
            uint64_t mx = 0;
            int cur = -1;
            uint32_t b0 = warp;
            for (uint32_t it = blockIdx.x; it < nitems; it += G) {
                const int ib = (int)(it / npairs);
                const uint32_t u0 = 2 * (it - ib * npairs);
                if (ib != cur) {
                    if (cur >= 0) batch_flush(dot, mx, accl[cur], &accm[cur]);
                    dot = 0;
                    mx = 0;
                    cur = ib;
                }
                const LzInst& I = s_inst[ib];
                const bool has1 = u0 + 1 < dimUP;
                const PairBuf P(xs, g, buf);
                const int64_t* const xq = I.basis + (size_t)j * f.stride;
                if (!tma::mbar_wait(&full[buf], parity)) {
                    if (lane == 0) atomicExch(a.err, 1);
                    give_up = 1;
                    break;
                }
                const int sb = I.bq_bits + kFxBits - 62;
                const int s_u = sb > 0 ? sb : 0;
                const bool unitU = I.unitUP != 0 && I.nclsUP == 1, unitD = I.unitDN != 0 && I.nclsDN == 1;
                const bool fold = MERGE && unitU && s_u > 0 && I.Fc >= s_u;
                int b = b0;
                for (; b < g.blocks; b += nc) {
                    const uint32_t c0 = 64u * b + (VEC ? 2u * lane : (uint32_t)lane), c1 = VEC ? c0 + 1 : c0 + 32;
                    if (c0 >= dimDN) continue;
                    const bool v1 = VEC || c1 < dimDN;  // the second column exists
                    Two dn[2], up[2];
                    pair_sums<VEC, SIGN, MERGE>(g, xq, P, has1, b, lane, c0, c1, v1, dn, up);
                    int64_t qo[2][2];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (h == 1 && !v1) break;
                        const uint32_t c = h ? c1 : c0;
                        int64_t xr[2];
                        lds2(P.x32 + pair_slot(c) * 16u, xr[0], xr[1]);
                        const int64_t ddn = __ldg(I.dDNq + c);
                        const uint64_t std_ = __ldg(a.stDN + c) & a.mask;
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            const PairRow& R = P.rows[has1 ? r : 0];
                            const int64_t x = xr[r], us = r ? up[h].b : up[h].a, ds = r ? dn[h].b : dn[h].a;
                            const int64_t dq = R.du + ddn + I.Uq * (int64_t)__popcll(R.st & std_);
                            if (fold) {
                                qo[r][h] = fold_round(us, mul_wide(dq, x), I.Fc, s_u);
                            } else {
                                i128 ar = mul_wide(dq, x);
                                if (MERGE) {
                                    ar += unitU ? ((i128)us) << I.Fc : mul_wide(us, I.coefUP);
                                } else {
                                    if (R.len) ar += unitU ? ((i128)us) << I.Fc : mul_wide(us, I.coefUP);
                                    if (I.nclsDN) ar += unitD ? ((i128)ds) << I.Fc : mul_wide(ds, I.coefDN);
                                }
                                qo[r][h] = shr_round_i64(ar, s_u);
                            }
                            if (r == 0 || has1) {
                                const int64_t q = qo[r][h];
                                dot += mul_wide(x, q) >> 24;
                                const uint64_t aq = (uint64_t)(q < 0 ? -q : q);
                                mx = aq > mx ? aq : mx;
                            }
                        }
                    }
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        if (r == 1 && !has1) break;
                        int64_t* o = I.u + (size_t)(u0 + r) * dimDN + c0;
                        if (VEC) {
                            *reinterpret_cast<longlong2*>(o) = make_longlong2(qo[r][0], qo[r][1]);
                        } else {
                            o[0] = qo[r][0];
                            if (v1) o[c1 - c0] = qo[r][1];
                        }
                    }
                }
                b0 = b - g.blocks;
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[buf]);
                if (++buf == nbuf) {
                    buf = 0;
                    parity ^= 1;
                }
            }
            __syncwarp();
            if (cur >= 0) batch_flush(dot, mx, accl[cur], &accm[cur]);
        }
        __syncthreads();
        if (give_up) return;  // (the staging warp has waited for its copies)
        if (tid < B) {
            red_push(&f.red[(rM % 4) * B + tid], batch_total(accl[tid]), accm[tid]);
            accl[tid][0] = accl[tid][1] = accl[tid][2] = 0;
            accm[tid] = 0;
        }
        if (!grid_sync(f.gbar, target, &give_up, a.err, f.wait)) return;
        if (warp < B) {
            const int b = warp;
            i128 s;
            uint64_t m;
            red_pull(&f.red[(rM % 4) * B + b], s, m);
            const LzInst& I = s_inst[b];
            const int sb = I.bq_bits + kFxBits - 62;
            const int s_u = sb > 0 ? sb : 0;
            const int e_u = sX[b].e - I.Fc + s_u;
            const LzCoefs c = lz_coefs_warp(j, s, e_u, m, sX[b].e, sX[b].m, sX[b].beta, sX[b].ib, sP[b].e, sP[b].m,
                                            sP[b].ib, s_status[b]);
            if (lane == 0) {
                s_coef[b] = c;
                s_ew[b] = c.e_w;
                if (blockIdx.x == 0) {
                    if (rM >= 2) f.red[((rM - 2) % 4) * B + b] = LzRedSet{0, 0, 0, 0};
                    LzState* lz = I.lz;
                    lz->s_u = s_u;
                    lz->e_u = e_u;
                    lz->m_u = m;
                    lz_store_coefs(lz, j, c);
                }
            }
        }
        __syncthreads();

        // ---- phase A: w_{j+1} of every instance ----------------------------
        // Vectors shorter than a pass of the grid: the instances side by side, a
        // share of the CTAs each (eight of 63,504 elements: one latency for eight, 7.0 ->
        // 5.1 us a step and instance).  Longer ones in turn, the last instance
        // first: the rows phase ended on it, so its u and w_j are the vectors still
        // in L2, and the next rows phase starts on instance 0, whose w_{j+1} this
        // phase writes last.
        const int64_t npair = f.n >> 1;
        const bool split = npair < (int64_t)G * kBatchThreads;
        const uint32_t nb = split ? G / (uint32_t)B : G, q = split ? blockIdx.x % nb : blockIdx.x;
        for (int k = 0; k < (split ? 1 : B); ++k) {
            const int b = split ? (int)(blockIdx.x / nb) : B - 1 - k;
            if (b >= B) break;
            const LzInst& I = s_inst[b];
            const int64_t* xq = I.basis + (size_t)j * f.stride;
            const int64_t* pq = j > 0 ? I.basis + (size_t)(j - 1) * f.stride : xq;
            int64_t* wq = I.basis + (size_t)(j + 1) * f.stride;
            const int64_t a0 = s_coef[b].at[0], a1 = s_coef[b].at[1], a2 = s_coef[b].at[2];
            const int Fa = s_coef[b].Fa;
            i128 ss = 0;
            uint64_t mw = 0;
            const longlong2* u2 = reinterpret_cast<const longlong2*>(I.u);
            const longlong2* x2 = reinterpret_cast<const longlong2*>(xq);
            const longlong2* p2 = reinterpret_cast<const longlong2*>(pq);
            longlong2* w2 = reinterpret_cast<longlong2*>(wq);
            for (int64_t i = (int64_t)q * kBatchThreads + tid; i < npair; i += (int64_t)nb * kBatchThreads) {
                const longlong2 uu = __ldcg(u2 + i), xx = __ldcg(x2 + i), pp = __ldcg(p2 + i);
                longlong2 w;
                w.x = shr_round_i64(mul_wide(a0, uu.x) + mul_wide(a1, xx.x) + mul_wide(a2, pp.x), Fa);
                w.y = shr_round_i64(mul_wide(a0, uu.y) + mul_wide(a1, xx.y) + mul_wide(a2, pp.y), Fa);
                w2[i] = w;
                ss += (mul_wide(w.x, w.x) >> 16) + (mul_wide(w.y, w.y) >> 16);
                const uint64_t ax = (uint64_t)(w.x < 0 ? -w.x : w.x), ay = (uint64_t)(w.y < 0 ? -w.y : w.y);
                mw = ax > mw ? ax : mw;
                mw = ay > mw ? ay : mw;
            }
            if ((f.n & 1) && q == 0 && tid == 0) {
                const int64_t i = f.n - 1;
                const int64_t w = shr_round_i64(
                    mul_wide(a0, __ldcg(I.u + i)) + mul_wide(a1, __ldcg(xq + i)) + mul_wide(a2, __ldcg(pq + i)), Fa);
                wq[i] = w;
                ss += mul_wide(w, w) >> 16;
                const uint64_t aw = (uint64_t)(w < 0 ? -w : w);
                mw = aw > mw ? aw : mw;
            }
            batch_flush(ss, mw, accl[b], &accm[b]);
        }
        __syncthreads();
        if (tid < B) {
            red_push(&f.red[(rA % 4) * B + tid], batch_total(accl[tid]), accm[tid]);
            accl[tid][0] = accl[tid][1] = accl[tid][2] = 0;
            accm[tid] = 0;
        }
        if (!grid_sync(f.gbar, target, &give_up, a.err, f.wait)) return;
        if (tid < B && blockIdx.x == 0) {
            const int b = tid;
            if (rA >= 2) f.red[((rA - 2) % 4) * B + b] = LzRedSet{0, 0, 0, 0};
            if (j + 1 == f.j1) {
                i128 ss;
                uint64_t mw;
                red_pull(&f.red[(rA % 4) * B + b], ss, mw);
                slot_done(s_inst[b].lz, j + 1, s_coef[b].e_w, ss, mw, sX[b], sP[b], s_status[b], s_min_bits[b], true);
            }
        }
        __syncthreads();
    }
}

// Cooperative launch of the batch, a CTA an SM, with the first operator's tables.
// cudaErrorNotSupported when the grid cannot be co-resident or two row pairs do not
// fit shared memory.
cudaError_t launch_lz_batch(const ed_op* op, const LzBatchArgs& f, bool merge, cudaStream_t s) {
    int nbuf = op->pair_nbuf;
    const int smem = nbuf * pair_buf_bytes(op->pair_args.zbase);
    if (op->pair_smem == 0 || nbuf < 2) return cudaErrorNotSupported;
    const void* fn;
    if (op->dimDN % 2 == 0)
        fn = op->pair_args.sign == 0 ? (merge ? (const void*)k_lz_batch<true, true, true> : (const void*)k_lz_batch<true, true, false>)
                                     : (merge ? (const void*)k_lz_batch<true, false, true> : (const void*)k_lz_batch<true, false, false>);
    else
        fn = op->pair_args.sign == 0 ? (merge ? (const void*)k_lz_batch<false, true, true> : (const void*)k_lz_batch<false, true, false>)
                                     : (merge ? (const void*)k_lz_batch<false, false, true> : (const void*)k_lz_batch<false, false, false>);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0, sms = 0, coop = 0;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kBatchThreads, smem)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, op->device)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, op->device)) != cudaSuccess) return e;
    if (!coop || per_sm < 1) return cudaErrorNotSupported;
    MvArgs av = op->mv;
    PairArgs gv = op->pair_args;
    LzBatchArgs fv = f;
    void* args[] = {&av, &gv, &fv, &nbuf};
    return cudaLaunchCooperativeKernel(fn, dim3((unsigned)sms), dim3(kBatchThreads), args, (size_t)smem, s);
}

}  // namespace ed

// ed_krylov.cu — Krylov time evolution psi(t) = exp(-i H t) psi0.
//
// The reference (Krylov<C>, MBL_test/include/HubMatrix_GPU.cuh:619-728)
// builds the tridiagonal T of psi0 with up to 1000 Lanczos steps, stopping
// at b < 1e-10, diagonalises it with LAPACK dsted, and for every time step
// regenerates the Krylov vectors with one Hubbard_mv each while adding
// (sum_j e^{-i m_j t} z_j[0] z_j[i]) v_i into phi.
//
// Here the recurrence is the Lanczos run of ed_lanczos.cu (the persistent
// kernel where the operator has one), its basis kept in device memory in the
// FX format (v_k = q_k 2^e_k / beta_k); T's propagator column
// exp(-i T t) e_0 comes from the host QR solver (ed_tridiag.cpp); and one
// kernel forms psi(t) = beta_0 sum_k c_k(t) v_k for up to kKrTimes times per
// pass over the basis.  Each time costs a quarter of a read of the basis
// instead of the reference's n matvecs.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "../../include/ed_hubbard.h"
#include "ed_device.cuh"
#include "ed_internal.hpp"
#include "ed_tridiag.hpp"

namespace ed {
namespace {

constexpr int kKrThreads = 256;
constexpr int kKrTimes = 4;  // times formed per pass over the basis
constexpr int kKcThreads = 128;
constexpr int kKcGroup = 8;    // basis vectors per copy group
constexpr int kKcChunk = 128;  // basis vectors whose coefficients are staged at a time
constexpr int kKcCarry = dev::kLimbRun / 2;  // vectors between carries (a complex product adds two terms)
static_assert(kKcCarry % kKcGroup == 0 && kKcChunk % kKcGroup == 0, "carry interval");
constexpr int kKrBlocks = 152 * 8;

int kr_grid(int64_t n) {
    int64_t g = (n + kKrThreads - 1) / kKrThreads;
    return (int)std::max<int64_t>(1, std::min<int64_t>(g, kKrBlocks));
}

// per block: sum of squares of the real and of the imaginary parts
__global__ void k_part_norms(const double* __restrict__ z, int64_t n, double* __restrict__ part) {
    double s0 = 0.0, s1 = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double2 v = reinterpret_cast<const double2*>(z)[i];
        s0 = fma(v.x, v.x, s0);
        s1 = fma(v.y, v.y, s1);
    }
    __shared__ double r0[kKrThreads], r1[kKrThreads];
    r0[threadIdx.x] = s0;
    r1[threadIdx.x] = s1;
    __syncthreads();
    for (int w = kKrThreads / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
            r0[threadIdx.x] += r0[threadIdx.x + w];
            r1[threadIdx.x] += r1[threadIdx.x + w];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = r0[0];
        part[2 * blockIdx.x + 1] = r1[0];
    }
}

// real vector of part p (0: re, 1: im) of n complex values
__global__ void k_part(const double* __restrict__ z, int64_t n, int p, double* __restrict__ out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = z[2 * i + p];
}

// out[t] = (accumulate ? out[t] : 0) + f * sum_k c_k(t) q_k for t < NT,
// f = i when times_i, else 1; q_k real (CPLX false) or complex.  coef holds
// for each k the NT times' (re high, re low, im high, im low) limbs, scaled
// by 2^F[t].
//
// Bound by instruction issue: the sums are exact integers (limb_mac, three
// 32-bit multiplies and their 64-bit adds per real product; four, before the
// cross products came from one, took 594 us for 470 at 140 vectors of 853,776
// elements and 4 times), where FP64 multiply-adds issue at 1/64 of the FP32 rate.  A thread forms two adjacent
// real elements (or one complex one) at NT = 4 times from 16 bytes of every
// basis vector; at the 48 accumulator registers x 2 that takes, 12 warps an
// SM are resident, too few to hide load latency, so each thread copies its
// own words of the next kKcGroup vectors into shared memory (cp.async, no
// barrier: only the copying thread reads them) while it sums the current
// ones, and the coefficients are staged for the block kKcChunk vectors at a
// time.
struct KrShift {
    int F[kKrTimes];
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(bytes)
                 : "memory");
}

template <bool CPLX, int NT>
__global__ void __launch_bounds__(kKcThreads, 3) k_krylov_combine(const int64_t* __restrict__ basis, int64_t stride,
                                                                  int64_t n, int nk, const int4* __restrict__ coef,
                                                                  const KrShift sh, double2* __restrict__ out,
                                                                  int64_t out_stride, int accumulate, int times_i) {
    using namespace dev;
    constexpr int E = CPLX ? 1 : 2;  // elements per thread
    __shared__ longlong2 sq[2][kKcGroup][kKcThreads];
    __shared__ int4 sc[kKcChunk * NT];
    const int tid = threadIdx.x;
    const int64_t items = (n + E - 1) / E;
    const int ngroups = (nk + kKcGroup - 1) / kKcGroup;
    // every thread of the block runs the same iterations (the coefficient
    // staging has barriers); threads past the end sum nothing and write nothing
    for (int64_t i0 = (int64_t)blockIdx.x * kKcThreads; i0 < items; i0 += (int64_t)gridDim.x * kKcThreads) {
        const int64_t i = i0 + tid;
        const bool live = i < items;
        const bool pair = CPLX || 2 * i + 1 < n;  // the second 8-byte word exists
        const int bytes = live ? (pair ? 16 : 8) : 0;
        const int64_t* q = basis + (live ? 2 * i : 0);
        LimbSum re[E][NT], im[E][NT];
#pragma unroll
        for (int e = 0; e < E; ++e)
#pragma unroll
            for (int t = 0; t < NT; ++t) re[e][t] = im[e][t] = LimbSum{0, 0, 0};
        auto fetch = [&](int g) {
#pragma unroll
            for (int kk = 0; kk < kKcGroup; ++kk) {
                const int k = g * kKcGroup + kk;
                if (k < nk) cp_async16(&sq[g & 1][kk][tid], q + (int64_t)k * stride, bytes);  // zero past `bytes`
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        fetch(0);
        for (int g = 0; g < ngroups; ++g) {
            const int k0 = g * kKcGroup;
            if (k0 % kKcChunk == 0) {
                __syncthreads();  // the previous chunk is no longer read
                const int m = min(kKcChunk, nk - k0) * NT;
                for (int c = tid; c < m; c += kKcThreads) sc[c] = __ldg(coef + (size_t)k0 * NT + c);
                __syncthreads();
            }
            if (g + 1 < ngroups) {
                fetch(g + 1);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            const int4* cg = sc + (size_t)(k0 % kKcChunk) * NT;
            const int kn = min(kKcGroup, nk - k0);
#pragma unroll 2
            for (int kk = 0; kk < kn; ++kk) {
                const longlong2 v = sq[g & 1][kk][tid];
                int xh, xl, yh, yl, nh = 0, nl = 0;
                limb_split(v.x, xh, xl);
                limb_split(v.y, yh, yl);
                if (CPLX) limb_split(-v.y, nh, nl);
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const int4 c = cg[kk * NT + t];
                    limb_mac(re[0][t], xh, xl, c.x, c.y);
                    limb_mac(im[0][t], xh, xl, c.z, c.w);
                    if (CPLX) {
                        limb_mac(re[0][t], nh, nl, c.z, c.w);
                        limb_mac(im[0][t], yh, yl, c.x, c.y);
                    } else {
                        limb_mac(re[E - 1][t], yh, yl, c.x, c.y);
                        limb_mac(im[E - 1][t], yh, yl, c.z, c.w);
                    }
                }
            }
            if ((k0 + kKcGroup) % kKcCarry == 0 || g + 1 == ngroups) {
#pragma unroll
                for (int e = 0; e < E; ++e)
#pragma unroll
                    for (int t = 0; t < NT; ++t) {
                        limb_carry(re[e][t]);
                        limb_carry(im[e][t]);
                    }
            }
        }
        if (!live) continue;
#pragma unroll
        for (int t = 0; t < NT; ++t) {
#pragma unroll
            for (int e = 0; e < E; ++e) {
                if (e == 1 && !pair) break;
                double2 v;
                v.x = i128_to_f64(limb_total(re[e][t]), -sh.F[t]);
                v.y = i128_to_f64(limb_total(im[e][t]), -sh.F[t]);
                if (times_i) v = make_double2(-v.y, v.x);
                double2* o = out + (size_t)t * out_stride + E * i + e;
                if (accumulate) {
                    const double2 p = *o;
                    v.x += p.x;
                    v.y += p.y;
                }
                *o = v;
            }
        }
    }
}

template <bool CPLX>
void launch_combine(int nt, const int64_t* basis, int64_t stride, int64_t n, int nk, const int4* coef, const KrShift& sh,
                    double2* out, int64_t out_stride, int accumulate, int times_i, cudaStream_t s) {
    const int64_t items = CPLX ? n : (n + 1) / 2;
    const int g = (int)std::max<int64_t>(1, std::min<int64_t>((items + kKcThreads - 1) / kKcThreads, 152 * 32));
    if (nt == 4)
        k_krylov_combine<CPLX, 4><<<g, kKcThreads, 0, s>>>(basis, stride, n, nk, coef, sh, out, out_stride, accumulate, times_i);
    else if (nt == 2)
        k_krylov_combine<CPLX, 2><<<g, kKcThreads, 0, s>>>(basis, stride, n, nk, coef, sh, out, out_stride, accumulate, times_i);
    else
        k_krylov_combine<CPLX, 1><<<g, kKcThreads, 0, s>>>(basis, stride, n, nk, coef, sh, out, out_stride, accumulate, times_i);
}

// Two-pass-matvec operators (the basis is not kept): out[t][p(i)] +=
// f * coef[t] q[i] for the regenerated real vector q in the permuted down
// order, p(i) = u * dim_dn + perm[c] its table-order position, f = i when
// times_i; every position is touched by one thread.
__global__ void __launch_bounds__(kKrThreads) k_krylov_acc_perm(const int64_t* __restrict__ q, int64_t dimUP,
                                                               int64_t dimDN, const uint32_t* __restrict__ perm,
                                                               const double2* __restrict__ coef, int nt,
                                                               double2* __restrict__ out, int64_t out_stride,
                                                               int times_i) {
    const int64_t D = dimUP * dimDN;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < D; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t u = i / dimDN, c = i - u * dimDN;
        const int64_t p = u * dimDN + __ldg(perm + c);
        const double w = (double)__ldg(q + i);
        for (int t = 0; t < nt; ++t) {
            const double2 cf = __ldg(coef + t);
            double2* o = out + (size_t)t * out_stride + p;
            double2 v = *o;
            if (times_i) {
                v.x -= cf.y * w;
                v.y += cf.x * w;
            } else {
                v.x += cf.x * w;
                v.y += cf.y * w;
            }
            *o = v;
        }
    }
}

}  // namespace
}  // namespace ed

extern "C" {

ed_status ed_krylov_evolve(ed_op* op, const ed_krylov_cfg* cfg, const double* psi0, int psi0_mem, int n_times,
                           const double* times, double* psi_out, int out_mem, ed_krylov_result* res,
                           void* stream) {
    using namespace ed;
    if (!op || !cfg || !psi0 || n_times < 0 || (n_times > 0 && (!times || !psi_out))) return ED_ERR_ARG;
    if (cfg->max_steps < 1 || cfg->max_steps > 100000 || !(cfg->tol >= 0.0)) return ED_ERR_ARG;
    if (psi0_mem != ED_MEM_HOST && psi0_mem != ED_MEM_DEVICE) return ED_ERR_ARG;
    if (out_mem != ED_MEM_HOST && out_mem != ED_MEM_DEVICE) return ED_ERR_ARG;
    for (int t = 0; t < n_times; ++t)
        if (!std::isfinite(times[t])) return ED_ERR_ARG;
    if (cudaSetDevice(op->device) != cudaSuccess) return ED_ERR_CUDA;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const int64_t D = op->D;
    int64_t launches = 0;
    ed_status st = ED_OK;

    double *d0 = nullptr, *dout = nullptr, *tmp = nullptr, *part = nullptr;
    double2* dcoef = nullptr;
    auto release = [&]() {
        if (psi0_mem == ED_MEM_HOST) cudaFreeAsync(d0, s);
        if (out_mem == ED_MEM_HOST) cudaFreeAsync(dout, s);
        cudaFreeAsync(tmp, s);
        cudaFreeAsync(part, s);
        cudaFreeAsync(dcoef, s);
        cudaStreamSynchronize(s);
    };
#define KR_CK(x)                            \
    do {                                    \
        if ((x) != cudaSuccess) {           \
            release();                      \
            return ED_ERR_CUDA;             \
        }                                   \
    } while (0)

    const size_t vbytes = sizeof(double) * 2 * (size_t)D;
    if (psi0_mem == ED_MEM_HOST) {
        if (cudaMallocAsync(&d0, vbytes, s) != cudaSuccess) return ED_ERR_ALLOC;
        KR_CK(cudaMemcpyAsync(d0, psi0, vbytes, cudaMemcpyHostToDevice, s));
    } else {
        d0 = const_cast<double*>(psi0);
    }
    const bool acc = cfg->accumulate != 0;
    if (out_mem == ED_MEM_HOST) {
        if (n_times > 0 && cudaMallocAsync(&dout, vbytes * n_times, s) != cudaSuccess) { release(); return ED_ERR_ALLOC; }
        if (n_times > 0 && acc) KR_CK(cudaMemcpyAsync(dout, psi_out, vbytes * n_times, cudaMemcpyHostToDevice, s));
    } else {
        dout = psi_out;
    }
    // |re psi0|^2, |im psi0|^2 (block partials summed in order on the host)
    const int g = kr_grid(D);
    if (cudaMallocAsync(&part, sizeof(double) * 2 * g, s) != cudaSuccess) { release(); return ED_ERR_ALLOC; }
    k_part_norms<<<g, kKrThreads, 0, s>>>(d0, D, part);
    KR_CK(cudaGetLastError());
    ++launches;
    std::vector<double> hp(2 * g);
    KR_CK(cudaMemcpyAsync(hp.data(), part, sizeof(double) * 2 * g, cudaMemcpyDeviceToHost, s));
    KR_CK(cudaStreamSynchronize(s));
    double n2[2] = {0.0, 0.0};
    for (int b = 0; b < g; ++b) {
        n2[0] += hp[2 * b];
        n2[1] += hp[2 * b + 1];
    }
    if (!std::isfinite(n2[0]) || !std::isfinite(n2[1])) { release(); return ED_ERR_NONFINITE; }

    // one recurrence for a complex operator; one per nonzero part for a real one
    struct Run { const double* start; int part; };
    std::vector<Run> runs;
    if (op->cplx) {
        if (n2[0] + n2[1] > 0.0) runs.push_back({d0, -1});
    } else {
        if (D > 0 && cudaMallocAsync(&tmp, sizeof(double) * (size_t)D, s) != cudaSuccess) { release(); return ED_ERR_ALLOC; }
        for (int p = 0; p < 2; ++p)
            if (n2[p] > 0.0) runs.push_back({tmp, p});
    }
    if ((runs.empty() || op->striped) && n_times > 0 && !acc) KR_CK(cudaMemsetAsync(dout, 0, vbytes * n_times, s));

    ed_lanczos_cfg lc{};
    lc.max_steps = cfg->max_steps;
    lc.mode = ED_LANCZOS_FIXED;
    lc.reorth = cfg->reorth;
    // the two-pass matvec's sectors keep three vectors and regenerate the basis
    lc.ritz = op->striped ? ED_RITZ_NONE : ED_RITZ_STORED;
    lc.start = ED_START_USER;
    std::vector<double> alpha(cfg->max_steps + 2), beta(cfg->max_steps + 2);
    int max_n = 0;
    double err = 0.0;
    bool written = acc;
    if (n_times > 0 && cudaMallocAsync(&dcoef, sizeof(double2) * (size_t)n_times * (cfg->max_steps + 1), s) != cudaSuccess) {
        release();
        return ED_ERR_ALLOC;
    }
    for (const Run& run : runs) {
        if (run.part >= 0) {
            k_part<<<kr_grid(D), kKrThreads, 0, s>>>(d0, D, run.part, tmp);
            KR_CK(cudaGetLastError());
            ++launches;
        }
        ed_lanczos_result lr{};
        st = lanczos_run(op, lanczos_ws_slot(op), &lc, run.start, ED_MEM_DEVICE, nullptr, ED_MEM_DEVICE, alpha.data(),
                         beta.data(), &lr, s, cfg->tol);
        if (st != ED_OK) { release(); return st; }
        launches += lr.launches;
        const int n = lr.steps;
        max_n = std::max(max_n, n);
        if (n_times == 0) continue;
        std::vector<double> c((size_t)2 * n * n_times);
        if (!tridiag_expm_e0(n, alpha.data(), beta.data() + 1, n_times, times, c.data())) {
            release();
            return ED_ERR_BREAKDOWN;
        }
        const int64_t* basis;
        int64_t stride;
        const int* e_dev;
        lanczos_basis(*lanczos_ws_slot(op), &basis, &stride, &e_dev);
        std::vector<int> e(n);
        KR_CK(cudaMemcpyAsync(e.data(), e_dev, sizeof(int) * n, cudaMemcpyDeviceToHost, s));
        KR_CK(cudaStreamSynchronize(s));
        // psi(t) = beta_0 sum_k c_k(t) v_k,  v_k = q_k 2^e_k / beta_k
        std::vector<double2> coef((size_t)n * n_times);
        for (int t = 0; t < n_times; ++t) {
            for (int k = 0; k < n; ++k) {
                const double f = beta[0] * std::ldexp(1.0, e[k]) / beta[k];
                coef[(size_t)t * n + k] = make_double2(f * c[(size_t)2 * n * t + 2 * k], f * c[(size_t)2 * n * t + 2 * k + 1]);
            }
            const double* cl = c.data() + (size_t)2 * n * t + 2 * (n - 1);
            err = std::max(err, beta[n] * std::hypot(cl[0], cl[1]) * beta[0]);
        }
        if (op->striped) {
            // coefficients time-major per vector: coefk[k][t]
            std::vector<double2> coefk((size_t)n * n_times);
            for (int t = 0; t < n_times; ++t)
                for (int k = 0; k < n; ++k) coefk[(size_t)k * n_times + t] = coef[(size_t)t * n + k];
            KR_CK(cudaMemcpyAsync(dcoef, coefk.data(), sizeof(double2) * coefk.size(), cudaMemcpyHostToDevice, s));
            const int cg = kr_grid(D);
            const int ti = run.part == 1 ? 1 : 0;
            double2* o = reinterpret_cast<double2*>(dout);
            st = lanczos_replay(op, *lanczos_ws_slot(op), n, [&](int k, const int64_t* qk) -> cudaError_t {
                k_krylov_acc_perm<<<cg, kKrThreads, 0, s>>>(qk, op->dimUP, op->dimDN, op->d_permDN,
                                                             dcoef + (size_t)k * n_times, n_times, o, D, ti);
                ++launches;
                return cudaGetLastError();
            }, s);
            if (st != ED_OK) { release(); return st; }
            KR_CK(cudaStreamSynchronize(s));
            written = true;
            continue;
        }
        // groups of 4 times, then 2 and 1: (re, im) limbs, vector-major inside a group
        struct Group { int t0, nt; size_t at; KrShift sh; };
        std::vector<Group> groups;
        std::vector<int4> limbs((size_t)n * n_times);
        std::vector<double> r(2 * (size_t)n);
        std::vector<int32_t> hl(4 * (size_t)n);
        for (int t0 = 0; t0 < n_times;) {
            const int left = n_times - t0, nt = left >= 4 ? 4 : (left >= 2 ? 2 : 1);
            Group gr{t0, nt, (size_t)n * t0, {}};
            for (int t = 0; t < nt; ++t) {
                for (int k = 0; k < n; ++k) {
                    const double2 cf = coef[(size_t)(t0 + t) * n + k];
                    r[2 * k] = cf.x;
                    r[2 * k + 1] = cf.y;
                }
                gr.sh.F[t] = limb_coefs(r.data(), 2 * n, hl.data());
                for (int k = 0; k < n; ++k)
                    limbs[gr.at + (size_t)k * nt + t] = make_int4(hl[4 * k], hl[4 * k + 1], hl[4 * k + 2], hl[4 * k + 3]);
            }
            groups.push_back(gr);
            t0 += nt;
        }
        static_assert(sizeof(int4) == sizeof(double2), "dcoef holds either form");
        KR_CK(cudaMemcpyAsync(dcoef, limbs.data(), sizeof(int4) * limbs.size(), cudaMemcpyHostToDevice, s));
        for (const Group& gr : groups) {
            double2* o = reinterpret_cast<double2*>(dout) + (size_t)gr.t0 * D;
            const int4* cf = reinterpret_cast<const int4*>(dcoef) + gr.at;
            if (op->cplx)
                launch_combine<true>(gr.nt, basis, stride, D, n, cf, gr.sh, o, D, written ? 1 : 0, run.part == 1 ? 1 : 0, s);
            else
                launch_combine<false>(gr.nt, basis, stride, D, n, cf, gr.sh, o, D, written ? 1 : 0, run.part == 1 ? 1 : 0, s);
            KR_CK(cudaGetLastError());
            ++launches;
        }
        // the next run overwrites the basis and the coefficients
        KR_CK(cudaStreamSynchronize(s));
        written = true;
    }
    if (out_mem == ED_MEM_HOST && n_times > 0)
        KR_CK(cudaMemcpyAsync(psi_out, dout, vbytes * n_times, cudaMemcpyDeviceToHost, s));
    KR_CK(cudaStreamSynchronize(s));
#undef KR_CK
    release();
    if (res) {
        res->steps = max_n;
        res->runs = (int)runs.size();
        res->norm = std::sqrt(n2[0] + n2[1]);
        res->err_est = err;
        res->launches = launches;
    }
    return ED_OK;
}

}  // extern "C"

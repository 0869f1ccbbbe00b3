// ed_ee_bidiag.cu — singular values of the entanglement-matrix blocks:
// Householder bidiagonalisation on the device, one thread-block cluster per
// block, then the Golub-Kahan bidiagonal SVD on the host.
//
// cusolverDnDgesvd runs a block of a few hundred rows at one SM's FP64 rate
// (a 400 x 400 block: 8.5e7 FMA, 26 ms on GB300, where FP64 issues at 1/64
// of FP32).  Here the rows of a block are spread over the CTAs of a cluster
// (up to 16 SMs), each CTA holding its slab of rows in shared memory for the
// whole reduction; a step k of the alternating reflections (Golub & Van
// Loan, Matrix Computations, 4th ed., Algorithm 5.4.2) needs two cluster
// barriers: one after every CTA has written its partial column norm and its
// partial w' = A[k+1:, k]^T A[k+1:, k+1:] (summed by every CTA in rank order
// through distributed shared memory, so all CTAs hold identical reflectors),
// one after the owner of row k has formed the right reflector.  The right
// reflector's update is local to each CTA's rows.  Output: the bidiagonal
// (d, e) of every block; its singular values are those of the block up to
// eps |block| (the backward error of the reflections), the accuracy gesvd has.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "../../include/ed_hubbard.h"
#include "ed_ee_plan.hpp"
#include "ed_internal.hpp"
#include "ed_tridiag.hpp"

namespace cg = cooperative_groups;

namespace ed {
namespace {

constexpr int kBdThreads = 512;
constexpr int kBdWarps = kBdThreads / 32;

struct EeJob {
    int64_t off;  // block: column-major m x n (m >= n) at blocks + off
    int32_t m, n;
    int64_t de;   // d at dd + de (n values), e at ee + de (n - 1 values)
};

constexpr int kBdChunk = 8;  // rows of an update unit

// LAPACK dlarfg convention: H = I - tau v v^T, v_0 = 1, H [alpha; x] = [beta; 0]
__device__ __forceinline__ void bd_reflector(double alpha, double xnorm2, double* beta, double* tau, double* scale) {
    if (xnorm2 == 0.0) {
        *beta = alpha;
        *tau = 0.0;
        *scale = 0.0;
        return;
    }
    const double b = -copysign(sqrt(fma(alpha, alpha, xnorm2)), alpha);
    *beta = b;
    *tau = (b - alpha) / b;
    *scale = 1.0 / (alpha - b);
}

// part(g0) + ... + part(g0 + G - 1), neighbours first
template <int G, typename F>
__device__ __forceinline__ double tree_sum(int g0, const F& part) {
    if constexpr (G == 1) return part(g0);
    else return tree_sum<G / 2>(g0, part) + tree_sum<G / 2>(g0 + G / 2, part);
}

// The arithmetic (four multiply-adds an element and step) is bound by the FP64
// pipe, which takes a warp instruction in 64 cycles on each of an SM's four
// schedulers, so every phase deals equal units of (32 columns, a few rows) to
// the 16 warps: with a thread per column, 5 warps of a 150-column step left
// half the pipes idle, and a warp per row spent as much on its shuffle sums as
// on the products.
template <int CS>
__global__ void __launch_bounds__(kBdThreads, 1) k_ee_bidiag(const EeJob* __restrict__ jobs,
                                                             const double* __restrict__ blocks,
                                                             double* __restrict__ dd, double* __restrict__ ee) {
    cg::cluster_group cl = cg::this_cluster();
    constexpr int G = kBdGroups / CS;  // groups of this CTA
    static_assert(G >= 2, "wv lies on group 1's sums");
    const int rank = (int)cl.block_rank();
    const EeJob J = jobs[blockIdx.x / CS];
    const int m = J.m, n = J.n;
    const int Rg = bd_group_rows(m), R = Rg * G;
    const int r0 = min(m, rank * R), r1 = min(m, r0 + R);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    extern __shared__ double sm[];
    double* slab = sm;                    // own rows, row-major, stride n
    double* pg = slab + (size_t)R * n;    // [g][j]: group g's part of the column sums
    double* part = pg;                    // [j] = sum over own rows i > k of A_ik A_ij, j >= k (on group 0's)
    double* wv = pg + n;                  // tau w_j of the left reflector (on group 1's, read by then)
    double* uu = wv;                      // local copy of u, once wv has been used
    double* rowk = pg + (size_t)G * n;    // row k (columns >= k), written by its owner
    double* ubuf = rowk + n;              // right reflector u_j (j > k), tau' at [n]
    double* zz = ubuf + n + 1;            // v_i of the left reflector, then tau' z_i of the right one
    double* sc = zz + R;                  // tau, scale of the left reflector
    const double* src = blocks + J.off;
    for (int64_t idx = tid; idx < (int64_t)(r1 - r0) * n; idx += kBdThreads) {
        const int i = (int)(idx % (r1 - r0)), j = (int)(idx / (r1 - r0));
        slab[(size_t)i * n + j] = src[(size_t)j * m + r0 + i];
    }
    __syncthreads();
    // own rows ilo .. r1-1: A_ij -= z_i c_j for j >= j0
    auto rank1 = [&](int ilo, int j0, const double* c) {
        const int jb = (n - j0 + 31) / 32, nc = (r1 - ilo + kBdChunk - 1) / kBdChunk;
        for (int u = warp; u < jb * nc; u += kBdWarps) {
            const int q = u / jb, j = j0 + (u - q * jb) * 32 + lane;
            if (j >= n) continue;
            const double cj = -c[j];
            const int i0 = ilo + q * kBdChunk, i1 = min(r1, i0 + kBdChunk);
            double* a = slab + (size_t)(i0 - r0) * n + j;
            for (int i = i0; i < i1; ++i, a += n) *a = fma(cj, zz[i - r0], *a);
        }
    };
    for (int k = 0; k < n; ++k) {
        const int owner = k / R;
        const int ilo = max(r0, k + 1);
        // (1) partials over own rows below k, group by group; part[k] is the
        // column's sigma'
        {
            const int jb = (n - k + 31) / 32;
            for (int u = warp; u < jb * G; u += kBdWarps) {
                const int g = u / jb, j = k + (u - g * jb) * 32 + lane;
                if (j >= n) continue;
                const int ib = max(ilo, r0 + g * Rg), ie = min(r1, r0 + (g + 1) * Rg);
                const double* a = slab + (size_t)(ib - r0) * n;
                double w = 0.0;
                for (int i = ib; i < ie; ++i, a += n) w = fma(a[k], a[j], w);
                pg[(size_t)g * n + j] = w;
            }
            __syncthreads();
            for (int j = k + tid; j < n; j += kBdThreads)
                part[j] = tree_sum<G>(0, [&](int g) { return pg[(size_t)g * n + j]; });
        }
        if (rank == owner)
            for (int j = k + tid; j < n; j += kBdThreads) rowk[j] = slab[(size_t)(k - r0) * n + j];
        cl.sync();  // A: partials and row k visible cluster-wide
        const double* rk = cl.map_shared_rank(rowk, owner);
        // (2) one warp forms the left reflector (the same tree over the ranks in
        // every CTA)
        if (warp == 0) {
            double sg = lane < CS ? cl.map_shared_rank(part, lane)[k] : 0.0;
#pragma unroll
            for (int o = 1; o < CS; o <<= 1) sg += __shfl_xor_sync(0xffffffffu, sg, o);
            if (lane == 0) {
                double beta, tau, scale;
                bd_reflector(rk[k], sg, &beta, &tau, &scale);
                sc[0] = tau;
                sc[1] = scale;
                if (rank == owner) dd[J.de + k] = beta;
            }
        }
        __syncthreads();
        const double tau = sc[0], scale = sc[1];
        for (int j = k + 1 + tid; j < n; j += kBdThreads) {
            const double w = tree_sum<CS>(0, [&](int r) { return cl.map_shared_rank(part, r)[j]; });
            wv[j] = tau * fma(scale, w, rk[j]);
        }
        const int il = max(r0, k);
        for (int i = il + tid; i < r1; i += kBdThreads)
            zz[i - r0] = (i == k) ? 1.0 : slab[(size_t)(i - r0) * n + k] * scale;
        __syncthreads();
        // (3) left update of own rows i >= k: A_ij -= tau v_i w_j
        if (tau != 0.0) rank1(il, k + 1, wv);
        __syncthreads();
        if (k + 1 >= n) break;
        // (4) one warp of the owner of row k forms the right reflector of A[k, k+1:]
        if (rank == owner && warp == 0) {
            const double* ak = slab + (size_t)(k - r0) * n;
            double x2 = 0.0;
            for (int j = k + 2 + lane; j < n; j += 32) x2 = fma(ak[j], ak[j], x2);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x2 += __shfl_xor_sync(0xffffffffu, x2, o);
            double b2, t2, s2;
            bd_reflector(ak[k + 1], x2, &b2, &t2, &s2);
            for (int j = k + 2 + lane; j < n; j += 32) ubuf[j] = ak[j] * s2;
            if (lane == 0) {
                ubuf[k + 1] = 1.0;
                ubuf[n] = t2;
                ee[J.de + k] = b2;
            }
        }
        cl.sync();  // B: the right reflector visible cluster-wide
        // (5) right update of own rows below k: z_i = tau' A[i, k+1:] u, A -= z u^T
        const double* ur = cl.map_shared_rank(ubuf, owner);
        const double tau2 = ur[n];
        for (int j = k + 1 + tid; j < n; j += kBdThreads) uu[j] = ur[j];
        __syncthreads();
        if (tau2 != 0.0) {
            // eight lanes a row, four rows a warp
            const int sub = lane >> 3, l8 = lane & 7;
            for (int i0 = ilo + 4 * warp; i0 < r1; i0 += 4 * kBdWarps) {
                const int i = i0 + sub;
                const double* ai = slab + (size_t)(min(i, r1 - 1) - r0) * n;
                double z = 0.0;
                for (int j = k + 1 + l8; j < n; j += 8) z = fma(ai[j], uu[j], z);
#pragma unroll
                for (int o = 1; o < 8; o <<= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
                if (l8 == 0 && i < r1) zz[i - r0] = tau2 * z;
            }
            __syncthreads();
            rank1(ilo, k + 1, uu);
        }
        __syncthreads();
    }
    cl.sync();  // no CTA leaves while another may still read its shared memory
}

// Launch one cluster of CS CTAs per job; false when this device cannot run it.
template <int CS>
bool launch_bidiag(const std::vector<EeJob>& jobs, const double* blocks, double* dd, double* ee, cudaStream_t s,
                   EeJob* djobs, size_t smem_bytes) {
    if (jobs.empty()) return true;
    const auto fn = k_ee_bidiag<CS>;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes) != cudaSuccess) return false;
    if (CS > 8 && cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return false;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)(jobs.size() * CS), 1, 1);
    lc.blockDim = dim3(kBdThreads, 1, 1);
    lc.dynamicSmemBytes = smem_bytes;
    lc.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CS;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    lc.attrs = at;
    lc.numAttrs = 1;
    int nclusters = 0;
    if (cudaOccupancyMaxActiveClusters(&nclusters, fn, &lc) != cudaSuccess || nclusters < 1) {
        cudaGetLastError();
        return false;
    }
    if (cudaLaunchKernelEx(&lc, fn, (const EeJob*)djobs, blocks, dd, ee) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return true;
}

}  // namespace

// Streams for the per-cluster-size launches (created once per device).
cudaStream_t bd_stream(int device, int i) {
    static std::mutex mu;
    static std::vector<std::vector<cudaStream_t>> st;
    std::lock_guard<std::mutex> g(mu);
    if ((int)st.size() <= device) st.resize(device + 1);
    while ((int)st[device].size() <= i) {
        cudaStream_t x = nullptr;
        if (cudaStreamCreateWithFlags(&x, cudaStreamNonBlocking) != cudaSuccess) return nullptr;
        st[device].push_back(x);
    }
    return st[device][i];
}

// Singular values of the blocks that fit the cluster kernel: handled[k] = 1
// and their values (descending) in sv_host[svo[k] ..).  The others are left
// for the cuSOLVER path.  Cluster size per block in proportion to its work.
// The largest block's is the one with the smallest estimate: a state by itself
// leaves SMs idle, so 16 CTAs end soonest ((7,5) of 12 sites: 3.3 ms, 5.8 ms
// on 4), while the blocks of a batch fill the GPU and wider clusters only add
// waiting (eight states: 14.7 ms on 16, 6.3 ms on 4).  One launch per cluster
// size, on its own stream.
ed_status ee_bidiag_blocks(int device, cudaStream_t s, const double* blocks, const std::vector<int64_t>& off,
                           const std::vector<int>& mm, const std::vector<int>& nn, const std::vector<int64_t>& svo,
                           std::vector<double>* sv_host, std::vector<char>* handled) {
    const char* env = std::getenv("ED_EE_METHOD");
    handled->assign(off.size(), 0);
    if (env && std::string(env) == "gesvd") return ED_OK;
    int max_smem = 0;
    cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    const size_t cap = (size_t)max_smem / sizeof(double);
    double wmax = 0.0;
    for (size_t k = 0; k < off.size(); ++k) wmax = std::max(wmax, (double)mm[k] * nn[k] * nn[k]);
    auto cluster = [&](size_t k, int top) {
        return bd_cluster(mm[k], nn[k], (double)mm[k] * nn[k] * nn[k] / wmax, top, cap);
    };
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    int top = 16;
    double best = 1e300;
    for (int t = 16; t >= 1; t /= 2) {
        double longest = 0.0, area = 0.0;
        for (size_t k = 0; k < off.size(); ++k) {
            const int g = nn[k] > 0 ? cluster(k, t) : kBdSizes;
            if (g >= kBdSizes) continue;
            const double sec = bd_seconds(mm[k], nn[k], g);
            longest = std::max(longest, sec);
            area += sec * (1 << g);
        }
        const double est = std::max(longest, area / sms);
        if (est < best) {
            best = est;
            top = t;
        }
    }
    constexpr int kSizes = kBdSizes;
    std::vector<EeJob> group[kSizes];
    size_t smem[kSizes] = {};
    std::vector<int> tag(off.size(), -1);
    for (size_t k = 0; k < off.size(); ++k) {
        const int m = mm[k], n = nn[k];
        if (n <= 0) { (*handled)[k] = 1; continue; }
        const int g = cluster(k, top);
        if (g >= kSizes) continue;  // too large for a cluster: cuSOLVER
        tag[k] = g;
        group[g].push_back(EeJob{off[k], m, n, svo[k]});
        smem[g] = std::max(smem[g], bd_smem_doubles(m, n, kBdGroups >> g));
    }
    size_t njobs = 0;
    for (int g = 0; g < kSizes; ++g) njobs += group[g].size();
    if (njobs == 0) return ED_OK;
    const int64_t total = svo.back();
    double *dd = nullptr, *ee = nullptr;
    EeJob* djobs = nullptr;
    if (cudaMalloc(&dd, sizeof(double) * std::max<int64_t>(total, 1)) != cudaSuccess ||
        cudaMalloc(&ee, sizeof(double) * std::max<int64_t>(total, 1)) != cudaSuccess ||
        cudaMalloc(&djobs, sizeof(EeJob) * njobs) != cudaSuccess) {
        cudaFree(dd); cudaFree(ee); cudaFree(djobs);
        return ED_ERR_ALLOC;
    }
    std::vector<EeJob> all;
    size_t first[kSizes];
    for (int g = kSizes - 1; g >= 0; --g) {
        first[g] = all.size();
        all.insert(all.end(), group[g].begin(), group[g].end());
    }
    ed_status st = ED_OK;
    if (cudaMemcpyAsync(djobs, all.data(), sizeof(EeJob) * njobs, cudaMemcpyHostToDevice, s) != cudaSuccess)
        st = ED_ERR_CUDA;
    cudaEvent_t ready = nullptr;
    if (st == ED_OK && (cudaEventCreateWithFlags(&ready, cudaEventDisableTiming) != cudaSuccess ||
                        cudaEventRecord(ready, s) != cudaSuccess))
        st = ED_ERR_CUDA;
    bool ok[kSizes] = {true, true, true, true, true};
    std::vector<cudaEvent_t> done_ev;
    for (int g = kSizes - 1; st == ED_OK && g >= 0; --g) {
        if (group[g].empty()) continue;
        cudaStream_t gs = bd_stream(device, g);
        cudaEvent_t ev = nullptr;
        if (!gs || cudaStreamWaitEvent(gs, ready, 0) != cudaSuccess ||
            cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) {
            st = ED_ERR_CUDA;
            break;
        }
        const size_t bytes = smem[g] * sizeof(double);
        EeJob* const dj = djobs + first[g];
        switch (g) {
            case 0: ok[g] = launch_bidiag<1>(group[g], blocks, dd, ee, gs, dj, bytes); break;
            case 1: ok[g] = launch_bidiag<2>(group[g], blocks, dd, ee, gs, dj, bytes); break;
            case 2: ok[g] = launch_bidiag<4>(group[g], blocks, dd, ee, gs, dj, bytes); break;
            case 3: ok[g] = launch_bidiag<8>(group[g], blocks, dd, ee, gs, dj, bytes); break;
            default: ok[g] = launch_bidiag<16>(group[g], blocks, dd, ee, gs, dj, bytes); break;
        }
        cudaEventRecord(ev, gs);
        cudaStreamWaitEvent(s, ev, 0);
        done_ev.push_back(ev);
    }
    std::vector<double> hd(std::max<int64_t>(total, 1)), he(std::max<int64_t>(total, 1));
    if (st == ED_OK && (cudaMemcpyAsync(hd.data(), dd, sizeof(double) * total, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
                        cudaMemcpyAsync(he.data(), ee, sizeof(double) * total, cudaMemcpyDeviceToHost, s) != cudaSuccess ||
                        cudaStreamSynchronize(s) != cudaSuccess))
        st = ED_ERR_CUDA;
    for (cudaEvent_t ev : done_ev) cudaEventDestroy(ev);
    if (ready) cudaEventDestroy(ready);
    cudaFree(dd); cudaFree(ee); cudaFree(djobs);
    if (st != ED_OK) return st;
    // the bidiagonal SVDs on host threads, largest first
    std::vector<int> todo;
    for (size_t k = 0; k < off.size(); ++k)
        if (tag[k] >= 0 && ok[tag[k]]) todo.push_back((int)k);
    std::stable_sort(todo.begin(), todo.end(), [&](int a, int b) { return nn[a] > nn[b]; });
    std::vector<char> ok_sv(off.size(), 0);
    const int nth = std::max(1, std::min<int>((int)todo.size(), (int)std::thread::hardware_concurrency()));
    // dealt in turn, largest first; a thread sweeps several of its matrices at a time
    auto work = [&](int t0) {
        std::vector<int> mine, n;
        std::vector<double*> d, e;
        for (size_t t = t0; t < todo.size(); t += nth) {
            const int k = todo[t];
            mine.push_back(k);
            n.push_back(nn[k]);
            d.push_back(hd.data() + svo[k]);
            e.push_back(he.data() + svo[k]);
        }
        std::vector<char> good(mine.size(), 0);
        bidiag_singular_values_many((int)mine.size(), n.data(), d.data(), e.data(), good.data());
        for (size_t i = 0; i < mine.size(); ++i) {
            const int k = mine[i];
            ok_sv[k] = good[i];
            if (!good[i]) continue;
            std::sort(d[i], d[i] + n[i], [](double x, double y) { return x > y; });
            std::copy(d[i], d[i] + n[i], sv_host->data() + svo[k]);
        }
    };
    std::vector<std::thread> th;
    for (int i = 1; i < nth; ++i) th.emplace_back(work, i);
    work(0);
    for (std::thread& t : th) t.join();
    for (int k : todo)
        if (ok_sv[k]) (*handled)[k] = 1;
    return ED_OK;
}

}  // namespace ed

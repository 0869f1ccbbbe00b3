// ed_matvec_tma.cu — one-launch matvec for spin sectors whose down-spin
// tables fit in shared memory (dim_dn up to a few thousand: chains and
// clusters up to ~14 sites, Kagome/Lieb 12).  The row engine lives in
// ed_matvec_tma.cuh; this file adds the kernel around it, the shared-memory
// plan and the launchers.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <functional>
#include <queue>
#include <vector>

#include "ed_matvec_tma.cuh"

namespace ed {
using namespace dev;

constexpr double kRowCostUp = 0.8;  // up-term share of a row's cost at the mean up-row length

// The Lanczos matvec: FX u with the step's partials.
template <bool CPLX, bool FAST, bool SCHED, bool SEG = false>
__global__ void __launch_bounds__(kTmaThreads, 2) k_matvec_tma(const MvArgs a) {
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ uint32_t uoff[kTmaUpStage];
    __shared__ uint32_t uent[kTmaUpStage];
    __shared__ int give_up;
    constexpr bool kGen = !FAST && !SEG;
    __shared__ int64_t s_cls[kGen ? 4 * kMaxCls : 1];
    TmaSmem S = tma_view(a, sm, uoff, uent, &give_up);
    tma_stage_classes<kGen>(a, s_cls, S);
    uint32_t u0 = 0;
    const bool has_row = tma_first_row(a, &u0);
    if (threadIdx.x == 0) {
        tma_init(S);
        tma_issue_tables(a, S);
        if (has_row) tma_issue_row<CPLX>(a, S, a.xq, u0, 0);
    }
    if (SCHED || (CPLX && SEG)) tma_zero_slots(a, S);
    __syncthreads();
    if (!tma::mbar_wait(&S.bar[2], 0)) {
        if (threadIdx.x == 0) atomicExch(a.err, 1);
        give_up = 1;
    }
    __syncthreads();

    const int b = a.bq_bits + bitlen_u64(*a.p_mx) - 62;
    const int s_u = b > 0 ? b : 0;
    i128 dot = 0;
    uint64_t mx = 0;
    uint32_t rc = 0;
    if (!give_up) {
        tma_rows<CPLX, 1, FAST, false, SCHED, false, SEG>(a, S, a.xq, a.uq, nullptr, rc, 0, s_u, dot, mx);
    } else if (threadIdx.x == 0) {
        // the table copy (the wait that gave up, once more) and the first row
        // copy must land before the CTA exits (bounded waits)
        tma::mbar_wait(&S.bar[2], 0);
        if (has_row) tma::mbar_wait(&S.bar[0], 0);
    }
    mv_lanczos_epilogue(a, dot, mx, s_u);
}

// The FP64 apply in one cooperative launch: largest exponent of x, grid
// barrier, FX copy of x, grid barrier, rows from the unit queue (as in the
// persistent Lanczos kernel).  As five stream operations (two memsets, the
// exponent pass, the conversion, the matvec) a Kagome12 apply spent 17 of its
// 42 us outside the matvec, and an 8-site one 16 us on launches alone; here the
// down tables land during the first pass, the last rows are split over the
// CTAs, and nothing is cleared by the host.  The conversion reads x again from
// L2.  The barriers are the runtime's (cooperative launch: every CTA is
// resident), so a CTA whose table copy gave up still takes part in both.
// Kagome12 42.0 -> 30.7 us, Kagome12 with flux 95 -> 84 us (69 with the class
// schedule and split rows), 8-site ring 17.0 -> 10.2 us (calls in a row, host and device).
template <bool CPLX, bool FAST, bool SCHED, bool SEG = false>
__global__ void __launch_bounds__(kTmaThreads, 2) k_apply(const MvArgs a, const ApplyArgs f) {
    extern __shared__ __align__(128) unsigned char sm[];
    __shared__ uint32_t uoff[kTmaUpStage];
    __shared__ uint32_t uent[kTmaUpStage];
    __shared__ int give_up, s_emax, s_red[32];
    __shared__ uint32_t s_next;
    constexpr bool kGen = !FAST && !SEG;
    __shared__ int64_t s_cls[kGen ? 4 * kMaxCls : 1];
    TmaSmem S = tma_view(a, sm, uoff, uent, &give_up);
    tma_stage_classes<kGen>(a, s_cls, S);
    const int tid = threadIdx.x;
    const int64_t gt = (int64_t)blockIdx.x * kTmaThreads + tid, GT = (int64_t)gridDim.x * kTmaThreads;
    uint32_t u0 = 0;
    const bool has_row = tma_first_row_dyn<true>(a, &u0);
    if (tid == 0) {
        tma_init(S);
        tma_issue_tables(a, S);
    }
    if (SCHED || (CPLX && SEG)) tma_zero_slots(a, S);
    {
        int e = 0;
#pragma unroll 4
        for (int64_t i = gt; i < f.n; i += GT) e = max(e, f64_biased_exp(__ldg(f.x + i)));
        e = block_max_int(e, s_red);
        if (tid == 0) {
            f.part[blockIdx.x] = e;
            if (blockIdx.x == 0) *f.taken = 0;
        }
    }
    cooperative_groups::this_grid().sync();
    {
        int e = 0;
        for (int b = tid; b < (int)gridDim.x; b += kTmaThreads) e = max(e, __ldcg(f.part + b));
        e = block_max_int(e, s_red);
        if (tid == 0) {
            s_emax = e;
            if (blockIdx.x == 0) {
                *f.emax = e;
                *f.flag = e == 2047 ? 1 : 0;
            }
        }
        __syncthreads();
    }
    const int E = fx_exp_from_emax(s_emax);
#pragma unroll 4
    for (int64_t i = gt; i < f.n; i += GT) f.xq[i] = f64_to_fx(__ldg(f.x + i), E);
    if (!tma::mbar_wait(&S.bar[2], 0)) {
        if (tid == 0) {
            atomicExch(a.err, 1);
            tma::mbar_wait(&S.bar[2], 0);  // the table copy must land before the CTA exits (bounded)
        }
        give_up = 1;
    }
    cooperative_groups::this_grid().sync();
    if (give_up) return;
    tma::fence_proxy_async_global();  // xq was written by other CTAs; its rows are read by bulk copies
    if (tid == 0 && has_row) {
        tma::fence_proxy_async_smem();
        tma_issue_row<CPLX>(a, S, f.xq, u0, 0);
    }
    uint32_t rc = 0;
    i128 dot = 0;
    uint64_t mx = 0;
    tma_rows<CPLX, 0, FAST, true, SCHED, true, SEG, false, true>(a, S, f.xq, nullptr, a.y, rc, E - a.Fc, 0, dot, mx,
                                                                  f.taken, &s_next);
}

static const void* apply_kernel(const ed_op* op) {
    if (op->cplx)
        return op->mv_fast ? (const void*)k_apply<true, true, false>
               : seg_kernels(op->mv) ? (const void*)k_apply<true, false, false, true>
                               : (const void*)k_apply<true, false, false>;
    if (!op->mv_fast)
        return seg_kernels(op->mv) ? (const void*)k_apply<false, false, false, true> : (const void*)k_apply<false, false, false>;
    return op->mv.dnSched ? (const void*)k_apply<false, true, true> : (const void*)k_apply<false, true, false>;
}

int apply_grid(const ed_op* op) {
    const void* fn = apply_kernel(op);
    // the kernel's shared-memory limit at the device's largest (never lowered
    // by a smaller operator), so that a call sets no attribute
    int per_sm = 0, sms = 0, coop = 0, optin = 0;
    cudaFuncAttributes fa;
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, op->device) != cudaSuccess ||
        cudaFuncGetAttributes(&fa, fn) != cudaSuccess ||
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kTmaThreads, op->tma_smem) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, op->device) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, op->device) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    // a CTA for every unit of work, as many as are resident together
    const int64_t units = op->mv.nunits;
    const int64_t g = std::min<int64_t>({(int64_t)per_sm * sms, op->tma_grid, std::max<int64_t>(units, 1), kApplyPart});
    return coop ? (int)g : 0;
}

cudaError_t launch_apply_rows(const ed_op* op, const MvArgs& a, const ApplyArgs& f, cudaStream_t s) {
    MvArgs av = a;
    ApplyArgs fv = f;
    void* args[] = {&av, &fv};
    return cudaLaunchCooperativeKernel(apply_kernel(op), dim3((unsigned)op->apply_grid), dim3(kTmaThreads), args,
                                       (size_t)op->tma_smem, s);
}

// Shared-memory plan: returns the dynamic bytes (0 when the sector does not
// fit or rows are not 16-byte multiples).
int tma_plan(const ed_op* op, MvArgs* a) {
    const int W = op->cplx ? 2 : 1;
    const int64_t dimDN = op->dimDN;
    // an odd real row is copied with one element before or after it
    // (a complex row has its zero slot there)
    const int64_t row_bytes = ((dimDN * W + 2) & ~(int64_t)1) * 8;
    // the gather schedule serves the single-class real kernel only
    if (op->cplx || !op->mv_fast) {
        a->dnSched = nullptr;
        a->dnSteps = nullptr;
    }
    auto up128 = [](int64_t v) { return (v + 127) / 128 * 128; };
    // with the schedule a row buffer holds [x | -x | 16 zeros]
    const int64_t buf_bytes = a->dnSched ? ((int64_t)2 * a->schedNeg + 18) * 8 : row_bytes;
    int64_t off = 128;  // mbarriers
    a->sm_row0 = (int)off;
    off += up128(buf_bytes);
    a->sm_row1 = (int)off;
    off += up128(buf_bytes);
    if (a->dnSched) {
        a->sm_sched = (int)off;
        off += up128((int64_t)a->schedSteps * a->dimDNp * 2);
        a->sm_steps = (int)off;
        off += up128(a->dimDNp / 32);
    } else if (a->clsSched) {
        a->sm_sched = (int)off;
        off += up128((int64_t)a->schedSteps * a->dimDNp * 2);
        a->sm_steps = (int)off;
        off += up128(a->dimDNp / 32 * 4);
        a->sm_dnnpos = (int)off;
        off += up128((int64_t)a->dimDNp * 4);
    } else {
        a->sm_dnptr = (int)off;
        off += up128((dimDN + 1) * 4);
        a->sm_dnent = (int)off;
        off += up128(op->tdn.nnz * 4);
        a->sm_dnnpos = (int)off;
        off += up128(dimDN);
    }
    a->sm_ddnq = (int)off;
    off += up128(dimDN * 8);
    a->sm_stdn = (int)off;
    off += up128(dimDN * 8);
    // uoff, uent, reduction scratch; the general kernels' coefficient classes
    const int64_t static_bytes = 2 * kTmaUpStage * 4 + 64 + 24 * 64 + (op->mv_fast || seg_kernels(*a) ? 0 : 4 * kMaxCls * 8);
    if (off + static_bytes > 227 * 1024) return 0;
    return (int)off;
}

static const void* matvec_kernel(const ed_op* op) {
    if (op->cplx)
        return op->mv_fast ? (const void*)k_matvec_tma<true, true, false>
               : seg_kernels(op->mv) ? (const void*)k_matvec_tma<true, false, false, true>
                               : (const void*)k_matvec_tma<true, false, false>;
    if (!op->mv_fast)
        return seg_kernels(op->mv) ? (const void*)k_matvec_tma<false, false, false, true>
                             : (const void*)k_matvec_tma<false, false, false>;
    return op->mv.dnSched ? (const void*)k_matvec_tma<false, true, true> : (const void*)k_matvec_tma<false, true, false>;
}

cudaError_t launch_matvec_tma(const ed_op* op, const MvArgs& a, cudaStream_t s) {
    const void* fn = matvec_kernel(op);
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, op->tma_smem);
    if (e != cudaSuccess) return e;
    MvArgs av = a;
    void* args[] = {&av};
    return cudaLaunchKernel(fn, dim3((unsigned)op->tma_grid), dim3(kTmaThreads), args, (size_t)op->tma_smem, s);
}

int tma_grid(const ed_op* op) {
    int per_sm = 0;
    const void* f = matvec_kernel(op);
    cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, op->tma_smem);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, kTmaThreads, op->tma_smem) != cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    if (per_sm > 2) per_sm = 2;
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, op->device);
    // every CTA is resident at once (the persistent Lanczos kernel relies on
    // it); rows are spread over them by row_plan, some CTAs may have none
    return sms * per_sm;
}

void row_plan(const SpinTable& up, int G, std::vector<uint32_t>* start, std::vector<uint32_t>* list,
              std::vector<uint32_t>* queue, double w) {
    const int64_t n = up.count;
    if (w < 0.0) {
        w = kRowCostUp;
        if (const char* e = std::getenv("ED_ROW_COST_UP")) w = std::atof(e);
    }
    double mean = 0.0;
    for (int64_t u = 0; u < n; ++u) mean += up.len[u];
    mean = n ? mean / (double)n : 0.0;
    std::vector<double> cost(n);
    for (int64_t u = 0; u < n; ++u) cost[u] = 1.0 + (mean > 0.0 ? w * up.len[u] / mean : 0.0);
    std::vector<uint32_t> order(n);
    for (int64_t u = 0; u < n; ++u) order[u] = (uint32_t)u;
    std::stable_sort(order.begin(), order.end(), [&](uint32_t x, uint32_t y) { return cost[x] > cost[y]; });
    *queue = order;
    // least-loaded CTA first; ties to the lowest index
    using Slot = std::pair<double, int>;
    std::priority_queue<Slot, std::vector<Slot>, std::greater<Slot>> heap;
    for (int b = 0; b < G; ++b) heap.push({0.0, b});
    std::vector<std::vector<uint32_t>> rows(G);
    for (uint32_t u : order) {
        Slot sl = heap.top();
        heap.pop();
        rows[sl.second].push_back(u);
        sl.first += cost[u];
        heap.push(sl);
    }
    start->assign(G + 1, 0);
    list->clear();
    list->reserve(n);
    for (int b = 0; b < G; ++b) {
        std::sort(rows[b].begin(), rows[b].end());
        (*start)[b] = (uint32_t)list->size();
        list->insert(list->end(), rows[b].begin(), rows[b].end());
    }
    (*start)[G] = (uint32_t)list->size();
}

}  // namespace ed

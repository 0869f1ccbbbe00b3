// ed_capi.cu — the extern "C" boundary (include/ed_hubbard.h).
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <list>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "../../include/ed_hubbard.h"
#include "ed_device.cuh"
#include "ed_tridiag.hpp"
#include "ed_internal.hpp"

namespace ed {

void lanczos_free_ws(void* p);
cudaError_t launch_random(double* f, int64_t n, uint64_t seed, cudaStream_t s);

// ------------------------------------------------------- device rank/unrank --
__global__ void k_unrank(const int64_t* __restrict__ ranks, int64_t count, uint64_t* __restrict__ words, int n_sites,
                         int n_part, const int64_t* __restrict__ bt) {
    const int kdim = n_part + 2;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) {
        int64_t r = ranks[i];
        uint64_t w = 0;
        int p = n_sites - 1;
        for (int k = n_part; k >= 1; --k) {
            while (p >= 0 && bt[p * kdim + k] > r) --p;
            if (p < 0) break;
            w |= 1ULL << p;
            r -= bt[p * kdim + k];
            --p;
        }
        words[i] = w;
    }
}

__global__ void k_rank(const uint64_t* __restrict__ words, int64_t count, int64_t* __restrict__ ranks, int n_sites,
                       int n_part, const int64_t* __restrict__ bt) {
    const int kdim = n_part + 2;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) {
        uint64_t w = words[i];
        if (__popcll(w) != n_part || (n_sites < 64 && (w >> n_sites))) {
            ranks[i] = -1;
            continue;
        }
        int64_t r = 0;
        int k = 0;
        while (w) {
            const int p = __ffsll((long long)w) - 1;
            r += bt[p * kdim + k + 1];
            ++k;
            w &= w - 1;
        }
        ranks[i] = r;
    }
}

}  // namespace ed

namespace {

int ceil_log2(double x) {
    if (!(x > 0.0)) return 0;
    int k;
    const double f = std::frexp(x, &k);  // x = f 2^k, f in [0.5, 1)
    return f == 0.5 ? k - 1 : k;
}

struct OpExtra {
    void* lz_ws = nullptr;
};

// Device copy of a host table; the allocation is rounded up to 16 bytes and
// the tail zeroed, so a table can be moved with 16-byte bulk copies.
template <typename T>
cudaError_t upload(T** dst, const T* src, size_t n) {
    const size_t bytes = (sizeof(T) * std::max<size_t>(n, 1) + 15) / 16 * 16;
    cudaError_t e = cudaMalloc(dst, bytes);
    if (e != cudaSuccess) return e;
    e = cudaMemset(*dst, 0, bytes);
    if (e == cudaSuccess && n) e = cudaMemcpy(*dst, src, sizeof(T) * n, cudaMemcpyHostToDevice);
    return e;
}

}  // namespace

// Plans and uploads the two-pass matvec when the down index's bandwidth
// leaves a useful window in shared memory; leaves op->striped false otherwise.
// ---- spin-table cache ----------------------------------------------------
// A sweep over disorder realisations builds operators whose hopping terms
// are identical and whose on-site (Make_N) terms differ.  The off-diagonal
// part of a spin table and its gather schedule depend only on (N, Q, real or
// complex, the ordered list of two-site terms); they are kept for the last
// few keys, and on a hit only the folded diagonal is recomputed, adding the
// Make_N values in term order exactly as build_spin does.
namespace {

struct SpinKey {
    int n = 0, q = 0;
    bool cplx = false;
    std::vector<uint64_t> words;  // kind, (i, j), bits of value and phase of every two-site term, in order
    bool operator==(const SpinKey& o) const { return n == o.n && q == o.q && cplx == o.cplx && words == o.words; }
};

struct SpinEntry {
    SpinKey key;
    ed::SpinTable table;
    int sched_state = 0;  // 0 not built, 1 built, -1 the table takes no schedule
    ed::GatherSchedule sched;
    int pair_state = 0;   // the same of the row-pair schedule
    ed::PairSchedule pair;
};

std::mutex g_spin_mu;
std::list<SpinEntry> g_spin_cache;  // most recent first
constexpr size_t kSpinCacheMax = 8;

SpinKey spin_key(int n, int q, bool cplx, const ed_term* t, int nt) {
    SpinKey k;
    k.n = n;
    k.q = q;
    k.cplx = cplx;
    for (int i = 0; i < nt; ++i) {
        if (t[i].kind == ED_TERM_DENSITY) continue;
        uint64_t v, ph;
        std::memcpy(&v, &t[i].value, 8);
        std::memcpy(&ph, &t[i].phase, 8);
        k.words.push_back((uint64_t)(uint32_t)t[i].kind);
        k.words.push_back(((uint64_t)(uint32_t)t[i].i << 32) | (uint32_t)t[i].j);
        k.words.push_back(v);
        k.words.push_back(ph);
    }
    return k;
}

// diag_re/diag_im/max_diag_abs of a table whose off-diagonal part is set
ed_status fold_diagonal(const ed::SpinBasis& b, const ed_term* t, int nt, ed::SpinTable* tab) {
    const int64_t count = b.count;
    tab->diag_re.assign(count, 0.0);
    tab->diag_im.assign(count, 0.0);
    tab->max_diag_abs = 0.0;
    for (int i = 0; i < nt; ++i)
        if (t[i].kind == ED_TERM_DENSITY && (t[i].i < 0 || t[i].i >= b.n_sites)) return ED_ERR_ARG;
    for (int64_t a = 0; a < count; ++a) {
        const uint64_t w = b.state[a];
        for (int i = 0; i < nt; ++i)
            if (t[i].kind == ED_TERM_DENSITY && ((w >> t[i].i) & 1ULL)) {
                tab->diag_re[a] += t[i].value;
                tab->diag_im[a] += 0.0;
            }
        tab->max_diag_abs = std::max(tab->max_diag_abs, std::abs(std::complex<double>(tab->diag_re[a], tab->diag_im[a])));
    }
    return ED_OK;
}

ed_status build_spin_cached(const ed::SpinBasis& b, const ed_term* t, int nt, bool cplx, ed::SpinTable* out,
                            std::string* err) {
    if (nt < 0 || (nt > 0 && !t)) return ED_ERR_ARG;
    const SpinKey k = spin_key(b.n_sites, b.n_part, cplx, t, nt);
    {
        std::lock_guard<std::mutex> g(g_spin_mu);
        for (auto it = g_spin_cache.begin(); it != g_spin_cache.end(); ++it)
            if (it->key == k) {
                *out = it->table;
                g_spin_cache.splice(g_spin_cache.begin(), g_spin_cache, it);
                return fold_diagonal(b, t, nt, out);
            }
    }
    const ed_status st = ed::build_spin(b, t, nt, cplx, out, nullptr, err);
    if (st != ED_OK) return st;
    std::lock_guard<std::mutex> g(g_spin_mu);
    g_spin_cache.push_front(SpinEntry{k, *out, 0, {}});
    if (g_spin_cache.size() > kSpinCacheMax) g_spin_cache.pop_back();
    return ED_OK;
}

// A schedule of a table built through the cache, kept in its entry.
template <typename S, typename F>
bool schedule_cached(const SpinKey& k, int SpinEntry::*state, S SpinEntry::*kept, S* out, const F& build) {
    {
        std::lock_guard<std::mutex> g(g_spin_mu);
        for (SpinEntry& e : g_spin_cache)
            if (e.key == k && e.*state != 0) {
                if (e.*state < 0) return false;
                *out = e.*kept;
                return true;
            }
    }
    const bool ok = build();
    std::lock_guard<std::mutex> g(g_spin_mu);
    for (SpinEntry& e : g_spin_cache)
        if (e.key == k) {
            e.*state = ok ? 1 : -1;
            if (ok) e.*kept = *out;
            break;
        }
    return ok;
}

// The row engine's gather schedule.
bool gather_schedule_cached(const SpinKey& k, const ed::SpinTable& td, ed::GatherSchedule* gs, std::string* err) {
    return schedule_cached(k, &SpinEntry::sched_state, &SpinEntry::sched, gs,
                           [&] { return ed::build_gather_schedule(td, gs, err); });
}

// The row pairs' (adjacent: an even count, part of the key).
bool pair_schedule_cached(const SpinKey& k, const ed::SpinTable& td, ed::PairSchedule* g) {
    std::string err;
    return schedule_cached(k, &SpinEntry::pair_state, &SpinEntry::pair, g,
                           [&] { return ed::build_pair_schedule(td, td.count % 2 == 0, g, &err); });
}

}  // namespace

// The Lanczos workspace pointer rides on the op (opaque to the header), and the
// cache's key of the down table.
struct ed_op_ext : ed_op {
    OpExtra extra;
    SpinKey dn_key;
};

constexpr int kDegreeBlock = 256;  // columns reordered by hop count within each block

static ed_status plan_striped(ed_op* op, bool forced, int64_t chunk_cap = 16384) {
    std::vector<uint32_t> perm, inv;
    int64_t bw = 0;
    ed::rcm_order(op->tdn, &perm, &inv, &bw);
    // lanes of a warp with similar hop counts: pass D's steps follow the
    // largest count among a warp's columns
    ed::sort_blocks_by_degree(op->tdn, kDegreeBlock, &perm, &inv, &bw);
    // window of chunk + 2 bw columns (+ alignment) in at most ~220 KB
    const int64_t max_win = 220 * 1024 / 8;
    int64_t chunk = (max_win - 2 * bw - 64) / 1024 * 1024;
    if (chunk > chunk_cap) chunk = chunk_cap / 1024 * 1024;
    const int64_t dn_pad = (op->dimDN + 1023) / 1024 * 1024;
    if (chunk > dn_pad) chunk = dn_pad;
    if (chunk < 1024) return ED_OK;  // too wide: the generic kernel stays
    if (!forced && op->dimDN * 8 <= 160 * 1024) return ED_OK;
    // Pass D's schedule: one step per hop of a column, at most two targets
    // per bank pair in a step, as 16-bit offsets into each chunk's window
    // (ed::window_schedule16)
    ed::GatherSchedule32 g;
    std::string err;
    if (!ed::build_gather_schedule32(op->tdn, perm, inv, &g, &err, -1, 2)) return ED_OK;
    std::vector<uint16_t> s16;
    int64_t zbase = 0;
    if (!ed::window_schedule16(g, op->dimDN, chunk, bw, &s16, &zbase)) return ED_OK;
    const std::vector<uint8_t> negc = ed::schedule_negcount(g);
    const int64_t sched_steps = std::max(g.steps, 1);
    const std::vector<uint16_t> s16bm = ed::lane_packed16(s16, g.count_pad, sched_steps, zbase);
    const int Fc = op->mv.Fc;
    std::vector<int64_t> dq((size_t)op->dimDN);
    std::vector<uint64_t> st((size_t)op->dimDN);
    for (int64_t c = 0; c < op->dimDN; ++c) {
        dq[c] = (int64_t)std::llrint(std::ldexp(op->tdn.diag_re[perm[c]], Fc));
        st[c] = op->bdn.state[perm[c]];
    }
    // a re-plan (the autotuner's chunk axis) replaces the previous tables
    cudaFree(op->d_permDN); cudaFree(op->d_sched16); cudaFree(op->d_steps32); cudaFree(op->d_dDNqP);
    cudaFree(op->d_stDNp); cudaFree(op->d_negDN);
    op->d_permDN = nullptr; op->d_sched16 = nullptr; op->d_steps32 = nullptr; op->d_dDNqP = nullptr;
    op->d_stDNp = nullptr; op->d_negDN = nullptr;
    if (upload(&op->d_permDN, perm.data(), perm.size()) != cudaSuccess ||
        upload(&op->d_sched16, s16bm.data(), s16bm.size()) != cudaSuccess ||
        upload(&op->d_steps32, g.steps32.data(), g.steps32.size()) != cudaSuccess ||
        upload(&op->d_negDN, negc.data(), negc.size()) != cudaSuccess ||
        upload(&op->d_dDNqP, dq.data(), dq.size()) != cudaSuccess ||
        upload(&op->d_stDNp, st.data(), st.size()) != cudaSuccess)
        return ED_ERR_ALLOC;
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, op->device);
    op->striped = true;
    op->st_grid = sms;
    op->st_bw = bw;
    op->st_chunk = (int)chunk;
    op->st_win = (int)(zbase + 16);
    op->st_zbase = (int)zbase;
    op->st_cpad = g.count_pad;
    op->st_s8 = (int)((sched_steps + 7) / 8);
    return ED_OK;
}

// Real single-class sectors: the row-pair kernel where the row engine's tables
// leave it no shared memory (from about 3,000 down states), and for vectors that
// are large enough to pay for its launches where they do.  A Lanczos step (100
// steps, open chains), row engine -> pairs, with two row CTAs an SM: 14-site 7+4
// (3.4 M elements) 87 -> 85 us, 15-site 5+4 (4.1 M) 104 -> 94, 16-site 6+3 (4.5 M)
// 152 -> 117, 15-site 7+4 (8.8 M) 214 -> 172, but 13-site 6+5 (2.2 M) 59 -> 62;
// with one, whose 16 warps leave the loads' latency open: 13-site 4+6 (1.2 M)
// 44 -> 46, 15 sites in a 3 x 5 torus 4+4 (1.9 M) 86 -> 71, 14-site 4+5 (2.0 M)
// 64 -> 63, 13-site 5+6 (2.2 M) 76 -> 61, 13-site 6+6 (2.9 M) 102 -> 75, 16-site
// 8+4 (23 M) 894 -> 403.
static bool prefer_pair(const ed_op* op) {
    if (op->tma_smem == 0) return true;
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, op->device);
    return op->D >= (op->tma_grid >= 2 * sms ? 4000000 : 1500000);
}

static ed_status set_pair(ed_op* op, const ed::PairSchedule& g) {
    cudaFree(op->d_pairTab);  // of an upload that failed
    op->d_pairTab = nullptr;
    // one upload: words (512 bytes a group of a half block), steps, negative counts
    const size_t at_steps = g.words.size() * sizeof(uint16_t), at_neg = at_steps + g.steps.size();
    std::vector<uint8_t> all(at_neg + g.negcnt.size());
    std::memcpy(all.data(), g.words.data(), at_steps);
    std::copy(g.steps.begin(), g.steps.end(), all.begin() + at_steps);
    std::copy(g.negcnt.begin(), g.negcnt.end(), all.begin() + at_neg);
    if (upload(&op->d_pairTab, all.data(), all.size()) != cudaSuccess) return ED_ERR_ALLOC;
    op->pair_args = {reinterpret_cast<const uint16_t*>(op->d_pairTab), op->d_pairTab + at_steps, op->d_pairTab + at_neg,
                     g.groups, (int)g.blocks, (int)g.zbase, g.sign};
    op->pair_smem = ed::pair_smem_bytes(g.zbase);
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, op->device);
    // one CTA of 1,024 threads an SM
    op->pair_nbuf = ed::pair_buffers((int)g.zbase, g.blocks);
    op->pair_threads = 1024;
    op->pair_grid = sms;
    return ED_OK;
}

// Plans and uploads the row-pair matvec where two rows fit shared memory;
// leaves op->pair false otherwise.
static ed_status plan_pair(ed_op_ext* op) {
    if (ed::pair_smem_bytes((op->dimDN + 7) / 8 * 8) == 0) return ED_OK;
    ed::PairSchedule g;
    if (!pair_schedule_cached(op->dn_key, op->tdn, &g)) return ED_OK;
    const ed_status st = set_pair(op, g);
    op->pair = st == ED_OK;
    return st;
}

namespace ed {
// The row-pair schedule of an operator that its matvec does not use (the batched
// Lanczos kernel's); false when it has none.
bool ensure_pair(ed_op* op) {
    if (op->pair_smem > 0) return true;
    if (pair_smem_bytes((op->dimDN + 7) / 8 * 8) == 0) return false;
    PairSchedule g;
    return pair_schedule_cached(static_cast<ed_op_ext*>(op)->dn_key, op->tdn, &g) && set_pair(op, g) == ED_OK;
}

void** lanczos_ws_slot(ed_op* op) { return &static_cast<ed_op_ext*>(op)->extra.lz_ws; }
}  // namespace ed

extern "C" {

const char* ed_status_string(ed_status s) {
    switch (s) {
        case ED_OK: return "ok";
        case ED_ERR_ARG: return "invalid argument";
        case ED_ERR_CUDA: return "CUDA error";
        case ED_ERR_ALLOC: return "allocation failed";
        case ED_ERR_TABLE: return "table row overflows its slots";
        case ED_ERR_RANGE: return "size beyond the supported range";
        case ED_ERR_NONFINITE: return "non-finite value in an input vector";
        case ED_ERR_BREAKDOWN: return "Lanczos breakdown (invariant subspace)";
        case ED_ERR_NOT_CONVERGED: return "not converged";
        case ED_ERR_TIMEOUT: return "bounded device wait gave up";
        case ED_ERR_NOT_BUILT: return "feature not available";
        default: return "unknown status";
    }
}

int ed_version(void) { return 100; }

int64_t ed_binom(int n, int k) { return ed::binom(n, k); }

ed_status ed_basis_unrank(int n_sites, int n_part, const int64_t* ranks, int64_t count, uint64_t* words) {
    if (n_sites < 1 || n_sites > 62 || n_part < 0 || n_part > n_sites || (count && (!ranks || !words)))
        return ED_ERR_ARG;
    ed::SpinBasis b;
    b.n_sites = n_sites;
    b.n_part = n_part;
    b.count = ed::binom(n_sites, n_part);
    const int kdim = n_part + 2;
    b.binom_tab.assign((size_t)(n_sites + 1) * kdim, 0);
    for (int p = 0; p <= n_sites; ++p)
        for (int k = 0; k < kdim; ++k) b.binom_tab[(size_t)p * kdim + k] = ed::binom(p, k);
    for (int64_t i = 0; i < count; ++i) {
        if (ranks[i] < 0 || ranks[i] >= b.count) return ED_ERR_ARG;
        words[i] = b.unrank(ranks[i]);
    }
    return ED_OK;
}

ed_status ed_basis_rank(int n_sites, int n_part, const uint64_t* words, int64_t count, int64_t* ranks) {
    if (n_sites < 1 || n_sites > 62 || n_part < 0 || n_part > n_sites || (count && (!ranks || !words)))
        return ED_ERR_ARG;
    ed::SpinBasis b;
    b.n_sites = n_sites;
    b.n_part = n_part;
    const int kdim = n_part + 2;
    b.binom_tab.assign((size_t)(n_sites + 1) * kdim, 0);
    for (int p = 0; p <= n_sites; ++p)
        for (int k = 0; k < kdim; ++k) b.binom_tab[(size_t)p * kdim + k] = ed::binom(p, k);
    ed_status st = ED_OK;
    for (int64_t i = 0; i < count; ++i) {
        ranks[i] = b.rank(words[i]);
        if (ranks[i] < 0) st = ED_ERR_ARG;
    }
    return st;
}

static ed_status device_rank_common(int n_sites, int n_part, const void* in, int64_t count, void* out, void* stream,
                                    bool rank) {
    if (n_sites < 1 || n_sites > 62 || n_part < 0 || n_part > n_sites || (count && (!in || !out))) return ED_ERR_ARG;
    if (count == 0) return ED_OK;
    const int kdim = n_part + 2;
    std::vector<int64_t> bt((size_t)(n_sites + 1) * kdim);
    for (int p = 0; p <= n_sites; ++p)
        for (int k = 0; k < kdim; ++k) bt[(size_t)p * kdim + k] = ed::binom(p, k);
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    int64_t* d_bt = nullptr;
    if (cudaMallocAsync(&d_bt, sizeof(int64_t) * bt.size(), s) != cudaSuccess) return ED_ERR_ALLOC;
    cudaMemcpyAsync(d_bt, bt.data(), sizeof(int64_t) * bt.size(), cudaMemcpyHostToDevice, s);
    int64_t blocks = (count + 255) / 256;
    if (blocks > 152 * 16) blocks = 152 * 16;
    if (rank)
        ed::k_rank<<<(int)blocks, 256, 0, s>>>(reinterpret_cast<const uint64_t*>(in), count,
                                               reinterpret_cast<int64_t*>(out), n_sites, n_part, d_bt);
    else
        ed::k_unrank<<<(int)blocks, 256, 0, s>>>(reinterpret_cast<const int64_t*>(in), count,
                                                 reinterpret_cast<uint64_t*>(out), n_sites, n_part, d_bt);
    cudaError_t e = cudaGetLastError();
    cudaFreeAsync(d_bt, s);
    return e == cudaSuccess ? ED_OK : ED_ERR_CUDA;
}

ed_status ed_basis_unrank_device(int n_sites, int n_part, const int64_t* ranks, int64_t count, uint64_t* words,
                                 void* stream) {
    return device_rank_common(n_sites, n_part, ranks, count, words, stream, false);
}

ed_status ed_basis_rank_device(int n_sites, int n_part, const uint64_t* words, int64_t count, int64_t* ranks,
                               void* stream) {
    return device_rank_common(n_sites, n_part, words, count, ranks, stream, true);
}

ed_status ed_tables_ell(int n_sites, int n_part, const ed_term* terms, int n_terms, double* ax, int64_t* aj,
                        uint64_t* state) {
    if (n_sites < 1 || n_sites > 62 || n_part < 0 || n_part > n_sites || (n_terms && !terms)) return ED_ERR_ARG;
    for (int t = 0; t < n_terms; ++t)
        if (terms[t].kind == ED_TERM_PEIERLS) return ED_ERR_ARG;
    ed::SpinBasis b;
    b.build(n_sites, n_part);
    ed::SpinEll ell;
    std::string err;
    ed_status st = ed::build_spin(b, terms, n_terms, false, nullptr, &ell, &err);
    if (st != ED_OK && st != ED_ERR_TABLE) return st;
    if (ax) std::memcpy(ax, ell.ax.data(), sizeof(double) * ell.ax.size());
    if (aj) std::memcpy(aj, ell.aj.data(), sizeof(int64_t) * ell.aj.size());
    if (state) std::memcpy(state, b.state.data(), sizeof(uint64_t) * b.state.size());
    return ell.overflow ? ED_ERR_TABLE : ED_OK;
}

ed_status ed_op_create(ed_op** out, const ed_model_desc* desc, int device) {
    if (!out || !desc) return ED_ERR_ARG;
    *out = nullptr;
    const int N = desc->n_sites;
    if (N < 1 || N > 62 || desc->n_up < 0 || desc->n_up > N || desc->n_dn < 0 || desc->n_dn > N) return ED_ERR_ARG;
    if ((desc->n_up_terms && !desc->up_terms) || (desc->n_dn_terms && !desc->dn_terms)) return ED_ERR_ARG;
    if (!std::isfinite(desc->U)) return ED_ERR_ARG;
    const bool cplx = (desc->flags & ED_OP_COMPLEX) != 0;
    ed_op_ext* op = new (std::nothrow) ed_op_ext();
    if (!op) return ED_ERR_ALLOC;
    op->device = device;
    op->n_sites = N;
    op->n_up = desc->n_up;
    op->n_dn = desc->n_dn;
    op->cplx = cplx;
    op->U = desc->U;
    const uint64_t all = (N >= 64) ? ~0ULL : ((1ULL << N) - 1ULL);
    op->mask = desc->interaction_mask ? (desc->interaction_mask & all) : all;
    op->bup.build(N, desc->n_up);
    op->bdn.build(N, desc->n_dn);
    op->dimUP = op->bup.count;
    op->dimDN = op->bdn.count;
    if (op->dimUP > (1LL << 24) || op->dimDN > (1LL << 24)) { delete op; return ED_ERR_RANGE; }
    op->D = op->dimUP * op->dimDN;
    if (op->D >= (1LL << 32)) { delete op; return ED_ERR_RANGE; }  // 32-bit element offsets
    std::string err;
    ed_status st = build_spin_cached(op->bup, desc->up_terms, desc->n_up_terms, cplx, &op->tup, &err);
    if (st == ED_OK) st = build_spin_cached(op->bdn, desc->dn_terms, desc->n_dn_terms, cplx, &op->tdn, &err);
    if (st != ED_OK) { delete op; return st; }
    op->dn_key = spin_key(N, desc->n_dn, cplx, desc->dn_terms, desc->n_dn_terms);

    // ---- fixed-point scale of the coefficients ----------------------------
    const ed::SpinTable& tu = op->tup;
    const ed::SpinTable& td = op->tdn;
    double cmax = 0.0;
    for (auto& c : tu.coef) cmax = std::max({cmax, std::fabs(c.real()), std::fabs(c.imag())});
    for (auto& c : td.coef) cmax = std::max({cmax, std::fabs(c.real()), std::fabs(c.imag())});
    double dmax_u = 0.0, dmax_d = 0.0;
    for (double v : tu.diag_re) dmax_u = std::max(dmax_u, std::fabs(v));
    for (double v : td.diag_re) dmax_d = std::max(dmax_d, std::fabs(v));
    const int nU = std::min({desc->n_up, desc->n_dn, __builtin_popcountll(op->mask)});
    const double diag_bound = dmax_u + dmax_d + std::fabs(desc->U) * nU;
    const double Bc = std::max({cmax, diag_bound, 1e-300});
    const int nterms = ((int)tu.coef.size() + (int)td.coef.size()) * (cplx ? 2 : 1) + 1;
    const int extra = std::max(0, ceil_log2((double)nterms) - 4);
    const int Fc = 61 - ceil_log2(Bc) - extra;
    ed::MvArgs& a = op->mv;
    std::memset(&a, 0, sizeof(a));
    a.dimUP = op->dimUP;
    a.dimDN = op->dimDN;
    a.Fc = Fc;
    a.mask = op->mask;
    a.Uq = (int64_t)std::llrint(std::ldexp(desc->U, Fc));
    a.nclsUP = (int)tu.coef.size();
    a.nclsDN = (int)td.coef.size();
    op->mv_fast = a.nclsUP <= 1 && a.nclsDN <= 1;
    for (int c = 0; c < a.nclsUP; ++c) {
        a.coefUP[2 * c] = (int64_t)std::llrint(std::ldexp(tu.coef[c].real(), Fc));
        a.coefUP[2 * c + 1] = (int64_t)std::llrint(std::ldexp(tu.coef[c].imag(), Fc));
    }
    for (int c = 0; c < a.nclsDN; ++c) {
        a.coefDN[2 * c] = (int64_t)std::llrint(std::ldexp(td.coef[c].real(), Fc));
        a.coefDN[2 * c + 1] = (int64_t)std::llrint(std::ldexp(td.coef[c].imag(), Fc));
    }
    a.unitUP = (a.nclsUP == 1 && tu.coef[0] == std::complex<double>(1.0, 0.0)) ? 1 : 0;
    a.unitDN = (a.nclsDN == 1 && td.coef[0] == std::complex<double>(1.0, 0.0)) ? 1 : 0;
    a.mergeUD = (a.nclsUP == 1 && a.nclsDN == 1 && tu.coef[0] == td.coef[0]) ? 1 : 0;
    if (a.nclsUP == 0 && a.nclsDN == 0) a.mergeUD = 0;
    // |acc| <= (row sums + diagonal) * 2^Fc * max|x_q|
    const double rowb = (tu.max_row_abs + td.max_row_abs) * (cplx ? 2.0 : 1.0) + diag_bound;
    a.bq_bits = ceil_log2(std::ldexp(std::max(rowb, 1e-300), Fc) + 1.0) + 1;

    // ---- device upload -------------------------------------------------------
    if (cudaSetDevice(device) != cudaSuccess) { delete op; return ED_ERR_CUDA; }
    std::vector<int64_t> dq_u(op->dimUP), dq_d(op->dimDN);
    for (int64_t i = 0; i < op->dimUP; ++i) dq_u[i] = (int64_t)std::llrint(std::ldexp(tu.diag_re[i], Fc));
    for (int64_t i = 0; i < op->dimDN; ++i) dq_d[i] = (int64_t)std::llrint(std::ldexp(td.diag_re[i], Fc));
    bool ok = upload(&op->d_upEnt, tu.ent.data(), tu.ent.size()) == cudaSuccess &&
              upload(&op->d_dnEnt, td.ent.data(), td.ent.size()) == cudaSuccess &&
              upload(&op->d_upLen, tu.len.data(), tu.len.size()) == cudaSuccess &&
              upload(&op->d_dnLen, td.len.data(), td.len.size()) == cudaSuccess &&
              upload(&op->d_upNpos, tu.npos.data(), tu.npos.size()) == cudaSuccess &&
              upload(&op->d_dnNpos, td.npos.data(), td.npos.size()) == cudaSuccess &&
              upload(&op->d_dUPq, dq_u.data(), dq_u.size()) == cudaSuccess &&
              upload(&op->d_dDNq, dq_d.data(), dq_d.size()) == cudaSuccess &&
              upload(&op->d_stUP, op->bup.state.data(), op->bup.state.size()) == cudaSuccess &&
              upload(&op->d_stDN, op->bdn.state.data(), op->bdn.state.size()) == cudaSuccess &&
              cudaMalloc(&op->d_emax, sizeof(int) * (4 + ed::kApplyPart + 1)) == cudaSuccess &&
              cudaMemset(op->d_emax, 0, 4 * sizeof(int)) == cudaSuccess;
    // one allocation for the small words
    op->d_flag = op->d_emax + 1;
    op->d_err = op->d_emax + 2;
    op->d_apply = op->d_emax + 4;
    // CSR copies (row-contiguous entries) for the shared-memory kernel
    auto csr = [](const ed::SpinTable& t, std::vector<uint32_t>* ptr, std::vector<uint32_t>* ent) {
        ptr->assign(t.count + 1, 0);
        ent->clear();
        ent->reserve((size_t)t.nnz);
        for (int64_t r = 0; r < t.count; ++r) {
            for (int k = 0; k < t.len[r]; ++k) ent->push_back(t.ent[(size_t)k * t.count + r]);
            (*ptr)[r + 1] = (uint32_t)ent->size();
        }
    };
    std::vector<uint32_t> up_ptr, up_ent, dn_ptr, dn_ent;
    csr(tu, &up_ptr, &up_ent);
    csr(td, &dn_ptr, &dn_ent);
    ok = ok && upload(&op->d_upPtr, up_ptr.data(), up_ptr.size()) == cudaSuccess &&
         upload(&op->d_upEntC, up_ent.data(), up_ent.size()) == cudaSuccess &&
         upload(&op->d_dnPtr, dn_ptr.data(), dn_ptr.size()) == cudaSuccess &&
         upload(&op->d_dnEntC, dn_ent.data(), dn_ent.size()) == cudaSuccess;
    if (!ok) { ed_op_destroy(op); return ED_ERR_ALLOC; }
    // at most kSegCls classes: class segments of the rows (real) or a class
    // schedule of the columns (complex; without one, and where the row engine
    // cannot hold two rows, the general path)
    a.mergeMC = a.perEntry = 0;
    a.upSegE = a.upSegP = a.dnSegE = a.dnSegP = nullptr;
    const bool few = a.nclsUP <= ed::kSegCls && a.nclsDN <= ed::kSegCls && !std::getenv("ED_NO_SEG");
    if (!op->mv_fast && few && !cplx) {
        auto segments = [](const ed::SpinTable& t, std::vector<uint32_t>* se, std::vector<uint32_t>* sp) {
            se->assign(t.count, 0u);
            sp->assign(t.count, 0u);
            for (int64_t r = 0; r < t.count; ++r) {
                int k = 0;
                uint32_t e = 0, p = 0;
                for (int c = 0; c < ed::kSegCls; ++c) {
                    while (k < t.len[r] && ((t.ent[(size_t)k * t.count + r] >> ed::kClassShift) & ed::kClassMask) == (uint32_t)c &&
                           !(t.ent[(size_t)k * t.count + r] & ed::kSignBit))
                        ++k;
                    p |= (uint32_t)k << (8 * c);
                    while (k < t.len[r] && ((t.ent[(size_t)k * t.count + r] >> ed::kClassShift) & ed::kClassMask) == (uint32_t)c)
                        ++k;
                    e |= (uint32_t)k << (8 * c);
                }
                (*se)[r] = e;
                (*sp)[r] = p;
            }
        };
        std::vector<uint32_t> use, usp, dse, dsp;
        segments(tu, &use, &usp);
        segments(td, &dse, &dsp);
        if (upload(&op->d_upSegE, use.data(), use.size()) != cudaSuccess ||
            upload(&op->d_upSegP, usp.data(), usp.size()) != cudaSuccess ||
            upload(&op->d_dnSegE, dse.data(), dse.size()) != cudaSuccess ||
            upload(&op->d_dnSegP, dsp.data(), dsp.size()) != cudaSuccess) {
            ed_op_destroy(op);
            return ED_ERR_ALLOC;
        }
        a.upSegE = op->d_upSegE;
        a.upSegP = op->d_upSegP;
        a.dnSegE = op->d_dnSegE;
        a.dnSegP = op->d_dnSegP;
    }
    // (48 bytes a column: two rows, diagonal and state)
    if (!op->mv_fast && few && cplx && 48 * op->dimDN < 227 * 1024) {
        ed::ClassSchedule cs;
        std::string cerr;
        if (ed::build_class_schedule(td, &cs, &cerr)) {
            // one upload: words (64 bytes a step of a block), counts, steps
            std::vector<uint32_t> all(cs.words.size() / 2 + cs.negcnt.size() + cs.steps4.size());
            std::memcpy(all.data(), cs.words.data(), cs.words.size() * 2);
            std::copy(cs.negcnt.begin(), cs.negcnt.end(), all.begin() + cs.words.size() / 2);
            std::copy(cs.steps4.begin(), cs.steps4.end(), all.begin() + cs.words.size() / 2 + cs.negcnt.size());
            if (upload(&op->d_clsSched, all.data(), all.size()) != cudaSuccess) {
                ed_op_destroy(op);
                return ED_ERR_ALLOC;
            }
                a.clsSched = reinterpret_cast<const uint16_t*>(op->d_clsSched);
            a.clsNeg = op->d_clsSched + cs.words.size() / 2;
            a.clsSteps = a.clsNeg + cs.negcnt.size();
            a.schedSteps = cs.steps;
            a.dimDNp = (int)cs.cpad;
        }
        auto partners = [](const int64_t* coef, int n, int8_t* part) {
            for (int c = 0; c < ed::kSegCls; ++c) part[c] = (int8_t)c;
            for (int c = 0; c < n; ++c) {
                if (part[c] != c || coef[2 * c + 1] == 0) continue;
                for (int q = c + 1; q < n; ++q)
                    if (part[q] == q && coef[2 * q] == coef[2 * c] && coef[2 * q + 1] == -coef[2 * c + 1]) {
                        part[c] = (int8_t)q;
                        part[q] = -1;
                        break;
                    }
            }
        };
        partners(a.coefUP, a.nclsUP, a.partUP);
        partners(a.coefDN, a.nclsDN, a.partDN);
    }
    if (ed::seg_kernels(a)) a.mergeMC = (a.nclsUP == a.nclsDN && tu.coef == td.coef) ? 1 : 0;
    // the general path: entries per (row, class) run of the two tables; below 2, a
    // product per entry replaces the running class sums
    if (!op->mv_fast && !ed::seg_kernels(a)) {
        int64_t runs = 0;
        for (const ed::SpinTable* t : {&tu, &td})
            for (int64_t r = 0; r < t->count; ++r) {
                uint32_t last = ~0u;
                for (int k = 0; k < t->len[r]; ++k) {
                    const uint32_t c = (t->ent[(size_t)k * t->count + r] >> ed::kClassShift) & ed::kClassMask;
                    runs += c != last;
                    last = c;
                }
            }
        a.perEntry = tu.nnz + td.nnz < 2 * runs ? 1 : 0;
    }
    a.upPtr = op->d_upPtr;
    a.upEntC = op->d_upEntC;
    a.dnPtr = op->d_dnPtr;
    a.dnEntC = op->d_dnEntC;
    a.dnNnz = (uint32_t)dn_ent.size();
    // conflict-free gather schedule for the shared-memory kernels (real,
    // single class); ED_NO_SCHED=1 keeps the CSR gathers
    a.dnSched = nullptr;
    a.dnSteps = nullptr;
    if (!cplx && td.coef.size() <= 1 && !std::getenv("ED_NO_SCHED")) {
        ed::GatherSchedule gs;
        std::string serr;
        if (gather_schedule_cached(op->dn_key, td, &gs, &serr)) {
            if (upload(&op->d_dnSched, gs.ent.data(), gs.ent.size()) != cudaSuccess ||
                upload(&op->d_dnSteps, gs.steps32.data(), gs.steps32.size()) != cudaSuccess) {
                ed_op_destroy(op);
                return ED_ERR_ALLOC;
            }
            a.dnSched = op->d_dnSched;
            a.dnSteps = op->d_dnSteps;
            a.schedSteps = gs.steps;
            a.dimDNp = (int)gs.count_pad;
            a.schedNeg = (int)gs.neg_base;
        }
    }
    a.err = op->d_err;
    a.upEnt = op->d_upEnt;
    a.dnEnt = op->d_dnEnt;
    a.upLen = op->d_upLen;
    a.dnLen = op->d_dnLen;
    a.upNpos = op->d_upNpos;
    a.dnNpos = op->d_dnNpos;
    a.dUPq = op->d_dUPq;
    a.dDNq = op->d_dDNq;
    a.stUP = op->d_stUP;
    a.stDN = op->d_stDN;
    const int W = cplx ? 2 : 1;
    const int64_t row_bytes = op->dimDN * W * 8;
    op->stage_smem = row_bytes <= 160 * 1024 ? (int)row_bytes : 0;
    op->grid = ed::matvec_grid(op);
    op->mv_threads = ed::matvec_threads(op->dimDN);
    // kernel choice: the row-staged TMA kernel where the down table fits in
    // shared memory, else the generic kernel; ED_MATVEC=generic forces the
    // generic kernel (tests compare the two)
    const char* pick = std::getenv("ED_MATVEC");
    const std::string want = pick ? pick : "";
    if (want != "generic" && want != "striped" && want != "pair") op->tma_smem = ed::tma_plan(op, &a);
    if (op->tma_smem > 0) op->tma_grid = ed::tma_grid(op);
    if (!cplx && op->mv_fast && (want.empty() || want == "pair") && prefer_pair(op)) {
        const ed_status pst = plan_pair(op);
        if (pst != ED_OK) {
            ed_op_destroy(op);
            return pst;
        }
    }
    // sectors whose down rows exceed shared memory: the two-pass matvec over
    // a bandwidth-reducing order of the down index (ED_MATVEC=striped forces
    // it where it applies)
    if (op->tma_smem == 0 && !op->pair && want != "generic" && !cplx && op->mv_fast && op->dimDN % 2 == 0) {
        const ed_status sst = plan_striped(op, want == "striped");
        if (sst != ED_OK) {
            ed_op_destroy(op);
            return sst;
        }
    }
    if (op->tma_smem > 0) {
        std::vector<uint32_t> rs, rl, rq;
        ed::row_plan(op->tup, op->tma_grid, &rs, &rl, &rq);
        const std::vector<uint32_t> uq = ed::unit_queue(rq, op->dimDN, op->tma_grid);
        // room for the unit queue at any row plan (at most 4 units a row)
        if (upload(&op->d_rowStart, rs.data(), rs.size()) != cudaSuccess ||
            upload(&op->d_rowList, rl.data(), rl.size()) != cudaSuccess ||
            upload(&op->d_rowQueue, rq.data(), rq.size()) != cudaSuccess ||
            cudaMalloc(&op->d_unitQueue, sizeof(uint32_t) * (rq.size() + 3 * (size_t)op->tma_grid + 4)) != cudaSuccess ||
            cudaMemcpy(op->d_unitQueue, uq.data(), sizeof(uint32_t) * uq.size(), cudaMemcpyHostToDevice) != cudaSuccess) {
            ed_op_destroy(op);
            return ED_ERR_ALLOC;
        }
        op->mv.rowStart = op->d_rowStart;
        op->mv.rowList = op->d_rowList;
        op->mv.rowQueue = op->d_rowQueue;
        op->mv.unitQueue = op->d_unitQueue;
        op->mv.nunits = (uint32_t)uq.size();
        op->apply_grid = op->pair ? 0 : ed::apply_grid(op);
    }
    *out = op;
    return ED_OK;
}

ed_status ed_op_destroy(ed_op* op) {
    if (!op) return ED_OK;
    cudaSetDevice(op->device);
    ed_op_ext* ox = static_cast<ed_op_ext*>(op);
    ed::lanczos_free_ws(ox->extra.lz_ws);
    cudaFree(op->d_upEnt); cudaFree(op->d_dnEnt); cudaFree(op->d_upLen); cudaFree(op->d_dnLen);
    cudaFree(op->d_upNpos); cudaFree(op->d_dnNpos);
    cudaFree(op->d_upPtr); cudaFree(op->d_upEntC); cudaFree(op->d_dnPtr); cudaFree(op->d_dnEntC);
    cudaFree(op->d_dnSched); cudaFree(op->d_dnSteps); cudaFree(op->d_rowStart); cudaFree(op->d_rowList); cudaFree(op->d_rowQueue);
    cudaFree(op->d_unitQueue);
    cudaFree(op->d_upSegE); cudaFree(op->d_upSegP); cudaFree(op->d_dnSegE); cudaFree(op->d_dnSegP);
    cudaFree(op->d_permDN); cudaFree(op->d_sched16); cudaFree(op->d_steps32); cudaFree(op->d_dDNqP);
    cudaFree(op->d_stDNp); cudaFree(op->d_sdn); cudaFree(op->d_negDN);
    cudaFree(op->d_clsSched);
    cudaFree(op->d_pairTab);
    cudaFree(op->d_dUPq); cudaFree(op->d_dDNq); cudaFree(op->d_stUP); cudaFree(op->d_stDN);
    cudaFree(op->d_xq); cudaFree(op->d_emax); cudaFree(op->d_io);
    if (op->h_stage) cudaFreeHost(op->h_stage);
    delete ox;
    return ED_OK;
}

int64_t ed_op_rows(const ed_op* op) { return op ? op->D : 0; }
int64_t ed_op_cols(const ed_op* op) { return op ? op->D : 0; }
int64_t ed_op_dim_up(const ed_op* op) { return op ? op->dimUP : 0; }
int64_t ed_op_dim_dn(const ed_op* op) { return op ? op->dimDN : 0; }
int ed_op_is_complex(const ed_op* op) { return op && op->cplx ? 1 : 0; }

int ed_op_matvec_kind(const ed_op* op) {
    if (!op) return -1;
    return op->striped ? ED_MV_TWO_PASS : (op->tma_smem > 0 ? ED_MV_ROWS : ED_MV_GENERIC);
}

int ed_op_row_pairs(const ed_op* op) { return op && op->pair ? 1 : 0; }

ed_status ed_op_perform(ed_op* op, const double* x, double* y, int mem, void* stream) {
    if (!op || !x || !y || (mem != ED_MEM_HOST && mem != ED_MEM_DEVICE)) return ED_ERR_ARG;
    if (cudaSetDevice(op->device) != cudaSuccess) return ED_ERR_CUDA;
    cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
    const int W = op->cplx ? 2 : 1;
    const int64_t DW = op->D * W;
    // two elements of padding: the row engine copies whole 16-byte words around a row
    if (!op->d_xq && cudaMalloc(&op->d_xq, sizeof(int64_t) * ((size_t)DW + 2)) != cudaSuccess) return ED_ERR_ALLOC;
    const double* dx = x;
    double* dy = y;
    if (mem == ED_MEM_HOST) {
        const size_t need = sizeof(double) * (size_t)DW * 2;
        if (op->d_io_bytes < need) {
            cudaFree(op->d_io);
            op->d_io = nullptr;
            op->d_io_bytes = 0;
            if (cudaMalloc(&op->d_io, need) != cudaSuccess) return ED_ERR_ALLOC;
            op->d_io_bytes = need;
        }
        if (cudaMemcpyAsync(op->d_io, x, sizeof(double) * DW, cudaMemcpyHostToDevice, s) != cudaSuccess)
            return ED_ERR_CUDA;
        dx = op->d_io;
        dy = op->d_io + DW;
    }
    const cudaError_t e = ed::launch_apply(op, dx, dy, op->d_xq, op->d_emax, op->d_flag, op->d_apply, s);
    if (e != cudaSuccess) { op->last_error = cudaGetErrorString(e); return ED_ERR_CUDA; }
    if (mem == ED_MEM_HOST) {
        int flag = 0, err = 0;
        if (cudaMemcpyAsync(y, dy, sizeof(double) * DW, cudaMemcpyDeviceToHost, s) != cudaSuccess) return ED_ERR_CUDA;
        if (cudaMemcpyAsync(&flag, op->d_flag, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess) return ED_ERR_CUDA;
        if (cudaMemcpyAsync(&err, op->d_err, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess) return ED_ERR_CUDA;
        if (cudaStreamSynchronize(s) != cudaSuccess) return ED_ERR_CUDA;
        // the bounded-wait flag is sticky: a device-pointer call that gave up
        // is reported by the next call that synchronises
        if (err) {
            cudaMemset(op->d_err, 0, sizeof(int));
            return ED_ERR_TIMEOUT;
        }
        if (flag) return ED_ERR_NONFINITE;
    }
    return ED_OK;
}

ed_status ed_lanczos_run(ed_op* op, const ed_lanczos_cfg* cfg, const double* start, int start_mem, double* evec,
                         int evec_mem, double* alpha, double* beta, ed_lanczos_result* res, void* stream) {
    if (!op || !cfg) return ED_ERR_ARG;
    if (cudaSetDevice(op->device) != cudaSuccess) return ED_ERR_CUDA;
    ed_op_ext* ox = static_cast<ed_op_ext*>(op);
    return ed::lanczos_run(op, &ox->extra.lz_ws, cfg, start, start_mem, evec, evec_mem, alpha, beta, res,
                           reinterpret_cast<cudaStream_t>(stream));
}

ed_status ed_lanczos_batch(ed_op* const* ops, int n_ops, const ed_lanczos_cfg* cfg, const double* starts, int start_mem,
                           double* evecs, int evec_mem, double* alpha, double* beta, ed_lanczos_result* res,
                           void* stream) {
    if (!ops || n_ops < 1 || !ops[0] || !cfg) return ED_ERR_ARG;
    if (cudaSetDevice(ops[0]->device) != cudaSuccess) return ED_ERR_CUDA;
    return ed::lanczos_batch_run(ops, n_ops, cfg, starts, start_mem, evecs, evec_mem, alpha, beta, res,
                                 reinterpret_cast<cudaStream_t>(stream));
}

// Rebuild and upload the persistent kernel's row plan with row-cost weight w.
static ed_status set_row_plan(ed_op* op, double w) {
    std::vector<uint32_t> rs, rl, rq;
    ed::row_plan(op->tup, op->tma_grid, &rs, &rl, &rq, w);
    const std::vector<uint32_t> uq = ed::unit_queue(rq, op->dimDN, op->lz_grid > 0 ? op->lz_grid : op->tma_grid);
    if (cudaMemcpy(op->d_rowStart, rs.data(), sizeof(uint32_t) * rs.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(op->d_rowList, rl.data(), sizeof(uint32_t) * rl.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(op->d_rowQueue, rq.data(), sizeof(uint32_t) * rq.size(), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(op->d_unitQueue, uq.data(), sizeof(uint32_t) * uq.size(), cudaMemcpyHostToDevice) != cudaSuccess)
        return ED_ERR_CUDA;
    op->mv.nunits = (uint32_t)uq.size();
    op->row_cost = w;
    return ED_OK;
}

ed_status ed_op_autotune(ed_op* op, const ed_tune_cfg* cfg, ed_tune_result* res, void* stream) {
    if (!op || !cfg || cfg->steps < 2 || cfg->steps > 10000) return ED_ERR_ARG;
    if (cudaSetDevice(op->device) != cudaSuccess) return ED_ERR_CUDA;
    ed_tune_result r{};
    ed_lanczos_cfg lc{};
    lc.max_steps = cfg->steps;
    lc.mode = ED_LANCZOS_FIXED;
    lc.ritz = ED_RITZ_NONE;
    lc.start = ED_START_RANDOM;
    const int saved_mode = op->lz_mode;
    const double saved_w = op->row_cost;
    // one candidate: a warm-up run, then the best of two timed runs
    auto time_run = [&](double* us) -> ed_status {
        ed_status st = ed_lanczos_run(op, &lc, nullptr, ED_MEM_DEVICE, nullptr, ED_MEM_DEVICE, nullptr, nullptr,
                                      nullptr, stream);
        double best = 1e300;
        for (int rep = 0; st == ED_OK && rep < 2; ++rep) {
            const auto t0 = std::chrono::steady_clock::now();
            st = ed_lanczos_run(op, &lc, nullptr, ED_MEM_DEVICE, nullptr, ED_MEM_DEVICE, nullptr, nullptr, nullptr,
                                stream);
            const double dt = std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t0).count();
            best = std::min(best, dt);
        }
        *us = best / cfg->steps;
        return st;
    };
    ed_status st = ED_OK;
    op->lz_mode = 1;
    st = time_run(&r.per_step_us);
    ++r.candidates;
    r.persistent = 0;
    r.us_per_step = r.per_step_us;
    r.row_cost = saved_w;
    const double weights[3] = {0.4, 0.8, 1.2};
    if (st == ED_OK && op->tma_smem > 0) {
        op->lz_mode = 2;
        for (int k = 0; k < 3 && st == ED_OK; ++k) {
            st = set_row_plan(op, weights[k]);
            if (st == ED_OK) st = time_run(&r.persistent_us[k]);
            ++r.candidates;
            if (st == ED_OK && r.persistent_us[k] < r.us_per_step) {
                r.us_per_step = r.persistent_us[k];
                r.persistent = 1;
                r.row_cost = weights[k];
            }
        }
    }
    // rows per CTA: the persistent kernel at one CTA per SM (each CTA takes
    // twice the rows of the two-per-SM grid), at the best weight
    const int saved_grid = op->lz_grid;
    r.ctas_per_sm = r.persistent ? 2 : 0;
    if (st == ED_OK && op->tma_smem > 0 && op->tma_grid > 1) {
        int sms = 152;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, op->device);
        if (op->tma_grid >= 2 * sms) {
            op->lz_mode = 2;
            op->lz_grid = sms;
            const double w_best = r.persistent ? r.row_cost : weights[1];
            st = set_row_plan(op, w_best);
            if (st == ED_OK) st = time_run(&r.one_cta_us);
            ++r.candidates;
            if (st == ED_OK && r.one_cta_us < r.us_per_step) {
                r.us_per_step = r.one_cta_us;
                r.persistent = 1;
                r.row_cost = w_best;
                r.ctas_per_sm = 1;
            }
        }
    }
    op->lz_grid = saved_grid;
    // two-pass sectors: pass D's window, the largest chunk and half of it
    // (the plan is rebuilt for each; the per-step kernels run these sectors)
    const int saved_chunk = op->striped ? op->st_chunk : 0;
    if (st == ED_OK && op->striped && saved_chunk >= 2048) {
        const int chunks[2] = {saved_chunk, saved_chunk / 2};
        double best = 1e300;
        int pick = saved_chunk;
        for (int k = 0; k < 2 && st == ED_OK; ++k) {
            if (k > 0) st = plan_striped(op, true, chunks[k]);
            if (st == ED_OK && (!op->striped || op->st_chunk != chunks[k])) break;  // no such plan
            if (st == ED_OK) st = time_run(&r.chunk_us[k]);
            ++r.candidates;
            if (st == ED_OK && r.chunk_us[k] < best) {
                best = r.chunk_us[k];
                pick = chunks[k];
            }
        }
        r.chunk = pick;
        if (st == ED_OK && best < r.us_per_step) r.us_per_step = best;
        const int keep = (st == ED_OK && cfg->apply) ? pick : saved_chunk;
        if (op->st_chunk != keep) {
            const ed_status s2 = plan_striped(op, true, keep);
            if (st == ED_OK) st = s2;
        }
    }
    if (st == ED_OK && cfg->apply) {
        op->lz_mode = r.persistent ? 2 : 1;
        op->lz_grid = r.ctas_per_sm == 1 ? op->tma_grid / 2 : 0;
        if (op->tma_smem > 0) st = set_row_plan(op, r.persistent ? r.row_cost : saved_w);
    } else {
        op->lz_mode = saved_mode;
        if (op->tma_smem > 0) {
            const ed_status s2 = set_row_plan(op, saved_w);
            if (st == ED_OK) st = s2;
        }
    }
    if (res) *res = r;
    return st;
}

ed_status ed_op_set_tuning(ed_op* op, const ed_tune_result* tuned) {
    if (!op || !tuned) return ED_ERR_ARG;
    if (cudaSetDevice(op->device) != cudaSuccess) return ED_ERR_CUDA;
    op->lz_mode = tuned->persistent ? 2 : 1;
    op->lz_grid = (tuned->persistent && tuned->ctas_per_sm == 1) ? op->tma_grid / 2 : 0;
    if (op->striped && tuned->chunk > 0 && tuned->chunk != op->st_chunk) {
        const ed_status st = plan_striped(op, true, tuned->chunk);
        if (st != ED_OK) return st;
    }
    if (op->tma_smem > 0 && tuned->persistent) return set_row_plan(op, tuned->row_cost);
    return ED_OK;
}

ed_status ed_random_vector(int64_t n, uint64_t seed, double* out_host) {
    if (n < 0 || (n && !out_host)) return ED_ERR_ARG;
    for (int64_t b = 0; b * 4 < n; ++b) {
        const ed::dev::Philox4 r = ed::dev::philox4x64_10((uint64_t)b, seed);
        for (int w = 0; w < 4; ++w) {
            const int64_t k = b * 4 + w;
            if (k < n) out_host[k] = ed::dev::uniform_pm1(r.v[w]);
        }
    }
    return ED_OK;
}

ed_status ed_random_vector_device(int64_t n, uint64_t seed, double* out_device, void* stream) {
    if (n < 0 || (n && !out_device)) return ED_ERR_ARG;
    if (n == 0) return ED_OK;
    return ed::launch_random(out_device, n, seed, reinterpret_cast<cudaStream_t>(stream)) == cudaSuccess ? ED_OK
                                                                                                       : ED_ERR_CUDA;
}

ed_status ed_tridiag_lowest(int n, const double* alpha, const double* offdiag, double* e0, double* z) {
    if (n < 1 || !alpha || (n > 1 && !offdiag) || !e0) return ED_ERR_ARG;
    *e0 = ed::tridiag_lowest_host(n, alpha, offdiag, z);
    return ED_OK;
}

ed_status ed_tridiag_eigen(int n, const double* alpha, const double* offdiag, double* evals, double* z) {
    if (n < 1 || !alpha || (n > 1 && !offdiag) || !evals) return ED_ERR_ARG;
    std::vector<double> m;
    std::vector<ed::TriRot> rots;
    if (!ed::tridiag_eigen_rotations(n, alpha, offdiag, &m, &rots)) return ED_ERR_BREAKDOWN;
    std::vector<int> order(n);
    for (int i = 0; i < n; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return m[x] < m[y]; });
    std::vector<double> col(n);
    for (int j = 0; j < n; ++j) {
        evals[j] = m[order[j]];
        if (!z) continue;
        std::fill(col.begin(), col.end(), 0.0);
        col[order[j]] = 1.0;
        ed::tri_apply_z(rots, col.data());
        std::copy(col.begin(), col.end(), z + (size_t)j * n);
    }
    return ED_OK;
}

ed_status ed_bidiag_singular_values(int n, const double* d, const double* e, double* s) {
    if (n < 1 || !d || (n > 1 && !e) || !s) return ED_ERR_ARG;
    std::vector<double> dd(d, d + n), ee(std::max(n - 1, 1), 0.0);
    for (int i = 0; i + 1 < n; ++i) ee[i] = e[i];
    if (!ed::bidiag_singular_values(n, dd.data(), ee.data())) return ED_ERR_NOT_CONVERGED;
    std::sort(dd.begin(), dd.end(), [](double x, double y) { return x > y; });
    std::copy(dd.begin(), dd.end(), s);
    return ED_OK;
}

ed_status ed_tridiag_expm(int n, const double* alpha, const double* offdiag, int n_times, const double* times,
                          double* out) {
    if (n < 1 || !alpha || (n > 1 && !offdiag) || n_times < 0 || (n_times && (!times || !out))) return ED_ERR_ARG;
    return ed::tridiag_expm_e0(n, alpha, offdiag, n_times, times, out) ? ED_OK : ED_ERR_BREAKDOWN;
}

}  // extern "C"

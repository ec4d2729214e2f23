// C ABI of the GB300 powder-FID engine (declared in include/spinach_gpu.h).
//
// Host part: converts the caller's CSC matrices (the I and Q{r}{k,m} that
// kernel/hamiltonian.m returns) into Hermitised value streams on one union
// sparsity pattern, reorders the basis by row length into a 32-row sliced
// ELL layout, uploads it once, and launches the propagation and powder-sum
// kernels of kernels.cuh for every orientation grid.  Also here: the launch
// configuration (one CTA or a cluster per orientation), the autotuner, the
// no-allocation entry point and batched CUDA graphs over many handles.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <tuple>
#include <new>
#include <stdexcept>
#include <string>
#include <vector>

#include "spinach_gpu.h"
#include "block.cuh"
#include "block_plan.h"
#include "builder.h"
#include "dense.cuh"
#include "kernels.cuh"

namespace {

struct SpxError : std::runtime_error {
    spx_status code;
    SpxError(spx_status c, const std::string &m) : std::runtime_error(m), code(c) {}
};

#define SPX_CUDA(call)                                                                    \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess) {                                                          \
            throw SpxError(e_ == cudaErrorMemoryAllocation ? SPX_ERR_OUT_OF_MEMORY         \
                                                           : SPX_ERR_CUDA,                \
                           std::string(#call) + ": " + cudaGetErrorString(e_));          \
        }                                                                                 \
    } while (0)

template <class T>
struct DevBuf {
    T *p = nullptr;
    size_t n = 0;
    DevBuf() = default;
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    ~DevBuf() { release(); }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
    void reserve(size_t count) {
        if (count <= n && p) return;
        release();
        SPX_CUDA(cudaMalloc(&p, std::max<size_t>(count, 1) * sizeof(T)));
        n = count;
    }
    void upload(const std::vector<T> &v, cudaStream_t s) {
        reserve(v.size());
        if (!v.empty()) SPX_CUDA(cudaMemcpyAsync(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s));
    }
};

// Pinned host memory of a handle for what a run copies to and from the device,
// at most kStage bytes, kept until the handle goes.
constexpr size_t kStage = 8 << 20;
struct HostStage {
    unsigned char *p = nullptr;
    size_t n = 0;
    HostStage() = default;
    HostStage(const HostStage &) = delete;
    HostStage &operator=(const HostStage &) = delete;
    ~HostStage() { if (p) cudaFreeHost(p); }
    // at least `bytes`; copies under way on s end before memory is given back
    unsigned char *get(size_t bytes, cudaStream_t s) {
        if (bytes <= n && p) return p;
        if (p) {
            SPX_CUDA(cudaStreamSynchronize(s));
            SPX_CUDA(cudaFreeHost(p));
            p = nullptr;
            n = 0;
        }
        SPX_CUDA(cudaMallocHost(&p, std::max<size_t>(bytes, 64 << 10)));
        n = std::max<size_t>(bytes, 64 << 10);
        return p;
    }
};

struct Cplx {
    double re = 0.0, im = 0.0;
};

// Coupled states of a run (block.cuh): their rows and a few lane layouts per
// precision, in one device allocation.
struct BlockPlan {
    bool ok = false;                 // false: the whole system runs (kernels.cuh)
    int n = 0, nv = 0;
    std::vector<int> rows;           // system rows (sliced order), ascending
    struct Layout {
        spx::BlockLayout dev{};
        spx::BlockCost cost;
        int warps = 0, ecap = 0;
    };
    std::vector<Layout> layouts[2];  // FP32, FP64
    spx::DenseSystem dense{};        // the same rows for the dense kernels (dense.cuh)
    int ncoil = 0;                   // coil entries among them
    const int *coil_row = nullptr, *coil_chan = nullptr;
    const double2 *coil_val = nullptr;
    double bound = 0.0;              // on |L| over all orientations, these rows alone
    DevBuf<unsigned char> mem;
};

// Device buffers of a run of the dense kernels.
struct DenseBufs {
    DevBuf<double2> M, V, Y;         // six matrices, states, detection rows
    DevBuf<int> sym;                 // whether an orientation's matrix is symmetric
};

// Device buffers of the kernels of block.cuh for one run.
struct BlockBufs {
    DevBuf<double> centre, halfwidth, lev_half, table, saved;   // halfwidth: sequences only
    DevBuf<float> tablef;
    DevBuf<unsigned long long> extent;
    DevBuf<int> lev, kcut;           // lev: steps per chunk | table rows | series lengths
};

// What the autotuner chose for a system: `shape` is what spx_autotune returns.
struct TunedShape {
    spx_options shape{};             // whole-system launch shape (threads, cluster, chunk_target)
    bool coupled = false;            // the coupled states run: shape is the whole system's default
    double blk_target = 0.0;         // and this their series argument of a chunk (0: the default)
};

// A pulse superoperator as CSR rows in the sliced order, with its 1-norm.
struct PulseOp {
    DevBuf<int> ptr, col;
    DevBuf<double2> val;
    double norm1 = 0.0;
};

}  // namespace

struct spx_handle {
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
    std::string err;
    int sm_count = 0;
    size_t smem_optin = 0, smem_sm = 0;     // shared memory of a CTA at most, and of an SM

    // uploaded system
    bool have_system = false;
    int n = 0, n_pad = 0, nslices = 0, ell_len = 0, nstreams = 0, nterms = 0;
    bool cplx = false;
    int64_t nnz = 0;
    double g_upper = 0.0;      // upper bound of the spectral radius of H over all orientations
    double max_im_diag = 0.0;
    double max_growth = 0.0;   // largest rate at which a state grows (relaxation of the wrong sign)
    double lo_scale = 1.0;     // power of two scaling every assembled off-diagonal entry into (-1, 1)
    DevBuf<int> d_slice_off, d_stream_coef, d_term_rkm;
    std::vector<int> slice_off_host;
    DevBuf<uint16_t> d_ell_col;
    DevBuf<double> d_ell_re, d_ell_im;
    DevBuf<double2> d_diag, d_rho0, d_coil, d_coil_vals;
    DevBuf<int> d_coil_rows, d_coil_chan;
    int ncoil = -1;                 // non-zero coil entries if at most 32, else -1
    int nchan = 1;                  // detection channels
    DevBuf<double2> d_rho0s;        // per-orientation initial states (sliced order)
    DevBuf<double2> d_seq[2], d_seq_rho;   // pulse sequences: states between segments
    DevBuf<int> d_seq_status;              // and the statuses of every launch of one
    std::vector<std::unique_ptr<PulseOp>> pulses;   // pulse superoperators of the last sequence
    DevBuf<double> d_neg_re, d_neg_im;     // echo detection: the adjoint generator's streams
    DevBuf<double2> d_neg_diag;
    DevBuf<double2> d_traj[2], d_echo_f;   // forward / adjoint trajectories, per-orientation echoes
    DevBuf<int> d_echo_ptr, d_echo_col;    // exp(-1i pi P) as CSR (sliced order)
    DevBuf<double2> d_echo_val;
    int64_t n_states = 0;           // their count (0: one initial state for all)
    std::vector<int> row_of;        // sliced-ELL row of every basis state
    int64_t revision = 0;           // counts uploads: systems, coils, initial states

    // coupled states of the plain acquisition (rebuilt with the coils and the
    // initial states) and what finding them takes
    std::vector<uint16_t> ell_col_host;
    std::vector<unsigned char> ell_parts;       // per ELL entry: 1 a real part, 2 an imaginary part in some stream
    std::vector<int> component;     // connected component of every row under L
    std::vector<double2> rho0_host;             // sliced order
    std::vector<int> coil_row_host, coil_chan_host;
    std::vector<double2> coil_val_host;
    std::vector<char> state_rows;   // rows with a non-zero per-orientation initial state
    BlockPlan plan;
    BlockBufs blk, chk_blk;
    DenseBufs dense, chk_dense;
    std::vector<double> row_bound;  // per row: sum of its entries' magnitudes over the value streams

    // run buffers
    DevBuf<double> d_grid;       // alpha | beta | gamma | weight
    DevBuf<double> d_table;
    DevBuf<unsigned char> d_fids;
    DevBuf<double2> d_part, d_fid;
    DevBuf<int> d_status, d_kused, d_mused;
    DevBuf<long long> d_matvecs;
    DevBuf<double> d_halfwidth;
    DevBuf<int> d_counter;           // orientation work counter of the propagation kernel

    int64_t launches = 0;           // kernels launched by this handle (spx_stats.kernel_launches)

    // FP64 check of FP32 runs: a few orientations re-run in FP64 on a second
    // stream while the FP32 run proceeds (spx_stats.fp32_rel_error)
    cudaStream_t check_stream = nullptr;     // of the highest priority: its launches depend on each other
    int high_priority = 0;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    DevBuf<double> d_chk_grid;       // alpha | beta | gamma of the checked orientations
    DevBuf<double2> d_chk_rho0s;     // their initial states when per-orientation states are set
    DevBuf<unsigned char> d_chk_fids;
    DevBuf<double> d_chk_table, d_chk_halfwidth;
    DevBuf<int> d_chk_status, d_chk_kused, d_chk_mused, d_chk_counter;
    DevBuf<long long> d_chk_matvecs;
    HostStage stage;
    int chk_pending = 0;             // checked orientations of the pending run (0: none)
    std::vector<int> chk_index;      // their grid indices
    const double2 *chk_out = nullptr;    // the pending run's powder FID (device)
    const double *chk_w = nullptr;       // and its grid weights (device)
    int64_t chk_nsteps = 0;

    // last run
    spx_stats stats{};
    bool stats_pending = false;
    bool stats_timed = true;        // kernel events recorded (not inside a captured graph)
    int64_t last_norient = 0;

    // the autotuner's choice per precision
    bool has_tuned[2] = {false, false};
    TunedShape tuned[2];
};

namespace {

// ---------------------------------------------------------------------------
// Upload: CSC -> Hermitised streams -> sliced ELL
// ---------------------------------------------------------------------------
void check_csc(const spx_csc *A, int64_t n, const char *name) {
    if (!A) throw SpxError(SPX_ERR_INVALID_ARGUMENT, std::string(name) + " is NULL");
    if (A->n != n) throw SpxError(SPX_ERR_INVALID_ARGUMENT, std::string(name) + " has the wrong dimension");
    if (!A->colptr) throw SpxError(SPX_ERR_INVALID_ARGUMENT, std::string(name) + ": NULL colptr");
    const int64_t nnz = A->colptr[n];
    if (A->colptr[0] != 0 || nnz < 0) throw SpxError(SPX_ERR_INVALID_ARGUMENT, std::string(name) + ": bad colptr");
    if (nnz > 0 && (!A->rowidx || !A->values))
        throw SpxError(SPX_ERR_INVALID_ARGUMENT, std::string(name) + ": NULL rowidx/values");
    for (int64_t c = 0; c < n; ++c)
        if (A->colptr[c + 1] < A->colptr[c]) throw SpxError(SPX_ERR_INVALID_ARGUMENT, std::string(name) + ": colptr decreases");
    for (int64_t p = 0; p < nnz; ++p) {
        if (A->rowidx[p] < 0 || A->rowidx[p] >= n)
            throw SpxError(SPX_ERR_INVALID_ARGUMENT, std::string(name) + ": row index out of range");
        if (!std::isfinite(A->values[2 * p]) || !std::isfinite(A->values[2 * p + 1]))
            throw SpxError(SPX_ERR_INVALID_ARGUMENT, std::string(name) + ": non-finite value");
    }
}

template <class F>
void for_each_entry(const spx_csc *A, F f) {
    for (int64_t c = 0; c < A->n; ++c)
        for (int64_t p = A->colptr[c]; p < A->colptr[c + 1]; ++p)
            f(A->rowidx[p], c, Cplx{A->values[2 * p], A->values[2 * p + 1]});
}

// f(row, column, ELL entry) for every off-diagonal entry of the pattern (sliced order).
template <class F>
void for_each_coupling(const spx_handle *h, F f) {
    for (int s = 0; s < h->nslices; ++s)
        for (int e = h->slice_off_host[s]; e < h->slice_off_host[s + 1]; ++e) {
            const int row = s * 32 + ((e - h->slice_off_host[s]) & 31), col = h->ell_col_host[e];
            if (row < h->n && col != row) f(row, col, e);         // padding points at its own row
        }
}

// The plan for the given rows (closed under L's couplings, ascending):
// state_pos their places in the run's state arrays (null: the system's rows),
// detect: with detection rows for the handle's coils.
void build_plan(spx_handle *h, const std::vector<int> &rows, const std::vector<int> *state_pos, bool detect,
                BlockPlan &plan) {
    plan.ok = false;
    plan.n = plan.nv = 0;
    plan.layouts[0].clear();
    plan.layouts[1].clear();
    plan.rows = rows;
    if (rows.empty() || rows.size() > (size_t)spx::kBlockRows) return;
    std::vector<int> own(h->n, -1);
    for (size_t i = 0; i < rows.size(); ++i) own[rows[i]] = (int)i;
    spx::BlockPattern P;
    P.rows = rows;
    P.n = (int)rows.size();
    P.entries.resize(P.n);
    std::vector<int> ent, esrc;                   // the whole entries, for the dense kernels
    for_each_coupling(h, [&](int r, int c, int e) {
        if (own[r] < 0) return;
        ent.push_back(own[c] * P.n + own[r]);
        esrc.push_back(e);
        if (h->ell_parts[e] & 1) P.entries[own[r]].push_back({own[c], e});
        if (h->ell_parts[e] & 2) P.entries[own[r]].push_back({P.n + own[c], h->ell_len + e});
    });
    // detection rows conj(coil): a complex coil on real values takes a row for
    // its real and one for its imaginary parts (times -1i)
    for (int ch = 0; ch < (detect ? h->nchan : 0); ++ch)
        for (int im = 0; im < (h->cplx ? 1 : 2); ++im) {
            std::vector<spx::BlockPattern::Entry> row;
            for (size_t i = 0; i < h->coil_row_host.size(); ++i) {
                const int r = own[h->coil_row_host[i]];
                const double2 v = h->coil_val_host[i];
                if (h->coil_chan_host[i] != ch || r < 0) continue;
                auto add = [&](int col, double x) {
                    if (x == 0.0) return;
                    row.push_back({col, -2 - (int)P.values.size()});
                    P.values.push_back(x);
                };
                if (h->cplx) { add(r, v.x); add(P.n + r, -v.y); }
                else add(r, im ? v.y : v.x);
            }
            if (im && row.empty()) continue;
            P.entries.push_back(row);
            P.vchan.push_back(ch);
            P.vfac.push_back(im);
            ++P.nv;
        }
    std::vector<int> crow, cchan;
    std::vector<double2> cval;
    if (detect)
        for (size_t i = 0; i < h->coil_row_host.size(); ++i)
            if (own[h->coil_row_host[i]] >= 0) {
                crow.push_back(own[h->coil_row_host[i]]);
                cchan.push_back(h->coil_chan_host[i]);
                cval.push_back(h->coil_val_host[i]);
            }
    plan.bound = 0.0;
    for (int r : rows) plan.bound = std::max(plan.bound, h->row_bound[r]);
    // layouts: the best warp count for a few grid sizes, each precision
    std::vector<unsigned char> blob;
    auto put = [&](const void *p, size_t bytes) {
        const size_t at = (blob.size() + 15) & ~size_t(15);
        blob.resize(at + std::max<size_t>(bytes, 16));
        if (bytes) std::memcpy(blob.data() + at, p, bytes);
        return at;
    };
    const size_t o_rows = put(P.rows.data(), P.rows.size() * sizeof(int));
    const size_t o_pos = state_pos ? put(state_pos->data(), state_pos->size() * sizeof(int)) : o_rows;
    const size_t o_val = put(P.values.data(), P.values.size() * sizeof(double));
    const size_t o_chan = put(P.vchan.data(), P.vchan.size() * sizeof(int));
    const size_t o_fac = put(P.vfac.data(), P.vfac.size() * sizeof(int));
    const size_t o_ent = put(ent.data(), ent.size() * sizeof(int)), o_esrc = put(esrc.data(), esrc.size() * sizeof(int));
    const size_t o_crow = put(crow.data(), crow.size() * sizeof(int)), o_cchan = put(cchan.data(), cchan.size() * sizeof(int));
    const size_t o_cval = put(cval.data(), cval.size() * sizeof(double2));
    struct At { size_t row, part, shape, src, col; };
    std::vector<At> at[2];
    for (int p = 0; p < 2; ++p) {
        const int ecap_max = p == 1 ? 32 : spx::kBlockMaxEntries;
        int widest = 1;
        for (auto &r : P.entries) widest = std::max(widest, (int)r.size());
        std::vector<spx::BlockLanes> lanes;
        std::vector<spx::BlockCost> costs;
        for (int e = 1; e <= std::min(widest, ecap_max); ++e) {
            const size_t cnt = block_lane_count(P, e);
            const int w = (int)((cnt + 31) / 32);                 // more warps than this only idle
            if (w > spx::kBlockRows / 32) continue;
            spx::BlockLanes L;
            spx::BlockCost c;
            if (block_lanes(P, w, e, p == 1, h->max_im_diag > 0.0, h->cplx, L, c)) {
                lanes.push_back(std::move(L));
                costs.push_back(c);
            }
        }
        if (lanes.empty()) { plan.layouts[0].clear(); return; }
        std::vector<size_t> keep;
        for (double per_sm : {0.5, 1.5, 2.5, 4.5, 7.0, 13.0, 27.0}) {
            size_t best = 0;
            for (size_t i = 1; i < lanes.size(); ++i)
                if (costs[i].time(per_sm) < costs[best].time(per_sm)) best = i;
            if (std::find(keep.begin(), keep.end(), best) == keep.end()) keep.push_back(best);
        }
        for (size_t i : keep) {
            const spx::BlockLanes &L = lanes[i];
            at[p].push_back({put(L.row.data(), L.row.size() * 4), put(L.part.data(), L.part.size() * 4),
                             put(L.shape.data(), L.shape.size() * 4), put(L.src.data(), L.src.size() * 4),
                             put(L.col.data(), L.col.size() * 2)});
            BlockPlan::Layout o;
            o.cost = costs[i];
            o.warps = L.warps;
            o.ecap = L.ecap;
            plan.layouts[p].push_back(o);
        }
    }
    plan.mem.reserve(blob.size());
    SPX_CUDA(cudaMemcpyAsync(plan.mem.p, blob.data(), blob.size(), cudaMemcpyHostToDevice, h->stream));
    SPX_CUDA(cudaStreamSynchronize(h->stream));              // blob is pageable
    const unsigned char *d = plan.mem.p;
    for (int p = 0; p < 2; ++p)
        for (size_t i = 0; i < at[p].size(); ++i) {
            spx::BlockLayout &b = plan.layouts[p][i].dev;
            b.n = P.n;
            b.nv = P.nv;
            b.threads = 32 * plan.layouts[p][i].warps;
            b.ecap = plan.layouts[p][i].ecap;
            b.lane_row = reinterpret_cast<const int *>(d + at[p][i].row);
            b.lane_part = reinterpret_cast<const int *>(d + at[p][i].part);
            b.warp_shape = reinterpret_cast<const int *>(d + at[p][i].shape);
            b.src = reinterpret_cast<const int *>(d + at[p][i].src);
            b.col = reinterpret_cast<const uint16_t *>(d + at[p][i].col);
            b.row_src = reinterpret_cast<const int *>(d + o_rows);
            b.state_pos = reinterpret_cast<const int *>(d + o_pos);
            b.vval = reinterpret_cast<const double *>(d + o_val);
            b.vchan = reinterpret_cast<const int *>(d + o_chan);
            b.vfac = reinterpret_cast<const int *>(d + o_fac);
        }
    plan.n = P.n;
    plan.nv = P.nv;
    plan.dense = {P.n, (int)ent.size(), reinterpret_cast<const int *>(d + o_ent), reinterpret_cast<const int *>(d + o_esrc),
                  reinterpret_cast<const int *>(d + o_rows)};
    plan.ncoil = (int)crow.size();
    plan.coil_row = reinterpret_cast<const int *>(d + o_crow);
    plan.coil_chan = reinterpret_cast<const int *>(d + o_cchan);
    plan.coil_val = reinterpret_cast<const double2 *>(d + o_cval);
    plan.ok = true;
}

// Rows with a non-zero initial state (of any orientation).
std::vector<char> start_rows(const spx_handle *h) {
    if (h->n_states > 0) return h->state_rows;
    std::vector<char> start(h->n);
    for (int i = 0; i < h->n; ++i) start[i] = h->rho0_host[i].x != 0.0 || h->rho0_host[i].y != 0.0;
    return start;
}

// Rows whose component (label[i]) holds both a coil entry and a start row.
std::vector<int> live_rows(const spx_handle *h, const std::vector<int> &label, const std::vector<char> &start) {
    std::vector<char> seen(h->n, 0), live(h->n, 0);
    for (int r : h->coil_row_host) seen[label[r]] = 1;
    for (int i = 0; i < h->n; ++i)
        if (start[i] && seen[label[i]]) live[label[i]] = 1;
    std::vector<int> rows;
    for (int i = 0; i < h->n; ++i)
        if (live[label[i]]) rows.push_back(i);
    return rows;
}

// The plan of the plain acquisition for the handle's coils and initial states.
// It lies where the plan before it lay if it fits there, so a graph that was
// captured with that one (spx_batch) may not run any more: hence the revision.
void rebuild_plan(spx_handle *h) {
    ++h->revision;
    build_plan(h, live_rows(h, h->component, start_rows(h)), nullptr, true, h->plan);
}

void upload_system(spx_handle *h, const spx_csc *I, int32_t n_terms, const int32_t *rank,
                   const int32_t *kk, const int32_t *mm, const spx_csc *Q, const spx_csc *R,
                   const double *rho0, const double *coil) {
    if (!I) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "I is NULL");
    const int64_t n = I->n;
    if (n < 1) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "dimension must be positive");
    if (n > 65535) throw SpxError(SPX_ERR_UNSUPPORTED, "Liouville dimension above 65535");
    if (n_terms < 0 || n_terms > (spx::kMaxCoef - 1) / 2)
        throw SpxError(SPX_ERR_UNSUPPORTED, "too many rotational-basis terms");
    if (n_terms > 0 && (!rank || !kk || !mm || !Q)) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "NULL term arrays");
    if (!rho0 || !coil) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "rho0/coil is NULL");
    check_csc(I, n, "I");
    for (int t = 0; t < n_terms; ++t) {
        if (rank[t] < 1 || rank[t] > 2) throw SpxError(SPX_ERR_UNSUPPORTED, "only spherical ranks 1 and 2 are supported");
        if (kk[t] < 0 || kk[t] > 2 * rank[t] || mm[t] < 0 || mm[t] > 2 * rank[t])
            throw SpxError(SPX_ERR_INVALID_ARGUMENT, "term projection index out of range");
        check_csc(&Q[t], n, "Q");
    }
    if (R) check_csc(R, n, "R");
    for (int64_t i = 0; i < 2 * n; ++i)
        if (!std::isfinite(rho0[i]) || !std::isfinite(coil[i]))
            throw SpxError(SPX_ERR_INVALID_ARGUMENT, "non-finite rho0/coil");

    // off-diagonal entries at or below 1e-14 of the largest input value are
    // rounding residues of cancelled commutators (a host builder that sums
    // operator products in another order leaves them): they are dropped, so
    // that they neither widen the pattern nor cost matvec work
    double vin2 = 0.0;                                  // squared magnitudes
    auto scan = [&](const spx_csc *A) {
        for_each_entry(A, [&](int64_t, int64_t, Cplx v) { vin2 = std::max(vin2, v.re * v.re + v.im * v.im); });
    };
    scan(I);
    for (int t = 0; t < n_terms; ++t) scan(&Q[t]);
    const double residue2 = 1e-28 * vin2;
    auto kept = [&](int64_t r, int64_t c, Cplx v) { return r == c || v.re * v.re + v.im * v.im > residue2; };

    // union pattern (structurally symmetric, full diagonal) as sorted keys
    // r*n + c: a bitmap of the n x n positions when it is small (a few MB),
    // else a sort of every entry and its transpose
    std::vector<int64_t> keys;
    if (n <= 8192) {
        const int64_t wpr = (n + 63) / 64;                 // 64-bit words per row
        std::vector<uint64_t> bits((size_t)(n * wpr), 0);
        auto mark = [&](int64_t r, int64_t c) { bits[(size_t)(r * wpr + (c >> 6))] |= 1ull << (c & 63); };
        for (int64_t i = 0; i < n; ++i) mark(i, i);
        auto add = [&](const spx_csc *A) {
            for_each_entry(A, [&](int64_t r, int64_t c, Cplx v) {
                if (!kept(r, c, v)) return;
                mark(r, c);
                mark(c, r);
            });
        };
        add(I);
        for (int t = 0; t < n_terms; ++t) add(&Q[t]);
        size_t cnt_bits = 0;
        for (uint64_t w : bits) cnt_bits += (size_t)__builtin_popcountll(w);
        keys.reserve(cnt_bits);
        for (int64_t r = 0; r < n; ++r)
            for (int64_t q = 0; q < wpr; ++q) {
                uint64_t w = bits[(size_t)(r * wpr + q)];
                while (w) {
                    const int b = __builtin_ctzll(w);
                    keys.push_back(r * n + q * 64 + b);
                    w &= w - 1;
                }
            }
    } else {
        keys.reserve((size_t)n * 4);
        for (int64_t i = 0; i < n; ++i) keys.push_back(i * n + i);
        auto add = [&](const spx_csc *A) {
            for_each_entry(A, [&](int64_t r, int64_t c, Cplx v) {
                if (!kept(r, c, v)) return;
                keys.push_back(r * n + c);
                keys.push_back(c * n + r);
            });
        };
        add(I);
        for (int t = 0; t < n_terms; ++t) add(&Q[t]);
        std::sort(keys.begin(), keys.end());
        keys.erase(std::unique(keys.begin(), keys.end()), keys.end());
    }
    const size_t nk = keys.size();
    // row and column of every key (one division each, not one per use)
    std::vector<int32_t> krow(nk), kcol(nk);
    for (size_t p = 0; p < nk; ++p) {
        krow[p] = (int32_t)(keys[p] / n);
        kcol[p] = (int32_t)(keys[p] - (int64_t)krow[p] * n);
    }
    // row start of each row in the key list; a position is found within its row
    std::vector<size_t> rstart(n + 1, 0);
    for (size_t p = 0; p < nk; ++p) rstart[krow[p] + 1]++;
    for (int64_t i = 0; i < n; ++i) rstart[i + 1] += rstart[i];
    auto pos = [&](int64_t r, int64_t c) -> size_t {
        return (size_t)(std::lower_bound(keys.begin() + rstart[r], keys.begin() + rstart[r + 1], r * n + c) -
                        keys.begin());
    };
    // position of the transposed key: (c, r) for key p = (r, c).  Keys come
    // row by row in column order, so the keys of one column c are met in
    // increasing row r, the order of row c's keys (the pattern is symmetric).
    std::vector<size_t> tpos(nk);
    {
        std::vector<size_t> cur(rstart.begin(), rstart.end() - 1);
        for (size_t p = 0; p < nk; ++p) tpos[p] = cur[kcol[p]]++;
    }
    // every kept entry (r, c) of A with the positions p of key (r, c) and q of
    // (c, r): the rows of column c are walked along row c's keys (MATLAB's CSC
    // rows ascend; a binary search where they do not)
    auto for_each_key = [&](const spx_csc *A, auto &&f) {
        for (int64_t c = 0; c < n; ++c) {
            size_t cur = rstart[c];
            const size_t end = rstart[c + 1];
            for (int64_t i = A->colptr[c]; i < A->colptr[c + 1]; ++i) {
                const int64_t r = A->rowidx[i];
                const Cplx v{A->values[2 * i], A->values[2 * i + 1]};
                if (!kept(r, c, v)) continue;
                while (cur < end && kcol[cur] < r) ++cur;
                const size_t q = (cur < end && kcol[cur] == r) ? cur : pos(c, r);
                f(tpos[q], q, r, c, v);
            }
        }
    };

    // streams: 0 = Ih + iR (coefficient 1), then S_t, A_t per term
    const int nst_all = 1 + 2 * n_terms;
    std::vector<std::vector<Cplx>> st(nst_all, std::vector<Cplx>(nk));
    for_each_key(I, [&](size_t p, size_t q, int64_t, int64_t, Cplx v) {
        Cplx &a = st[0][p];
        a.re += 0.5 * v.re; a.im += 0.5 * v.im;
        Cplx &b = st[0][q];
        b.re += 0.5 * v.re; b.im -= 0.5 * v.im;
    });
    for (int t = 0; t < n_terms; ++t) {
        auto &S = st[1 + 2 * t];
        auto &A = st[2 + 2 * t];
        for_each_key(&Q[t], [&](size_t p, size_t q, int64_t, int64_t, Cplx v) {
            // S = (Q + Q^H)/2,  A = 1i (Q - Q^H)/2
            S[p].re += 0.5 * v.re; S[p].im += 0.5 * v.im;
            S[q].re += 0.5 * v.re; S[q].im -= 0.5 * v.im;
            A[p].re -= 0.5 * v.im; A[p].im += 0.5 * v.re;
            A[q].re -= 0.5 * v.im; A[q].im -= 0.5 * v.re;
        });
    }
    double max_im_diag = 0.0;
    if (R) {
        for_each_entry(R, [&](int64_t r, int64_t c, Cplx v) {
            if (r != c) {
                if (v.re != 0.0 || v.im != 0.0)
                    throw SpxError(SPX_ERR_UNSUPPORTED, "only diagonal relaxation superoperators are supported");
                return;
            }
            Cplx &a = st[0][pos(r, r)];      // L = H + 1i*R
            a.re -= v.im;
            a.im += v.re;
        });
    }
    // scale of everything, real/complex off-diagonal decision
    double vmax = 0.0;
    for (auto &s : st)
        for (auto &v : s) vmax = std::max(vmax, std::max(std::fabs(v.re), std::fabs(v.im)));
    const double im_tol = 1e-14 * vmax;
    bool cplx = false;
    for (auto &s : st)
        for (size_t p = 0; p < nk && !cplx; ++p) {
            if (krow[p] != kcol[p] && std::fabs(s[p].im) > im_tol) cplx = true;
        }
    // drop streams that are zero up to rounding (1e-14 of the largest value:
    // e.g. the anti-Hermitian part of a term whose commutators cancel only to
    // the last bits in the caller's summation order)
    std::vector<int> keep;
    for (int s = 0; s < nst_all; ++s) {
        bool nz = (s == 0);
        for (size_t p = 0; p < nk && !nz; ++p) nz = std::fabs(st[s][p].re) > im_tol || std::fabs(st[s][p].im) > im_tol;
        if (nz) keep.push_back(s);
    }
    const int nst = (int)keep.size();

    // rows: count off-diagonals, order by count (descending, stable)
    std::vector<int> cnt(n, 0);
    for (size_t p = 0; p < nk; ++p) {
        const int32_t r = krow[p], c = kcol[p];
        if (r != c) ++cnt[r];
    }
    std::vector<int> perm(n);  // new -> old
    for (int i = 0; i < n; ++i) perm[i] = i;
    std::stable_sort(perm.begin(), perm.end(), [&](int a, int b) { return cnt[a] > cnt[b]; });
    std::vector<int> inv(n);
    for (int i = 0; i < n; ++i) inv[perm[i]] = i;
    const int nslices = (int)((n + 31) / 32), n_pad = nslices * 32;
    std::vector<int> slice_off(nslices + 1, 0);
    for (int s = 0; s < nslices; ++s) {
        int w = 0;
        for (int l = 0; l < 32; ++l) {
            const int row = s * 32 + l;
            if (row < n) w = std::max(w, cnt[perm[row]]);
        }
        slice_off[s + 1] = slice_off[s] + 32 * w;
    }
    const int ell_len = slice_off[nslices];

    std::vector<uint16_t> ell_col(std::max(ell_len, 1), 0);
    std::vector<double> ell_re((size_t)nst * std::max(ell_len, 1), 0.0), ell_im;
    if (cplx) ell_im.assign((size_t)nst * std::max(ell_len, 1), 0.0);
    std::vector<double2> diag((size_t)nst * n_pad, make_double2(0.0, 0.0));
    double g_upper = 0.0;
    std::vector<double> row_bound(n_pad, 0.0);
    for (int s = 0; s < nslices; ++s) {
        for (int l = 0; l < 32; ++l) {
            const int row = s * 32 + l;
            int c = 0;
            double rowsum = 0.0;
            if (row < n) {
                const int old = perm[row];
                for (size_t p = rstart[old]; p < rstart[old + 1]; ++p) {
                    const int64_t oc = kcol[p];
                    if (oc == old) {
                        for (int q = 0; q < nst; ++q) {
                            const Cplx v = st[keep[q]][p];
                            diag[(size_t)q * n_pad + row] = make_double2(v.re, v.im);
                            rowsum += (keep[q] == 0) ? std::fabs(v.re) : std::hypot(v.re, v.im);
                        }
                        continue;
                    }
                    const size_t e = (size_t)slice_off[s] + (size_t)c * 32 + l;
                    ell_col[e] = (uint16_t)inv[oc];
                    for (int q = 0; q < nst; ++q) {
                        const Cplx v = st[keep[q]][p];
                        ell_re[(size_t)q * ell_len + e] = v.re;
                        if (cplx) ell_im[(size_t)q * ell_len + e] = v.im;
                        rowsum += std::hypot(v.re, v.im);
                    }
                    ++c;
                }
            }
            // padding entries point at the row itself with zero value
            const int w = (slice_off[s + 1] - slice_off[s]) / 32;
            for (; c < w; ++c) ell_col[(size_t)slice_off[s] + (size_t)c * 32 + l] = (uint16_t)std::min(row, n_pad - 1);
            g_upper = std::max(g_upper, rowsum);
            row_bound[row] = rowsum;
        }
    }
    double max_growth = 0.0;
    for (int i = 0; i < n; ++i) {
        max_im_diag = std::max(max_im_diag, std::fabs(diag[i].y));
        max_growth = std::max(max_growth, diag[i].y);
    }
    std::vector<int> stream_coef(nst);
    for (int q = 0; q < nst; ++q) stream_coef[q] = keep[q];     // slot in the coefficient vector
    std::vector<int> term_rkm(3 * std::max(n_terms, 1), 0);
    for (int t = 0; t < n_terms; ++t) {
        term_rkm[3 * t] = rank[t];
        term_rkm[3 * t + 1] = kk[t];
        term_rkm[3 * t + 2] = mm[t];
    }
    std::vector<double2> r0(n_pad, make_double2(0, 0)), cl(n_pad, make_double2(0, 0));
    for (int i = 0; i < n; ++i) {
        r0[inv[i]] = make_double2(rho0[2 * i], rho0[2 * i + 1]);
        cl[inv[i]] = make_double2(coil[2 * i], coil[2 * i + 1]);
    }

    SPX_CUDA(cudaSetDevice(h->device));
    h->have_system = false;
    ++h->revision;
    h->d_slice_off.upload(slice_off, h->stream);
    h->slice_off_host = slice_off;
    h->d_ell_col.upload(ell_col, h->stream);
    h->d_ell_re.upload(ell_re, h->stream);
    if (cplx) h->d_ell_im.upload(ell_im, h->stream); else h->d_ell_im.release();
    h->d_diag.upload(diag, h->stream);
    h->d_stream_coef.upload(stream_coef, h->stream);
    h->d_term_rkm.upload(term_rkm, h->stream);
    h->d_rho0.upload(r0, h->stream);
    h->d_coil.upload(cl, h->stream);
    // sparse coil: at most 32 non-zero rows -> moments read straight from the state
    std::vector<int> crow;
    std::vector<double2> cval;
    for (int i = 0; i < n_pad; ++i)
        if (cl[i].x != 0.0 || cl[i].y != 0.0) { crow.push_back(i); cval.push_back(cl[i]); }
    h->ncoil = (crow.size() <= 32) ? (int)crow.size() : -1;
    if (h->ncoil > 0) {
        h->d_coil_rows.upload(crow, h->stream);
        h->d_coil_vals.upload(cval, h->stream);
        h->d_coil_chan.upload(std::vector<int>(crow.size(), 0), h->stream);
    }
    h->nchan = 1;
    h->n_states = 0;
    h->row_of = inv;
    h->n = (int)n;
    h->n_pad = n_pad;
    h->nslices = nslices;
    h->ell_len = ell_len;
    h->nstreams = nst;
    h->nterms = n_terms;
    h->cplx = cplx;
    h->nnz = (int64_t)nk;
    h->g_upper = g_upper;
    // every assembled off-diagonal entry is at most g_upper in magnitude (the
    // rotational coefficients are at most 1): 2^-(floor(log2 g_upper) + 1)
    // scales them into (-1, 1) for the packed FP32 layout
    h->lo_scale = g_upper > 0.0 ? std::ldexp(1.0, -std::ilogb(g_upper) - 1) : 1.0;
    h->max_im_diag = max_im_diag;
    h->max_growth = max_growth;
    h->ell_parts.assign(std::max(ell_len, 1), 0);
    for (int q = 0; q < nst; ++q)
        for (int e = 0; e < ell_len; ++e) {
            if (std::fabs(ell_re[(size_t)q * ell_len + e]) > im_tol) h->ell_parts[e] |= 1;
            if (cplx && std::fabs(ell_im[(size_t)q * ell_len + e]) > im_tol) h->ell_parts[e] |= 2;
        }
    h->ell_col_host = std::move(ell_col);
    h->row_bound = std::move(row_bound);
    h->rho0_host = std::move(r0);
    h->coil_row_host = std::move(crow);
    h->coil_val_host = std::move(cval);
    h->coil_chan_host.assign(h->coil_row_host.size(), 0);
    spx::Components comp((int)n);
    for_each_coupling(h, [&](int r, int c, int) { comp.join(r, c); });
    h->component.resize(n);
    for (int i = 0; i < (int)n; ++i) h->component[i] = comp.find(i);
    rebuild_plan(h);
    SPX_CUDA(cudaStreamSynchronize(h->stream));
    h->have_system = true;
}

// Several detection states (evolution.m 'multichannel'): column c of the
// n x nchan column-major complex array is channel c.
void upload_coils(spx_handle *h, int32_t nchan, const double *coils) {
    if (!h->have_system) throw SpxError(SPX_ERR_NO_SYSTEM, "no spin system uploaded");
    if (!coils) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "coils is NULL");
    if (nchan < 1 || nchan > 8) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "channels must be 1..8");
    const int n = h->n;
    for (int64_t i = 0; i < 2 * (int64_t)n * nchan; ++i)
        if (!std::isfinite(coils[i])) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "non-finite coil");
    std::vector<int> crow, cchan;
    std::vector<double2> cval;
    for (int c = 0; c < nchan; ++c)
        for (int i = 0; i < n; ++i) {
            const double re = coils[2 * ((size_t)c * n + i)], im = coils[2 * ((size_t)c * n + i) + 1];
            if (re != 0.0 || im != 0.0) {
                crow.push_back(h->row_of[i]);
                cval.push_back(make_double2(re, im));
                cchan.push_back(c);
            }
        }
    if (nchan > 1 && crow.size() > 32)
        throw SpxError(SPX_ERR_UNSUPPORTED, "several channels need at most 32 non-zero coil entries in total");
    SPX_CUDA(cudaSetDevice(h->device));
    if (nchan == 1) {                               // dense copy for the per-row projection path
        std::vector<double2> cl(h->n_pad, make_double2(0, 0));
        for (size_t e = 0; e < crow.size(); ++e) cl[crow[e]] = cval[e];
        h->d_coil.upload(cl, h->stream);
    }
    h->ncoil = crow.size() <= 32 ? (int)crow.size() : -1;
    if (h->ncoil > 0) {
        h->d_coil_rows.upload(crow, h->stream);
        h->d_coil_vals.upload(cval, h->stream);
        h->d_coil_chan.upload(cchan, h->stream);
    }
    h->nchan = nchan;
    h->coil_row_host = std::move(crow);
    h->coil_val_host = std::move(cval);
    h->coil_chan_host = std::move(cchan);
    rebuild_plan(h);
    SPX_CUDA(cudaStreamSynchronize(h->stream));
}

// Per-orientation initial states (powder.m:244-254: 'aniso_eq' or a function
// handle rho0 evaluated at every orientation): states holds n_states
// Liouville vectors, orientation after orientation, interleaved complex.
void set_initial_states(spx_handle *h, int64_t n_states, const double *states) {
    if (!h->have_system) throw SpxError(SPX_ERR_NO_SYSTEM, "no spin system uploaded");
    if (n_states == 0) {
        const bool had = h->n_states != 0;
        h->n_states = 0;
        SPX_CUDA(cudaSetDevice(h->device));
        if (had) rebuild_plan(h);
        return;
    }
    if (n_states < 0 || !states) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "bad initial-state array");
    const int n = h->n;
    std::vector<double2> st((size_t)n_states * h->n_pad, make_double2(0, 0));
    std::vector<char> rows(n, 0);
    for (int64_t o = 0; o < n_states; ++o)
        for (int i = 0; i < n; ++i) {
            const double re = states[2 * ((size_t)o * n + i)], im = states[2 * ((size_t)o * n + i) + 1];
            if (!std::isfinite(re) || !std::isfinite(im)) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "non-finite initial state");
            st[(size_t)o * h->n_pad + h->row_of[i]] = make_double2(re, im);
            if (re != 0.0 || im != 0.0) rows[h->row_of[i]] = 1;
        }
    SPX_CUDA(cudaSetDevice(h->device));
    h->d_rho0s.upload(st, h->stream);
    SPX_CUDA(cudaStreamSynchronize(h->stream));
    h->n_states = n_states;
    h->state_rows = std::move(rows);
    rebuild_plan(h);
}

// ---------------------------------------------------------------------------
// Launch configuration
// ---------------------------------------------------------------------------
constexpr int kPowderGroup = 64;    // orientations per partial sum of the powder reduction

// The options of a run: the caller's, and what the autotuner adds.  A run whose
// caller set a shape, or a chunk length beside the tuner's, takes the whole
// system in that shape; one in a shape of the engine's own may still take the
// coupled-state kernels.
struct RunOptions : spx_options {
    bool own = false;                // threads, cluster and chunk_target are the tuner's
    double blk_target = 0.0;         // TunedShape::blk_target
    RunOptions() : spx_options{} {}
    RunOptions(const spx_options &o) : spx_options(o) {}
};

struct Config {
    int threads, rmax, M, Kmax, grid;
    bool fixed;
    double chunk_x;
    size_t smem;
    double tol;
    int cl = 1;                                   // CTAs per cluster
    int slices[spx::kMaxCluster + 1] = {};        // row blocks of the cluster's CTAs
    int nsl_loc = 0, ell_loc = 0;                 // largest block (slices, ELL entries)
    int traj_m = 1;                               // trajectory outputs: chunk length (1: none)
    bool traj = false;                            // the kernels with trajectory outputs
    // the coupled-state kernels (block.cuh), if they run: their layout and that
    // of the spectral bounds, chunk target, chunk cap, series cap, ladder steps and shared memory
    const BlockPlan::Layout *blk = nullptr, *blk_bounds = nullptr;
    double blk_x = 0.0;
    int blk_M = 0, blk_K = 0, blk_lev = 0;
    int blk_which = 0, blk_bounds_which = 0;      // the propagation and bounds kernels (spx_block_kernel_*)
    // by dense matrices (dense.cuh): states and detection rows kept,
    // squarings of the scaled exponential
    const BlockPlan *dense = nullptr;
    int dense_m = 0, dense_rows = 0, dense_scale = 0;
    bool dense_one = false;                       // one CTA per orientation
    size_t blk_smem = 0, blk_even = 0;            // blk_even: no SM takes more CTAs than its share
};

double host_series_terms(double x, double lg, double tol) {
    if (!(x > 0.0)) return 1;
    const double ltol = std::log(tol);
    int k = std::max(1, (int)std::ceil(x) + 1);
    while (k < 200000) {
        const double lt = -0.5 * std::log(2.0 * M_PI * k) + k * std::log(M_E * x / (2.0 * k)) + k * lg;
        if (lt < ltol) break;
        ++k;
    }
    return k;
}

template <bool F64, bool CPLX>
size_t smem_bytes(const spx_handle *h, int nsl_loc, int ell_loc, int Kmax, int M, int threads, int traj_m, int cl) {
    // cluster launches of FP32 real values keep each column in its value
    const bool packed = !F64 && !CPLX && cl > 1;
    spx::SmemLayout<F64, CPLX> L(h->n_pad, nsl_loc, ell_loc, Kmax, M, threads, h->nchan, traj_m, packed);
    return L.total;
}

size_t smem_for(const spx_handle *h, bool f64, int nsl_loc, int ell_loc, int Kmax, int M, int threads,
                int traj_m, int cl) {
    if (f64)
        return h->cplx ? smem_bytes<true, true>(h, nsl_loc, ell_loc, Kmax, M, threads, traj_m, cl)
                       : smem_bytes<true, false>(h, nsl_loc, ell_loc, Kmax, M, threads, traj_m, cl);
    return h->cplx ? smem_bytes<false, true>(h, nsl_loc, ell_loc, Kmax, M, threads, traj_m, cl)
                   : smem_bytes<false, false>(h, nsl_loc, ell_loc, Kmax, M, threads, traj_m, cl);
}

}  // namespace
// Kernel addresses from the translation units that instantiate them
// (kern_<precision><value type>_<sc: listed coil | dc: dense coil>.cu).
const void *spx_kernel_f32r_sc(int rmax, bool cluster, bool wide);
const void *spx_kernel_f32c_sc(int rmax, bool cluster, bool wide);
const void *spx_kernel_f64r_sc(int rmax, bool cluster, bool wide);
const void *spx_kernel_f64c_sc(int rmax, bool cluster, bool wide);
const void *spx_kernel_f32r_dc(int rmax, bool cluster, bool wide);
const void *spx_kernel_f32c_dc(int rmax, bool cluster, bool wide);
const void *spx_kernel_f64r_dc(int rmax, bool cluster, bool wide);
const void *spx_kernel_f64c_dc(int rmax, bool cluster, bool wide);
const void *spx_kernel_f32r_sc_t(int rmax, bool cluster, bool wide);     // with trajectory outputs
const void *spx_kernel_f32c_sc_t(int rmax, bool cluster, bool wide);
const void *spx_kernel_f64r_sc_t(int rmax, bool cluster, bool wide);
const void *spx_kernel_f64c_sc_t(int rmax, bool cluster, bool wide);
const void *spx_kernel_f32r_dc_t(int rmax, bool cluster, bool wide);
const void *spx_kernel_f32c_dc_t(int rmax, bool cluster, bool wide);
const void *spx_kernel_f64r_dc_t(int rmax, bool cluster, bool wide);
const void *spx_kernel_f64c_dc_t(int rmax, bool cluster, bool wide);
// Kernels of block.cuh (kern_block_<value type>.cu): which 0 the FP32 and 5 the
// FP64 spectral bounds, 1 the FP32 and 2 the FP64 propagation.
const void *spx_block_kernel_r(int ecap, int which);
const void *spx_block_kernel_c(int ecap, int which);
namespace {

// Single-CTA kernels for RMAX 1, 2, 4, 6; cluster kernels for RMAX 1, 2, 4;
// sc: the coil is listed (at most 32 non-zeros), else the dense projection.
const void *select_kernel(bool f64, bool cplx, int rmax, bool clu, bool sc, bool traj = false, bool wide = false) {
    const void *k;
    if (traj) {
        if (sc) {
            if (f64) k = cplx ? spx_kernel_f64c_sc_t(rmax, clu, wide) : spx_kernel_f64r_sc_t(rmax, clu, wide);
            else k = cplx ? spx_kernel_f32c_sc_t(rmax, clu, wide) : spx_kernel_f32r_sc_t(rmax, clu, wide);
        } else {
            if (f64) k = cplx ? spx_kernel_f64c_dc_t(rmax, clu, wide) : spx_kernel_f64r_dc_t(rmax, clu, wide);
            else k = cplx ? spx_kernel_f32c_dc_t(rmax, clu, wide) : spx_kernel_f32r_dc_t(rmax, clu, wide);
        }
    } else if (sc) {
        if (f64) k = cplx ? spx_kernel_f64c_sc(rmax, clu, wide) : spx_kernel_f64r_sc(rmax, clu, wide);
        else k = cplx ? spx_kernel_f32c_sc(rmax, clu, wide) : spx_kernel_f32r_sc(rmax, clu, wide);
    } else {
        if (f64) k = cplx ? spx_kernel_f64c_dc(rmax, clu, wide) : spx_kernel_f64r_dc(rmax, clu, wide);
        else k = cplx ? spx_kernel_f32c_dc(rmax, clu, wide) : spx_kernel_f32r_dc(rmax, clu, wide);
    }
    if (!k) throw SpxError(SPX_ERR_INTERNAL, "no kernel for this launch shape");
    return k;
}

// Split the slices into cl contiguous blocks of about equal cost (ELL entries
// plus a per-row share); returns false if cl exceeds the slice count.
bool partition_slices(const spx_handle *h, int cl, Config &c) {
    if (cl > h->nslices) return false;
    const std::vector<int> &off = h->slice_off_host;
    auto cost = [&](int sl) { return (double)(off[sl + 1] - off[sl]) + 32.0 * 4; };
    double total = 0;
    for (int sl = 0; sl < h->nslices; ++sl) total += cost(sl);
    c.cl = cl;
    c.slices[0] = 0;
    double acc = 0;
    int r = 1;
    for (int sl = 0; sl < h->nslices && r < cl; ++sl) {
        acc += cost(sl);
        // cut once the running cost reaches r/cl of the total, leaving a slice for every later block
        if (acc >= total * r / cl || h->nslices - (sl + 1) == cl - r) c.slices[r++] = sl + 1;
    }
    c.slices[cl] = h->nslices;
    c.nsl_loc = 0;
    c.ell_loc = 0;
    for (int j = 0; j < cl; ++j) {
        if (c.slices[j + 1] <= c.slices[j]) return false;
        c.nsl_loc = std::max(c.nsl_loc, c.slices[j + 1] - c.slices[j]);
        c.ell_loc = std::max(c.ell_loc, off[c.slices[j + 1]] - off[c.slices[j]]);
    }
    return true;
}

const void *block_kernel(bool cplx, int ecap, int which) {
    const void *k = cplx ? spx_block_kernel_c(ecap, which) : spx_block_kernel_r(ecap, which);
    if (!k) throw SpxError(SPX_ERR_INTERNAL, "no coupled-state kernel for this layout");
    return k;
}

size_t block_smem_for(bool f64, bool cplx, int K, int M, const BlockPlan::Layout &l, bool traj) {
    return f64 ? spx::block_smem64(K, M, l.dev.nv, l.dev.threads, l.dev.ecap, l.dev.n, cplx, traj)
               : spx::block_smem32(K, M, l.dev.nv, l.dev.threads, traj);
}

// The layout with the least modelled time for a grid.
const BlockPlan::Layout *best_layout(const std::vector<BlockPlan::Layout> &ls, double per_sm) {
    const BlockPlan::Layout *best = nullptr;
    for (const auto &l : ls)
        if (!best || l.cost.time(per_sm) < best->cost.time(per_sm)) best = &l;
    return best;
}

// How the coupled-state kernels run a plan: its layout with the least modelled
// time for this grid, the chunk and the tables; false if they cannot.
bool configure_block(spx_handle *h, const BlockPlan &plan, int64_t n_orient, double dt, int64_t nsteps, bool f64,
                     double chunk_target, int kmax_override, int m_cap, bool traj, Config &c) {
    if (!plan.ok) return false;
    const double per_sm = (double)n_orient / h->sm_count;
    const BlockPlan::Layout *best = best_layout(plan.layouts[f64 ? 1 : 0], per_sm);
    if (!best) return false;
    c.blk_x = chunk_target > 0 ? chunk_target : 300.0;
    const double lg = (h->g_upper > 0) ? 2.0 * h->max_im_diag / (h->g_upper / 4.0) : 0.0;
    int K = (int)host_series_terms(std::max(c.blk_x, h->g_upper * dt), std::min(lg, 0.05), c.tol) + 16;
    c.blk_K = std::min(std::max(K, kmax_override), 8192);
    // a table's columns: at most 2^18 entries a table (long series come with short chunks)
    c.blk_M = (int)std::min<int64_t>(std::min(m_cap, std::max(1, (1 << 18) / c.blk_K)), nsteps + 1);
    c.blk_lev = (int)std::max<int64_t>(4, std::min<int64_t>(spx::kBlockLevels, n_orient / 16));
    c.blk_smem = block_smem_for(f64, h->cplx, c.blk_K, c.blk_M, *best, traj);
    c.blk_which = (f64 ? 2 : 1) + (traj ? 2 : 0);
    const void *kfn = block_kernel(h->cplx, best->ecap, c.blk_which);
    cudaFuncAttributes fa{};
    SPX_CUDA(cudaFuncGetAttributes(&fa, kfn));
    if (c.blk_smem + fa.sharedSizeBytes > h->smem_optin) return false;
    SPX_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(h->smem_optin - fa.sharedSizeBytes)));
    const size_t even = (size_t)(n_orient + h->sm_count - 1) / h->sm_count, own = fa.sharedSizeBytes + 1024;
    const size_t part = (h->smem_sm / (even + 1) + 256) & ~(size_t)15;
    c.blk_even = part > own ? std::max(c.blk_smem, part - own) : c.blk_smem;
    c.blk = best;
    c.blk_bounds = best;
    if (f64) {
        // the FP64 bounds run on any layout of at most kBlockMaxEntries a lane
        c.blk_bounds = nullptr;
        for (const auto &ls : plan.layouts)
            for (const auto &l : ls)
                if (l.ecap <= spx::kBlockMaxEntries &&
                    (!c.blk_bounds || l.cost.bounds_time(per_sm) < c.blk_bounds->cost.bounds_time(per_sm)))
                    c.blk_bounds = &l;
    }
    c.blk_bounds_which = f64 ? 5 : 0;
    return true;
}

// Chooses the dense kernels for a run on the coupled states when their modelled
// time is below the series': both in cycles, by FP64 instructions (2 lanes a
// cycle on each SM) or by latency (6000 cycles and 470 a state from one of the
// dense launches to the next; the layout's latency for each series term).
// Measured sides (coupled states, orientations, steps): FP64 52, 1, 2048: dense
// 0.5 ms, series 2.3 ms; 52, 1000, 2048: 16 and 11 ms; 8, 400, 1024: 0.2 and
// 1.4 ms.  FP32 6, 200, 1024: 0.07 and 0.65 ms (one CTA an orientation); 20, 200, 1024: 0.56 and 1.02;
// 20, 1000, 1024: 1.86 and 1.28; 52, 1, 1024: 0.50 and 0.36; 70, 1, 1024: 0.67
// and 1.09.
void choose_dense(const spx_handle *h, const BlockPlan &plan, int64_t n_orient, double dt, int64_t nsteps, bool f64, Config &c) {
    const double n = plan.n, npts = (double)nsteps + 1.0;
    // rounding doubles with every squaring; and the matrices take memory
    if (nsteps > 8192 || 6.0 * n_orient * n * n * sizeof(double2) > 1e9) return;
    int m = 1, rows = 1, squarings = 0;
    while ((int64_t)m * rows < nsteps + 1) {
        if (m <= rows) m *= 2; else rows *= 2;
        ++squarings;
    }
    int scale = 0;
    while (std::ldexp(plan.bound * dt, -scale) > 0.5) ++scale;
    const bool one = plan.n <= spx::kDenseOne && spx::dense_one_smem(plan.n, m, rows, h->nchan) <= 96 * 1024;
    const double products = 6.0 + scale + squarings;
    const double half = h->cplx || n < spx::kDenseTri ? 1.0 : 0.5;    // real couplings: symmetric products
    const double work = 4.0 * n * n * (half * products * n + m + rows * h->nchan) + 4.0 * n * npts * h->nchan;
    const double chain = products + squarings + 4.0;
    const double dense = one ? work * std::ceil((double)n_orient / h->sm_count) / 2.0 + 800.0 * chain + 2e4
                             : work * n_orient / (2.0 * h->sm_count) + (6000.0 + 470.0 * n) * chain;
    const double per_sm = (double)n_orient / h->sm_count;
    // the spectral half-width is about an eighth of the row bound (5.6 to 11.5
    // on the benchmark systems), a chunk's series a quarter longer than its
    // argument, and an FP64 term takes twice the model's cycles alone, 1.5 times
    // in company; FP32 terms 0.85 to 1.5 times, after 130 us of bounds and tables
    const double terms = 1.25 * plan.bound / 8.0 * dt * npts + 30.0;
    const double factor = f64 ? (per_sm > 2.0 ? 1.5 : 2.0) : per_sm > 2.0 ? 1.5 : per_sm > 1.0 ? 1.2 : 0.85;
    const double series = terms * factor * c.blk->cost.time(per_sm) + (f64 ? 1e5 : 2.5e5);
    if (dense > series) return;
    c.dense = &plan;
    c.dense_m = m;
    c.dense_rows = rows;
    c.dense_scale = scale;
    c.dense_one = one;
}

bool forced_shape(const RunOptions &o) {
    return o.chunk_steps > 0 || ((o.threads > 0 || o.cluster > 0 || o.chunk_target > 0) && !o.own);
}

// The caller's options (null: the defaults).
spx_options given_options(const spx_options *opt) {
    spx_options o{};
    if (opt) o = *opt;
    if (o.precision != SPX_FP32 && o.precision != SPX_FP64)
        throw SpxError(SPX_ERR_INVALID_ARGUMENT, "unknown precision");
    return o;
}

// Whether the state could grow to more than four times its norm, which the
// whole-system kernel refuses as diverged (its chunks' norm check).  The dense
// matrices watch no norm, and the coupled-state kernels neither the other states
// nor chunks as long, so a run that this may happen to is the whole system's.
bool may_diverge(const spx_handle *h, double dt, int64_t nsteps) {
    return h->max_growth * dt * (double)nsteps > 1.3862943611198906;       // ln 4
}

// Whether a powder run takes the coupled-state kernels.  c holds the whole
// system's launch shape (so what is refused does not depend on them).
void choose_block(spx_handle *h, const BlockPlan *plan, int64_t n_orient, double dt, int64_t nsteps,
                  const RunOptions &opt, int kmax_override, int m_cap, Config &c) {
    const bool f64 = opt.precision == SPX_FP64;
    if (!plan || !plan->ok || forced_shape(opt) || may_diverge(h, dt, nsteps)) return;
    // FP32 runs of more than 8192 undamped steps keep the whole system: there
    // FP32 nears the 1e-5 bar and its error decides whether the run is repeated
    // in FP64, so the decision stays the one it has been (a three-spin system,
    // 16384 steps: 1.2e-5 on the whole system, 3.5e-6 on its coupled states)
    if (!f64 && h->max_im_diag == 0.0 && nsteps > 8192) return;
    if (configure_block(h, *plan, n_orient, dt, nsteps, f64, opt.blk_target, kmax_override, m_cap, false, c) &&
        kmax_override == 0 && m_cap == 256)
        choose_dense(h, *plan, n_orient, dt, nsteps, f64, c);
}

// traj: the run writes the state at every step (chunks of opt.chunk_steps
// steps, their intermediate states accumulated in shared memory).  plan: the
// run's coupled states, if it may be restricted to them.
Config choose_config(spx_handle *h, int64_t n_orient, double dt, int64_t nsteps, const RunOptions &opt,
                     int kmax_override, int m_cap = 256, bool traj = false, const BlockPlan *plan = nullptr) {
    Config c{};
    c.traj = traj;
    const bool f64 = opt.precision == SPX_FP64;
    if (opt.cluster != 0 && opt.cluster != 1 && opt.cluster != 2 && opt.cluster != 4 && opt.cluster != 8)
        throw SpxError(SPX_ERR_INVALID_ARGUMENT, "cluster must be 0 (auto), 1, 2, 4 or 8");
    if (opt.lanczos_its != 0 && (opt.lanczos_its < 2 || opt.lanczos_its > spx::kMaxLanczos))
        throw SpxError(SPX_ERR_INVALID_ARGUMENT, "lanczos_its must be 0 or 2..48");
    c.tol = opt.series_tol > 0 ? opt.series_tol : (f64 ? 1e-16 : 1e-11);
    // chunk: each orientation picks the step count whose series argument
    // s*M*dt is about chunk_x (kernel side); M here is the cap.  The first
    // layout that fits one SM's shared memory is used: one CTA per orientation
    // with the longest chunk target, else clusters of 2, 4, 8 CTAs sharing an
    // orientation (rows split between them).
    c.fixed = opt.chunk_steps > 0;
    const double lg = (h->g_upper > 0) ? 2.0 * h->max_im_diag / (h->g_upper / 4.0) : 0.0;
    // c1 (chunks of any length): x_c = 300 -> 76.8 ms, 450 -> 81.0 ms, 600 -> 84.3 ms
    std::vector<double> targets = {300.0, 200.0, 150.0, 100.0, 60.0, 30.0};
    if (opt.chunk_target > 0) targets = {opt.chunk_target};
    bool placed = false;
    const int cls[] = {1, 2, 4, 8};
    // up to 6 rows per lane on one CTA, at most 4 on a cluster (c4 on one CTA
    // with 6 rows per lane: 323 ms per powder when compared, 183 ms since; on
    // 2-CTA clusters with 3: 344 ms -- a cluster pays a barrier across SMs
    // per term)
    for (int cl : cls) {
        if (opt.cluster > 0 && cl != opt.cluster) continue;       // cluster size set by the caller
        if (!partition_slices(h, cl, c)) continue;
        // warps: one per 32-row slice, at most 16 (c1 on an older kernel: 16
        // warps 118.9 ms, 13 warps 121.3 ms per 1000-orientation powder; c2
        // dim 4096 on 8-CTA clusters: 16 warps 536 ms, 9 warps 584 ms), then
        // half as many; a smaller CTA is tried before a larger cluster (its
        // reconstruction scratch is smaller), if the rows per lane stay within
        // the limit.  FP32 with 33-46 slices on a CTA first tries 2 rows per
        // lane on up to 24 warps (the wide kernels; one warp more than the
        // rows need: c1 on 20 warps 60.4 ms against 63.8 on 16 with 3 rows)
        const bool wide_ok = !f64 && !traj;
        std::vector<int> nws = {std::min(16, std::max(1, c.nsl_loc))};
        if (opt.threads > 0) nws = {std::max(1, std::min(wide_ok ? 24 : 16, opt.threads / 32))};
        else {
            if (nws[0] > 4) nws.push_back((nws[0] + 1) / 2);
            if (wide_ok && c.nsl_loc > 32 && c.nsl_loc <= 46) nws.insert(nws.begin(), std::min(24, c.nsl_loc / 2 + 2));
        }
        for (int nwarps : nws) {
        const int rows = (c.nsl_loc + nwarps - 1) / nwarps;
        if (rows > (cl > 1 ? 4 : 6)) continue;
        if (nwarps > 16 && rows > 2) continue;                       // the wide kernel has 2 rows per lane
        c.rmax = (rows <= 1 && nwarps <= 16) ? 1 : rows <= 2 ? 2 : rows <= 4 ? 4 : 6;   // wide: always RMAX 2
        c.threads = nwarps * 32;
        // dynamic shared memory may use what the kernel's static arrays leave
        cudaFuncAttributes fa{};
        SPX_CUDA(cudaFuncGetAttributes(&fa, select_kernel(f64, h->cplx, c.rmax, cl > 1, h->ncoil > 0, traj, c.threads > 512)));
        const size_t budget = h->smem_optin > fa.sharedSizeBytes ? h->smem_optin - fa.sharedSizeBytes : 0;
        for (double tx : targets) {
            c.chunk_x = tx;
            int M = c.fixed ? opt.chunk_steps : m_cap;
            M = (int)std::min<int64_t>(M, nsteps + 1);
            M = std::max(M, 1);
            c.M = M;
            // a single step whose series argument exceeds the target (long
            // delays of a pulse program) still gets a table that holds its series
            const double xu = c.fixed ? std::max(h->g_upper * M * dt, 1.0) : std::max(c.chunk_x, h->g_upper * dt);
            int K = (int)host_series_terms(xu, std::min(lg, 0.05), c.tol) + 16;
            if (kmax_override > 0) K = std::max(K, kmax_override);
            c.Kmax = std::min(K, 8192);
            c.traj_m = traj ? c.M : 1;
            c.smem = smem_for(h, f64, c.nsl_loc, c.ell_loc, c.Kmax, c.M, c.threads, c.traj_m, cl);
            if (c.smem <= budget) { placed = true; break; }
            if (c.fixed) break;
        }
        if (placed) break;
        }
        if (placed) break;
    }
    if (!placed)
        throw SpxError(SPX_ERR_UNSUPPORTED, "system does not fit the shared memory of a cluster of 8 SMs (" +
                                                std::to_string(c.smem) + " bytes per SM)");
    const void *kfn = select_kernel(f64, h->cplx, c.rmax, c.cl > 1, h->ncoil > 0, c.traj, c.threads > 512);
    {
        // allow the whole budget: several configurations of one kernel may be
        // prepared before any of them launches (batched graphs)
        cudaFuncAttributes fa{};
        SPX_CUDA(cudaFuncGetAttributes(&fa, kfn));
        SPX_CUDA(cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)(h->smem_optin - fa.sharedSizeBytes)));
    }
    if (c.cl == 1) {
        int per_sm = 0;
        SPX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, c.threads, c.smem));
        per_sm = std::max(per_sm, 1);
        c.grid = (int)std::min<int64_t>(n_orient, (int64_t)h->sm_count * per_sm);
    } else {
        cudaLaunchConfig_t lc{};
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)c.cl;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        lc.gridDim = dim3((unsigned)(c.cl * h->sm_count));
        lc.blockDim = dim3((unsigned)c.threads);
        lc.dynamicSmemBytes = c.smem;
        lc.attrs = at;
        lc.numAttrs = 1;
        int nclusters = 0;
        SPX_CUDA(cudaOccupancyMaxActiveClusters(&nclusters, kfn, &lc));
        if (nclusters < 1) throw SpxError(SPX_ERR_UNSUPPORTED, "no cluster of " + std::to_string(c.cl) + " CTAs fits");
        c.grid = (int)std::min<int64_t>(n_orient, nclusters) * c.cl;
    }
    choose_block(h, plan, n_orient, dt, nsteps, opt, kmax_override, m_cap, c);
    return c;
}

// FP32 runs hand the assembled L of every orientation from the bounds to the
// propagation (both on one layout) while it takes at most 512 MB; larger grids
// assemble it twice (a radical's 4000 orientations: 96 MB).
size_t saved_block(const Config &c) {
    return spx::block_saved(c.blk->dev.ecap, c.blk->dev.threads);
}
bool saves_block(int64_t n_orient, bool f64, const Config &c) {
    return !f64 && (double)n_orient * (double)saved_block(c) <= 64e6;
}

size_t block_table_entries(const Config &c) { return (size_t)c.blk_lev * c.blk_K * spx::block_row(c.blk_M); }

void reserve_block(BlockBufs &b, int64_t n_orient, bool f64, const Config &c) {
    b.centre.reserve(n_orient);
    b.extent.reserve(2);
    b.lev_half.reserve(c.blk_lev);
    b.lev.reserve(3 * (size_t)c.blk_lev);
    b.kcut.reserve((size_t)c.blk_lev * (c.blk_M + 1));
    b.table.reserve(block_table_entries(c));
    if (!f64) b.tablef.reserve(block_table_entries(c));
    if (saves_block(n_orient, f64, c)) b.saved.reserve(n_orient * saved_block(c));
}

// The buffers' addresses and the configuration in a run descriptor.
void block_run_buffers(spx::BlockRun &r, const Config &c, double *centre, unsigned long long *extent, double *lev_half,
                       int *lev, int *kcut, double *table, float *tablef) {
    r.centre = centre;
    r.extent = extent;
    r.lev_half = lev_half;
    r.nlev = c.blk_lev;
    r.lev_m = lev;
    r.lev_k = lev + c.blk_lev;
    r.lev_raw = lev + 2 * c.blk_lev;
    r.kcut = kcut;
    r.table = table;
    r.tablef = tablef;
    r.Mcap = c.blk_M;
    r.Kmax = c.blk_K;
    r.chunk_x = c.blk_x;
    r.tol = c.tol;
}

// The three launches of a run over the coupled states: spectral bounds (of
// every orientation), Bessel tables (for one time step) and propagation.
void launch_bounds(spx_handle *h, const Config &c, spx::DevSystem &sys, spx::BlockRun &r, cudaStream_t stream) {
    spx::BlockLayout lay = c.blk_bounds->dev;
    SPX_CUDA(cudaMemsetAsync(r.extent, 0, 2 * sizeof(unsigned long long), stream));
    void *args[] = {&sys, &lay, &r};
    SPX_CUDA(cudaLaunchKernel(block_kernel(h->cplx, c.blk_bounds->ecap, c.blk_bounds_which), dim3((unsigned)r.n_orient),
                              dim3((unsigned)lay.threads), args, 0, stream));
    ++h->launches;
}
void launch_tables(spx_handle *h, const Config &c, spx::BlockRun &r, cudaStream_t stream) {
    spx::block_tables_kernel<<<dim3((unsigned)(c.blk_M / 32 + 1), (unsigned)c.blk_lev), 128, 0, stream>>>(r);
    SPX_CUDA(cudaGetLastError());
    ++h->launches;
}
void launch_propagation(spx_handle *h, const Config &c, spx::DevSystem &sys, spx::BlockRun &r, cudaStream_t stream) {
    spx::BlockLayout lay = c.blk->dev;
    void *args[] = {&sys, &lay, &r};
    const bool f64 = c.blk_which % 2 == 0;
    SPX_CUDA(cudaLaunchKernel(block_kernel(h->cplx, c.blk->ecap, c.blk_which), dim3((unsigned)r.n_orient),
                              dim3((unsigned)(lay.threads * (f64 ? 2 : 1))), args, c.blk_smem, stream));
    ++h->launches;
}
void launch_block(spx_handle *h, const Config &c, spx::DevSystem &sys, spx::BlockRun &r, cudaStream_t stream) {
    launch_bounds(h, c, sys, r, stream);
    launch_tables(h, c, r, stream);
    launch_propagation(h, c, sys, r, stream);
}

// Launch the propagation kernel (plain or cluster launch) on the handle's stream.
void launch_chebyshev(spx_handle *h, bool f64, const Config &c, spx::DevSystem &sys, spx::DevRun &run,
                      cudaStream_t stream = nullptr) {
    if (!stream) stream = h->stream;
    SPX_CUDA(cudaMemsetAsync(run.next_orient, 0, sizeof(int), stream));
    run.cl = c.cl;
    run.nsl_loc = c.nsl_loc;
    run.ell_loc = c.ell_loc;
    for (int j = 0; j <= spx::kMaxCluster; ++j) run.cl_slices[j] = j <= c.cl ? c.slices[j] : 0;
    const void *kfn = select_kernel(f64, h->cplx, c.rmax, c.cl > 1, h->ncoil > 0, c.traj, c.threads > 512);
    void *args[] = {&sys, &run};
    ++h->launches;
    if (c.cl == 1) {
        SPX_CUDA(cudaLaunchKernel(kfn, dim3(c.grid), dim3(c.threads), args, c.smem, stream));
        return;
    }
    cudaLaunchConfig_t lc{};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)c.cl;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    lc.gridDim = dim3((unsigned)c.grid);
    lc.blockDim = dim3((unsigned)c.threads);
    lc.dynamicSmemBytes = c.smem;
    lc.stream = stream;
    lc.attrs = at;
    lc.numAttrs = 1;
    SPX_CUDA(cudaLaunchKernelExC(&lc, kfn, args));
}

void reserve_dense(const spx_handle *h, DenseBufs &b, int64_t n_orient, const Config &c) {
    if (c.dense_one) return;
    const size_t n = (size_t)c.dense->n;
    b.M.reserve(6 * (size_t)n_orient * n * n);
    b.sym.reserve(n_orient);
    b.V.reserve((size_t)n_orient * c.dense_m * n);
    b.Y.reserve((size_t)n_orient * h->nchan * c.dense_rows * n);
}

// A run by dense matrices: out (of type Vec) and the status words as the
// propagation kernels write them.  pick: see BlockRun.
template <class Vec>
void launch_dense(spx_handle *h, const Config &c, spx::DevSystem &sys, DenseBufs &b, int64_t n_orient, int pick,
                  const double *d_al, const double *d_be, const double *d_ga, double dt, int64_t nsteps, Vec *out,
                  const spx::DevRun &words, cudaStream_t stream, const spx::DenseCheck &check = spx::DenseCheck{}) {
    const BlockPlan &plan = *c.dense;
    const int n = plan.n, m = c.dense_m, rows = c.dense_rows;
    spx::DenseStart st{};
    st.n_orient = (int)n_orient; st.pick = pick;
    st.alpha = d_al; st.beta = d_be; st.gamma = d_ga;
    st.h = std::ldexp(dt, -c.dense_scale);
    st.m = m; st.nchan = h->nchan; st.rows = rows;
    st.rho0 = sys.rho0; st.rho0s = sys.rho0s; st.state_stride = (size_t)h->n_pad;
    st.ncoil = plan.ncoil; st.coil_row = plan.coil_row; st.coil_chan = plan.coil_chan; st.coil_val = plan.coil_val;
    st.status = words.status; st.kused = words.kused; st.mused = words.mused; st.matvecs = words.matvecs;
    st.halfwidth = words.halfwidth; st.bound = plan.bound;
    st.products = 6 + c.dense_scale;
    const int64_t npts = nsteps + 1;
    double f[17];
    f[0] = 1.0;
    for (int k = 1; k <= 16; ++k) f[k] = f[k - 1] / k;
    if (c.dense_one) {
        spx::DenseOne one{c.dense_scale, (int)npts, {}};
        std::copy(f, f + 17, one.f);
        const size_t smem = spx::dense_one_smem(n, m, rows, h->nchan);
        if (smem > 40 * 1024)
            SPX_CUDA(cudaFuncSetAttribute(spx::dense_one_kernel<Vec>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)(96 * 1024)));
        spx::dense_one_kernel<Vec><<<dim3((unsigned)n_orient), spx::kDenseOneThreads, smem, stream>>>(sys, plan.dense, st, one,
                                                                                                    out, check);
        SPX_CUDA(cudaGetLastError());
        ++h->launches;
        return;
    }
    const int64_t total = n_orient * n * n;
    double2 *M[6];
    for (int q = 0; q < 6; ++q) M[q] = b.M.p + (size_t)q * total;
    auto grid = [&](int64_t items) {
        return dim3((unsigned)std::max<int64_t>(1, std::min<int64_t>((items + spx::kDenseThreads - 1) / spx::kDenseThreads,
                                                                      (int64_t)h->sm_count * 64)));
    };
    st.A = M[0]; st.V = b.V.p; st.Y = b.Y.p;
    const bool tri = n >= spx::kDenseTri && !h->cplx;
    st.sym = tri ? b.sym.p : nullptr;
    spx::dense_start_kernel<<<dim3((unsigned)n_orient), n < spx::kDenseTri ? spx::kDenseThreads : 256, 0, stream>>>(sys, plan.dense, st);
    ++h->launches;
    auto product = [&](const double2 *A, const double2 *B, double2 *C, const spx::DenseSum &t = spx::DenseSum{}) {
        if (tri) spx::dense_product_kernel<true><<<grid(total), spx::kDenseThreads, 0, stream>>>(total, n, b.sym.p, A, B, C, t);
        else spx::dense_product_kernel<false><<<grid(total), spx::kDenseThreads, 0, stream>>>(total, n, nullptr, A, B, C, t);
        ++h->launches;
    };
    // exp(A) to degree 16 in powers of A^4: M = A, A^2, A^3, A^4
    product(M[0], M[0], M[1]);
    product(M[1], M[0], M[2]);
    product(M[1], M[1], M[3]);
    auto quarter = [&](int q) { return spx::DenseSum{M[0], M[1], M[2], f[4 * q], f[4 * q + 1], f[4 * q + 2], f[4 * q + 3]}; };
    spx::dense_sum_kernel<<<grid(total), spx::kDenseThreads, 0, stream>>>(total, n, quarter(3), M[3], f[16], M[4]);
    ++h->launches;
    product(M[3], M[4], M[5], quarter(2));
    product(M[3], M[5], M[4], quarter(1));
    // without the identity while the step is scaled down: exp(A) - 1 = Z keeps
    // its digits, and (1 + Z)^2 - 1 = 2 Z + Z^2
    if (c.dense_scale > 0) f[0] = 0.0;
    product(M[3], M[4], M[5], quarter(0));
    double2 *U = M[5], *W = M[4];
    for (int q = 0; q < c.dense_scale; ++q) {
        product(U, U, W, spx::DenseSum{U, U, U, q + 1 == c.dense_scale ? 1.0 : 0.0, 2.0, 0.0, 0.0});
        std::swap(U, W);
    }
    auto square = [&] { product(U, U, W); std::swap(U, W); };
    // states 0 .. m-1 with U, U^2, U^4, ...; then detection rows with U^m, U^2m, ...
    for (int have = 1; have < m; have *= 2) {
        spx::dense_states_kernel<<<grid(n_orient * have * n), spx::kDenseThreads, 0, stream>>>(n_orient, n, m, have, have, U,
                                                                                                b.V.p);
        ++h->launches;
        if (2 * have < m || rows > 1) square();
    }
    for (int have = 1; have < rows; have *= 2) {
        spx::dense_rows_kernel<<<grid(n_orient * h->nchan * have * n), spx::kDenseThreads, 0, stream>>>(
            n_orient, n, h->nchan, rows, have, have, U, b.Y.p);
        ++h->launches;
        if (2 * have < rows) square();
    }
    spx::dense_points_kernel<Vec><<<grid(n_orient * h->nchan * npts), spx::kDenseThreads, 0, stream>>>(
        n_orient, n, h->nchan, rows, m, (int)npts, b.Y.p, b.V.p, out, words.status, check);
    ++h->launches;
    SPX_CUDA(cudaGetLastError());
}

// Device buffers of one run (idempotent; called before graph capture too).
void reserve_run(spx_handle *h, int64_t n_orient, int64_t nsteps, bool f64, const Config &c) {
    const size_t npts = ((size_t)nsteps + 1) * h->nchan;       // every channel's points
    const size_t vec_bytes = f64 ? sizeof(double2) : sizeof(float2);
    h->d_fids.reserve(npts * n_orient * vec_bytes);
    if (c.dense) reserve_dense(h, h->dense, n_orient, c);
    else if (c.blk) reserve_block(h->blk, n_orient, f64, c);
    else h->d_table.reserve((size_t)c.grid * c.Kmax * (c.M + 1));
    h->d_status.reserve(n_orient);
    h->d_kused.reserve(n_orient);
    h->d_mused.reserve(n_orient);
    h->d_matvecs.reserve(n_orient);
    h->d_halfwidth.reserve(n_orient);
    h->d_counter.reserve(1);
    const int ngroups = (int)((n_orient + kPowderGroup - 1) / kPowderGroup);
    h->d_part.reserve((size_t)ngroups * npts);
}

// The statistics known at launch (finish_run adds the rest).
void describe_run(spx_handle *h, int64_t n_orient, int64_t nsteps, int32_t precision, const Config &c) {
    h->stats = spx_stats{};
    h->stats.n_orientations = n_orient;
    h->stats.nsteps = nsteps;
    h->stats.chunk_steps = c.M;
    h->stats.threads = c.threads;
    h->stats.precision = precision;
    h->stats.dim = h->n;
    h->stats.nnz = h->nnz;
    h->stats.ell_entries = h->ell_len;
    h->stats.value_streams = h->nstreams;
    h->stats.real_offdiag = h->cplx ? 0 : 1;
    h->stats.cluster = c.cl;
    h->stats.channels = h->nchan;
    h->stats.smem_bytes = (int32_t)c.smem;
    h->stats.coupled_dim = c.blk ? c.blk->dev.n : 0;
}

// Weighted sum of the orientations' FIDs: deterministic FP64, fixed groups of
// orientations in a fixed order.
void launch_powder_sum(spx_handle *h, bool f64, const void *fids, const double *d_w, int64_t n_orient, size_t npts,
                       double2 *part, double2 *d_out) {
    const int group = kPowderGroup;
    const int ngroups = (int)((n_orient + group - 1) / group);
    // small CTAs: a point takes four FP64 instructions an orientation, which only
    // more SMs do faster (a whole run of 200 orientations and 1025 points: 179 us
    // with 256 threads, 171 with 64)
    const dim3 pb(64), pg((unsigned)((npts + 63) / 64), (unsigned)ngroups);
    if (f64)
        spx::powder_partial_kernel<double2><<<pg, pb, 0, h->stream>>>(
            reinterpret_cast<const double2 *>(fids), d_w, (int)n_orient, (int)npts, group, part);
    else
        spx::powder_partial_kernel<float2><<<pg, pb, 0, h->stream>>>(
            reinterpret_cast<const float2 *>(fids), d_w, (int)n_orient, (int)npts, group, part);
    SPX_CUDA(cudaGetLastError());
    spx::powder_combine_kernel<<<dim3(pg.x), pb, 0, h->stream>>>(part, ngroups,
                                                                                             (int)npts, d_out);
    SPX_CUDA(cudaGetLastError());
    h->launches += 2;
}

// The uploaded system as the kernels take it.
spx::DevSystem device_system(const spx_handle *h) {
    spx::DevSystem sys{};
    sys.n = h->n; sys.n_pad = h->n_pad; sys.nslices = h->nslices; sys.ell_len = h->ell_len;
    sys.slice_off = h->d_slice_off.p; sys.ell_col = h->d_ell_col.p;
    sys.ell_re = h->d_ell_re.p; sys.ell_im = h->cplx ? h->d_ell_im.p : nullptr;
    sys.diag = h->d_diag.p; sys.stream_coef = h->d_stream_coef.p; sys.nstreams = h->nstreams;
    sys.ncoef = 1 + 2 * h->nterms; sys.nterms = h->nterms; sys.term_rkm = h->d_term_rkm.p;
    sys.rho0 = h->d_rho0.p; sys.coil = h->d_coil.p; sys.max_im_diag = h->max_im_diag; sys.lo_scale = h->lo_scale;
    sys.ncoil = h->ncoil; sys.coil_rows = h->d_coil_rows.p; sys.coil_vals = h->d_coil_vals.p;
    sys.coil_chan = h->d_coil_chan.p; sys.nchan = h->nchan;
    sys.rho0s = h->n_states > 0 ? h->d_rho0s.p : nullptr;
    return sys;
}

// Initial and final states of one run when they are not the handle's own
// (pulse sequences hand the state of one segment to the next).
struct RunIO {
    const double2 *rho0 = nullptr;     // one initial state for every orientation (sliced order)
    const double2 *rho0s = nullptr;    // one per orientation, n_orient x n_pad
    double2 *state_out = nullptr;      // the state after the last step, n_orient x n_pad
    double2 *traj_out = nullptr;       // the state at every step, n_orient x (nsteps+1) x n_pad (needs a
                                       // trajectory configuration: choose_config(..., traj = true))
    bool adjoint = false;              // propagate under -H + 1i R (the adjoint of L, negated)
};

RunOptions apply_tuned(const spx_handle *h, const spx_options &given);

constexpr int kCheckOrients = SPX_FP32_CHECKED_ORIENTATIONS;   // orientations of an FP32 run re-run in FP64

// Orientation indices checked in FP64: evenly spaced over the grid.
int check_index(int j, int S, int64_t n_orient) { return (int)(((2 * (int64_t)j + 1) * n_orient) / (2 * S)); }

// Enqueue the FP64 re-run of the checked orientations on the check stream
// (forked from the handle's stream) and return its CTA count, so that the
// FP32 launch can leave those SMs to it.
int launch_fp32_check(spx_handle *h, int64_t n_orient, const double *d_al, const double *d_be, const double *d_ga,
                      double dt, int64_t nsteps, const RunOptions &opt, const spx::DevSystem &sys32) {
    const int S = (int)std::min<int64_t>(kCheckOrients, n_orient);
    spx_options given{};
    given.precision = SPX_FP64;
    given.lanczos_its = opt.lanczos_its;
    const RunOptions o64 = apply_tuned(h, given);
    const Config c = choose_config(h, S, dt, nsteps, o64, 0, 256, false, &h->plan);
    const size_t npts = ((size_t)nsteps + 1) * h->nchan;
    if (!h->check_stream) {
        SPX_CUDA(cudaStreamCreateWithPriority(&h->check_stream, cudaStreamNonBlocking, h->high_priority));
        SPX_CUDA(cudaEventCreateWithFlags(&h->ev_fork, cudaEventDisableTiming));
        SPX_CUDA(cudaEventCreateWithFlags(&h->ev_join, cudaEventDisableTiming));
    }
    h->d_chk_grid.reserve(3 * (size_t)S);
    h->d_chk_fids.reserve(npts * S * sizeof(double2));
    if (c.dense) reserve_dense(h, h->chk_dense, S, c);
    else if (c.blk) reserve_block(h->chk_blk, S, true, c);
    else h->d_chk_table.reserve((size_t)c.grid * c.Kmax * (c.M + 1));
    h->d_chk_status.reserve(S);
    h->d_chk_kused.reserve(S);
    h->d_chk_mused.reserve(S);
    h->d_chk_matvecs.reserve(S);
    h->d_chk_halfwidth.reserve(S);
    h->d_chk_counter.reserve(1);
    if (sys32.rho0s) h->d_chk_rho0s.reserve((size_t)S * h->n_pad);
    std::vector<int> &idx = h->chk_index;
    idx.resize(S);
    for (int j = 0; j < S; ++j) idx[j] = check_index(j, S, n_orient);
    SPX_CUDA(cudaEventRecord(h->ev_fork, h->stream));
    SPX_CUDA(cudaStreamWaitEvent(h->check_stream, h->ev_fork, 0));
    if (c.dense) {
        spx::DevSystem sys = sys32;
        spx::DevRun words{};
        words.status = h->d_chk_status.p; words.kused = h->d_chk_kused.p; words.mused = h->d_chk_mused.p;
        words.matvecs = h->d_chk_matvecs.p; words.halfwidth = h->d_chk_halfwidth.p;
        launch_dense(h, c, sys, h->chk_dense, S, (int)n_orient, d_al, d_be, d_ga, dt, nsteps,
                     reinterpret_cast<double2 *>(h->d_chk_fids.p), words, h->check_stream);
        SPX_CUDA(cudaEventRecord(h->ev_join, h->check_stream));
        return 0;
    }
    if (c.blk) {
        // the checked orientations are picked out of the whole grid on the device
        spx::DevSystem sys = sys32;
        spx::BlockRun r{};
        BlockBufs &b = h->chk_blk;
        block_run_buffers(r, c, b.centre.p, b.extent.p, b.lev_half.p, b.lev.p, b.kcut.p, b.table.p, nullptr);
        r.n_orient = S; r.alpha = d_al; r.beta = d_be; r.gamma = d_ga; r.pick = (int)n_orient;
        r.dt = dt; r.nsteps = (int)nsteps;
        r.lanczos_its = o64.lanczos_its > 0 ? o64.lanczos_its : 32;
        r.halfwidth = h->d_chk_halfwidth.p; r.max_im_diag = h->max_im_diag;
        r.rho0 = sys.rho0; r.rho0s = sys.rho0s; r.state_stride = (size_t)h->n_pad;
        r.fids = h->d_chk_fids.p; r.nchan = h->nchan;
        r.status = h->d_chk_status.p; r.kused = h->d_chk_kused.p; r.mused = h->d_chk_mused.p;
        r.matvecs = h->d_chk_matvecs.p;
        launch_block(h, c, sys, r, h->check_stream);
        SPX_CUDA(cudaEventRecord(h->ev_join, h->check_stream));
        return 0;
    }
    double *g = h->d_chk_grid.p;
    for (int j = 0; j < S; ++j) {
        SPX_CUDA(cudaMemcpyAsync(g + j, d_al + idx[j], sizeof(double), cudaMemcpyDeviceToDevice, h->check_stream));
        SPX_CUDA(cudaMemcpyAsync(g + S + j, d_be + idx[j], sizeof(double), cudaMemcpyDeviceToDevice, h->check_stream));
        SPX_CUDA(cudaMemcpyAsync(g + 2 * S + j, d_ga + idx[j], sizeof(double), cudaMemcpyDeviceToDevice,
                                 h->check_stream));
        if (sys32.rho0s)
            SPX_CUDA(cudaMemcpyAsync(h->d_chk_rho0s.p + (size_t)j * h->n_pad, sys32.rho0s + (size_t)idx[j] * h->n_pad,
                                     h->n_pad * sizeof(double2), cudaMemcpyDeviceToDevice, h->check_stream));
    }
    spx::DevSystem sys = sys32;
    if (sys32.rho0s) sys.rho0s = h->d_chk_rho0s.p;
    spx::DevRun run{};
    run.traj_m = c.traj_m;
    run.n_orient = S; run.alpha = g; run.beta = g + S; run.gamma = g + 2 * S;
    run.dt = dt; run.nsteps = (int)nsteps; run.M = c.M; run.Kmax = c.Kmax; run.tol = c.tol;
    run.fixed_chunk = c.fixed ? 1 : 0; run.chunk_x = c.chunk_x;
    run.lanczos_its = o64.lanczos_its > 0 ? o64.lanczos_its : 32;
    run.safe_bounds = 0; run.fids = h->d_chk_fids.p; run.table = h->d_chk_table.p;
    run.status = h->d_chk_status.p; run.matvecs = h->d_chk_matvecs.p; run.halfwidth = h->d_chk_halfwidth.p;
    run.kused = h->d_chk_kused.p; run.mused = h->d_chk_mused.p; run.next_orient = h->d_chk_counter.p;
    launch_chebyshev(h, true, c, sys, run, h->check_stream);
    SPX_CUDA(cudaEventRecord(h->ev_join, h->check_stream));
    return c.grid;
}

void launch_powder(spx_handle *h, int64_t n_orient, const double *d_al, const double *d_be,
                   const double *d_ga, const double *d_w, double dt, int64_t nsteps,
                   const RunOptions &opt, double2 *d_out, const Config &c_in, int safe_bounds = 0, bool timed = true,
                   const RunIO &io = RunIO{}, bool fp32_check = false) {
    const bool f64 = opt.precision == SPX_FP64;
    Config c = c_in;
    const size_t npts = ((size_t)nsteps + 1) * h->nchan;   // the powder sum treats channels as more points
    reserve_run(h, n_orient, nsteps, f64, c);

    spx::DevSystem sys = device_system(h);
    if (io.rho0) sys.rho0 = io.rho0;
    if (io.rho0s) sys.rho0s = io.rho0s;
    if (io.adjoint) {
        sys.ell_re = h->d_neg_re.p;
        sys.ell_im = h->cplx ? h->d_neg_im.p : nullptr;
        sys.diag = h->d_neg_diag.p;
    }
    spx::DevRun run{};
    run.state_out = io.state_out;
    if (io.traj_out && !c.traj) throw SpxError(SPX_ERR_INTERNAL, "trajectory output needs a trajectory configuration");
    run.traj_out = io.traj_out;
    run.traj_m = c.traj_m;
    run.n_orient = (int)n_orient; run.alpha = d_al; run.beta = d_be; run.gamma = d_ga;
    run.dt = dt; run.nsteps = (int)nsteps; run.M = c.M; run.Kmax = c.Kmax; run.tol = c.tol;
    run.fixed_chunk = c.fixed ? 1 : 0; run.chunk_x = c.chunk_x;
    run.lanczos_its = opt.lanczos_its > 0 ? opt.lanczos_its : 32;
    run.safe_bounds = safe_bounds; run.fids = h->d_fids.p; run.table = h->d_table.p;
    run.status = h->d_status.p; run.matvecs = h->d_matvecs.p; run.halfwidth = h->d_halfwidth.p;
    run.kused = h->d_kused.p;
    run.mused = h->d_mused.p;
    run.next_orient = h->d_counter.p;

    int chk = 0;
    spx::DenseCheck kept{};
    if (fp32_check && !f64 && c.dense) {
        // an FP32 run by dense matrices is an FP64 run that is rounded at the
        // end: the check takes its unrounded points
        chk = (int)std::min<int64_t>(kCheckOrients, n_orient);
        h->d_chk_fids.reserve(npts * chk * sizeof(double2));
        h->d_chk_status.reserve(chk);
        h->chk_index.resize(chk);
        for (int j = 0; j < chk; ++j) h->chk_index[j] = check_index(j, chk, n_orient);
        static_assert(spx::kDevOk == 0, "status words start at zero");
        SPX_CUDA(cudaMemsetAsync(h->d_chk_status.p, 0, chk * sizeof(int), h->stream));
        kept = {reinterpret_cast<double2 *>(h->d_chk_fids.p), h->d_chk_status.p, chk};
    } else if (fp32_check && !f64) {
        // the FP64 re-run takes its CTAs' SMs; an FP32 run of several waves
        // keeps the rest (a single-wave grid keeps every CTA: fewer would add
        // a wave)
        const int chk_ctas = launch_fp32_check(h, n_orient, d_al, d_be, d_ga, dt, nsteps, opt, sys);
        chk = (int)std::min<int64_t>(kCheckOrients, n_orient);
        const int take = ((chk_ctas + c.cl - 1) / c.cl) * c.cl;
        const bool waves = n_orient * c.cl > c.grid;
        if (waves && c.grid - take >= std::max(c.cl, c.grid / 2)) c.grid -= take;
    }
    if (timed) SPX_CUDA(cudaEventRecord(h->ev[0], h->stream));
    if (c.dense) {
        if (f64)
            launch_dense(h, c, sys, h->dense, n_orient, 0, d_al, d_be, d_ga, dt, nsteps,
                         reinterpret_cast<double2 *>(h->d_fids.p), run, h->stream);
        else
            launch_dense(h, c, sys, h->dense, n_orient, 0, d_al, d_be, d_ga, dt, nsteps,
                         reinterpret_cast<float2 *>(h->d_fids.p), run, h->stream, kept);
    } else if (c.blk) {
        spx::BlockRun r{};
        BlockBufs &b = h->blk;
        block_run_buffers(r, c, b.centre.p, b.extent.p, b.lev_half.p, b.lev.p, b.kcut.p, b.table.p,
                          f64 ? nullptr : b.tablef.p);
        if (saves_block(n_orient, f64, c)) r.saved = b.saved.p;
        r.n_orient = (int)n_orient; r.alpha = d_al; r.beta = d_be; r.gamma = d_ga;
        r.dt = dt; r.nsteps = (int)nsteps; r.lanczos_its = run.lanczos_its; r.safe_bounds = safe_bounds;
        r.halfwidth = run.halfwidth; r.max_im_diag = h->max_im_diag;
        r.rho0 = sys.rho0; r.rho0s = sys.rho0s; r.state_stride = (size_t)h->n_pad;
        r.fids = run.fids; r.nchan = h->nchan;
        r.status = run.status; r.kused = run.kused; r.mused = run.mused; r.matvecs = run.matvecs;
        // launched beside the check's kernels, a grid of less than a wave piles up
        // on the SMs that are free first (200 orientations of a rotor-frame
        // system, 128 threads each: 3.3 to 5.8 ms, 3.3 with even shares); beside
        // other systems of a batch even shares would cost 8 %
        if (chk) c.blk_smem = c.blk_even;
        launch_block(h, c, sys, r, h->stream);
    } else {
        launch_chebyshev(h, f64, c, sys, run);
    }
    if (timed) SPX_CUDA(cudaEventRecord(h->ev[1], h->stream));
    launch_powder_sum(h, f64, h->d_fids.p, d_w, n_orient, npts, h->d_part.p, d_out);
    if (chk && !kept.count) SPX_CUDA(cudaStreamWaitEvent(h->stream, h->ev_join, 0));   // the FP64 re-run is part of the run
    if (timed) SPX_CUDA(cudaEventRecord(h->ev[2], h->stream));
    h->stats_timed = timed;

    describe_run(h, n_orient, nsteps, opt.precision, c);
    h->stats_pending = true;
    h->last_norient = n_orient;
    h->chk_pending = chk;
    h->chk_out = d_out;
    h->chk_w = d_w;
    h->chk_nsteps = nsteps;
}

// FP32 error of a run from its checked orientations (FP32 FIDs f32 and
// their FP64 re-runs f64, S x npts each, channel by channel), its powder FID
// pw and the sum of its squared grid weights w2:
//   orientation  the largest relative 2-norm error of the checked FIDs;
//   powder       the error these imply for the powder FID sum_o w_o f_o,
//                split into two parts added in quadrature.  The part that
//                follows the signal: an orientation's FP32 error acts like a
//                phase error growing with time, so phi(t), the larger of the
//                checked orientations' relative errors over [0, t], weighted
//                by the powder FID's intensity: sqrt(sum |pw|^2 phi^2 /
//                sum |pw|^2).  The part that does not: errors independent
//                across orientations add in quadrature, sqrt(w2) times the
//                checked orientations' rms error norm, over |pw|.
struct FP32Error {
    double orientation = 0.0, powder = 0.0;
};
FP32Error fp32_error(const std::vector<const float2 *> &f32, const double2 *f64, const double2 *pw,
                     double w2, int S, size_t len, int nchan) {
    FP32Error out;
    const size_t npts = len * nchan;
    std::vector<double> phi(len);
    for (int ch = 0; ch < nchan; ++ch) {
        std::fill(phi.begin(), phi.end(), 0.0);
        double err2 = 0.0;                  // sum over checked orientations of |delta f|^2
        for (int j = 0; j < S; ++j) {
            const size_t base = (size_t)j * npts + (size_t)ch * len;
            double num = 0.0, den = 0.0;
            for (size_t t = 0; t < len; ++t) {
                const double2 b = f64[base + t];
                const float2 a = f32[j][(size_t)ch * len + t];
                const double dx = (double)a.x - b.x, dy = (double)a.y - b.y;
                num += dx * dx + dy * dy;
                den += b.x * b.x + b.y * b.y;
                phi[t] = std::max(phi[t], den > 0.0 ? std::sqrt(num / den) : (num > 0.0 ? INFINITY : 0.0));
            }
            err2 += num;
            out.orientation = std::max(out.orientation, den > 0.0 ? std::sqrt(num / den) : (num > 0.0 ? INFINITY : 0.0));
        }
        double num = 0.0, den = 0.0;
        for (size_t t = 0; t < len; ++t) {
            const double2 p = pw[(size_t)ch * len + t];
            const double a = p.x * p.x + p.y * p.y;
            num += a * phi[t] * phi[t];
            den += a;
        }
        if (den > 0.0) {
            const double coherent2 = num / den;
            const double independent2 = w2 * (err2 / S) / den;
            out.powder = std::max(out.powder, std::sqrt(coherent2 + independent2));
        } else if (err2 > 0.0) {
            out.powder = INFINITY;
        }
    }
    return out;
}

// Synchronise, read per-orientation status and fill the statistics.  All results
// are copied behind the run into one pinned buffer of the handle (runs of more
// than kStage bytes of them: pageable memory) and waited for once: a copy of its
// own for each of the eleven took a 200-orientation run of three spins 271 us;
// it takes 181.  want_fid: also the powder FID of h->d_fid, which is returned in
// that buffer, where it lies until the handle's next run (null if it does not
// fit: then it is still in h->d_fid).  The caller's arrays are left to the
// caller, who writes them once nothing can fail any more.
const double *finish_run(spx_handle *h, bool want_fid = false) {
    if (!h->stats_pending) {
        SPX_CUDA(cudaStreamSynchronize(h->stream));
        return nullptr;
    }
    h->stats_pending = false;
    const int64_t no = h->last_norient;
    const int S = h->chk_pending;
    h->chk_pending = 0;
    const size_t len = (size_t)h->chk_nsteps + 1, npts = len * h->nchan;
    struct Piece { size_t at; const void *src; size_t bytes; };
    std::vector<Piece> pieces;
    size_t total = 0;
    auto piece = [&](const void *src, size_t bytes) {
        pieces.push_back({total, src, bytes});
        total += (bytes + 15) & ~(size_t)15;
        return pieces.size() - 1;
    };
    const size_t p_status = piece(h->d_status.p, no * sizeof(int)), p_kused = piece(h->d_kused.p, no * sizeof(int)),
                 p_mused = piece(h->d_mused.p, no * sizeof(int)), p_mv = piece(h->d_matvecs.p, no * sizeof(long long)),
                 p_hw = piece(h->d_halfwidth.p, no * sizeof(double));
    size_t p_cst = 0, p_f64 = 0, p_f32 = 0, p_pw = 0, p_w = 0;
    if (S > 0) {
        p_cst = piece(h->d_chk_status.p, S * sizeof(int));
        p_f64 = piece(h->d_chk_fids.p, S * npts * sizeof(double2));
        for (int j = 0; j < S; ++j) {
            const size_t q = piece(reinterpret_cast<const float2 *>(h->d_fids.p) + (size_t)h->chk_index[j] * npts,
                                   npts * sizeof(float2));
            if (j == 0) p_f32 = q;
        }
        p_pw = piece(h->chk_out, npts * sizeof(double2));
        p_w = piece(h->chk_w, no * sizeof(double));
    }
    want_fid = want_fid && total + npts * sizeof(double2) <= kStage;
    const size_t p_fid = want_fid ? piece(h->d_fid.p, npts * sizeof(double2)) : 0;
    std::vector<unsigned char> pageable;
    unsigned char *base;
    if (total <= kStage) {
        base = h->stage.get(total, h->stream);
    } else {
        pageable.resize(total);
        base = pageable.data();
    }
    for (const Piece &q : pieces)
        SPX_CUDA(cudaMemcpyAsync(base + q.at, q.src, q.bytes, cudaMemcpyDeviceToHost, h->stream));
    SPX_CUDA(cudaStreamSynchronize(h->stream));
    auto words = [&](size_t q) { return base + pieces[q].at; };
    const int *status = reinterpret_cast<const int *>(words(p_status)), *kused = reinterpret_cast<const int *>(words(p_kused)),
              *mused = reinterpret_cast<const int *>(words(p_mused));
    const long long *mv = reinterpret_cast<const long long *>(words(p_mv));
    const double *hw = reinterpret_cast<const double *>(words(p_hw));
    float ms0 = 0, ms1 = 0;
    if (h->stats_timed) {
        SPX_CUDA(cudaEventElapsedTime(&ms0, h->ev[0], h->ev[1]));
        SPX_CUDA(cudaEventElapsedTime(&ms1, h->ev[1], h->ev[2]));
    }
    h->stats.kernel_ms = ms0;
    h->stats.reduce_ms = ms1;
    int64_t failed = 0, matvecs = 0;
    int maxk = 0, maxm = 0;
    double hmin = INFINITY, hmax = 0.0;
    int first_bad = -1, first_code = 0;
    for (int64_t o = 0; o < no; ++o) {
        if (status[o] != spx::kDevOk) {
            ++failed;
            if (first_bad < 0) { first_bad = (int)o; first_code = status[o]; }
        }
        matvecs += mv[o];
        maxk = std::max(maxk, kused[o]);
        maxm = std::max(maxm, mused[o]);
        hmin = std::min(hmin, hw[o]);
        hmax = std::max(hmax, hw[o]);
    }
    h->stats.matvecs = matvecs;
    h->stats.max_terms = maxk;
    h->stats.chunk_steps = maxm;
    h->stats.orientations_failed = failed;
    h->stats.min_half_width = hmin;
    h->stats.max_half_width = hmax;
    if (S > 0) {
        const int *cst = reinterpret_cast<const int *>(words(p_cst));
        bool ok = true;
        for (int j = 0; j < S; ++j) ok = ok && cst[j] == spx::kDevOk;
        // an FP64 re-run that failed its own series checks measures nothing
        h->stats.fp32_checked = ok ? S : 0;
        if (ok) {
            std::vector<const float2 *> f32(S);
            for (int j = 0; j < S; ++j) f32[j] = reinterpret_cast<const float2 *>(words(p_f32 + j));
            const double *w = reinterpret_cast<const double *>(words(p_w));
            double w2 = 0.0;
            for (int64_t o = 0; o < no; ++o) w2 += w[o] * w[o];
            const FP32Error e = fp32_error(f32, reinterpret_cast<const double2 *>(words(p_f64)),
                                           reinterpret_cast<const double2 *>(words(p_pw)), w2, S, len, h->nchan);
            h->stats.fp32_rel_error = e.orientation;
            h->stats.fp32_powder_error = e.powder;
        }
    }
    if (failed) {
        static const char *why[] = {"ok", "series longer than the coefficient table", "state norm grew (spectral bound violated)",
                                    "non-finite state", "launch configuration has too few threads"};
        const char *w = (first_code >= 0 && first_code <= 4) ? why[first_code] : "unknown device status";
        throw SpxError(SPX_ERR_SERIES, std::to_string(failed) + " orientation(s) failed, first #" +
                                           std::to_string(first_bad) + ": " + w);
    }
    return want_fid ? reinterpret_cast<const double *>(words(p_fid)) : nullptr;
}

void validate_run(spx_handle *h, int64_t n_orient, double dt, int64_t nsteps) {
    if (!h->have_system) throw SpxError(SPX_ERR_NO_SYSTEM, "no spin system uploaded");
    if (h->n_states > 0 && h->n_states != n_orient)
        throw SpxError(SPX_ERR_INVALID_ARGUMENT, "the grid size differs from the number of per-orientation initial states");
    if (n_orient < 1 || n_orient > (1LL << 30)) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "bad orientation count");
    if (!(dt > 0.0) || !std::isfinite(dt)) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "dt must be positive and finite");
    if (nsteps < 0 || nsteps > (1LL << 28)) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "bad step count");
    if (h->g_upper * dt > 1e4)
        throw SpxError(SPX_ERR_NORM, "|L*dt| exceeds 1e4: check L and dt (kernel/step.m:230-233)");
}

template <class F>
spx_status guarded(spx_handle *h, F f) {
    try {
        f();
        if (h) h->err.clear();
        return SPX_OK;
    } catch (const SpxError &e) {
        if (h) h->err = e.what();
        return e.code;
    } catch (const std::bad_alloc &) {
        if (h) h->err = "host allocation failed";
        return SPX_ERR_OUT_OF_MEMORY;
    } catch (const std::exception &e) {
        if (h) h->err = e.what();
        return SPX_ERR_INTERNAL;
    } catch (...) {
        if (h) h->err = "unknown failure";
        return SPX_ERR_INTERNAL;
    }
}

// ---------------------------------------------------------------------------
// Pulse sequences
// ---------------------------------------------------------------------------
// exp(-1i * theta * P) applied to many states (kernel/step.m: a hard pulse
// step(spin_system, pulse_op, rho, angle)), FP64: nsub substeps of a Taylor
// series with nterms terms, each substep's argument at most 1 in the 1-norm.
// One CTA per state at a time; x (the sum), t (the term) and u in shared memory.
__global__ void pulse_kernel(int n_states, int n_pad, const int *__restrict__ ptr, const int *__restrict__ col,
                             const double2 *__restrict__ val, double theta_sub, int nsub, int nterms,
                             double2 *states) {
    extern __shared__ double2 ps[];
    double2 *x = ps, *t = ps + n_pad, *u = ps + 2 * n_pad;
    for (int st = blockIdx.x; st < n_states; st += gridDim.x) {
        double2 *sv = states + (size_t)st * n_pad;
        for (int i = threadIdx.x; i < n_pad; i += blockDim.x) x[i] = sv[i];
        __syncthreads();
        for (int sub = 0; sub < nsub; ++sub) {
            for (int i = threadIdx.x; i < n_pad; i += blockDim.x) t[i] = x[i];
            __syncthreads();
            for (int k = 1; k <= nterms; ++k) {
                // u = (-1i theta / k) P t
                const double f = theta_sub / k;
                for (int i = threadIdx.x; i < n_pad; i += blockDim.x) {
                    double re = 0.0, im = 0.0;
                    for (int e = ptr[i]; e < ptr[i + 1]; ++e) {
                        const double2 a = val[e], b = t[col[e]];
                        re = fma(a.x, b.x, fma(-a.y, b.y, re));
                        im = fma(a.x, b.y, fma(a.y, b.x, im));
                    }
                    u[i] = make_double2(f * im, -f * re);       // -1i * f * (re + 1i im)
                }
                __syncthreads();
                for (int i = threadIdx.x; i < n_pad; i += blockDim.x) {
                    t[i] = u[i];
                    x[i].x += u[i].x;
                    x[i].y += u[i].y;
                }
                __syncthreads();
            }
        }
        for (int i = threadIdx.x; i < n_pad; i += blockDim.x) sv[i] = x[i];
        __syncthreads();
    }
}

// Upload a pulse superoperator (CSC, the caller's basis order) as CSR rows in
// the sliced order of the uploaded system.
void upload_pulse(spx_handle *h, const spx_csc *P, PulseOp &op) {
    check_csc(P, h->n, "pulse_op");
    const int n_pad = h->n_pad;
    std::vector<std::vector<std::pair<int, double2>>> rows(n_pad);
    std::vector<double> colsum(h->n, 0.0);
    for_each_entry(P, [&](int64_t r, int64_t c, Cplx v) {
        if (v.re == 0.0 && v.im == 0.0) return;
        rows[h->row_of[r]].push_back({h->row_of[c], make_double2(v.re, v.im)});
        colsum[c] += std::hypot(v.re, v.im);
    });
    std::vector<int> ptr(n_pad + 1, 0), col;
    std::vector<double2> val;
    for (int i = 0; i < n_pad; ++i) {
        for (auto &e : rows[i]) { col.push_back(e.first); val.push_back(e.second); }
        ptr[i + 1] = (int)col.size();
    }
    if (col.empty()) { col.push_back(0); val.push_back(make_double2(0, 0)); }
    SPX_CUDA(cudaSetDevice(h->device));
    op.ptr.upload(ptr, h->stream);
    op.col.upload(col, h->stream);
    op.val.upload(val, h->stream);
    op.norm1 = colsum.empty() ? 0.0 : *std::max_element(colsum.begin(), colsum.end());
}

// exp(-1i * theta * P) on n_states states of n_pad entries (sliced order).
void apply_pulse(spx_handle *h, const PulseOp &op, double theta, int64_t n_states, double2 *states) {
    const double x = op.norm1 * std::fabs(theta);
    if (!(x < 2147483647.0)) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "pulse operator times angle overflows");
    const int nsub = std::max(1, (int)std::ceil(x));
    const int nterms = 25;                     // 1 / 25! < 1e-25 per substep
    const size_t smem = 3 * (size_t)h->n_pad * sizeof(double2);
    if (smem > h->smem_optin) throw SpxError(SPX_ERR_UNSUPPORTED, "pulse states do not fit shared memory");
    SPX_CUDA(cudaFuncSetAttribute(reinterpret_cast<const void *>(&pulse_kernel),
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int grid = (int)std::min<int64_t>(n_states, (int64_t)h->sm_count * 2);
    ++h->launches;
    pulse_kernel<<<grid, 256, smem, h->stream>>>((int)n_states, h->n_pad, op.ptr.p, op.col.p, op.val.p, theta / nsub,
                                                 nsub, nterms, states);
    SPX_CUDA(cudaGetLastError());
}

// A pulse program on the evolution core: hard pulses exp(-1i*angle*P) and
// evolution segments, each segment one powder run that starts from the
// previous segment's final states (per orientation; before the first segment
// the pulses act on the single rho0, or on the per-orientation initial
// states when they are set).  Recorded segments append their powder FID
// (nsteps+1 points) to fid.
void upload_grid(spx_handle *h, int64_t n_orient, const double *alphas, const double *betas, const double *gammas,
                 const double *weights) {
    h->d_grid.reserve(4 * (size_t)n_orient);
    double *g = h->d_grid.p;
    const size_t b = (size_t)n_orient * sizeof(double);
    SPX_CUDA(cudaMemcpyAsync(g, alphas, b, cudaMemcpyHostToDevice, h->stream));
    SPX_CUDA(cudaMemcpyAsync(g + n_orient, betas, b, cudaMemcpyHostToDevice, h->stream));
    SPX_CUDA(cudaMemcpyAsync(g + 2 * n_orient, gammas, b, cudaMemcpyHostToDevice, h->stream));
    SPX_CUDA(cudaMemcpyAsync(g + 3 * n_orient, weights, b, cudaMemcpyHostToDevice, h->stream));
}

// ---------------------------------------------------------------------------
// Pulse sequences on the coupled states: the rows that L and the pulses
// connect to both the coil and the initial state, in an order of their own
// (state arrays of n entries), propagated one set of L-connected rows at a
// time.  A hard pulse is one sparse product with its exponential.
// ---------------------------------------------------------------------------
struct HostCsr {
    std::vector<int> ptr, col;
    std::vector<double2> val;
};
struct SparseOp {
    DevBuf<int> ptr, col;
    DevBuf<double2> val;
    void upload(const HostCsr &m, cudaStream_t s) {
        ptr.upload(m.ptr, s);
        col.upload(m.col.empty() ? std::vector<int>{0} : m.col, s);
        val.upload(m.val.empty() ? std::vector<double2>{make_double2(0, 0)} : m.val, s);
        SPX_CUDA(cudaStreamSynchronize(s));           // pageable sources
    }
};

double2 cmul(double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }

constexpr int kPulseBlock = 64;        // largest set of states that a pulse operator couples here

// exp(-1i theta P) of a pulse operator given as rows, one connected set of
// states at a time (a spin's rotation couples a few): scaling and squaring of
// the Taylor series, 1/2^s scaled to a 1-norm of at most one half.  Of a rotation
// that was scaled down, entries at or below 1e-15 are rounding residues and are
// dropped; a smaller rotation's small entries are what it does.
// False if a set is larger than kPulseBlock.
bool pulse_exponential(const std::vector<std::vector<std::pair<int, double2>>> &rows, double theta, HostCsr &out) {
    const int n = (int)rows.size();
    spx::Components comp(n);
    for (int i = 0; i < n; ++i)
        for (auto &e : rows[i]) comp.join(i, e.first);
    std::vector<std::vector<int>> sets(n);
    for (int i = 0; i < n; ++i) sets[comp.find(i)].push_back(i);
    std::vector<std::vector<std::pair<int, double2>>> res(n);
    std::vector<int> at(n, -1);
    for (auto &set : sets) {
        const int m = (int)set.size();
        if (m == 0) continue;
        if (m > kPulseBlock) return false;
        for (int q = 0; q < m; ++q) at[set[q]] = q;
        std::vector<double2> A((size_t)m * m, make_double2(0, 0)), X(A), T(A), Y(A);
        for (int q = 0; q < m; ++q)
            for (auto &e : rows[set[q]]) {            // -1i theta P
                double2 &a = A[(size_t)q * m + at[e.first]];
                a.x += theta * e.second.y;
                a.y -= theta * e.second.x;
            }
        double norm = 0.0;
        for (int c = 0; c < m; ++c) {
            double sum = 0.0;
            for (int r = 0; r < m; ++r) sum += std::hypot(A[(size_t)r * m + c].x, A[(size_t)r * m + c].y);
            if (!(sum <= norm)) norm = sum;           // NaN too
        }
        if (!std::isfinite(norm)) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "pulse operator times angle overflows");
        int sq = 0;
        while (norm > 0.5) { norm *= 0.5; ++sq; }
        const double f = std::ldexp(1.0, -sq);
        for (auto &a : A) { a.x *= f; a.y *= f; }
        auto product = [&](const std::vector<double2> &a, const std::vector<double2> &b, std::vector<double2> &c) {
            for (int r = 0; r < m; ++r)
                for (int q = 0; q < m; ++q) {
                    double2 sum = make_double2(0, 0);
                    for (int k = 0; k < m; ++k) {
                        const double2 v = cmul(a[(size_t)r * m + k], b[(size_t)k * m + q]);
                        sum.x += v.x;
                        sum.y += v.y;
                    }
                    c[(size_t)r * m + q] = sum;
                }
        };
        for (int q = 0; q < m; ++q) X[(size_t)q * m + q] = T[(size_t)q * m + q] = make_double2(1, 0);
        for (int k = 1; k <= 18; ++k) {               // 0.5^19 / 19! < 1e-22
            product(T, A, Y);
            for (size_t e = 0; e < Y.size(); ++e) {
                T[e] = make_double2(Y[e].x / k, Y[e].y / k);
                X[e].x += T[e].x;
                X[e].y += T[e].y;
            }
        }
        for (int q = 0; q < sq; ++q) { product(X, X, Y); X.swap(Y); }
        const double residue = sq > 0 ? 1e-15 : 0.0;
        for (int r = 0; r < m; ++r)
            for (int c = 0; c < m; ++c) {
                const double2 v = X[(size_t)r * m + c];
                if (std::fabs(v.x) > residue || std::fabs(v.y) > residue) res[set[r]].push_back({set[c], v});
            }
    }
    out = HostCsr{};
    out.ptr.assign(n + 1, 0);
    for (int i = 0; i < n; ++i) {
        for (auto &e : res[i]) { out.col.push_back(e.first); out.val.push_back(e.second); }
        out.ptr[i + 1] = (int)out.col.size();
    }
    return true;
}

// y = M x for n_states states of n entries each.
__global__ void sparse_states_kernel(int64_t n_states, int n, const int *__restrict__ ptr, const int *__restrict__ col,
                                     const double2 *__restrict__ val, const double2 *__restrict__ x, double2 *y) {
    const int64_t total = n_states * n;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = q / n;
        const int i = (int)(q - o * n);
        double re = 0.0, im = 0.0;
        for (int e = ptr[i]; e < ptr[i + 1]; ++e) {
            const double2 a = val[e], b = x[o * n + col[e]];
            re = fma(a.x, b.x, fma(-a.y, b.y, re));
            im = fma(a.x, b.y, fma(a.y, b.x, im));
        }
        y[q] = make_double2(re, im);
    }
}

// out[o][i] = in[o][rows[i]], states of n_in entries.
__global__ void gather_states_kernel(int64_t n_states, int n, int n_in, const int *__restrict__ rows,
                                     const double2 *__restrict__ in, double2 *out) {
    const int64_t total = n_states * n;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = q / n;
        out[q] = in[o * n_in + rows[q - o * n]];
    }
}

unsigned state_blocks(const spx_handle *h, int64_t items) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((items + 255) / 256, (int64_t)h->sm_count * 16));
}

// The rows a sequence moves, and its pulse operators on them.
struct CoupledSequence {
    std::vector<int> rows, at;       // system rows; a row's place among them, or -1
    std::vector<std::vector<std::vector<std::pair<int, double2>>>> pulses;
    int n() const { return (int)rows.size(); }

    // Restrict the sequence to the rows that L and the pulses connect.
    CoupledSequence(spx_handle *h, const std::vector<const spx_csc *> &ops) {
        spx::Components comp(h->n);
        for (int i = 0; i < h->n; ++i) comp.join(i, h->component[i]);
        for (const spx_csc *P : ops) {
            check_csc(P, h->n, "pulse_op");
            for_each_entry(P, [&](int64_t r, int64_t c, Cplx v) {
                if (v.re != 0.0 || v.im != 0.0) comp.join(h->row_of[r], h->row_of[c]);
            });
        }
        std::vector<int> label(h->n);
        for (int i = 0; i < h->n; ++i) label[i] = comp.find(i);
        rows = live_rows(h, label, start_rows(h));
        at.assign(h->n, -1);
        for (size_t i = 0; i < rows.size(); ++i) at[rows[i]] = (int)i;
        for (const spx_csc *P : ops) {
            pulses.emplace_back(rows.size());
            for_each_entry(P, [&](int64_t r, int64_t c, Cplx v) {
                const int i = at[h->row_of[r]], j = at[h->row_of[c]];
                if (i >= 0 && j >= 0 && (v.re != 0.0 || v.im != 0.0)) pulses.back()[i].push_back({j, make_double2(v.re, v.im)});
            });
        }
    }
    // places of all rows of the L-components that hold one of these places
    std::vector<char> closure(const spx_handle *h, const std::vector<char> &places) const {
        std::vector<char> hit(h->n, 0), out(rows.size(), 0);
        for (size_t i = 0; i < rows.size(); ++i)
            if (places[i]) hit[h->component[rows[i]]] = 1;
        for (size_t i = 0; i < rows.size(); ++i) out[i] = hit[h->component[rows[i]]];
        return out;
    }
    std::vector<char> coil_places(const spx_handle *h) const {
        std::vector<char> p(rows.size(), 0);
        for (int r : h->coil_row_host)
            if (at[r] >= 0) p[at[r]] = 1;
        return closure(h, p);
    }
    void plan(spx_handle *h, const std::vector<char> &places, bool detect, BlockPlan &out) const {
        std::vector<int> r, pos;
        for (size_t i = 0; i < rows.size(); ++i)
            if (places[i]) { r.push_back(rows[i]); pos.push_back((int)i); }
        build_plan(h, r, &pos, detect, out);
    }
};

// Tables of a sequence hold for any step count: their chunks are as long as
// the tables allow.
constexpr int64_t kAnySteps = (int64_t)1 << 28;

// One set of rows of a sequence with its bounds and tables.
struct SequenceGroup {
    BlockPlan plan;
    BlockBufs bufs;
    Config c;
    double table_dt = 0.0;           // time step of the tables held (0: none)
    bool bounded = false;
};

// Propagates a group over nsteps steps of dt: bounds on the first call, tables
// whenever the time step changes.  first: place of the orientations among the
// call's (status and halfwidth are given where they start).  False, and nothing
// launched, if the series is too long for the coupled-state kernels' shared
// memory (|L| dt of several thousand): the whole call then starts again on the
// whole system.
bool run_group(spx_handle *h, SequenceGroup &g, spx::DevSystem &sys, spx::BlockRun r, int64_t n_orient,
               const double *const (&angles)[3], double dt, int64_t nsteps, double tol, int lanczos_its, bool f64, bool traj,
               int *status, double *halfwidth, int64_t first = 0) {
    if (!g.bounded || g.table_dt != dt) {
        Config c{};
        c.tol = tol;
        if (!configure_block(h, g.plan, n_orient, dt, kAnySteps, f64, 0.0, 0, traj ? spx::kBlockTraj : 256, traj, c))
            return false;
        g.c = c;
        reserve_block(g.bufs, n_orient, f64, c);
    }
    const Config &c = g.c;
    BlockBufs &b = g.bufs;
    block_run_buffers(r, c, b.centre.p, b.extent.p, b.lev_half.p, b.lev.p, b.kcut.p, b.table.p, f64 ? nullptr : b.tablef.p);
    if (saves_block(n_orient, f64, c)) r.saved = b.saved.p;
    r.n_orient = (int)n_orient; r.alpha = angles[0]; r.beta = angles[1]; r.gamma = angles[2];
    r.dt = dt; r.lanczos_its = lanczos_its > 0 ? lanczos_its : 32;
    r.max_im_diag = h->max_im_diag; r.halfwidth = halfwidth;
    r.nchan = 1; r.status = status;
    r.kused = h->d_kused.p + first; r.mused = h->d_mused.p + first; r.matvecs = h->d_matvecs.p + first;
    if (!g.bounded) launch_bounds(h, c, sys, r, h->stream);
    g.bounded = true;
    if (g.table_dt != dt) {
        r.nsteps = (int)kAnySteps;
        launch_tables(h, c, r, h->stream);
        g.table_dt = dt;
    }
    r.nsteps = (int)nsteps;
    launch_propagation(h, c, sys, r, h->stream);
    return true;
}

// Statuses of a sequence's launches (after a synchronisation).
void check_statuses(spx_handle *h, int64_t n_orient, int64_t launches) {
    std::vector<int> st((size_t)(n_orient * launches));
    SPX_CUDA(cudaMemcpy(st.data(), h->d_seq_status.p, st.size() * sizeof(int), cudaMemcpyDeviceToHost));
    for (size_t q = 0; q < st.size(); ++q)
        if (st[q] != spx::kDevOk)
            throw SpxError(SPX_ERR_SERIES, "a segment failed its series checks (status " + std::to_string(st[q]) +
                                               ", orientation #" + std::to_string(q % n_orient) + ")");
}

// The run on the coupled states, or false if they do not qualify (the caller
// then runs the whole system).  Arguments are validated and the grid is on the
// device; total: recorded points.
bool run_coupled_sequence(spx_handle *h, int64_t n_orient, const std::vector<const spx_csc *> &pulse_ops,
                          const std::vector<spx_seq_op> &ops, const RunOptions &o, int64_t total, double *fid,
                          double *fids_per_orient) {
    if (forced_shape(o)) return false;
    for (auto &q : ops)
        if (q.kind == SPX_SEQ_EVOLVE && may_diverge(h, q.dt, q.nsteps)) return false;
    CoupledSequence seq(h, pulse_ops);
    const int n = seq.n();
    if (n == 0) return false;
    int last_evolve = -1;
    int64_t evolves = 0, max_steps = 0;
    for (size_t i = 0; i < ops.size(); ++i)
        if (ops[i].kind == SPX_SEQ_EVOLVE) {
            last_evolve = (int)i;
            ++evolves;
            max_steps = std::max(max_steps, ops[i].nsteps);
        }
    if (last_evolve < 0) return false;
    // sets of rows: the coil's components together, every other large
    // component alone, the small ones together
    std::vector<std::unique_ptr<SequenceGroup>> groups;
    const std::vector<char> coil = seq.coil_places(h);
    {
        std::vector<std::vector<int>> comps(h->n);
        for (int i = 0; i < n; ++i)
            if (!coil[i]) comps[h->component[seq.rows[i]]].push_back(i);
        std::vector<char> small(n, 0);
        int count = 0;
        auto flush = [&](std::vector<char> &places) {
            groups.push_back(std::make_unique<SequenceGroup>());
            seq.plan(h, places, false, groups.back()->plan);
            std::fill(places.begin(), places.end(), 0);
        };
        for (auto &c : comps) {
            if (c.empty()) continue;
            if (c.size() > 24) {
                std::vector<char> one(n, 0);
                for (int i : c) one[i] = 1;
                flush(one);
                continue;
            }
            if (count + (int)c.size() > spx::kBlockRows) { flush(small); count = 0; }
            for (int i : c) small[i] = 1;
            count += (int)c.size();
        }
        if (count) flush(small);
        groups.push_back(std::make_unique<SequenceGroup>());      // the coil's last
        seq.plan(h, coil, true, groups.back()->plan);
    }
    for (auto &g : groups)
        if (!g->plan.ok) return false;
    // the pulses' exponentials
    std::map<std::pair<int, double>, std::unique_ptr<SparseOp>> turns;
    for (auto &q : ops)
        if (q.kind == SPX_SEQ_PULSE && !turns.count({q.pulse, q.angle})) {
            HostCsr m;
            if (!pulse_exponential(seq.pulses[q.pulse], q.angle, m)) return false;
            auto op = std::make_unique<SparseOp>();
            op->upload(m, h->stream);
            turns[{q.pulse, q.angle}] = std::move(op);
        }
    const bool f64 = o.precision == SPX_FP64;
    const size_t vec = f64 ? sizeof(double2) : sizeof(float2);
    const double *g = h->d_grid.p;
    const double *const angles[3] = {g, g + n_orient, g + 2 * n_orient};
    const size_t ns = (size_t)n_orient * n;
    const bool own_states = h->n_states > 0;
    h->d_seq[0].reserve(ns);
    h->d_seq[1].reserve(ns);
    h->d_seq_rho.reserve(2 * (size_t)n);
    h->d_fid.reserve((size_t)std::max<int64_t>(total, 1));
    h->d_fids.reserve((size_t)(max_steps + 1) * n_orient * vec);
    h->d_part.reserve((size_t)((n_orient + kPowderGroup - 1) / kPowderGroup) * (max_steps + 1));
    h->d_status.reserve(n_orient);
    h->d_kused.reserve(n_orient);
    h->d_mused.reserve(n_orient);
    h->d_matvecs.reserve(n_orient);
    h->d_halfwidth.reserve(n_orient);
    h->d_seq_status.reserve((size_t)(n_orient * evolves * (int64_t)groups.size()));
    spx::DevSystem sys = device_system(h);
    DevBuf<int> drows;
    int cur = 0, rcur = 0;
    bool per_orient = own_states;
    if (own_states) {
        drows.upload(seq.rows, h->stream);
        ++h->launches;
        gather_states_kernel<<<state_blocks(h, ns), 256, 0, h->stream>>>(n_orient, n, h->n_pad, drows.p, h->d_rho0s.p,
                                                                          h->d_seq[0].p);
        SPX_CUDA(cudaGetLastError());
    } else {
        std::vector<double2> r0(n);
        for (int i = 0; i < n; ++i) r0[i] = h->rho0_host[seq.rows[i]];
        SPX_CUDA(cudaMemcpyAsync(h->d_seq_rho.p, r0.data(), n * sizeof(double2), cudaMemcpyHostToDevice, h->stream));
        SPX_CUDA(cudaStreamSynchronize(h->stream));
    }
    Config whole{};
    int64_t at = 0, launched = 0;
    std::vector<std::vector<unsigned char>> each;      // recorded segments, until all of them are known to be good
    SPX_CUDA(cudaEventRecord(h->ev[0], h->stream));
    for (size_t i = 0; i < ops.size(); ++i) {
        const spx_seq_op &q = ops[i];
        if (q.kind == SPX_SEQ_PULSE) {
            const SparseOp &op = *turns[{q.pulse, q.angle}];
            double2 *x = per_orient ? h->d_seq[cur].p : h->d_seq_rho.p + (size_t)rcur * n;
            double2 *y = per_orient ? h->d_seq[cur ^ 1].p : h->d_seq_rho.p + (size_t)(rcur ^ 1) * n;
            const int64_t cnt = per_orient ? n_orient : 1;
            ++h->launches;
            sparse_states_kernel<<<state_blocks(h, cnt * n), 256, 0, h->stream>>>(cnt, n, op.ptr.p, op.col.p, op.val.p, x, y);
            SPX_CUDA(cudaGetLastError());
            if (per_orient) cur ^= 1; else rcur ^= 1;
            continue;
        }
        // the whole system's configuration: what it refuses stays refused
        whole = choose_config(h, n_orient, q.dt, q.nsteps, o, 0);
        const bool last = (int)i == last_evolve;
        for (size_t k = 0; k < groups.size(); ++k) {
            const bool detects = k + 1 == groups.size();
            if (last && !detects) continue;                        // nothing after it reads these states
            spx::BlockRun r{};
            if (per_orient) r.rho0s = h->d_seq[cur].p;
            else r.rho0 = h->d_seq_rho.p + (size_t)rcur * n;
            r.state_stride = (size_t)n;
            r.state_out = last ? nullptr : h->d_seq[cur ^ 1].p;
            r.fids = h->d_fids.p;
            int *status = last ? h->d_status.p : h->d_seq_status.p + (size_t)(launched++) * n_orient;
            SequenceGroup &grp = *groups[k];
            double *half = h->d_halfwidth.p;
            if (!detects) {
                grp.bufs.halfwidth.reserve(n_orient);
                half = grp.bufs.halfwidth.p;
            }
            if (!run_group(h, grp, sys, r, n_orient, angles, q.dt, q.nsteps, whole.tol, o.lanczos_its, f64, false, status,
                           half))
                return false;
        }
        if (q.record) {
            const size_t np = (size_t)q.nsteps + 1;
            launch_powder_sum(h, f64, h->d_fids.p, g + 3 * n_orient, n_orient, np, h->d_part.p, h->d_fid.p + at);
            if (fids_per_orient) {
                // this segment's FIDs of every orientation
                each.emplace_back(np * (size_t)n_orient * vec);
                SPX_CUDA(cudaMemcpyAsync(each.back().data(), h->d_fids.p, each.back().size(), cudaMemcpyDeviceToHost,
                                         h->stream));
                SPX_CUDA(cudaStreamSynchronize(h->stream));
            }
            at += (int64_t)np;
        }
        cur ^= 1;
        per_orient = true;
    }
    SPX_CUDA(cudaEventRecord(h->ev[1], h->stream));
    SPX_CUDA(cudaEventRecord(h->ev[2], h->stream));
    h->stats_timed = true;
    whole.blk = groups.back()->c.blk;
    describe_run(h, n_orient, ops[last_evolve].nsteps, o.precision, whole);
    h->stats_pending = true;
    h->last_norient = n_orient;
    h->chk_pending = 0;
    finish_run(h);
    if (launched) check_statuses(h, n_orient, launched);
    if (total > 0) SPX_CUDA(cudaMemcpy(fid, h->d_fid.p, (size_t)total * sizeof(double2), cudaMemcpyDeviceToHost));
    at = 0;
    for (const std::vector<unsigned char> &seg : each) {
        // into each orientation's row
        const size_t np = seg.size() / ((size_t)n_orient * vec);
        for (int64_t w = 0; w < n_orient; ++w)
            for (size_t j = 0; j < np; ++j) {
                const size_t e = (size_t)w * np + j;
                double2 v;
                if (f64) v = reinterpret_cast<const double2 *>(seg.data())[e];
                else {
                    const float2 f = reinterpret_cast<const float2 *>(seg.data())[e];
                    v = make_double2(f.x, f.y);
                }
                fids_per_orient[2 * ((size_t)w * total + at + j)] = v.x;
                fids_per_orient[2 * ((size_t)w * total + at + j) + 1] = v.y;
            }
        at += (int64_t)np;
    }
    return true;
}

void run_sequence(spx_handle *h, int64_t n_orient, const double *alphas, const double *betas, const double *gammas,
                  const double *weights, int32_t n_pulse, const spx_csc *pulse_ops, int32_t n_ops,
                  const spx_seq_op *ops, const RunOptions &o, double *fid, double *fids_per_orient = nullptr) {
    if (h->nchan != 1) throw SpxError(SPX_ERR_UNSUPPORTED, "pulse sequences take one coil");
    if (h->n_states > 0 && h->n_states != n_orient)
        throw SpxError(SPX_ERR_INVALID_ARGUMENT, "the grid size differs from the number of per-orientation initial states");
    if (n_pulse < 0 || n_ops < 0 || (n_pulse > 0 && !pulse_ops) || (n_ops > 0 && !ops))
        throw SpxError(SPX_ERR_INVALID_ARGUMENT, "bad pulse or operation arrays");
    int64_t max_steps = 0, total = 0;
    for (int i = 0; i < n_ops; ++i) {
        const spx_seq_op &q = ops[i];
        if (q.kind == SPX_SEQ_EVOLVE && q.record) total += q.nsteps + 1;
        if (q.kind == SPX_SEQ_PULSE) {
            if (q.pulse < 0 || q.pulse >= n_pulse) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "pulse index out of range");
            if (!std::isfinite(q.angle)) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "non-finite pulse angle");
        } else if (q.kind == SPX_SEQ_EVOLVE) {
            validate_run(h, n_orient, q.dt, q.nsteps);
            max_steps = std::max(max_steps, q.nsteps);
        } else {
            throw SpxError(SPX_ERR_INVALID_ARGUMENT, "unknown sequence operation");
        }
    }
    if (n_orient < 1) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "bad orientation count");
    {
        std::vector<const spx_csc *> list;
        for (int k = 0; k < n_pulse; ++k) list.push_back(&pulse_ops[k]);
        upload_grid(h, n_orient, alphas, betas, gammas, weights);
        if (run_coupled_sequence(h, n_orient, list, std::vector<spx_seq_op>(ops, ops + n_ops), o, total, fid,
                                 fids_per_orient))
            return;
    }
    h->pulses.clear();
    for (int k = 0; k < n_pulse; ++k) {
        h->pulses.push_back(std::make_unique<PulseOp>());
        upload_pulse(h, &pulse_ops[k], *h->pulses.back());
    }
    double *g = h->d_grid.p;
    const size_t ns = (size_t)n_orient * h->n_pad;
    h->d_seq[0].reserve(ns);
    h->d_seq[1].reserve(ns);
    h->d_seq_rho.reserve(h->n_pad);
    h->d_fid.reserve((size_t)max_steps + 1);
    SPX_CUDA(cudaMemcpyAsync(h->d_seq_rho.p, h->d_rho0.p, h->n_pad * sizeof(double2), cudaMemcpyDeviceToDevice,
                             h->stream));
    // states differ per orientation after the first segment, or from the
    // start with per-orientation initial states (n_states == n_orient, checked)
    bool per_orient = h->n_states > 0;
    if (per_orient)
        SPX_CUDA(cudaMemcpyAsync(h->d_seq[0].p, h->d_rho0s.p, ns * sizeof(double2), cudaMemcpyDeviceToDevice,
                                 h->stream));
    int cur = 0;
    size_t at = 0;
    for (int i = 0; i < n_ops; ++i) {
        const spx_seq_op &q = ops[i];
        if (q.kind == SPX_SEQ_PULSE) {
            if (per_orient) apply_pulse(h, *h->pulses[q.pulse], q.angle, n_orient, h->d_seq[cur].p);
            else apply_pulse(h, *h->pulses[q.pulse], q.angle, 1, h->d_seq_rho.p);
            continue;
        }
        RunIO io;
        if (per_orient) io.rho0s = h->d_seq[cur].p;
        else io.rho0 = h->d_seq_rho.p;
        io.state_out = h->d_seq[cur ^ 1].p;
        const Config c = choose_config(h, n_orient, q.dt, q.nsteps, o, 0);
        launch_powder(h, n_orient, g, g + n_orient, g + 2 * n_orient, g + 3 * n_orient, q.dt, q.nsteps, o, h->d_fid.p,
                      c, 0, true, io);
        finish_run(h);
        if (q.record) {
            const size_t np = (size_t)q.nsteps + 1;
            SPX_CUDA(cudaMemcpy(fid + 2 * at, h->d_fid.p, np * sizeof(double2), cudaMemcpyDeviceToHost));
            if (fids_per_orient) {
                // this segment's FIDs of every orientation, into each orientation's row
                std::vector<double2> tmp(np * (size_t)n_orient);
                if (o.precision == SPX_FP64) {
                    SPX_CUDA(cudaMemcpy(tmp.data(), h->d_fids.p, tmp.size() * sizeof(double2), cudaMemcpyDeviceToHost));
                } else {
                    std::vector<float2> t32(tmp.size());
                    SPX_CUDA(cudaMemcpy(t32.data(), h->d_fids.p, t32.size() * sizeof(float2), cudaMemcpyDeviceToHost));
                    for (size_t i = 0; i < t32.size(); ++i) tmp[i] = make_double2(t32[i].x, t32[i].y);
                }
                for (int64_t or_ = 0; or_ < n_orient; ++or_)
                    for (size_t j = 0; j < np; ++j) {
                        const double2 v = tmp[(size_t)or_ * np + j];
                        fids_per_orient[2 * ((size_t)or_ * total + at + j)] = v.x;
                        fids_per_orient[2 * ((size_t)or_ * total + at + j) + 1] = v.y;
                    }
            }
            at += np;
        }
        cur ^= 1;
        per_orient = true;
    }
}

// experiments/cpmg.m: a 90-degree pulse, npoints-1 steps of acquisition, then
// nloops times (180-degree pulse, 2*npoints-1 steps), the FIDs concatenated
// (npoints + 2*npoints*nloops points).
void run_cpmg(spx_handle *h, int64_t n_orient, const double *alphas, const double *betas, const double *gammas,
              const double *weights, double dt, int64_t npoints, int32_t nloops, const spx_csc *pulse_op,
              const RunOptions &o, double *fid, double *fids_per_orient) {
    // experiments/cpmg.m:77-90: both positive integers
    if (npoints < 1 || nloops < 1) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "npoints and nloops must be positive");
    std::vector<spx_seq_op> prog;
    auto pulse = [&](double angle) {
        spx_seq_op q{};
        q.kind = SPX_SEQ_PULSE;
        q.pulse = 0;
        q.angle = angle;
        prog.push_back(q);
    };
    auto evolve = [&](int64_t nsteps) {
        spx_seq_op q{};
        q.kind = SPX_SEQ_EVOLVE;
        q.nsteps = nsteps;
        q.dt = dt;
        q.record = 1;
        prog.push_back(q);
    };
    pulse(M_PI / 2);
    evolve(npoints - 1);
    for (int n = 0; n < nloops; ++n) {
        pulse(M_PI);
        evolve(2 * npoints - 1);
    }
    run_sequence(h, n_orient, alphas, betas, gammas, weights, 1, pulse_op, (int32_t)prog.size(), prog.data(), o, fid,
                 fids_per_orient);
}

// Echo detection (experiments/esr_dipolar/eseem.m): the stack of half-echo
// states is pulsed and refocused, point n being coil' U^n Pi U^n rho1 with
// U = exp(-1i L tau), rho1 the 90-degree-pulsed rho0 and Pi = exp(-1i pi P).
// With v_n = (U')^n coil = exp(1i L' n tau) coil, point n is v_n' * Pi * u_n,
// u_n = U^n rho1: two trajectories (L, and -H + 1i R for the adjoint) and one
// sparse bilinear form per orientation and step, instead of the reference's
// n-step refocusing of every column.

// The adjoint generator -(H) + 1i R from the uploaded streams: every value is
// negated except the imaginary diagonal of stream 0 (the relaxation rates).
__global__ void negate_streams_kernel(int64_t n_ell, const double *re, const double *im, double *nre, double *nim,
                                      int64_t n_diag, int n_pad, const double2 *diag, double2 *ndiag) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_ell; i += stride) {
        nre[i] = -re[i];
        if (im) nim[i] = -im[i];
    }
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_diag; i += stride) {
        const double2 d = diag[i];
        ndiag[i] = make_double2(-d.x, i < n_pad ? d.y : -d.y);
    }
}

__global__ void identity_kernel(int n_pad, double2 *a) {
    const int64_t n2 = (int64_t)n_pad * n_pad;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += (int64_t)gridDim.x * blockDim.x)
        a[i] = make_double2(i / n_pad == i % n_pad ? 1.0 : 0.0, 0.0);
}

// out[o][n] = sum_i conj(v[o][n][i]) * (Pi u[o][n])[i], one warp per (o, n).
__global__ void echo_form_kernel(int n_orient, int npoints, int n_pad, const int *__restrict__ ptr,
                                 const int *__restrict__ col, const double2 *__restrict__ val,
                                 const double2 *__restrict__ u, const double2 *__restrict__ v, int reverse,
                                 double2 *out) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t)n_orient * npoints;
    for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nw;
         w += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        // v point npoints-1-j of the same orientation when reverse
        const int64_t wv = reverse ? w - 2 * (w % npoints) + npoints - 1 : w;
        const double2 *uu = u + w * n_pad, *vv = v + wv * n_pad;
        double re = 0.0, im = 0.0;
        for (int i = lane; i < n_pad; i += 32) {
            double wr = 0.0, wi = 0.0;
            for (int e = ptr[i]; e < ptr[i + 1]; ++e) {
                const double2 a = val[e], b = uu[col[e]];
                wr = fma(a.x, b.x, fma(-a.y, b.y, wr));
                wi = fma(a.x, b.y, fma(a.y, b.x, wi));
            }
            const double2 c = vv[i];                 // conj(c) * w
            re = fma(c.x, wr, fma(c.y, wi, re));
            im = fma(c.x, wi, fma(-c.y, wr, im));
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            re += __shfl_xor_sync(0xffffffffu, re, o);
            im += __shfl_xor_sync(0xffffffffu, im, o);
        }
        if (lane == 0) out[w] = make_double2(re, im);
    }
}

// fid[n] = sum_o w[o] f[o][n] in orientation order (powder.m:280-287).
__global__ void echo_powder_kernel(int n_orient, int npoints, const double2 *f, const double *w, double2 *fid) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= npoints) return;
    double re = 0.0, im = 0.0;
    for (int o = 0; o < n_orient; ++o) {
        const double2 v = f[(size_t)o * npoints + n];
        re = fma(w[o], v.x, re);
        im = fma(w[o], v.y, im);
    }
    fid[n] = make_double2(re, im);
}

constexpr int kTrajChunk = 4;       // steps per chunk of trajectory outputs (falls back to 2, 1)

// Pi = exp(-1i*theta*P) column by column, kept as CSR in the echo buffers
// (entries above 1e-15; Pi is unitary, so they are at most 1).
void upload_echo_propagator(spx_handle *h, const PulseOp &P, double theta) {
    const int n_pad = h->n_pad;
    DevBuf<double2> dense;
    dense.reserve((size_t)n_pad * n_pad);
    ++h->launches;
    identity_kernel<<<h->sm_count * 4, 256, 0, h->stream>>>(n_pad, dense.p);
    SPX_CUDA(cudaGetLastError());
    apply_pulse(h, P, theta, n_pad, dense.p);
    std::vector<double2> hd((size_t)n_pad * n_pad);
    SPX_CUDA(cudaMemcpyAsync(hd.data(), dense.p, hd.size() * sizeof(double2), cudaMemcpyDeviceToHost, h->stream));
    SPX_CUDA(cudaStreamSynchronize(h->stream));
    std::vector<int> ptr(n_pad + 1, 0), col;
    std::vector<double2> val;
    for (int i = 0; i < n_pad; ++i) {
        for (int j = 0; j < n_pad; ++j) {
            const double2 v = hd[(size_t)j * n_pad + i];         // column j holds Pi e_j
            if (std::fabs(v.x) > 1e-15 || std::fabs(v.y) > 1e-15) {
                col.push_back(j);
                val.push_back(v);
            }
        }
        ptr[i + 1] = (int)col.size();
    }
    if (col.empty()) { col.push_back(0); val.push_back(make_double2(0, 0)); }
    h->d_echo_ptr.upload(ptr, h->stream);
    h->d_echo_col.upload(col, h->stream);
    h->d_echo_val.upload(val, h->stream);
}

// The adjoint generator -H + 1i R in the d_neg_* streams: propagating under it
// is propagating under the adjoint of exp(-1i L dt).
void negate_generator(spx_handle *h) {
    const int64_t n_ell = (int64_t)h->nstreams * h->ell_len, n_diag = (int64_t)h->nstreams * h->n_pad;
    h->d_neg_re.reserve((size_t)std::max<int64_t>(n_ell, 1));
    if (h->cplx) h->d_neg_im.reserve((size_t)std::max<int64_t>(n_ell, 1));
    h->d_neg_diag.reserve((size_t)n_diag);
    ++h->launches;
    negate_streams_kernel<<<h->sm_count * 4, 256, 0, h->stream>>>(
        n_ell, h->d_ell_re.p, h->cplx ? h->d_ell_im.p : nullptr, h->d_neg_re.p, h->cplx ? h->d_neg_im.p : nullptr,
        n_diag, h->n_pad, h->d_diag.p, h->d_neg_diag.p);
    SPX_CUDA(cudaGetLastError());
}

// The echo core: the forward trajectory u from d_seq_rho and the adjoint
// trajectory v from the coil (adj0 null) or from per-orientation states adj0
// (n_orient x n_pad), nsteps steps of tau each; echo_f[o][j] =
// conj(v[o][k]) * Pi * u[o][j] with k = j, or k = nsteps - j when reverse;
// d_fid = their weighted sum in orientation order.
void echo_trajectories(spx_handle *h, int64_t n_orient, const double *g, double tau, int64_t nsteps,
                       const RunOptions &o, const double2 *adj0, bool reverse) {
    const int n_pad = h->n_pad;
    const int64_t npoints = nsteps + 1;
    // the states at every step come from chunks of a few steps (their
    // intermediate states accumulated in shared memory: one-step chunks spend
    // most of their series on the truncation tail); orientations in batches
    // whose two trajectories take a quarter of the free device memory (at
    // most 48 GB): few batches, so few partly filled waves
    RunOptions o1 = o;
    size_t free_b = 0, total_b = 0;
    SPX_CUDA(cudaMemGetInfo(&free_b, &total_b));
    const size_t budget = std::min<size_t>(free_b / 4, 48ull << 30);
    const size_t per_orient = 2 * (size_t)npoints * n_pad * sizeof(double2);
    const int64_t batch = std::max<int64_t>(1, std::min<int64_t>(n_orient, (int64_t)(budget / per_orient)));
    h->d_traj[0].reserve((size_t)batch * npoints * n_pad);
    h->d_traj[1].reserve((size_t)batch * npoints * n_pad);
    h->d_echo_f.reserve((size_t)n_orient * npoints);
    h->d_fid.reserve((size_t)npoints);
    for (int64_t b0 = 0; b0 < n_orient; b0 += batch) {
        const int64_t nb = std::min(batch, n_orient - b0);
        // the longest chunk among those needing the fewest CTAs per orientation
        // (FP64 accumulators of 4-step chunks push c4 from 2- to 4-CTA clusters)
        Config c{};
        bool have = false;
        for (int m : {kTrajChunk, 2, 1}) {
            o1.chunk_steps = m;
            try {
                const Config cm = choose_config(h, nb, tau, nsteps, o1, 0, 256, true);
                if (!have || cm.cl < c.cl) c = cm;
                have = true;
            } catch (const SpxError &e) {
                if (e.code != SPX_ERR_UNSUPPORTED) throw;
            }
        }
        if (!have) throw SpxError(SPX_ERR_UNSUPPORTED, "the trajectory does not fit a cluster of 8 SMs");
        o1.chunk_steps = c.M;
        for (int dir = 0; dir < 2; ++dir) {
            RunIO io;
            if (dir == 0) io.rho0 = h->d_seq_rho.p;
            else if (adj0) io.rho0s = adj0 + (size_t)b0 * n_pad;
            else io.rho0 = h->d_coil.p;
            io.traj_out = h->d_traj[dir].p;
            io.adjoint = dir == 1;
            launch_powder(h, nb, g + b0, g + n_orient + b0, g + 2 * n_orient + b0, g + 3 * n_orient + b0, tau, nsteps,
                          o1, h->d_fid.p, c, 0, true, io);
            finish_run(h);
        }
        const int64_t warps = nb * npoints;
        const int blocks = (int)std::min<int64_t>((warps + 7) / 8, (int64_t)h->sm_count * 16);
        ++h->launches;
        echo_form_kernel<<<blocks, 256, 0, h->stream>>>((int)nb, (int)npoints, n_pad, h->d_echo_ptr.p, h->d_echo_col.p,
                                                        h->d_echo_val.p, h->d_traj[0].p, h->d_traj[1].p,
                                                        reverse ? 1 : 0, h->d_echo_f.p + b0 * npoints);
        SPX_CUDA(cudaGetLastError());
    }
    ++h->launches;
    echo_powder_kernel<<<(unsigned)((npoints + 127) / 128), 128, 0, h->stream>>>(
        (int)n_orient, (int)npoints, h->d_echo_f.p, g + 3 * n_orient, h->d_fid.p);
    SPX_CUDA(cudaGetLastError());
}

// Copies the powder echo (and every orientation's) to the host, times scale.
void echo_outputs(spx_handle *h, int64_t n_orient, int64_t npoints, double scale, double *fid,
                  double *fids_per_orient) {
    SPX_CUDA(cudaMemcpyAsync(fid, h->d_fid.p, (size_t)npoints * sizeof(double2), cudaMemcpyDeviceToHost, h->stream));
    if (fids_per_orient)
        SPX_CUDA(cudaMemcpyAsync(fids_per_orient, h->d_echo_f.p, (size_t)n_orient * npoints * sizeof(double2),
                                 cudaMemcpyDeviceToHost, h->stream));
    SPX_CUDA(cudaStreamSynchronize(h->stream));
    if (scale != 1.0) {
        for (int64_t i = 0; i < 2 * npoints; ++i) fid[i] *= scale;
        if (fids_per_orient)
            for (int64_t i = 0; i < 2 * n_orient * npoints; ++i) fids_per_orient[i] *= scale;
    }
}

// out[o][j] = sum_i conj(v[o][j'][i]) (Pi u[o][j])[i], one warp per (o, j), with
// j' = j, or the last point minus j when reverse; Pi has v's rows and u's columns.
template <class Vec>
__global__ void coupled_echo_kernel(int n_orient, int npoints, int nu, int nv, const int *__restrict__ ptr,
                                    const int *__restrict__ col, const double2 *__restrict__ val,
                                    const Vec *__restrict__ u, const Vec *__restrict__ v, int reverse, double2 *out) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t)n_orient * npoints;
    for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nw;
         w += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int64_t wv = reverse ? w - 2 * (w % npoints) + npoints - 1 : w;
        const Vec *uu = u + w * nu, *vv = v + wv * nv;
        double re = 0.0, im = 0.0;
        for (int i = lane; i < nv; i += 32) {
            double wr = 0.0, wi = 0.0;
            for (int e = ptr[i]; e < ptr[i + 1]; ++e) {
                const double2 a = val[e];
                const Vec b = uu[col[e]];
                wr = fma(a.x, (double)b.x, fma(-a.y, (double)b.y, wr));
                wi = fma(a.x, (double)b.y, fma(a.y, (double)b.x, wi));
            }
            const Vec c = vv[i];                 // conj(c) * w
            re = fma((double)c.x, wr, fma((double)c.y, wi, re));
            im = fma((double)c.x, wi, fma(-(double)c.y, wr, im));
        }
#pragma unroll
        for (int q = 16; q; q >>= 1) {
            re += __shfl_xor_sync(0xffffffffu, re, q);
            im += __shfl_xor_sync(0xffffffffu, im, q);
        }
        if (lane == 0) out[w] = make_double2(re, im);
    }
}

// M x on the host.
std::vector<double2> apply_host(const HostCsr &m, const std::vector<double2> &x) {
    std::vector<double2> y(x.size(), make_double2(0, 0));
    for (size_t i = 0; i < x.size(); ++i)
        for (int e = m.ptr[i]; e < m.ptr[i + 1]; ++e) {
            const double2 v = cmul(m.val[e], x[m.col[e]]);
            y[i].x += v.x;
            y[i].y += v.y;
        }
    return y;
}

// The echo core (echo_trajectories) on the coupled states: the adjoint
// trajectory lives on the coil's rows (or those that `back`, a pulse on the
// adjoint state after nsteps steps, leads to), the forward one on the rows
// that the echo pulse connects to them.  out_back: DEER's first adjoint run.
// False if the states do not qualify.
bool run_coupled_echo(spx_handle *h, int64_t n_orient, const std::vector<const spx_csc *> &ops, double first_angle,
                      const double *back_angle, int echo_op, double tau, int64_t nsteps, const RunOptions &o,
                      bool reverse) {
    if (forced_shape(o) || may_diverge(h, tau, nsteps)) return false;
    CoupledSequence seq(h, ops);
    const int n = seq.n();
    if (n == 0) return false;
    HostCsr first, echo, back;
    if (!pulse_exponential(seq.pulses[0], first_angle, first) || !pulse_exponential(seq.pulses[echo_op], M_PI, echo)) return false;
    if (back_angle && !pulse_exponential(seq.pulses[0], *back_angle, back)) return false;
    std::vector<double2> rho(n), coil(n, make_double2(0, 0));
    for (int i = 0; i < n; ++i) rho[i] = h->rho0_host[seq.rows[i]];
    rho = apply_host(first, rho);
    for (size_t i = 0; i < h->coil_row_host.size(); ++i)
        if (seq.at[h->coil_row_host[i]] >= 0) coil[seq.at[h->coil_row_host[i]]] = h->coil_val_host[i];
    // the places a matrix's rows read, and those whose rows read the given places
    auto reads = [&](const HostCsr &m, const std::vector<char> &rows) {
        std::vector<char> p(n, 0);
        for (int i = 0; i < n; ++i)
            if (rows[i])
                for (int e = m.ptr[i]; e < m.ptr[i + 1]; ++e) p[m.col[e]] = 1;
        return p;
    };
    const std::vector<char> at_coil = seq.coil_places(h);
    std::vector<char> vp = at_coil;
    if (back_angle) {
        std::vector<char> p(n, 0);
        for (int i = 0; i < n; ++i)
            for (int e = back.ptr[i]; e < back.ptr[i + 1]; ++e) p[i] |= at_coil[back.col[e]];
        vp = seq.closure(h, p);
    }
    std::vector<char> excited(n, 0);
    for (int i = 0; i < n; ++i) excited[i] = rho[i].x != 0.0 || rho[i].y != 0.0;
    excited = seq.closure(h, excited);
    std::vector<char> up = seq.closure(h, reads(echo, vp));
    for (int i = 0; i < n; ++i) up[i] = up[i] && excited[i];
    SequenceGroup gu, gv, gb;
    seq.plan(h, up, false, gu.plan);
    seq.plan(h, vp, false, gv.plan);
    if (back_angle) seq.plan(h, at_coil, false, gb.plan);
    if (!gu.plan.ok || !gv.plan.ok || (back_angle && !gb.plan.ok)) return false;
    const int nu = gu.plan.n, nv = gv.plan.n;
    HostCsr form;                                   // echo's rows of v and columns of u
    {
        std::vector<int> own(n, -1);
        int q = 0;
        for (int i = 0; i < n; ++i)
            if (up[i]) own[i] = q++;
        form.ptr.push_back(0);
        for (int i = 0; i < n; ++i) {
            if (!vp[i]) continue;
            for (int e = echo.ptr[i]; e < echo.ptr[i + 1]; ++e)
                if (own[echo.col[e]] >= 0) { form.col.push_back(own[echo.col[e]]); form.val.push_back(echo.val[e]); }
            form.ptr.push_back((int)form.col.size());
        }
    }
    SparseOp dform, dback;
    dform.upload(form, h->stream);
    const bool f64 = o.precision == SPX_FP64;
    const size_t vec = f64 ? sizeof(double2) : sizeof(float2);
    const int64_t npoints = nsteps + 1;
    const double *g = h->d_grid.p;
    h->d_seq_rho.reserve(2 * (size_t)n);
    SPX_CUDA(cudaMemcpyAsync(h->d_seq_rho.p, rho.data(), n * sizeof(double2), cudaMemcpyHostToDevice, h->stream));
    SPX_CUDA(cudaMemcpyAsync(h->d_seq_rho.p + n, coil.data(), n * sizeof(double2), cudaMemcpyHostToDevice, h->stream));
    SPX_CUDA(cudaStreamSynchronize(h->stream));
    spx::DevSystem sys = device_system(h);
    h->d_status.reserve(n_orient);
    h->d_kused.reserve(n_orient);
    h->d_mused.reserve(n_orient);
    h->d_matvecs.reserve(n_orient);
    h->d_halfwidth.reserve(n_orient);
    h->d_echo_f.reserve((size_t)n_orient * npoints);
    h->d_fid.reserve((size_t)npoints);
    h->d_part.reserve((size_t)((n_orient + kPowderGroup - 1) / kPowderGroup) * npoints);
    h->d_seq_status.reserve(3 * (size_t)n_orient);
    SPX_CUDA(cudaEventRecord(h->ev[0], h->stream));
    const double2 *adj = h->d_seq_rho.p + n;
    bool adj_each = false;
    int *status[3];
    for (int q = 0; q < 3; ++q) status[q] = h->d_seq_status.p + (size_t)q * n_orient;
    if (back_angle) {
        const Config whole = choose_config(h, n_orient, tau, nsteps, o, 0);     // refusals of the whole system
        const size_t ns = (size_t)n_orient * n;
        h->d_seq[0].reserve(ns);
        h->d_seq[1].reserve(ns);
        SPX_CUDA(cudaMemsetAsync(h->d_seq[0].p, 0, ns * sizeof(double2), h->stream));
        spx::BlockRun r{};
        r.adjoint = 1;
        r.rho0 = adj;
        r.state_stride = (size_t)n;
        r.state_out = h->d_seq[0].p;
        const double *const angles[3] = {g, g + n_orient, g + 2 * n_orient};
        gb.bufs.halfwidth.reserve(n_orient);
        if (!run_group(h, gb, sys, r, n_orient, angles, tau, nsteps, whole.tol, o.lanczos_its, f64, false, status[2],
                       gb.bufs.halfwidth.p))
            return false;
        dback.upload(back, h->stream);
        ++h->launches;
        sparse_states_kernel<<<state_blocks(h, ns), 256, 0, h->stream>>>(n_orient, n, dback.ptr.p, dback.col.p, dback.val.p,
                                                                          h->d_seq[0].p, h->d_seq[1].p);
        SPX_CUDA(cudaGetLastError());
        adj = h->d_seq[1].p;
        adj_each = true;
    }
    // orientations in batches whose two trajectories take a quarter of the free
    // device memory, at most 48 GB
    size_t free_b = 0, total_b = 0;
    SPX_CUDA(cudaMemGetInfo(&free_b, &total_b));
    const size_t held = (h->d_traj[0].n + h->d_traj[1].n) * sizeof(double2);
    const size_t budget = std::min<size_t>((free_b + held) / 4, 48ull << 30);
    const int64_t batch = std::max<int64_t>(
        1, std::min<int64_t>(n_orient, (int64_t)(budget / ((size_t)npoints * (nu + nv) * vec))));
    auto traj = [&](int which, int rows) {
        h->d_traj[which].reserve(((size_t)batch * npoints * rows * vec + sizeof(double2) - 1) / sizeof(double2));
        return (void *)h->d_traj[which].p;
    };
    void *tu = traj(0, nu), *tv = traj(1, nv);
    Config whole{};
    for (int64_t b0 = 0; b0 < n_orient; b0 += batch) {
        const int64_t nb = std::min(batch, n_orient - b0);
        bool have = false;
        for (int m : {kTrajChunk, 2, 1}) {          // the whole system's configuration: its refusals stand
            RunOptions o1 = o;
            o1.chunk_steps = m;
            try {
                whole = choose_config(h, nb, tau, nsteps, o1, 0, 256, true);
                have = true;
                break;
            } catch (const SpxError &e) {
                if (e.code != SPX_ERR_UNSUPPORTED) throw;
            }
        }
        if (!have) throw SpxError(SPX_ERR_UNSUPPORTED, "the trajectory does not fit a cluster of 8 SMs");
        const double *const angles[3] = {g + b0, g + n_orient + b0, g + 2 * n_orient + b0};
        for (int dir = 0; dir < 2; ++dir) {
            SequenceGroup &grp = dir ? gv : gu;
            grp.bounded = false;
            grp.table_dt = 0.0;
            grp.bufs.halfwidth.reserve(nb);
            spx::BlockRun r{};
            r.adjoint = dir;
            r.state_stride = (size_t)n;
            if (dir == 0) r.rho0 = h->d_seq_rho.p;
            else if (adj_each) r.rho0s = adj + (size_t)b0 * n;
            else r.rho0 = adj;
            r.traj_out = dir ? tv : tu;
            const bool final = dir == 1;
            if (!run_group(h, grp, sys, r, nb, angles, tau, nsteps, whole.tol, o.lanczos_its, f64, true, status[dir] + b0,
                           final ? h->d_halfwidth.p + b0 : grp.bufs.halfwidth.p, b0))
                return false;
        }
        const int64_t warps = nb * npoints;
        const int blocks = (int)std::min<int64_t>((warps + 7) / 8, (int64_t)h->sm_count * 16);
        ++h->launches;
        if (f64)
            coupled_echo_kernel<double2><<<blocks, 256, 0, h->stream>>>(
                (int)nb, (int)npoints, nu, nv, dform.ptr.p, dform.col.p, dform.val.p, (const double2 *)tu,
                (const double2 *)tv, reverse ? 1 : 0, h->d_echo_f.p + b0 * npoints);
        else
            coupled_echo_kernel<float2><<<blocks, 256, 0, h->stream>>>(
                (int)nb, (int)npoints, nu, nv, dform.ptr.p, dform.col.p, dform.val.p, (const float2 *)tu,
                (const float2 *)tv, reverse ? 1 : 0, h->d_echo_f.p + b0 * npoints);
        SPX_CUDA(cudaGetLastError());
    }
    launch_powder_sum(h, true, h->d_echo_f.p, g + 3 * n_orient, n_orient, (size_t)npoints, h->d_part.p, h->d_fid.p);
    SPX_CUDA(cudaEventRecord(h->ev[1], h->stream));
    SPX_CUDA(cudaEventRecord(h->ev[2], h->stream));
    SPX_CUDA(cudaMemcpyAsync(h->d_status.p, status[1], n_orient * sizeof(int), cudaMemcpyDeviceToDevice, h->stream));
    h->stats_timed = true;
    whole.blk = gv.c.blk;
    describe_run(h, n_orient, nsteps, o.precision, whole);
    h->stats_pending = true;
    h->last_norient = n_orient;
    h->chk_pending = 0;
    finish_run(h);
    if (!back_angle) SPX_CUDA(cudaMemset(status[2], 0, n_orient * sizeof(int)));
    check_statuses(h, n_orient, 3);
    return true;
}

// first_angle: pi/2 for eseem.m, pi/4 for oopeseem.m (the out-of-phase echo).
void run_eseem(spx_handle *h, int64_t n_orient, const double *alphas, const double *betas, const double *gammas,
               const double *weights, double timestep, int64_t npoints, const spx_csc *pulse_op,
               double first_angle, const RunOptions &o, double *fid, double *fids_per_orient) {
    if (h->nchan != 1 || h->n_states != 0)
        throw SpxError(SPX_ERR_UNSUPPORTED, "pulse sequences take one coil and one initial state");
    if (npoints < 1) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "npoints must be positive");
    const double tau = timestep / 2;                // eseem.m: steps of timestep/2
    const int64_t nsteps = npoints - 1;
    validate_run(h, n_orient, tau, nsteps);
    if (h->n_pad > 8192) throw SpxError(SPX_ERR_UNSUPPORTED, "echo detection is limited to dimension 8192");
    upload_grid(h, n_orient, alphas, betas, gammas, weights);
    if (run_coupled_echo(h, n_orient, {pulse_op}, first_angle, nullptr, 0, tau, nsteps, o, false)) {
        echo_outputs(h, n_orient, npoints, 1.0, fid, fids_per_orient);
        return;
    }
    h->pulses.clear();
    h->pulses.push_back(std::make_unique<PulseOp>());
    upload_pulse(h, pulse_op, *h->pulses.back());
    const PulseOp &P = *h->pulses.back();
    // rho1 = exp(-1i first_angle P) rho0
    h->d_seq_rho.reserve(h->n_pad);
    SPX_CUDA(cudaMemcpyAsync(h->d_seq_rho.p, h->d_rho0.p, h->n_pad * sizeof(double2), cudaMemcpyDeviceToDevice,
                             h->stream));
    apply_pulse(h, P, first_angle, 1, h->d_seq_rho.p);
    upload_echo_propagator(h, P, M_PI);
    negate_generator(h);
    echo_trajectories(h, n_orient, h->d_grid.p, tau, nsteps, o, nullptr, false);
    echo_outputs(h, n_orient, npoints, 1.0, fid, fids_per_orient);
}

// Three-pulse DEER with hard pulses (experiments/esr_dipolar/deer_3p_hard_deer.m,
// 'brief' output): with U = exp(-1i L stepsize), N = nsteps and
// rho1 = exp(-1i (pi/2) X_prob) rho0,
//   trace[j] = coil' U^N P_prob U^(N-j) Pi_pump U^j rho1 / |coil|_2,  j = 0..N,
// P_prob = exp(-1i pi X_prob), Pi_pump = exp(-1i pi X_pump).  With
// w = P_prob' (U')^N coil (an adjoint run of N steps, then the pulse by -pi),
// trace[j] = conj((U')^(N-j) w) Pi_pump U^j rho1: the adjoint trajectory from
// w read backwards against the forward trajectory from rho1.
void run_deer(spx_handle *h, int64_t n_orient, const double *alphas, const double *betas, const double *gammas,
              const double *weights, double stepsize, int64_t nsteps, const spx_csc *ex_prob,
              const spx_csc *ex_pump, const RunOptions &o, double *fid, double *fids_per_orient) {
    if (h->nchan != 1 || h->n_states != 0)
        throw SpxError(SPX_ERR_UNSUPPORTED, "pulse sequences take one coil and one initial state");
    if (nsteps < 1) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "nsteps must be a positive integer");
    validate_run(h, n_orient, stepsize, nsteps);
    const int n_pad = h->n_pad;
    if (n_pad > 8192) throw SpxError(SPX_ERR_UNSUPPORTED, "echo detection is limited to dimension 8192");
    upload_grid(h, n_orient, alphas, betas, gammas, weights);
    const double back = -M_PI;
    if (run_coupled_echo(h, n_orient, {ex_prob, ex_pump}, M_PI / 2, &back, 1, stepsize, nsteps, o, true)) {
        double nrm = 0.0;
        for (const double2 &v : h->coil_val_host) nrm += v.x * v.x + v.y * v.y;
        if (!(nrm > 0.0)) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "the probe coil is zero");
        echo_outputs(h, n_orient, nsteps + 1, 1.0 / std::sqrt(nrm), fid, fids_per_orient);
        return;
    }
    h->pulses.clear();
    for (const spx_csc *q : {ex_prob, ex_pump}) {
        h->pulses.push_back(std::make_unique<PulseOp>());
        upload_pulse(h, q, *h->pulses.back());
    }
    const PulseOp &prob = *h->pulses[0], &pump = *h->pulses[1];
    const double *g = h->d_grid.p;
    h->d_seq_rho.reserve(n_pad);
    SPX_CUDA(cudaMemcpyAsync(h->d_seq_rho.p, h->d_rho0.p, n_pad * sizeof(double2), cudaMemcpyDeviceToDevice,
                             h->stream));
    apply_pulse(h, prob, M_PI / 2, 1, h->d_seq_rho.p);
    upload_echo_propagator(h, pump, M_PI);
    negate_generator(h);
    // w = P_prob' (U')^N coil for every orientation
    h->d_seq[0].reserve((size_t)n_orient * n_pad);
    h->d_fid.reserve((size_t)nsteps + 1);
    {
        RunIO io;
        io.rho0 = h->d_coil.p;
        io.state_out = h->d_seq[0].p;
        io.adjoint = true;
        const Config c = choose_config(h, n_orient, stepsize, nsteps, o, 0);
        launch_powder(h, n_orient, g, g + n_orient, g + 2 * n_orient, g + 3 * n_orient, stepsize, nsteps, o,
                      h->d_fid.p, c, 0, true, io);
        finish_run(h);
    }
    apply_pulse(h, prob, -M_PI, n_orient, h->d_seq[0].p);
    echo_trajectories(h, n_orient, g, stepsize, nsteps, o, h->d_seq[0].p, true);
    // deer_3p_hard_deer.m divides by the 2-norm of the probe coil
    std::vector<double2> coil(n_pad);
    SPX_CUDA(cudaMemcpyAsync(coil.data(), h->d_coil.p, n_pad * sizeof(double2), cudaMemcpyDeviceToHost, h->stream));
    SPX_CUDA(cudaStreamSynchronize(h->stream));
    double nrm = 0.0;
    for (const double2 &v : coil) nrm += v.x * v.x + v.y * v.y;
    if (!(nrm > 0.0)) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "the probe coil is zero");
    echo_outputs(h, n_orient, nsteps + 1, 1.0 / std::sqrt(nrm), fid, fids_per_orient);
}

// ---------------------------------------------------------------------------
// Autotuner
// ---------------------------------------------------------------------------
// shape of a tuning problem: systems with the same key get the same answer.
// First what describes the system and its coupled states, then the run.
using SystemKey = std::tuple<int, int, int, int, int, int, int, int>;
using TuneKey = std::pair<SystemKey, std::tuple<int, int, int>>;
std::mutex g_tune_mutex;
std::map<TuneKey, TunedShape> g_tune_cache;

SystemKey system_key(const spx_handle *h, int precision) {
    return SystemKey{h->n, h->ell_len, h->nslices, h->nstreams, h->cplx ? 1 : 0, precision,
                     h->plan.ok ? h->plan.n : 0, h->nchan};
}
// kernels: 0 the whole system's, 1 the coupled states', 2 the dense matrices.
TuneKey tune_key(const spx_handle *h, double dt, int64_t nsteps, int precision, int kernels) {
    // spectral scale in octaves: the series length per step follows it
    const int scale = (int)std::lround(std::log2(std::max(h->g_upper * dt, 1e-30)));
    return TuneKey{system_key(h, precision), {scale, (int)std::min<int64_t>(nsteps, 512), kernels}};
}

bool same_shape(const spx_options &a, const spx_options &b) {
    return a.threads == b.threads && a.cluster == b.cluster && a.chunk_target == b.chunk_target;
}

// The tuner's choice that options ask for: the handle's where they leave the
// shape at zero, else one that spx_autotune returned, for this handle or another
// one with such a system; null for neither.
const TunedShape *tuned_shape(const spx_handle *h, const spx_options &o) {
    const int p = o.precision == SPX_FP64 ? 1 : 0;
    const bool left = o.threads == 0 && o.cluster == 0 && o.chunk_target == 0.0;
    if (h->has_tuned[p] && (left || same_shape(o, h->tuned[p].shape))) return &h->tuned[p];
    if (left || o.threads == 0 || o.cluster == 0) return nullptr;
    const SystemKey key = system_key(h, o.precision);
    std::lock_guard<std::mutex> lk(g_tune_mutex);              // entries are never erased
    for (auto it = g_tune_cache.lower_bound(TuneKey{key, {INT_MIN, INT_MIN, INT_MIN}});
         it != g_tune_cache.end() && it->first.first == key; ++it)
        if (same_shape(o, it->second.shape)) return &it->second;
    return nullptr;
}

// The run's options with the tuner's choice in them.
RunOptions apply_tuned(const spx_handle *h, const spx_options &given) {
    RunOptions o(given);
    const TunedShape *t = tuned_shape(h, given);
    if (!t || (t->coupled && o.chunk_steps > 0)) return o;
    if (t->coupled) {
        o.threads = o.cluster = 0;             // the whole system's default, should it run after all
        o.chunk_target = 0.0;
        o.blk_target = t->blk_target;
    } else {
        o.threads = t->shape.threads;
        o.cluster = t->shape.cluster;
        o.chunk_target = t->shape.chunk_target;
    }
    o.own = true;
    return o;
}

// Kernel time of one candidate over the sample, or +inf if it cannot run.
double time_candidate(spx_handle *h, int64_t n, const double *d_al, const double *d_be, const double *d_ga,
                      const double *d_w, double dt, int64_t nsteps, const RunOptions &o, double2 *d_out) {
    double best = INFINITY;
    try {
        const Config c = choose_config(h, n, dt, nsteps, o, 0, 256, false, &h->plan);
        for (int rep = 0; rep < 2; ++rep) {           // first launch also loads the kernel
            launch_powder(h, n, d_al, d_be, d_ga, d_w, dt, nsteps, o, d_out, c);
            finish_run(h);
            best = std::min(best, h->stats.kernel_ms);
        }
    } catch (const SpxError &) {
        SPX_CUDA(cudaStreamSynchronize(h->stream));
        h->stats_pending = false;
        return INFINITY;
    }
    return best;
}

TunedShape autotune(spx_handle *h, int64_t n_orient, const double *d_al, const double *d_be, const double *d_ga,
                    double dt, int64_t nsteps, int precision) {
    RunOptions base;
    base.precision = precision;
    // sample: one wave of single-CTA orientations (at most 1024), at most 512
    // steps (several chunks, so long chunks are not penalised; a 256-step
    // sample picked shorter chunks and made the c2 graph 2 % slower)
    const int64_t ns = std::min<int64_t>(nsteps, 512);
    int64_t n = std::min<int64_t>(n_orient, 1024);
    Config c0{};                     // the default; a refused one leaves the shapes below to try
    try {
        c0 = choose_config(h, n, dt, ns, base, 0, 256, false, &h->plan);
        if (!c0.blk) n = std::min<int64_t>(n, c0.grid);
    } catch (const SpxError &) {
        c0 = Config{};
        n = std::min<int64_t>(n, h->sm_count);
    }
    const TuneKey key = tune_key(h, dt, nsteps, precision, c0.dense ? 2 : c0.blk ? 1 : 0);
    {
        std::lock_guard<std::mutex> lk(g_tune_mutex);
        auto it = g_tune_cache.find(key);
        if (it != g_tune_cache.end()) return it->second;
    }
    DevBuf<double> w;
    w.reserve((size_t)n);
    std::vector<double> hw((size_t)n, 1.0 / (double)n);
    SPX_CUDA(cudaMemcpyAsync(w.p, hw.data(), n * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    DevBuf<double2> out;
    out.reserve(((size_t)ns + 1) * h->nchan);
    auto time = [&](const RunOptions &o) { return time_candidate(h, n, d_al, d_be, d_ga, w.p, dt, ns, o, out.p); };
    // series length per chunk
    const double targets[] = {450.0, 300.0, 150.0, 60.0};
    TunedShape best;
    best.shape = base;
    double best_t = INFINITY;
    if (c0.blk) {
        // a run over the coupled states has its own layouts: only the series length
        // per chunk is tuned (the dense matrices have none); the whole system keeps
        // its default shape, which is the one returned
        best.coupled = true;
        best.shape.threads = c0.threads;
        best.shape.cluster = c0.cl;
        best.shape.chunk_target = c0.chunk_x;
        if (!c0.dense) {
            for (double tx : targets) {
                RunOptions o = base;
                o.blk_target = tx;
                const double t = time(o);
                if (t < best_t) { best_t = t; best.blk_target = tx; }
            }
            if (!std::isfinite(best_t)) throw SpxError(SPX_ERR_UNSUPPORTED, "no launch shape could run this system");
        }
    } else {
        const int cls[] = {1, 2, 4, 8};
        int cl_min = 0;              // smallest cluster that fits; it and twice it are tried
        for (int cl : cls) {
            if (cl_min && cl > 2 * cl_min) break;
            // warps: the default for this cluster size, half, and 16
            RunOptions o = base;
            o.cluster = cl;
            Config c{};
            try {
                c = choose_config(h, n, dt, ns, o, 0);
            } catch (const SpxError &) {
                continue;
            }
            if (!cl_min) cl_min = cl;
            const int nw0 = c.threads / 32;
            std::vector<int> nws = {nw0, std::max(1, nw0 / 2), 16};
            std::sort(nws.begin(), nws.end());
            nws.erase(std::unique(nws.begin(), nws.end()), nws.end());
            for (int nw : nws) {
                o.threads = nw * 32;
                const double t = time(o);
                if (t < best_t) { best_t = t; best.shape = o; }
            }
        }
        if (!std::isfinite(best_t)) throw SpxError(SPX_ERR_UNSUPPORTED, "no launch shape could run this system");
        const RunOptions shape = best.shape;
        for (double tx : targets) {
            RunOptions o = shape;
            o.chunk_target = tx;
            const double t = time(o);
            if (t < best_t) { best_t = t; best.shape = o; }
        }
    }
    std::lock_guard<std::mutex> lk(g_tune_mutex);
    g_tune_cache.emplace(key, best);
    return best;
}

// ---------------------------------------------------------------------------
// No-allocation variant: all intermediates in one static device array
// ---------------------------------------------------------------------------
constexpr int kNoallocChunkCap = 64;

__global__ void status_any_kernel(const int *status, int n, int *flag) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        if (status[i] != spx::kDevOk) atomicOr(flag, 1);
}

}  // namespace

static __device__ __align__(256) unsigned char g_noalloc_scratch[SPX_NOALLOC_SCRATCH_BYTES];

namespace {

std::mutex g_noalloc_mutex;
struct NoallocAddress {
    unsigned long long ctx_id = 0;   // context the address belongs to (0: none yet)
    void *ptr = nullptr;
};
NoallocAddress g_noalloc_address[256];

// Identifier of the current context (driver entry points fetched through the
// runtime, so the library needs no link against libcuda).  Context ids are
// never reused within a process, so a reset primary context gets a new one.
unsigned long long current_context_id() {
    typedef CUresult (*GetCurrent)(CUcontext *);
    typedef CUresult (*GetId)(CUcontext, unsigned long long *);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    if (!get_current || !get_id) {
        cudaDriverEntryPointQueryResult q1 = cudaDriverEntryPointSymbolNotFound, q2 = q1;
        void *f1 = nullptr, *f2 = nullptr;
        SPX_CUDA(cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f1, 12000, cudaEnableDefault, &q1));
        SPX_CUDA(cudaGetDriverEntryPointByVersion("cuCtxGetId", &f2, 12000, cudaEnableDefault, &q2));
        if (q1 != cudaDriverEntryPointSuccess || q2 != cudaDriverEntryPointSuccess || !f1 || !f2)
            throw SpxError(SPX_ERR_CUDA, "the driver lacks cuCtxGetCurrent/cuCtxGetId");
        get_current = reinterpret_cast<GetCurrent>(f1);
        get_id = reinterpret_cast<GetId>(f2);
    }
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (get_current(&ctx) != CUDA_SUCCESS || !ctx || get_id(ctx, &id) != CUDA_SUCCESS)
        throw SpxError(SPX_ERR_CUDA, "no current CUDA context");
    return id;
}

// Device address of g_noalloc_scratch on the current device.  Host code only
// sees a stand-in symbol, never the device address, so the address is looked
// up with cudaGetSymbolAddress once per device and context (again after
// another part of the process has reset the device and its context).
void *noalloc_scratch(int device) {
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (device < 0 || device >= 256) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "device ordinal out of range");
    const unsigned long long id = current_context_id();
    NoallocAddress &a = g_noalloc_address[device];
    if (!a.ptr || a.ctx_id != id) {
        void *ptr = nullptr;
        SPX_CUDA(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
        if (!ptr) throw SpxError(SPX_ERR_CUDA, "no device address for the static scratch array");
        a.ptr = ptr;
        a.ctx_id = id;
    }
    return a.ptr;
}

void run_powder_noalloc(spx_handle *h, int64_t n_orient, const double *d_al, const double *d_be,
                        const double *d_ga, const double *d_w, double dt, int64_t nsteps, int32_t precision,
                        double *d_fid) {
    validate_run(h, n_orient, dt, nsteps);
    if (!d_al || !d_be || !d_ga || !d_w || !d_fid) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "NULL device pointer");
    if (precision != SPX_FP32 && precision != SPX_FP64) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "unknown precision");
    SPX_CUDA(cudaSetDevice(h->device));
    spx_options opt{};
    opt.precision = precision;
    Config c = choose_config(h, n_orient, dt, nsteps, opt, 0, kNoallocChunkCap, false, &h->plan);
    const bool f64 = precision == SPX_FP64;
    const size_t npts = ((size_t)nsteps + 1) * h->nchan;   // all channels' points
    const int group = 64;
    const int ngroups = (int)((n_orient + group - 1) / group);
    // carve the scratch: sizes first, then check, then addresses
    constexpr int kParts = 14;
    size_t offs[kParts], total = 0;
    auto carve = [&] {
        const size_t tables = c.blk ? block_table_entries(c) : (size_t)c.grid * c.Kmax * (c.M + 1);
        const size_t sizes[kParts] = {
            tables * sizeof(double),                                      // Bessel tables
            npts * (size_t)n_orient * (f64 ? sizeof(double2) : sizeof(float2)),   // per-orientation FIDs
            (size_t)ngroups * npts * sizeof(double2),                     // FP64 partial sums
            (size_t)n_orient * sizeof(int), (size_t)n_orient * sizeof(int), (size_t)n_orient * sizeof(int),
            (size_t)n_orient * sizeof(long long) + (size_t)n_orient * sizeof(double),
            sizeof(int), sizeof(int),
            // coupled-state kernels: float tables, centres, extents, ladder, columns' terms
            c.blk && !f64 ? tables * sizeof(float) : 0, c.blk ? (size_t)n_orient * sizeof(double) : 0,
            c.blk ? 2 * sizeof(unsigned long long) : 0,
            c.blk ? (size_t)c.blk_lev * (sizeof(double) + 3 * sizeof(int)) : 0,
            c.blk ? (size_t)c.blk_lev * (c.blk_M + 1) * sizeof(int) : 0};
        total = 0;
        for (int i = 0; i < kParts; ++i) {
            offs[i] = total;
            total += (sizes[i] + 255) & ~(size_t)255;
        }
    };
    // what the whole system needs decides what is refused; the coupled states
    // run where they fit too
    const BlockPlan::Layout *coupled = c.blk;
    c.blk = nullptr;
    carve();
    if (total > SPX_NOALLOC_SCRATCH_BYTES)
        throw SpxError(SPX_ERR_UNSUPPORTED, "this run needs " + std::to_string(total) +
                                                " bytes of scratch; spx_run_powder_noalloc holds " +
                                                std::to_string((size_t)SPX_NOALLOC_SCRATCH_BYTES) +
                                                " (use spx_run_powder_device for larger runs)");
    c.blk = coupled;
    carve();
    if (total > SPX_NOALLOC_SCRATCH_BYTES) {
        c.blk = nullptr;
        carve();
    }
    unsigned char *base = static_cast<unsigned char *>(noalloc_scratch(h->device));
    int *flag = reinterpret_cast<int *>(base + offs[7]);
    spx::DevSystem sys = device_system(h);
    spx::DevRun run{};
    run.n_orient = (int)n_orient; run.alpha = d_al; run.beta = d_be; run.gamma = d_ga;
    run.dt = dt; run.nsteps = (int)nsteps; run.M = c.M; run.Kmax = c.Kmax; run.tol = c.tol;
    run.fixed_chunk = c.fixed ? 1 : 0; run.chunk_x = c.chunk_x;
    run.lanczos_its = opt.lanczos_its > 0 ? opt.lanczos_its : 32; run.safe_bounds = 0;
    run.table = reinterpret_cast<double *>(base + offs[0]);
    run.fids = base + offs[1];
    run.status = reinterpret_cast<int *>(base + offs[3]);
    run.kused = reinterpret_cast<int *>(base + offs[4]);
    run.mused = reinterpret_cast<int *>(base + offs[5]);
    run.matvecs = reinterpret_cast<long long *>(base + offs[6]);
    run.halfwidth = reinterpret_cast<double *>(base + offs[6] + (size_t)n_orient * sizeof(long long));
    run.next_orient = reinterpret_cast<int *>(base + offs[8]);
    double2 *part = reinterpret_cast<double2 *>(base + offs[2]);
    // values that must start at zero: the failure flag here, the work counter
    // (run.next_orient) in launch_chebyshev; everything else is written
    // before it is read
    SPX_CUDA(cudaMemsetAsync(flag, 0, sizeof(int), h->stream));
    if (c.blk) {
        spx::BlockRun r{};
        block_run_buffers(r, c, reinterpret_cast<double *>(base + offs[10]),
                          reinterpret_cast<unsigned long long *>(base + offs[11]),
                          reinterpret_cast<double *>(base + offs[12]),
                          reinterpret_cast<int *>(base + offs[12] + c.blk_lev * sizeof(double)),
                          reinterpret_cast<int *>(base + offs[13]), run.table,
                          f64 ? nullptr : reinterpret_cast<float *>(base + offs[9]));
        r.n_orient = run.n_orient; r.alpha = d_al; r.beta = d_be; r.gamma = d_ga;
        r.dt = dt; r.nsteps = (int)nsteps; r.lanczos_its = run.lanczos_its;
        r.halfwidth = run.halfwidth; r.max_im_diag = h->max_im_diag;
        r.rho0 = sys.rho0; r.rho0s = sys.rho0s; r.state_stride = (size_t)h->n_pad;
        r.fids = run.fids; r.nchan = h->nchan;
        r.status = run.status; r.kused = run.kused; r.mused = run.mused; r.matvecs = run.matvecs;
        launch_block(h, c, sys, r, h->stream);
    } else {
        launch_chebyshev(h, f64, c, sys, run);
    }
    launch_powder_sum(h, f64, run.fids, d_w, n_orient, npts, part, reinterpret_cast<double2 *>(d_fid));
    ++h->launches;
    status_any_kernel<<<dim3(64), dim3(256), 0, h->stream>>>(run.status, (int)n_orient, flag);
    SPX_CUDA(cudaGetLastError());
    int failed = 0;
    SPX_CUDA(cudaMemcpyAsync(&failed, flag, sizeof(int), cudaMemcpyDeviceToHost, h->stream));
    SPX_CUDA(cudaStreamSynchronize(h->stream));
    if (failed)
        throw SpxError(SPX_ERR_SERIES, "at least one orientation failed its series checks; "
                                       "spx_run_powder retries such runs with conservative bounds");
}

}  // namespace

extern "C" {

spx_status spx_run_powder_noalloc(spx_handle *h, int64_t n_orient, const double *d_alphas,
                                  const double *d_betas, const double *d_gammas, const double *d_weights,
                                  double dt, int64_t nsteps, int32_t precision, double *d_fid) {
    if (!h) return SPX_ERR_INVALID_ARGUMENT;
    return guarded(h, [&] {
        run_powder_noalloc(h, n_orient, d_alphas, d_betas, d_gammas, d_weights, dt, nsteps, precision, d_fid);
    });
}


spx_status spx_create(spx_handle **handle, int device) {
    if (!handle) return SPX_ERR_INVALID_ARGUMENT;
    *handle = nullptr;
    spx_handle *h = new (std::nothrow) spx_handle();
    if (!h) return SPX_ERR_OUT_OF_MEMORY;
    const spx_status st = guarded(h, [&] {
        int ndev = 0;
        SPX_CUDA(cudaGetDeviceCount(&ndev));
        if (device < 0 || device >= ndev) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "no such CUDA device");
        h->device = device;
        SPX_CUDA(cudaSetDevice(device));
        SPX_CUDA(cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking));
        for (auto &e : h->ev) SPX_CUDA(cudaEventCreate(&e));
        SPX_CUDA(cudaDeviceGetAttribute(&h->sm_count, cudaDevAttrMultiProcessorCount, device));
        int optin = 0;
        SPX_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
        h->smem_optin = (size_t)optin;
        SPX_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device));
        h->smem_sm = (size_t)optin;
        int least = 0;
        SPX_CUDA(cudaDeviceGetStreamPriorityRange(&least, &h->high_priority));
    });
    if (st != SPX_OK) {
        spx_destroy(h);
        return st;
    }
    *handle = h;
    return SPX_OK;
}

spx_status spx_destroy(spx_handle *h) {
    if (!h) return SPX_OK;
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    for (auto &e : h->ev)
        if (e) cudaEventDestroy(e);
    if (h->check_stream) cudaStreamSynchronize(h->check_stream);
    if (h->ev_fork) cudaEventDestroy(h->ev_fork);
    if (h->ev_join) cudaEventDestroy(h->ev_join);
    if (h->check_stream) cudaStreamDestroy(h->check_stream);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
    return SPX_OK;
}

spx_status spx_upload_system(spx_handle *h, const spx_csc *I, int32_t n_terms, const int32_t *rank,
                             const int32_t *k, const int32_t *m, const spx_csc *Q, const spx_csc *R,
                             const double *rho0, const double *coil) {
    if (!h) return SPX_ERR_INVALID_ARGUMENT;
    return guarded(h, [&] { upload_system(h, I, n_terms, rank, k, m, Q, R, rho0, coil); });
}

spx_status spx_run_powder(spx_handle *h, int64_t n_orient, const double *alphas, const double *betas,
                          const double *gammas, const double *weights, double dt, int64_t nsteps,
                          const spx_options *opt, double *fid, double *fids_per_orient) {
    if (!h) return SPX_ERR_INVALID_ARGUMENT;
    return guarded(h, [&] {
        validate_run(h, n_orient, dt, nsteps);
        if (!alphas || !betas || !gammas || !weights || !fid)
            throw SpxError(SPX_ERR_INVALID_ARGUMENT, "NULL grid or output pointer");
        for (int64_t o = 0; o < n_orient; ++o)
            if (!std::isfinite(alphas[o]) || !std::isfinite(betas[o]) || !std::isfinite(gammas[o]) ||
                !std::isfinite(weights[o]))
                throw SpxError(SPX_ERR_INVALID_ARGUMENT, "non-finite grid entry");
        RunOptions o = apply_tuned(h, given_options(opt));
        SPX_CUDA(cudaSetDevice(h->device));
        h->d_grid.reserve(4 * (size_t)n_orient);
        double *g = h->d_grid.p;
        const size_t b = (size_t)n_orient * sizeof(double);
        const double *parts[4] = {alphas, betas, gammas, weights};
        if (4 * b <= kStage) {
            unsigned char *t = h->stage.get(4 * b, h->stream);
            for (int q = 0; q < 4; ++q) std::memcpy(t + q * b, parts[q], b);
            SPX_CUDA(cudaMemcpyAsync(g, t, 4 * b, cudaMemcpyHostToDevice, h->stream));
        } else {
            for (int q = 0; q < 4; ++q)
                SPX_CUDA(cudaMemcpyAsync(g + q * n_orient, parts[q], b, cudaMemcpyHostToDevice, h->stream));
        }
        h->d_fid.reserve(((size_t)nsteps + 1) * h->nchan);
        Config c = choose_config(h, n_orient, dt, nsteps, o, 0, 256, false, &h->plan);
        const bool check = o.precision == SPX_FP32 && !(o.flags & SPX_FLAG_NO_FP32_CHECK);
        launch_powder(h, n_orient, g, g + n_orient, g + 2 * n_orient, g + 3 * n_orient, dt, nsteps, o, h->d_fid.p, c,
                      0, true, RunIO{}, check);
        bool retried = false;
        const double *staged = nullptr;
        try {
            staged = finish_run(h, true);
        } catch (const SpxError &e) {
            // one retry: a wider coefficient table if that was the only problem,
            // otherwise the conservative spectral bound
            std::vector<int> status(n_orient), kused(n_orient);
            SPX_CUDA(cudaMemcpy(status.data(), h->d_status.p, n_orient * sizeof(int), cudaMemcpyDeviceToHost));
            SPX_CUDA(cudaMemcpy(kused.data(), h->d_kused.p, n_orient * sizeof(int), cudaMemcpyDeviceToHost));
            bool retriable = true;
            int kneed = 0;
            for (int64_t i = 0; i < n_orient; ++i) {
                if (status[i] == spx::kDevTooManyRows) retriable = false;
                kneed = std::max(kneed, kused[i]);
            }
            if (!retriable) throw;
            c = choose_config(h, n_orient, dt, nsteps, o, 2 * kneed + 16, 256, false, &h->plan);
            retried = true;
            launch_powder(h, n_orient, g, g + n_orient, g + 2 * n_orient, g + 3 * n_orient, dt, nsteps, o,
                          h->d_fid.p, c, 1, true, RunIO{}, check);
            staged = finish_run(h, true);
        }
        h->stats.retries = retried ? 1 : 0;
        // the bar applies to what the caller receives: the powder FID, and
        // every orientation's FID when those are asked for too
        const double err32 = fids_per_orient ? std::max(h->stats.fp32_rel_error, h->stats.fp32_powder_error)
                                             : h->stats.fp32_powder_error;
        // the estimate comes from two orientations: it has tracked the measured
        // powder error within about 25 %, so the re-run starts at half the bar
        if (check && h->stats.fp32_checked > 0 && !(err32 <= 0.5 * SPX_FP32_ERROR_BAR) &&
            !(o.flags & SPX_FLAG_NO_PROMOTE)) {
            // the FP32 result misses the bar on the checked orientations: run
            // the whole grid again in FP64 and return that
            const spx_stats s32 = h->stats;
            spx_options given64 = o;
            given64.precision = SPX_FP64;
            given64.threads = given64.cluster = 0;
            given64.chunk_target = 0.0;
            const RunOptions o64 = apply_tuned(h, given64);
            const Config c64 = choose_config(h, n_orient, dt, nsteps, o64, 0, 256, false, &h->plan);
            launch_powder(h, n_orient, g, g + n_orient, g + 2 * n_orient, g + 3 * n_orient, dt, nsteps, o64,
                          h->d_fid.p, c64);
            staged = finish_run(h, true);
            h->stats.fp32_checked = s32.fp32_checked;
            h->stats.fp32_rel_error = s32.fp32_rel_error;
            h->stats.fp32_powder_error = s32.fp32_powder_error;
            h->stats.promoted_fp64 = 1;
            h->stats.retries = s32.retries;
            o.precision = SPX_FP64;
        }
        const size_t fid_bytes = ((size_t)nsteps + 1) * h->nchan * sizeof(double2);
        if (staged) std::memcpy(fid, staged, fid_bytes);
        else SPX_CUDA(cudaMemcpy(fid, h->d_fid.p, fid_bytes, cudaMemcpyDeviceToHost));
        if (fids_per_orient) {
            const size_t cnt = ((size_t)nsteps + 1) * h->nchan * n_orient;
            if (o.precision == SPX_FP64) {
                SPX_CUDA(cudaMemcpy(fids_per_orient, h->d_fids.p, cnt * sizeof(double2), cudaMemcpyDeviceToHost));
            } else {
                std::vector<float2> tmp(cnt);
                SPX_CUDA(cudaMemcpy(tmp.data(), h->d_fids.p, cnt * sizeof(float2), cudaMemcpyDeviceToHost));
                for (size_t i = 0; i < cnt; ++i) {
                    fids_per_orient[2 * i] = tmp[i].x;
                    fids_per_orient[2 * i + 1] = tmp[i].y;
                }
            }
        }
    });
}

spx_status spx_run_powder_device(spx_handle *h, int64_t n_orient, const double *d_alphas, const double *d_betas,
                                 const double *d_gammas, const double *d_weights, double dt, int64_t nsteps,
                                 const spx_options *opt, double *d_fid) {
    if (!h) return SPX_ERR_INVALID_ARGUMENT;
    return guarded(h, [&] {
        validate_run(h, n_orient, dt, nsteps);
        if (!d_alphas || !d_betas || !d_gammas || !d_weights || !d_fid)
            throw SpxError(SPX_ERR_INVALID_ARGUMENT, "NULL device pointer");
        RunOptions o = apply_tuned(h, given_options(opt));
        SPX_CUDA(cudaSetDevice(h->device));
        const Config c = choose_config(h, n_orient, dt, nsteps, o, 0, 256, false, &h->plan);
        const bool check = o.precision == SPX_FP32 && !(o.flags & SPX_FLAG_NO_FP32_CHECK);
        launch_powder(h, n_orient, d_alphas, d_betas, d_gammas, d_weights, dt, nsteps, o,
                      reinterpret_cast<double2 *>(d_fid), c, 0, true, RunIO{}, check);
    });
}

spx_status spx_synchronize(spx_handle *h) {
    if (!h) return SPX_ERR_INVALID_ARGUMENT;
    return guarded(h, [&] {
        SPX_CUDA(cudaSetDevice(h->device));
        finish_run(h);
    });
}

void *spx_get_stream(spx_handle *h) { return h ? (void *)h->stream : nullptr; }

spx_status spx_get_stats(spx_handle *h, spx_stats *stats) {
    if (!h || !stats) return SPX_ERR_INVALID_ARGUMENT;
    const spx_status st = guarded(h, [&] {
        SPX_CUDA(cudaSetDevice(h->device));
        finish_run(h);
    });
    *stats = h->stats;
    stats->kernel_launches = h->launches;
    return st;
}

const char *spx_status_string(spx_status s) {
    switch (s) {
        case SPX_OK: return "success";
        case SPX_ERR_INVALID_ARGUMENT: return "invalid argument";
        case SPX_ERR_NO_SYSTEM: return "no spin system uploaded";
        case SPX_ERR_CUDA: return "CUDA runtime error";
        case SPX_ERR_UNSUPPORTED: return "unsupported input";
        case SPX_ERR_SERIES: return "series did not converge";
        case SPX_ERR_NORM: return "|L*dt| too large";
        case SPX_ERR_OUT_OF_MEMORY: return "out of memory";
        case SPX_ERR_INTERNAL: return "internal error";
    }
    return "unknown status";
}

const char *spx_last_error(const spx_handle *h) { return h ? h->err.c_str() : "NULL handle"; }

const char *spx_version(void) { return "spinach-gb300 0.1 (sm_103a)"; }

spx_status spx_run_cpmg(spx_handle *h, int64_t n_orient, const double *alphas, const double *betas,
                        const double *gammas, const double *weights, double dt, int64_t npoints, int32_t nloops,
                        const spx_csc *pulse_op, const spx_options *opt, double *fid, double *fids_per_orient) {
    if (!h) return SPX_ERR_INVALID_ARGUMENT;
    return guarded(h, [&] {
        if (!alphas || !betas || !gammas || !weights || !fid || !pulse_op)
            throw SpxError(SPX_ERR_INVALID_ARGUMENT, "NULL argument");
        for (int64_t o = 0; o < n_orient; ++o)
            if (!std::isfinite(alphas[o]) || !std::isfinite(betas[o]) || !std::isfinite(gammas[o]) ||
                !std::isfinite(weights[o]))
                throw SpxError(SPX_ERR_INVALID_ARGUMENT, "non-finite grid entry");
        RunOptions o = apply_tuned(h, given_options(opt));
        SPX_CUDA(cudaSetDevice(h->device));
        run_cpmg(h, n_orient, alphas, betas, gammas, weights, dt, npoints, nloops, pulse_op, o, fid, fids_per_orient);
    });
}

spx_status spx_run_sequence(spx_handle *h, int64_t n_orient, const double *alphas, const double *betas,
                            const double *gammas, const double *weights, int32_t n_pulse, const spx_csc *pulse_ops,
                            int32_t n_ops, const spx_seq_op *ops, const spx_options *opt, double *fid,
                            double *fids_per_orient) {
    if (!h) return SPX_ERR_INVALID_ARGUMENT;
    return guarded(h, [&] {
        if (!alphas || !betas || !gammas || !weights || !fid) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "NULL argument");
        for (int64_t o = 0; o < n_orient; ++o)
            if (!std::isfinite(alphas[o]) || !std::isfinite(betas[o]) || !std::isfinite(gammas[o]) ||
                !std::isfinite(weights[o]))
                throw SpxError(SPX_ERR_INVALID_ARGUMENT, "non-finite grid entry");
        RunOptions o = apply_tuned(h, given_options(opt));
        SPX_CUDA(cudaSetDevice(h->device));
        run_sequence(h, n_orient, alphas, betas, gammas, weights, n_pulse, pulse_ops, n_ops, ops, o, fid,
                     fids_per_orient);
    });
}

namespace {
spx_status run_echo_entry(spx_handle *h, int64_t n_orient, const double *alphas, const double *betas,
                          const double *gammas, const double *weights, double timestep, int64_t npoints,
                          const spx_csc *pulse_op, double first_angle, const spx_options *opt, double *fid,
                          double *fids_per_orient) {
    if (!h) return SPX_ERR_INVALID_ARGUMENT;
    return guarded(h, [&] {
        if (!alphas || !betas || !gammas || !weights || !fid || !pulse_op)
            throw SpxError(SPX_ERR_INVALID_ARGUMENT, "NULL argument");
        for (int64_t o = 0; o < n_orient; ++o)
            if (!std::isfinite(alphas[o]) || !std::isfinite(betas[o]) || !std::isfinite(gammas[o]) ||
                !std::isfinite(weights[o]))
                throw SpxError(SPX_ERR_INVALID_ARGUMENT, "non-finite grid entry");
        spx_options o = given_options(opt);
        SPX_CUDA(cudaSetDevice(h->device));
        run_eseem(h, n_orient, alphas, betas, gammas, weights, timestep, npoints, pulse_op, first_angle, o, fid,
                  fids_per_orient);
    });
}
}  // namespace

spx_status spx_run_eseem(spx_handle *h, int64_t n_orient, const double *alphas, const double *betas,
                         const double *gammas, const double *weights, double timestep, int64_t npoints,
                         const spx_csc *pulse_op, const spx_options *opt, double *fid, double *fids_per_orient) {
    return run_echo_entry(h, n_orient, alphas, betas, gammas, weights, timestep, npoints, pulse_op, M_PI / 2, opt,
                          fid, fids_per_orient);
}

spx_status spx_run_oopeseem(spx_handle *h, int64_t n_orient, const double *alphas, const double *betas,
                            const double *gammas, const double *weights, double timestep, int64_t npoints,
                            const spx_csc *pulse_op, const spx_options *opt, double *fid, double *fids_per_orient) {
    return run_echo_entry(h, n_orient, alphas, betas, gammas, weights, timestep, npoints, pulse_op, M_PI / 4, opt,
                          fid, fids_per_orient);
}

spx_status spx_run_deer(spx_handle *h, int64_t n_orient, const double *alphas, const double *betas,
                        const double *gammas, const double *weights, double stepsize, int64_t nsteps,
                        const spx_csc *ex_prob, const spx_csc *ex_pump, const spx_options *opt, double *fid,
                        double *fids_per_orient) {
    if (!h) return SPX_ERR_INVALID_ARGUMENT;
    return guarded(h, [&] {
        if (!alphas || !betas || !gammas || !weights || !fid || !ex_prob || !ex_pump)
            throw SpxError(SPX_ERR_INVALID_ARGUMENT, "NULL argument");
        for (int64_t o = 0; o < n_orient; ++o)
            if (!std::isfinite(alphas[o]) || !std::isfinite(betas[o]) || !std::isfinite(gammas[o]) ||
                !std::isfinite(weights[o]))
                throw SpxError(SPX_ERR_INVALID_ARGUMENT, "non-finite grid entry");
        spx_options o = given_options(opt);
        SPX_CUDA(cudaSetDevice(h->device));
        run_deer(h, n_orient, alphas, betas, gammas, weights, stepsize, nsteps, ex_prob, ex_pump, o, fid,
                 fids_per_orient);
    });
}

spx_status spx_set_initial_states(spx_handle *h, int64_t n_states, const double *states) {
    if (!h) return SPX_ERR_INVALID_ARGUMENT;
    return guarded(h, [&] { set_initial_states(h, n_states, states); });
}

spx_status spx_build_system(spx_handle *h, int32_t n_spins, const int32_t *mults, int64_t dim,
                            const int64_t *basis_keys, const int64_t *radix, int32_t n_terms, const int32_t *rank,
                            const int32_t *k, const int32_t *m, int64_t n_mono, const int32_t *mono_term,
                            const int32_t *mono_spins, const int32_t *mono_codes, const double *mono_coefs,
                            const double *r_diag, const double *rho0, const double *coil, double *build_ms) {
    if (!h) return SPX_ERR_INVALID_ARGUMENT;
    return guarded(h, [&] {
        if (n_terms < 0 || n_terms > (spx::kMaxCoef - 1) / 2)
            throw SpxError(SPX_ERR_UNSUPPORTED, "too many rotational-basis terms");
        if (n_terms > 0 && (!rank || !k || !m)) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "NULL term arrays");
        if (!rho0 || !coil) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "rho0/coil is NULL");
        SPX_CUDA(cudaSetDevice(h->device));
        spx::BuildSpec spec;
        spec.n_spins = n_spins;
        spec.mults = mults;
        spec.dim = dim;
        spec.keys = basis_keys;
        spec.radix = radix;
        spec.n_terms = n_terms;
        spec.n_mono = n_mono;
        spec.mono_term = mono_term;
        spec.mono_spins = mono_spins;
        spec.mono_codes = mono_codes;
        spec.mono_coefs = mono_coefs;
        spx::BuildInfo info;
        std::vector<spx::HostCsc> mats;
        try {
            mats = spx::build_operators(spec, h->stream, &info);
        } catch (const std::invalid_argument &e) {
            throw SpxError(SPX_ERR_INVALID_ARGUMENT, e.what());
        } catch (const std::runtime_error &e) {
            throw SpxError(SPX_ERR_CUDA, e.what());
        }
        auto view = [&](spx::HostCsc &A) {
            spx_csc v{};
            v.n = dim;
            v.colptr = A.colptr.data();
            v.rowidx = A.rowidx.data();
            v.values = A.values.data();
            return v;
        };
        // terms whose matrix came out empty are dropped (as hamiltonian.m keeps
        // only the non-zero rotational components)
        spx_csc I = view(mats[0]);
        std::vector<spx_csc> Q;
        std::vector<int32_t> rk, kk, mm;
        for (int t = 0; t < n_terms; ++t) {
            if (mats[1 + t].rowidx.empty()) continue;
            Q.push_back(view(mats[1 + t]));
            rk.push_back(rank[t]);
            kk.push_back(k[t]);
            mm.push_back(m[t]);
        }
        spx::HostCsc R;
        if (r_diag) {
            R.colptr.resize(dim + 1);
            for (int64_t i = 0; i < dim; ++i) {
                if (!std::isfinite(r_diag[i])) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "non-finite relaxation rate");
                R.colptr[i] = (int64_t)R.rowidx.size();
                if (r_diag[i] != 0.0) {
                    R.rowidx.push_back(i);
                    R.values.push_back(r_diag[i]);
                    R.values.push_back(0.0);
                }
            }
            R.colptr[dim] = (int64_t)R.rowidx.size();
        }
        spx_csc Rv = view(R);
        upload_system(h, &I, (int32_t)Q.size(), rk.data(), kk.data(), mm.data(), Q.data(), r_diag ? &Rv : nullptr,
                      rho0, coil);
        if (build_ms) *build_ms = info.kernel_ms;
    });
}

spx_status spx_upload_coils(spx_handle *h, int32_t nchan, const double *coils) {
    if (!h) return SPX_ERR_INVALID_ARGUMENT;
    return guarded(h, [&] { upload_coils(h, nchan, coils); });
}

spx_status spx_autotune(spx_handle *h, int64_t n_orient, const double *d_alphas, const double *d_betas,
                        const double *d_gammas, double dt, int64_t nsteps, int32_t precision, spx_options *best) {
    if (!h) return SPX_ERR_INVALID_ARGUMENT;
    return guarded(h, [&] {
        validate_run(h, n_orient, dt, nsteps);
        if (!d_alphas || !d_betas || !d_gammas) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "NULL device pointer");
        if (precision != SPX_FP32 && precision != SPX_FP64) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "unknown precision");
        SPX_CUDA(cudaSetDevice(h->device));
        finish_run(h);
        const TunedShape t = autotune(h, n_orient, d_alphas, d_betas, d_gammas, dt, nsteps, precision);
        const int p = precision == SPX_FP64 ? 1 : 0;
        h->tuned[p] = t;
        h->has_tuned[p] = true;
        if (best) *best = t.shape;
    });
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Batched powders: one CUDA graph, one branch per system
// ---------------------------------------------------------------------------
struct spx_batch {
    // one system's run, as given to spx_batch_create
    struct Run {
        spx_handle *h;
        int64_t n_orient;
        const double *alphas, *betas, *gammas, *weights;
        double dt;
        int64_t nsteps;
        spx_options opt;
        double2 *fid;
        int64_t revision;                // of the handle when the graph was captured
    };
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaEvent_t ev[2] = {nullptr, nullptr};
    std::vector<cudaEvent_t> marks;      // fork / join events used while capturing
    std::vector<Run> runs;
    std::string err;
    bool launched = false;
};

namespace {

thread_local std::string g_batch_create_error;     // why the last spx_batch_create on this thread failed

template <class F>
spx_status batch_guarded(spx_batch *b, F f) {
    try {
        f();
        if (b) b->err.clear();
        return SPX_OK;
    } catch (const SpxError &e) {
        if (b) b->err = e.what();
        return e.code;
    } catch (const std::bad_alloc &) {
        if (b) b->err = "host allocation failed";
        return SPX_ERR_OUT_OF_MEMORY;
    } catch (const std::exception &e) {
        if (b) b->err = e.what();
        return SPX_ERR_INTERNAL;
    }
}

// Captures the batch's graph for what its handles hold now.
void capture_batch(spx_batch *b) {
    const size_t n = b->runs.size();
    // launch shapes and buffers first: nothing may allocate while capturing
    std::vector<Config> cfg(n);
    std::vector<RunOptions> os(n);
    for (size_t i = 0; i < n; ++i) {
        const spx_batch::Run &r = b->runs[i];
        os[i] = apply_tuned(r.h, r.opt);
        cfg[i] = choose_config(r.h, r.n_orient, r.dt, r.nsteps, os[i], 0, 256, false, &r.h->plan);
        reserve_run(r.h, r.n_orient, r.nsteps, os[i].precision == SPX_FP64, cfg[i]);
        SPX_CUDA(cudaStreamSynchronize(r.h->stream));
    }
    // load every kernel the graph will hold before capturing (lazy module loading
    // would otherwise happen inside the capture)
    {
        cudaFuncAttributes fa{};
        SPX_CUDA(cudaFuncGetAttributes(&fa, reinterpret_cast<const void *>(&spx::powder_partial_kernel<float2>)));
        SPX_CUDA(cudaFuncGetAttributes(&fa, reinterpret_cast<const void *>(&spx::powder_partial_kernel<double2>)));
        SPX_CUDA(cudaFuncGetAttributes(&fa, reinterpret_cast<const void *>(&spx::powder_combine_kernel)));
        SPX_CUDA(cudaFuncGetAttributes(&fa, reinterpret_cast<const void *>(&spx::block_tables_kernel)));
        for (size_t i = 0; i < n; ++i) {
            const spx_handle *h = b->runs[i].h;
            if (cfg[i].dense) {
                for (const void *k : {reinterpret_cast<const void *>(&spx::dense_start_kernel),
                                      reinterpret_cast<const void *>(&spx::dense_one_kernel<float2>),
                                      reinterpret_cast<const void *>(&spx::dense_one_kernel<double2>),
                                      reinterpret_cast<const void *>(&spx::dense_product_kernel<false>),
                                      reinterpret_cast<const void *>(&spx::dense_product_kernel<true>),
                                      reinterpret_cast<const void *>(&spx::dense_sum_kernel),
                                      reinterpret_cast<const void *>(&spx::dense_states_kernel),
                                      reinterpret_cast<const void *>(&spx::dense_rows_kernel),
                                      reinterpret_cast<const void *>(&spx::dense_points_kernel<float2>),
                                      reinterpret_cast<const void *>(&spx::dense_points_kernel<double2>)})
                    SPX_CUDA(cudaFuncGetAttributes(&fa, k));
                continue;
            }
            if (cfg[i].blk) {
                SPX_CUDA(cudaFuncGetAttributes(&fa, block_kernel(h->cplx, cfg[i].blk_bounds->ecap, cfg[i].blk_bounds_which)));
                SPX_CUDA(cudaFuncGetAttributes(&fa, block_kernel(h->cplx, cfg[i].blk->ecap, cfg[i].blk_which)));
                continue;
            }
            SPX_CUDA(cudaFuncGetAttributes(&fa, select_kernel(os[i].precision == SPX_FP64, h->cplx, cfg[i].rmax,
                                                              cfg[i].cl > 1, h->ncoil > 0, false,
                                                              cfg[i].threads > 512)));
        }
    }
    cudaGraph_t graph = nullptr;
    SPX_CUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
    try {
        SPX_CUDA(cudaEventRecord(b->marks[n], b->stream));             // fork
        for (size_t i = 0; i < n; ++i) {
            const spx_batch::Run &r = b->runs[i];
            SPX_CUDA(cudaStreamWaitEvent(r.h->stream, b->marks[n], 0));
            launch_powder(r.h, r.n_orient, r.alphas, r.betas, r.gammas, r.weights, r.dt, r.nsteps, os[i], r.fid, cfg[i],
                          0, false);
            SPX_CUDA(cudaEventRecord(b->marks[i], r.h->stream));        // join
            SPX_CUDA(cudaStreamWaitEvent(b->stream, b->marks[i], 0));
        }
    } catch (...) {
        cudaStreamEndCapture(b->stream, &graph);
        if (graph) cudaGraphDestroy(graph);
        throw;
    }
    SPX_CUDA(cudaStreamEndCapture(b->stream, &graph));
    cudaGraphExec_t exec = nullptr;
    const cudaError_t ie = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    SPX_CUDA(ie);
    if (b->exec) cudaGraphExecDestroy(b->exec);
    b->exec = exec;
    for (spx_batch::Run &r : b->runs) {
        r.h->stats_pending = false;
        r.revision = r.h->revision;
    }
}

}  // namespace

extern "C" {

spx_status spx_batch_destroy(spx_batch *b) {
    if (!b) return SPX_OK;
    cudaSetDevice(b->device);
    if (b->stream) cudaStreamSynchronize(b->stream);
    if (b->exec) cudaGraphExecDestroy(b->exec);
    for (auto e : b->marks) cudaEventDestroy(e);
    for (auto e : b->ev)
        if (e) cudaEventDestroy(e);
    if (b->stream) cudaStreamDestroy(b->stream);
    delete b;
    return SPX_OK;
}

spx_status spx_batch_create(spx_batch **out, int32_t n, spx_handle *const *handles, const int64_t *n_orient,
                            const double *const *d_alphas, const double *const *d_betas,
                            const double *const *d_gammas, const double *const *d_weights, const double *dt,
                            const int64_t *nsteps, const spx_options *opts, double *const *d_fids) {
    if (!out || n < 1 || !handles || !n_orient || !d_alphas || !d_betas || !d_gammas || !d_weights || !dt ||
        !nsteps || !d_fids)
        return SPX_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    spx_batch *b = new (std::nothrow) spx_batch();
    if (!b) return SPX_ERR_OUT_OF_MEMORY;
    const spx_status st = batch_guarded(b, [&] {
        for (int i = 0; i < n; ++i) {
            spx_handle *h = handles[i];
            if (!h) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "NULL handle #" + std::to_string(i));
            if (h->device != handles[0]->device) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "handles on different devices");
            if (!d_alphas[i] || !d_betas[i] || !d_gammas[i] || !d_weights[i] || !d_fids[i])
                throw SpxError(SPX_ERR_INVALID_ARGUMENT, "NULL device pointer for system #" + std::to_string(i));
            validate_run(h, n_orient[i], dt[i], nsteps[i]);
            for (int j = 0; j < i; ++j)
                if (handles[j] == h) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "a handle appears twice");
        }
        b->device = handles[0]->device;
        SPX_CUDA(cudaSetDevice(b->device));
        SPX_CUDA(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
        for (auto &e : b->ev) SPX_CUDA(cudaEventCreate(&e));
        for (int i = 0; i < n; ++i) {
            finish_run(handles[i]);
            const spx_options o = given_options(opts ? &opts[i] : nullptr);
            b->runs.push_back({handles[i], n_orient[i], d_alphas[i], d_betas[i], d_gammas[i], d_weights[i], dt[i],
                               nsteps[i], o, reinterpret_cast<double2 *>(d_fids[i]), 0});
        }
        b->marks.resize(n + 1, nullptr);
        for (auto &e : b->marks) SPX_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        capture_batch(b);
    });
    if (st != SPX_OK) {
        g_batch_create_error = b->err;
        for (int i = 0; i < n && handles; ++i)
            if (handles[i]) handles[i]->stats_pending = false;
        spx_batch_destroy(b);
        return st;
    }
    g_batch_create_error.clear();
    *out = b;
    return SPX_OK;
}

spx_status spx_batch_launch(spx_batch *b, void *stream) {
    if (!b) return SPX_ERR_INVALID_ARGUMENT;
    return batch_guarded(b, [&] {
        SPX_CUDA(cudaSetDevice(b->device));
        cudaStream_t s = stream ? (cudaStream_t)stream : b->stream;
        // a system, coils or initial states uploaded since: the graph's launches
        // hold the sizes and places of what was there before
        bool stale = false;
        for (const spx_batch::Run &r : b->runs) stale = stale || r.revision != r.h->revision;
        if (stale) {
            if (b->launched) SPX_CUDA(cudaEventSynchronize(b->ev[1]));
            for (const spx_batch::Run &r : b->runs) validate_run(r.h, r.n_orient, r.dt, r.nsteps);
            capture_batch(b);
        }
        SPX_CUDA(cudaEventRecord(b->ev[0], s));
        SPX_CUDA(cudaGraphLaunch(b->exec, s));
        SPX_CUDA(cudaEventRecord(b->ev[1], s));
        for (const spx_batch::Run &r : b->runs) {
            r.h->stats_pending = true;
            r.h->stats_timed = false;
            r.h->last_norient = r.n_orient;
        }
        b->launched = true;
    });
}

spx_status spx_batch_synchronize(spx_batch *b, double *ms) {
    if (!b) return SPX_ERR_INVALID_ARGUMENT;
    return batch_guarded(b, [&] {
        SPX_CUDA(cudaSetDevice(b->device));
        if (!b->launched) throw SpxError(SPX_ERR_INVALID_ARGUMENT, "batch not launched");
        SPX_CUDA(cudaEventSynchronize(b->ev[1]));
        float t = 0.f;
        SPX_CUDA(cudaEventElapsedTime(&t, b->ev[0], b->ev[1]));
        if (ms) *ms = t;
        for (size_t i = 0; i < b->runs.size(); ++i) {
            try {
                finish_run(b->runs[i].h);
            } catch (const SpxError &e) {
                throw SpxError(e.code, "system #" + std::to_string(i) + ": " + e.what());
            }
        }
    });
}

const char *spx_batch_last_error(const spx_batch *b) { return b ? b->err.c_str() : g_batch_create_error.c_str(); }

}  // extern "C"

// Propagation of the states that couple to the detection states.
//
// The Liouvillian of a powder is block diagonal over the connected components
// of its sparsity pattern (coherence orders and, in restricted bases, further
// product states never mix), and an orientation's FID coil' exp(-1i L t) rho0
// depends only on the components that hold coil entries and rho0 entries.
// The engine finds those rows once per system (block_plan.h) and these kernels
// run the same chunked Chebyshev expansion as kernels.cuh on them alone: 52 of
// 1156 states for a seven-spin IK-0(3) system, 252 of 4096 for six spins, 144
// of 2736 for the radical with ten protons.
//
// At these sizes a term's cost is latency and issue slots, not memory, so the
// layout differs from kernels.cuh: one small CTA per orientation, many CTAs
// per SM; every lane keeps its share of one row (values, columns, diagonal) in
// registers for the whole orientation and only the state is read from shared
// memory; a wide row is split over 2-32 neighbouring lanes, whose partial sums
// meet in shuffles; the detection states are extra rows of the matrix, so a
// term's product yields the moments too.  Spectral bounds and Bessel tables
// are separate launches: the bounds of every orientation come first, and the
// tables are shared by all orientations whose half-widths fall into the same
// step of a geometric ladder (at most 32 tables instead of one per
// orientation).
#pragma once

#include "kernels.cuh"

namespace spx {

constexpr int kBlockRows = 512;        // largest number of coupled states
constexpr int kBlockLevels = 32;       // steps of the half-width ladder (Bessel tables)
constexpr int kBlockMaxEntries = 24;   // entries of one lane
constexpr int kBlockTraj = 4;          // steps per chunk of runs that write the state at every step

// One layout of the rows on a CTA's lanes (device pointers).
struct BlockLayout {
    int n;                      // coupled states
    int nv;                     // detection rows
    int threads;                // lanes (the CTA of the FP64 kernel has two threads for each)
    int ecap;                   // entries per lane
    const int *lane_row;        // [threads] state row, n + v for detection row v, -1: none
    const int *lane_part;       // [threads] lanes of the row | part index << 8
    const int *warp_shape;      // [threads/32] entries per lane | shuffle rounds << 8
    const int *src;             // [ecap][threads] real part of an ELL entry of the system, its imaginary part
                                // (ell_len later), -1 none, -2-i: value i of the detection rows
    const uint16_t *col;        // [ecap][threads] state row the entry reads, n + row: 1i times that
    const int *row_src;         // [n] row of the system (sliced order)
    const int *state_pos;       // [n] place of the row in the run's state arrays
    const double *vval;         // entry values of the detection rows
    const int *vchan;           // [nv] channel of a detection row
    const int *vfac;            // [nv] 0: times 1, 1: times -1i (imaginary parts of a complex coil)
};

struct BlockRun {
    int n_orient;
    const double *alpha, *beta, *gamma;
    int pick;                   // 0: orientation o of the grid; else orientation ((2 o + 1) pick) / (2 n_orient)
    double dt;
    int nsteps;
    int Mcap;                   // largest chunk (steps)
    double chunk_x;             // series argument of one chunk
    int Kmax;                   // largest series
    double tol;
    int lanczos_its, safe_bounds;
    // bounds and ladder
    double *centre;             // [n_orient]
    double *halfwidth;          // [n_orient]
    unsigned long long *extent; // [2] largest half-width's bits, complement of the smallest's (zeroed)
    int nlev;                   // ladder steps in use, 1..kBlockLevels
    double *lev_half;           // [nlev]
    int *lev_m, *lev_k, *lev_raw;   // [nlev] steps per chunk, table rows, series length before the cap
    int *kcut;                  // [nlev][Mcap+1] terms a column needs
    double *table;              // [nlev][Kmax][block_row(M)] (2 - delta_k0) J_k(half j dt)
    float *tablef;              // the same in float, times block_sign(k), or null
    double max_im_diag;
    int adjoint;                // propagate under -H + 1i R: the adjoint of exp(-1i L dt)
    // states (read and written at state_pos)
    const double2 *rho0;        // one initial state
    const double2 *rho0s;       // or one per orientation, state_stride apart
    size_t state_stride;
    double2 *state_out;         // or null: the state after the last step, state_stride apart
    void *traj_out;             // or null: [n_orient][nsteps+1][n] the state at every step, in the run's precision
    void *fids;                 // [n_orient][nchan][nsteps+1]; not written when nv == 0
    int nchan;
    double *saved;              // or null: every orientation's assembled L, in lane order (block_saved)
    int *status, *kused, *mused;
    long long *matvecs;
};

// FP32 entries of one lane: values as hi + lo floats, and the byte offset of
// the state they multiply.  All values are real: a complex system (EXT) keeps
// 1i x beside x, its entries' real and imaginary parts are entries of their own
// that read one or the other, and a part that is zero for every orientation is
// left out (of 1904 entries of a magic-angle-spinning block none has both).
template <int ECAP> struct BlockEntries {
    float hi[ECAP], lo[ECAP];
    int col[ECAP];
    __device__ __forceinline__ void set(int i, double v) { split(v, hi[i], lo[i]); }
    // (Y, L, P) += v * x: Y + L + P is the sum.  The product is exact inside the
    // fused multiply-adds, so the low-order part L keeps the product's rounding
    // as well as the sum's; P sums the products of the values' low parts.  Each
    // of the three takes one dependent operation per entry.
    __device__ __forceinline__ void mac(int i, f2x &Y, f2x &L, f2x &P, f2x X) const {
        const f2x H = f2pk(hi[i], hi[i]);
        const f2x S = fma2(H, X, Y);
        L = add2(L, fma2(H, X, sub2(Y, S)));
        Y = S;
        P = fma2(f2pk(lo[i], lo[i]), X, P);
    }
    __device__ __forceinline__ void plain(int i, float2 &y, float2 x) const {
        y.x = fmaf(hi[i], x.x, y.x);
        y.y = fmaf(hi[i], x.y, y.y);
    }
    __device__ __forceinline__ float mag(int i) const { return fabsf(hi[i]); }
};

// The CTA's barrier for the terms, whose loops differ between warps (each warp
// arrives from its own instance of the loop).
static __device__ __forceinline__ void block_sync() { asm volatile("barrier.sync 0;" ::: "memory"); }
static __device__ __forceinline__ void st_shared(uint32_t a, f2x v) {
    asm volatile("st.shared.b64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}

// What a lane knows about its row.
struct BlockLane {
    int row;                    // state row, n + v, or -1
    int parts, part;            // lanes of the row, this lane's index among them
    int ew, rounds;             // entries per lane and shuffle rounds of the warp
    bool own;                   // holds the row's diagonal and state
    bool state;                 // own and a state row (not a detection row)
};
static __device__ __forceinline__ BlockLane block_lane(const BlockLayout &B, int t) {
    BlockLane l;
    l.row = B.lane_row[t];
    const int p = B.lane_part[t], w = B.warp_shape[t >> 5];
    l.parts = p & 0xff;
    l.part = p >> 8;
    l.ew = w & 0xff;
    l.rounds = w >> 8;
    l.own = l.row >= 0 && l.part == 0;
    l.state = l.own && l.row < B.n;
    return l;
}

// The thread whose part of the layout a thread plays.  An SM's warp slots belong
// to its four units by turns, so CTAs of two warps would all put their first
// warp, the one with the wide rows, on the same two units: every other pair of
// CTAs plays the parts the other way round (seven spins, 1000 orientations: 1.54
// -> 1.38 ms; CTAs of three warps and more are spread well enough, and turning
// those too costs 3 to 15 %).  Ends with a barrier where it takes one.
static __device__ __forceinline__ int block_role(int nwarps) {
    if (nwarps != 2) return threadIdx.x;
    __shared__ int s_turned;
    if (threadIdx.x == 0) {
        unsigned slot;
        asm volatile("mov.u32 %0, %%warpid;" : "=r"(slot));
        s_turned = (slot >> 2) & 1;
    }
    __syncthreads();
    return threadIdx.x ^ (32 * s_turned);
}

// One lane's entries of an orientation's L: FP64 sums over the value streams
// (coef: the rotational coefficients), stream by stream, so that the loads of
// all entries are in flight together; detection rows keep their values.
// sign: -1 for the adjoint generator -H + 1i R.
template <int ECAP>
static __device__ __forceinline__ void block_assemble(const DevSystem &sys, const BlockLayout &B, int ew, int t,
                                                      const double *coef, double sign, double (&v)[ECAP]) {
    int src[ECAP];
    const double *at[ECAP];
#pragma unroll
    for (int i = 0; i < ECAP; ++i) {
        src[i] = i < ew ? B.src[i * B.threads + t] : -1;
        at[i] = src[i] < sys.ell_len ? sys.ell_re + src[i] : sys.ell_im + (src[i] - sys.ell_len);
        v[i] = 0.0;
    }
    for (int s = 0; s < sys.nstreams; ++s) {
        const double c = coef[sys.stream_coef[s]];
        const size_t off = (size_t)s * sys.ell_len;
#pragma unroll
        for (int i = 0; i < ECAP; ++i)
            if (src[i] >= 0) v[i] = fma(c, at[i][off], v[i]);
    }
#pragma unroll
    for (int i = 0; i < ECAP; ++i) {
        v[i] *= sign;
        if (src[i] <= -2) v[i] = B.vval[-2 - src[i]];
    }
}

// Diagonal entry of system row r.
static __device__ __forceinline__ double2 block_diagonal(const DevSystem &sys, int r, const double *coef, double sign) {
    double2 dg = make_double2(0.0, 0.0);
    for (int s = 0; s < sys.nstreams; ++s) {
        const double c = coef[sys.stream_coef[s]];
        const double2 d = sys.diag[(size_t)s * sys.n_pad + r];
        dg.x = fma(c, d.x, dg.x);
        dg.y = fma(c, d.y, dg.y);
    }
    dg.x *= sign;
    return dg;
}

// Doubles of one orientation in BlockRun::saved: the lanes' entries, then
// their diagonals.
static __host__ __device__ inline size_t block_saved(int ecap, int threads) { return (size_t)threads * (ecap + 2); }

// Index in the grid of the run's orientation o.
static __device__ __forceinline__ int block_grid_index(const BlockRun &R, int o) {
    return R.pick ? (int)(((2 * (long long)o + 1) * R.pick) / (2 * (long long)R.n_orient)) : o;
}

// Rotational coefficients of the run's orientation o into coef (all threads call).
static __device__ __forceinline__ void block_coefficients(const DevSystem &sys, const BlockRun &R, int o, double *coef) {
    o = block_grid_index(R, o);
    wigner_coefficients(sys, R.alpha[o], R.beta[o], R.gamma[o], coef);
}

// Extreme eigenvalues (low, high) of the tridiagonal matrix (al, be), by one
// warp: lanes 0-15 bracket the lowest, lanes 16-31 the highest, each round
// counting the eigenvalues below 16 interior points (Sturm sequences) and
// shrinking its bracket 17-fold, to 1e-6 of its size.  The counts stay right to
// the division's rounding; the interval is widened by far more afterwards.
static __device__ __forceinline__ double2 tridiag_ends(const float *al, const float *be, int m, int lane) {
    float a = CUDART_INF_F, b = -CUDART_INF_F;
    for (int i = lane; i < m; i += 32) {
        const float r = (i > 0 ? fabsf(be[i - 1]) : 0.f) + (i < m - 1 ? fabsf(be[i]) : 0.f);
        a = fminf(a, al[i] - r);
        b = fmaxf(b, al[i] + r);
    }
#pragma unroll
    for (int q = 16; q; q >>= 1) {
        a = fminf(a, __shfl_xor_sync(0xffffffffu, a, q));
        b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, q));
    }
    const bool high = lane >= 16;
    const int target = high ? m : 1;                             // count >= target: right of the wanted one
    for (int it = 0; it < 8; ++it) {
        const float step = (b - a) * (1.f / 17.f), x = a + (float)((lane & 15) + 1) * step;
        int cnt = 0;
        float q = al[0] - x;
        cnt += q < 0.f;
        for (int i = 1; i < m; ++i) {
            const float e = be[i - 1];
            q = al[i] - x - __fdividef(e * e, q == 0.f ? 1e-30f : q);
            cnt += q < 0.f;
        }
        const unsigned mask = (__ballot_sync(0xffffffffu, cnt >= target) >> (high ? 16 : 0)) & 0xffffu;
        const int j = mask ? __ffs(mask) - 1 : 16;
        b = mask ? a + (float)(j + 1) * step : b;
        a = a + (float)j * step;
        const bool done = !(b - a > 1e-6f * fmaxf(fabsf(a), fabsf(b)) + 1e-30f);
        if (__all_sync(0xffffffffu, done)) break;
    }
    // the outer end of each bracket
    return make_double2((double)__shfl_sync(0xffffffffu, a, 0), (double)__shfl_sync(0xffffffffu, b, 31));
}

// |last component| of the tridiagonal matrix's unit eigenvector at theta, by
// two steps of inverse iteration (one thread; w: work arrays).
static __device__ float ritz_last(const float *al, const float *be, int m, float theta, float (*w)[kMaxLanczos]) {
    if (m <= 1) return 1.f;
    float *y = w[0], *c = w[1], *d = w[2];
    const float shift = theta + 1e-5f * (fabsf(theta) + 1e-30f);
    for (int i = 0; i < m; ++i) y[i] = 1.f;
    for (int it = 0; it < 2; ++it) {
        float den = al[0] - shift, cp, dp;                       // (T - shift) x = y
        den = den == 0.f ? 1e-30f : den;
        cp = c[0] = __fdividef(be[0], den);
        dp = d[0] = __fdividef(y[0], den);
        for (int i = 1; i < m; ++i) {
            const float e = be[i - 1];
            den = al[i] - shift - e * cp;
            den = den == 0.f ? 1e-30f : den;
            const float inv = __fdividef(1.f, den);
            cp = c[i] = i < m - 1 ? be[i] * inv : 0.f;
            dp = d[i] = (y[i] - e * dp) * inv;
        }
        float x = dp, nrm = x * x;
        y[m - 1] = x;
        for (int i = m - 2; i >= 0; --i) {
            x = d[i] - c[i] * x;
            y[i] = x;
            nrm += x * x;
        }
        if (!(nrm > 0.f) || !isfinite(nrm)) return 1.f;
        const float inv = rsqrtf(nrm);
        for (int i = 0; i < m; ++i) y[i] *= inv;
    }
    return fabsf(y[m - 1]);
}

// ---------------------------------------------------------------------------
// Spectral bounds of every orientation of FP32 runs: Gershgorin discs, and Lanczos
// on the Hermitian part, in FP32 (the interval is widened by the Ritz residuals
// and 2% of its width, and the propagation watches the norm).
// The matrix is taken about the middle of its discs, so that alpha is no larger
// than the spread.  The assembled L goes to R.saved for the FP32 propagation, which
// runs on the same layout.
// ---------------------------------------------------------------------------
template <bool EXT, int ECAP>
__global__ void __launch_bounds__(kBlockRows, ECAP <= 16 ? 2 : 1) block_bounds_kernel(const DevSystem sys, const BlockLayout B,
                                                                     const BlockRun R) {
    __shared__ double s_coef[kMaxCoef];
    __shared__ float2 s_x[2][(EXT ? 2 : 1) * kBlockRows + 1];
    __shared__ float2 s_part[2][kBlockRows / 32];
    __shared__ float s_al[kMaxLanczos], s_be[kMaxLanczos];
    __shared__ float s_work[2][3][kMaxLanczos];
    const int o = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const BlockLane l = block_lane(B, tid);
    block_coefficients(sys, R, o, s_coef);
    BlockEntries<ECAP> E;
    double2 dg = make_double2(0.0, 0.0);
    {
        const double sign = R.adjoint ? -1.0 : 1.0;
        double *save = R.saved ? R.saved + (size_t)o * block_saved(B.ecap, B.threads) : nullptr;
        // four entries at a time: more FP64 sums in registers cost resident CTAs
#pragma unroll
        for (int i0 = 0; i0 < ECAP; i0 += 4) {
            double v[4];
            BlockLayout Bi = B;
            Bi.src = B.src + (size_t)i0 * B.threads;
            block_assemble<4>(sys, Bi, l.ew - i0, tid, s_coef, sign, v);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int i = i0 + q;
                E.set(i, v[q]);
                E.col[i] = i < l.ew ? B.col[i * B.threads + tid] * (int)sizeof(float2) : 0;
                if (save && i < l.ew) save[(size_t)i * B.threads + tid] = v[q];
            }
        }
        if (l.state) dg = block_diagonal(sys, B.row_src[l.row], s_coef, sign);
        if (save) {
            double *sd = save + (size_t)B.ecap * B.threads;
            sd[tid] = dg.x;
            sd[B.threads + tid] = dg.y;
        }
    }
    int par = 0;
    // sums (op 0) or maxima (op 1) of both components over the CTA; the slots
    // alternate, so one barrier each
    auto reduce = [&](float2 v, int op) {
#pragma unroll
        for (int q = 16; q; q >>= 1) {
            const float ux = __shfl_xor_sync(0xffffffffu, v.x, q), uy = __shfl_xor_sync(0xffffffffu, v.y, q);
            v.x = op ? fmaxf(v.x, ux) : v.x + ux;
            v.y = op ? fmaxf(v.y, uy) : v.y + uy;
        }
        if (nwarps == 1) return v;
        if (lane == 0) s_part[par][warp] = v;
        __syncthreads();
        v = s_part[par][0];
        for (int w = 1; w < nwarps; ++w) {
            const float2 u = s_part[par][w];
            v.x = op ? fmaxf(v.x, u.x) : v.x + u.x;
            v.y = op ? fmaxf(v.y, u.y) : v.y + u.y;
        }
        par ^= 1;
        return v;
    };
    auto join = [&](float v) {                                // sum over the parts of a row
        for (int r = 0; r < l.rounds; ++r) {
            const float u = __shfl_xor_sync(0xffffffffu, v, 1 << r);
            if ((l.parts >> r) > 1) v += u;
        }
        return v;
    };
    float rad = 0.f;
#pragma unroll
    for (int i = 0; i < ECAP; ++i) rad += E.mag(i);
    rad = join(rad);
    // float sums: 4e-6 of the row covers their rounding
    const float dgf = (float)dg.x, slack = 4e-6f * (fabsf(dgf) + rad);
    const float2 g = reduce(l.state ? make_float2(dgf + rad + slack, -(dgf - rad - slack))
                                    : make_float2(-CUDART_INF_F, -CUDART_INF_F), 1);
    const double gmax = g.x, gmin = -g.y, mid = 0.5 * (gmax + gmin);
    const float dre = (float)(dg.x - mid);

    float2 q_cur = make_float2(0.f, 0.f), q_prev = q_cur;
    if (l.state) q_cur.x = 1.0f + 0.37f * __sinf(1.7f * (float)l.row + 0.3f);
    {
        const float inv = rsqrtf(reduce(make_float2(q_cur.x * q_cur.x, 0.f), 0).x);
        q_cur.x *= inv;
    }
    float beta_prev = 0.f;
    int m_eff = 0;
    // also beyond n steps: FP32 vectors lose their orthogonality on clustered
    // spectra, and n steps then miss the ends (more only find them again)
    const int lits = min(R.lanczos_its, kMaxLanczos);
    const int slot = l.state ? l.row : (EXT ? 2 : 1) * kBlockRows, slot2 = l.state ? B.n + l.row : slot;
    for (int j = 0; j < lits; ++j) {
        float2 *x = s_x[j & 1];
        x[slot] = q_cur;
        if (EXT) x[slot2] = make_float2(-q_cur.y, q_cur.x);
        __syncthreads();
        float2 y = make_float2(0.f, 0.f);
        const char *xb = reinterpret_cast<const char *>(x);
#pragma unroll
        for (int i = 0; i < ECAP; ++i) E.plain(i, y, *reinterpret_cast<const float2 *>(xb + E.col[i]));
        y.x = join(y.x);
        y.y = join(y.y);
        if (l.state) {
            y.x += dre * q_cur.x - beta_prev * q_prev.x;
            y.y += dre * q_cur.y - beta_prev * q_prev.y;
        } else {
            y = make_float2(0.f, 0.f);
        }
        const float alpha = reduce(make_float2(q_cur.x * y.x + q_cur.y * y.y, 0.f), 0).x;
        y.x -= alpha * q_cur.x;
        y.y -= alpha * q_cur.y;
        // beta from the residual itself: |w|^2 - alpha^2 would hide directions
        // that the start vector holds little of
        const float beta = sqrtf(reduce(make_float2(y.x * y.x + y.y * y.y, 0.f), 0).x);
        if (tid == 0) { s_al[j] = alpha; s_be[j] = beta; }
        m_eff = j + 1;
        if (!(beta > 1e-12f * (fabsf(alpha) + 1e-30f))) break;      // invariant subspace
        const float inv = 1.f / beta;
        q_prev = q_cur;
        q_cur.x = y.x * inv;
        q_cur.y = y.y * inv;
        beta_prev = beta;
    }
    __syncthreads();
    if (tid < 32) {
        const double2 ends = tridiag_ends(s_al, s_be, m_eff, lane);
        const double tlo = ends.x, thi = ends.y;
        float rr = 0.f;                                          // lane 0 the top, lane 1 the bottom
        if (!R.safe_bounds && lane < 2)
            rr = fabsf(s_be[m_eff - 1]) * ritz_last(s_al, s_be, m_eff, lane == 0 ? (float)thi : (float)tlo, s_work[lane]);
        const double rhi = __shfl_sync(0xffffffffu, rr, 0), rlo = __shfl_sync(0xffffffffu, rr, 1);
        if (lane == 0) {
            double hi = gmax, lo = gmin;
            if (!R.safe_bounds) {
                const double wid = thi - tlo;
                hi = fmin(mid + thi + rhi + 0.02 * wid, gmax);
                lo = fmax(mid + tlo - rlo - 0.02 * wid, gmin);
                if (!(hi >= lo)) { hi = gmax; lo = gmin; }
            }
            const double scale = fmax(fabs(hi), fabs(lo));
            const double half = fmax(0.5 * (hi - lo) * 1.01 + 1e-9 * scale, R.max_im_diag) + 1e-30;
            R.centre[o] = 0.5 * (hi + lo);
            R.halfwidth[o] = half;
            const unsigned long long bits = (unsigned long long)__double_as_longlong(half);   // half > 0
            atomicMax(R.extent, bits);
            atomicMax(R.extent + 1, ~bits);
        }
    }
}

// The same in FP64 for FP64 runs.  Real couplings keep real vectors.  Bound by
// latency: a step is one product and two sums over the CTA, 32 times, and an FP64
// instruction takes a warp 64 cycles, so it runs just its warp's entries, on the
// layout that the host finds cheapest for it (with FP32 bounds and with these:
// seven spins, 1000 orientations, 2048 steps in FP64 13.67 and 13.58 ms; one
// orientation of a radical with three protons, 127 steps, 0.35 and 0.39 ms).
template <bool EXT, int ECAP>
__global__ void __launch_bounds__(kBlockRows, 1)
    block_bounds64_kernel(const DevSystem sys, const BlockLayout B, const BlockRun R) {
    using Vec = std::conditional_t<EXT, double2, double>;          // a state's part of a Lanczos vector
    constexpr int XN = (EXT ? 2 : 1) * kBlockRows;            // the last slot takes what no one reads
    __shared__ double s_coef[kMaxCoef];
    __shared__ Vec s_x[2][XN + 1];
    __shared__ double2 s_part[2][kBlockRows / 32];
    __shared__ float s_al[kMaxLanczos], s_be[kMaxLanczos];
    __shared__ float s_work[2][3][kMaxLanczos];
    const int o = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const BlockLane l = block_lane(B, tid);
    block_coefficients(sys, R, o, s_coef);
    double val[ECAP];
    int col[ECAP];                                            // byte offsets
    double2 dg = make_double2(0.0, 0.0);
    {
        const double sign = R.adjoint ? -1.0 : 1.0;
        // four entries at a time: more FP64 sums in registers cost resident CTAs
#pragma unroll
        for (int i0 = 0; i0 < ECAP; i0 += 4) {
            double v[4];
            BlockLayout Bi = B;
            Bi.src = B.src + (size_t)i0 * B.threads;
            block_assemble<4>(sys, Bi, l.ew - i0, tid, s_coef, sign, v);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int i = i0 + q;
                val[i] = v[q];
                col[i] = i < l.ew ? B.col[i * B.threads + tid] * (int)sizeof(Vec) : 0;
            }
        }
        if (l.state) dg = block_diagonal(sys, B.row_src[l.row], s_coef, sign);
    }
    int par = 0;
    // sum over the CTA; the slots alternate, so one barrier each
    auto sum = [&](double v) {
#pragma unroll
        for (int q = 16; q; q >>= 1) v += __shfl_xor_sync(0xffffffffu, v, q);
        if (nwarps == 1) return v;
        if (lane == 0) s_part[par][warp].x = v;
        __syncthreads();
        v = lane < nwarps ? s_part[par][lane].x : 0.0;        // log2 of the warps' additions
        for (int q = 1; q < nwarps; q *= 2) v += __shfl_xor_sync(0xffffffffu, v, q);
        v = __shfl_sync(0xffffffffu, v, 0);
        par ^= 1;
        return v;
    };
    // largest of both components over the CTA
    auto largest = [&](double2 v) {
#pragma unroll
        for (int q = 16; q; q >>= 1) {
            const double ux = __shfl_xor_sync(0xffffffffu, v.x, q), uy = __shfl_xor_sync(0xffffffffu, v.y, q);
            v.x = ux > v.x ? ux : v.x;
            v.y = uy > v.y ? uy : v.y;
        }
        if (nwarps == 1) return v;
        if (lane == 0) s_part[par][warp] = v;
        __syncthreads();
        for (int w = 0; w < nwarps; ++w) {
            const double2 u = s_part[par][w];
            v.x = u.x > v.x ? u.x : v.x;
            v.y = u.y > v.y ? u.y : v.y;
        }
        par ^= 1;
        return v;
    };
    auto join = [&](double v) {                                 // sum over the parts of a row
        for (int r = 0; r < l.rounds; ++r) {
            const double u = __shfl_xor_sync(0xffffffffu, v, 1 << r);
            if ((l.parts >> r) > 1) v += u;
        }
        return v;
    };
    double rad = 0;
#pragma unroll
    for (int i = 0; i < ECAP; ++i)
        if (i < l.ew) rad += fabs(val[i]);
    rad = join(rad);
    const double2 ends = largest(l.state ? make_double2(dg.x + rad, rad - dg.x) : make_double2(-CUDART_INF, -CUDART_INF));
    const double gmax = ends.x, gmin = -ends.y, mid = 0.5 * (gmax + gmin);
    const double dre = dg.x - mid;

    Vec q_cur{}, q_prev{};
    auto re = [](Vec &v) -> double & { if constexpr (EXT) return v.x; else return v; };
    // over the real and, where there are any, the imaginary parts of two vectors
    auto dot = [](const Vec &a, const Vec &b) -> double {
        if constexpr (EXT) return a.x * b.x + a.y * b.y;
        else return a * b;
    };
    if (l.state) re(q_cur) = (double)(1.0f + 0.37f * __sinf(1.7f * (float)l.row + 0.3f));
    re(q_cur) *= rsqrt(sum(re(q_cur) * re(q_cur)));
    double beta_prev = 0;
    int m_eff = 0;
    const int lits = min(R.lanczos_its, min(kMaxLanczos, B.n));
    const int slot = l.state ? l.row : XN, slot2 = l.state ? B.n + l.row : slot;
    for (int j = 0; j < lits; ++j) {
        Vec *x = s_x[j & 1];
        x[slot] = q_cur;
        if constexpr (EXT) {
            Vec turned;
            turned.x = -q_cur.y;
            turned.y = q_cur.x;
            x[slot2] = turned;
        }
        __syncthreads();
        Vec y{};
        const char *xb = reinterpret_cast<const char *>(x);
#pragma unroll
        for (int i = 0; i < ECAP; ++i)
            if (i < l.ew) {
                const Vec xi = *reinterpret_cast<const Vec *>(xb + col[i]);
                if constexpr (EXT) { y.x = fma(val[i], xi.x, y.x); y.y = fma(val[i], xi.y, y.y); }
                else y = fma(val[i], xi, y);
            }
        if constexpr (EXT) { y.x = join(y.x); y.y = join(y.y); }
        else y = join(y);
        if (!l.state) y = Vec{};
        else if constexpr (EXT) {
            y.x += dre * q_cur.x - beta_prev * q_prev.x;
            y.y += dre * q_cur.y - beta_prev * q_prev.y;
        } else {
            y += dre * q_cur - beta_prev * q_prev;
        }
        const double alpha = sum(dot(q_cur, y));
        if constexpr (EXT) { y.x -= alpha * q_cur.x; y.y -= alpha * q_cur.y; }
        else y -= alpha * q_cur;
        // beta from the residual itself: |w|^2 - alpha^2 would hide directions
        // that the start vector holds little of
        const double beta2 = sum(dot(y, y));
        double beta, inv;
        if (beta2 > 1e-30 && beta2 < 1e30) {
            // a float's reciprocal root and one Newton step (to 5e-15): a third of the
            // FP64 instructions of sqrt and a division, which were half of a step's
            const double r = (double)rsqrtf((float)beta2);
            inv = r * fma(-0.5 * beta2, r * r, 1.5);
            beta = beta2 * inv;
        } else {
            beta = sqrt(beta2);
            inv = 1.0 / beta;
        }
        if (tid == 0) { s_al[j] = (float)alpha; s_be[j] = (float)beta; }
        m_eff = j + 1;
        if (!(beta > 1e-12 * (fabs(alpha) + 1e-30))) break;      // invariant subspace
        q_prev = q_cur;
        if constexpr (EXT) { q_cur.x = y.x * inv; q_cur.y = y.y * inv; }
        else q_cur = y * inv;
        beta_prev = beta;
    }
    __syncthreads();
    if (tid < 32) {
        const double2 ritz = tridiag_ends(s_al, s_be, m_eff, lane);
        const double tlo = ritz.x, thi = ritz.y;
        float rr = 0.f;                                          // lane 0 the top, lane 1 the bottom
        if (!R.safe_bounds && lane < 2)
            rr = fabsf(s_be[m_eff - 1]) * ritz_last(s_al, s_be, m_eff, lane == 0 ? (float)thi : (float)tlo, s_work[lane]);
        const double rhi = __shfl_sync(0xffffffffu, rr, 0), rlo = __shfl_sync(0xffffffffu, rr, 1);
        if (lane == 0) {
            double hi = gmax, lo = gmin;
            if (!R.safe_bounds) {
                const double wid = thi - tlo;
                hi = fmin(mid + thi + rhi + 0.02 * wid, gmax);
                lo = fmax(mid + tlo - rlo - 0.02 * wid, gmin);
                if (!(hi >= lo)) { hi = gmax; lo = gmin; }
            }
            const double scale = fmax(fabs(hi), fabs(lo));
            const double half = fmax(0.5 * (hi - lo) * 1.01 + 1e-9 * scale, R.max_im_diag) + 1e-30;
            R.centre[o] = 0.5 * (hi + lo);
            R.halfwidth[o] = half;
            const unsigned long long bits = (unsigned long long)__double_as_longlong(half);   // half > 0
            atomicMax(R.extent, bits);
            atomicMax(R.extent + 1, ~bits);
        }
    }
}

// ---------------------------------------------------------------------------
// Bessel tables of the ladder: step i has half-width hmax * exp(-i * step);
// an orientation takes the last step that still covers its own half-width, so
// it runs at most e^step more terms than with a table of its own (16 steps to
// an octave: 2 % on average).  Grid (columns / 32, steps); only steps that an
// orientation takes are tabulated.
// ---------------------------------------------------------------------------
static __device__ __noinline__ double ladder_half(const unsigned long long *extent, int nlev, int lev) {
    const double hmax = __longlong_as_double((long long)extent[0]);
    const double hmin = __longlong_as_double((long long)~extent[1]);
    double step = 0.69314718055994531 / 16;
    if (nlev > 1) step = fmax(step, log(hmax / hmin) / (nlev - 1));
    return lev == 0 ? hmax : hmax * exp(-lev * step);
}

// (-1i)^k is this sign times 1 (even k) or -1i (odd k).
static __device__ __forceinline__ double block_sign(int k) { return (k & 2) ? -1.0 : 1.0; }

// Table rows are a multiple of 16 bytes long, so that a thread takes the
// values of neighbouring columns in one load.
static __host__ __device__ inline int block_row(int M) { return (M + 4) & ~3; }

// Column j of a table by Miller's backward recurrence (bessel_column of
// kernels.cuh), unnormalised; returns the factor that normalises it and the
// number of terms that are not zero (kn).
static __device__ double block_column(double *tab, int M, int j, int K, double half, double dt, int &kn) {
    const size_t ld = (size_t)block_row(M);
    double *col = tab + j;
    const double x = half * j * dt;
    kn = min(K, 3);
    if (x < 1e-6) {
        // half the leading terms (every term but the first is doubled later)
        col[0] = 1.0 - 0.25 * x * x;
        if (K > 1) col[ld] = 0.5 * x;
        if (K > 2) col[2 * ld] = 0.125 * x * x;
        return 1.0;
    }
    kn = min(K, series_terms(x, 0.0, 1e-40, K + 64) + 1);
    const int base = max(kn, (int)ceil(x));
    int kst = base + 20 + (int)sqrtf(160.f * base);
    kst += kst & 1;
    const double two_over_x = 2.0 / x;
    const float ftx = (float)two_over_x;
    float fjp1 = 0.f, fjk = 1e-30f;
    int k = kst;
    for (; k > kn; --k) {
        const float fjm1 = ((float)k * ftx) * fjk - fjp1;
        fjp1 = fjk;
        fjk = fjm1;
        if (fabsf(fjk) > 1e20f) { fjk *= 1e-20f; fjp1 *= 1e-20f; }
    }
    // an FP64 instruction takes a warp 64 cycles: one conversion and product
    // for two terms, and only even orders enter the norm
    double jp1 = fjp1, jk = fjk, even = 0.0;
    if (k & 1) {                                      // an odd number of terms: one alone first
        const double jm1 = (k * two_over_x) * jk - jp1;
        jp1 = jk;
        jk = jm1;
        --k;
        if (k > 0) even += jk;
        col[(size_t)k * ld] = jk;
    }
    for (; k >= 2; k -= 2) {
        const double f = k * two_over_x;
        const double a = f * jk - jp1;                // J_{k-1}
        const double b = (f - two_over_x) * a - jk;   // J_{k-2}
        col[(size_t)(k - 1) * ld] = a;
        col[(size_t)(k - 2) * ld] = b;
        if (k > 2) even += b;
        jp1 = a;
        jk = b;
    }
    return 1.0 / (2.0 * even + jk);                   // J_0 + 2 sum J_2k = 1
}

static __global__ void __launch_bounds__(128) block_tables_kernel(const BlockRun R) {
    const int lev = blockIdx.y, tid = threadIdx.x;
    const double half = ladder_half(R.extent, R.nlev, lev);
    const double next = lev + 1 < R.nlev ? ladder_half(R.extent, R.nlev, lev + 1) : 0.0;
    __shared__ int s_k, s_raw;
    if (tid == 0) s_k = 0;
    __syncthreads();
    for (int o = tid; o < R.n_orient; o += blockDim.x) {
        const double h = R.halfwidth[o];
        if (h <= half && !(h <= next)) { s_k = 1; break; }
    }
    __syncthreads();
    const bool used = s_k != 0;
    __syncthreads();
    const double target = R.chunk_x / (half * R.dt);
    // a chunk damps the state by at most e^2: the terms grow with Im L, and
    // their sum loses the digits they gained
    const double damped = R.max_im_diag > 0.0 ? floor(2.0 / (R.max_im_diag * R.dt)) : (double)R.Mcap;
    const int M = min((int)fmax(1.0, fmin((double)R.Mcap, fmin(damped, floor(target)))), R.nsteps + 1);
    const double lg = 2.0 * R.max_im_diag / half;
    if (tid == 0) {
        s_raw = used ? series_terms(half * M * R.dt, lg, R.tol, R.Kmax + 1) : 0;
        s_k = used ? min(R.Kmax, max(2, s_raw) + 2) : 0;        // 0: no table
        if (blockIdx.x == 0) {
            R.lev_half[lev] = half;
            R.lev_m[lev] = M;
            R.lev_k[lev] = s_k;
            R.lev_raw[lev] = s_raw;
        }
    }
    __syncthreads();
    if (!used || blockIdx.x * 32 > M) return;
    __shared__ double s_inv[32];
    __shared__ int s_kn[32];
    const int lane = tid & 31, warp = tid >> 5, j = blockIdx.x * 32 + lane;
    const int K = s_k;
    const size_t ld = (size_t)block_row(M), at = (size_t)lev * R.Kmax * block_row(R.Mcap);
    double *tab = R.table + at;
    float *tf = R.tablef ? R.tablef + at : nullptr;
    // one warp runs the columns' recurrences; all four scale and round them,
    // eight values of a column in flight
    if (warp == 0 && j <= M) s_inv[lane] = block_column(tab, M, j, K, half, R.dt, s_kn[lane]);
    __syncthreads();
    if (j > M) return;
    const double inv = s_inv[lane], two = 2.0 * inv;
    const int kn = s_kn[lane];
    for (int k0 = 8 * warp; k0 < K; k0 += 32) {
        double v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = k0 + q < kn ? tab[(size_t)(k0 + q) * ld + j] : 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int k = k0 + q;
            if (k < K) {
                v[q] *= k == 0 ? inv : two;
                tab[(size_t)k * ld + j] = v[q];
                if (tf) tf[(size_t)k * ld + j] = (float)((k == 0 ? 2.0 : block_sign(k)) * v[q]);   // FP32 moments 0 are halved
            }
        }
    }
    __syncthreads();
    if (warp != 0) return;
    // terms the column needs: the last one above the tolerance (with the growth
    // e^{k lg} that Im L allows), plus two
    int last = 2;
    double grow = exp((kn - 1) * lg);
    const double shrink = exp(-lg);
    for (int k0 = kn - 1; k0 >= 2 && last == 2; k0 -= 8) {
        double v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = k0 - q >= 2 ? tab[(size_t)(k0 - q) * ld + j] : 0.0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            if (last == 2 && k0 - q >= 2 && !(fabs(v[q]) * grow <= R.tol)) last = k0 - q + 1;
            if (lg > 0.0) grow *= shrink;
        }
    }
    R.kcut[(size_t)lev * (R.Mcap + 1) + j] = min(last + 2, K);
}

constexpr int kBlockPoints32 = 4, kBlockPoints64 = 1;      // points a thread sums together (block_points)

// Shared memory for the points' partial sums, and all dynamic shared memory of
// the propagation kernels.
static __host__ __device__ inline size_t block_rec(int Mcap, int threads, int points) {
    return (size_t)points * (size_t)(threads > Mcap / points + 1 ? threads : Mcap / points + 1);
}
static __host__ __device__ inline size_t block_smem32(int Kmax, int Mcap, int nv, int threads, bool traj) {
    return 8 * ((size_t)(Kmax + 2) * (1 + nv + (traj ? kBlockTraj - 1 : 0)) + (size_t)(Mcap + 1) +
                block_rec(Mcap, threads, kBlockPoints32));
}
static __host__ __device__ inline size_t block_smem64(int Kmax, int Mcap, int nv, int lanes, int ecap, int n, bool ext,
                                                      bool traj) {
    return 16 * (block_rec(Mcap, 2 * lanes, kBlockPoints64) + (size_t)(Mcap + 1) + (size_t)(Kmax + 2) * nv) +
           8 * (size_t)(Kmax + 2) * (traj ? kBlockTraj : 1) +
           8 * (size_t)ecap * lanes + 8 * 4 * ((ext ? 2 : 1) * (size_t)n + 1) + 2 * (size_t)ecap * lanes;
}

// (-1i) * t as a packed pair
static __device__ __forceinline__ f2x turn2(f2x t) {
    const float2 f = f2up(t);
    return f2pk(f.y, -f.x);
}

// 1i * t
static __device__ __forceinline__ f2x rot2(f2x t) {
    const float2 f = f2up(t);
    return f2pk(-f.y, f.x);
}

// What a CTA knows of its orientation's series.
struct BlockSeries {
    double cen, half;
    int M, K, nchunks, j_last;
    size_t ld;                  // table row length
    const double *tab;
    const float *tabf;
    const int *kcut;
    bool ok;
};
// The ladder step of orientation o; a series longer than the table sets the
// orientation's status and ok = false.
static __device__ __forceinline__ BlockSeries block_series(const BlockRun &R, int o) {
    BlockSeries S;
    const double own = R.halfwidth[o];
    int lev = 0;
    while (lev + 1 < R.nlev && R.lev_half[lev + 1] >= own) ++lev;
    S.cen = R.centre[o];
    S.half = R.lev_half[lev];
    S.M = R.lev_m[lev];
    const int Kb = R.lev_k[lev];
    const size_t at = (size_t)lev * R.Kmax * block_row(R.Mcap);
    S.kcut = R.kcut + (size_t)lev * (R.Mcap + 1);
    S.K = Kb > 0 ? S.kcut[S.M] : 0;
    S.tab = R.table + at;
    S.tabf = R.tablef ? R.tablef + at : nullptr;
    S.ld = (size_t)block_row(S.M);
    S.nchunks = (R.nsteps + S.M) / S.M;
    S.j_last = R.nsteps - (S.nchunks - 1) * S.M;
    S.ok = !(Kb == 0 || (R.lev_raw[lev] + 2 > R.Kmax && S.K >= Kb - 2));
    if (!S.ok && threadIdx.x == 0) {
        R.status[o] = kDevTableTooSmall;
        R.kused[o] = R.Kmax + 1;
        R.mused[o] = S.M;
        R.matvecs[o] = 0;
    }
    return S;
}

// size e^{-i c j dt}, j < M: one sine and cosine per thread, turned on by
// blockDim.x steps at a time (FP64 transcendentals are slow here), and the
// phases of a whole and of the last chunk.
template <class Vec>
static __device__ __forceinline__ void block_phases(const BlockRun &R, const BlockSeries &S, double size, Vec *phase,
                                                    double2 *turn) {
    const int tid = threadIdx.x, nt = (int)blockDim.x;
    if (tid < S.M) {
        double sn, cs, rs = 0.0, rc = 1.0;
        sincos(-S.cen * tid * R.dt, &sn, &cs);
        if (S.M > nt) sincos(-S.cen * nt * R.dt, &rs, &rc);
        for (int j = tid; j < S.M; j += nt) {
            phase[j] = tovec(make_double2(size * cs, size * sn), Vec());
            const double c2 = cs * rc - sn * rs;
            sn = sn * rc + cs * rs;
            cs = c2;
        }
    }
    if (tid < 2) {
        double sn, cs;
        sincos(-S.cen * (tid == 0 ? S.M : S.j_last) * R.dt, &sn, &cs);
        turn[tid] = make_double2(cs, sn);
    }
}

// FID points of chunk a: f_j = e^{-i c j dt} sum_k J_k(s j dt) (-1i)^k mu_k.
// tr: the table in the run's precision.  After a barrier; the caller's next
// barrier ends it.  An FP32 thread sums four neighbouring points over a part of
// the terms: one 16-byte table load (from L2) and one moment serve all of them
// (three spins, 200 orientations: 0.78 ms with one point a thread, 0.66 with
// two, 0.65 with four; seven spins 1.68, 1.60, 1.54).  FP64 is bound by its
// instructions and takes one point.
template <class Vec, class Real>
static __device__ __forceinline__ void block_points(const BlockLayout &B, const BlockRun &R, const BlockSeries &S,
                                                    const Real *tr, int a, int Kc, const Vec *s_mu, const Vec *s_phase,
                                                    Vec *s_rec, Vec *fid_out) {
    constexpr int N = sizeof(Real) == 4 ? kBlockPoints32 : kBlockPoints64, UN = 8;
    using Wide = std::conditional_t<sizeof(Real) == 4, float4, double>;
    const int M = S.M, tid = threadIdx.x, nt = blockDim.x;
    const int np = min(M, R.nsteps + 1 - a * M);                // points of this chunk
    const int cols = (np + N - 1) / N;                           // threads for all of them
    const int parts = max(1, nt / cols);
    const int kper = ((Kc + parts - 1) / parts + 3) & ~3;
    const size_t ld = S.ld;
    for (int v = 0; v < B.nv; ++v) {
        const Vec *mu = s_mu + (size_t)v * (R.Kmax + 2);
        if (v > 0) __syncthreads();                              // s_rec reused
        for (int jj = tid; jj < cols * parts; jj += nt) {
            const int j = (jj % cols) * N, part = jj / cols;
            const int k0 = part * kper, k1 = min(min(Kc, k0 + kper), S.kcut[min(j + N - 1, M - 1)]);
            Vec e[N], d[N];                                      // even and odd terms
#pragma unroll
            for (int q = 0; q < N; ++q) e[q] = d[q] = vzero<Vec>();
            const Real *col = tr + j;
            // the float table holds the signs of (-1i)^k, the double one does not
            auto term = [&](int k, int odd, bool minus, const Wide &w) {
                const Vec m = mu[k];
                const Real *J = reinterpret_cast<const Real *>(&w);
#pragma unroll
                for (int q = 0; q < N; ++q) {
                    const Real b = sizeof(Real) == 8 && minus ? -J[q] : J[q];
                    Vec &t = odd ? d[q] : e[q];
                    t.x += b * m.x;
                    t.y += b * m.y;
                }
            };
            int k = k0;
            for (; k + UN <= k1; k += UN) {
                Wide w[UN];
#pragma unroll
                for (int u = 0; u < UN; ++u) w[u] = *reinterpret_cast<const Wide *>(col + (size_t)(k + u) * ld);
#pragma unroll
                for (int u = 0; u < UN; ++u) term(k + u, u & 1, u & 2, w[u]);
            }
            for (; k < k1; ++k) {
                const Wide w = *reinterpret_cast<const Wide *>(col + (size_t)k * ld);
                if (k & 1) term(k, 1, k & 2, w);
                else term(k, 0, k & 2, w);
            }
#pragma unroll
            for (int q = 0; q < N; ++q) {
                Vec f;                                           // e - 1i d
                f.x = e[q].x + d[q].y;
                f.y = e[q].y - d[q].x;
                s_rec[part * cols * N + j + q] = f;
            }
        }
        __syncthreads();
        Vec *out = fid_out + (size_t)B.vchan[v] * (R.nsteps + 1) + (size_t)a * M;
        const bool first = v == 0 || B.vchan[v] != B.vchan[v - 1];
        for (int j = tid; j < np; j += nt) {
            Vec f = s_rec[j];
            for (int q = 1; q < parts; ++q) {
                f.x += s_rec[q * cols * N + j].x;
                f.y += s_rec[q * cols * N + j].y;
            }
            const Vec ph = s_phase[j];
            Vec g;
            g.x = ph.x * f.x - ph.y * f.y;
            g.y = ph.x * f.y + ph.y * f.x;
            if (B.vfac[v]) { const Real t = g.x; g.x = g.y; g.y = -t; }
            if (!first) { g.x += out[j].x; g.y += out[j].y; }
            out[j] = g;
        }
    }
}

// Calls f(entries per lane, shuffle rounds), both compile-time, with the
// smallest instance that covers this warp (every count up to 8, then steps of
// an eighth of the kernel's largest): straight-line code, so that a term's
// loads all start before its sums (a loop that left after the warp's own entry
// count waited 70 cycles for every entry).
template <int ECAP, int EW = ECAP, class F>
static __device__ __forceinline__ void block_dispatch(const BlockLane &l, F &&f) {
    constexpr int step = ECAP <= 8 ? 1 : ECAP / 8;
    if constexpr (EW == ECAP) {
        if (l.rounds == 1) return f(std::integral_constant<int, ECAP>{}, std::integral_constant<int, 1>{});
        if (l.rounds == 2) return f(std::integral_constant<int, ECAP>{}, std::integral_constant<int, 2>{});
        if (l.rounds > 2) return f(std::integral_constant<int, ECAP>{}, std::integral_constant<int, 5>{});
    }
    if constexpr (EW > step) {
        if (l.ew <= EW - step) return block_dispatch<ECAP, EW - step>(l, f);
    }
    f(std::integral_constant<int, EW>{}, std::integral_constant<int, 0>{});
}

// ---------------------------------------------------------------------------
// Propagation, FP32: values in registers, (re, im) in packed f32x2 operations.
// ---------------------------------------------------------------------------
// TRJ: also the state at every step (R.traj_out), from chunks of at most
// kBlockTraj steps whose inner states are summed beside the chunk-end state.
// The launch bounds set the registers: 96 up to 16 entries (80 for 8 gives
// seven spins, 1000 orientations, 1.62 ms for 1.54), 128 for 24.
template <bool EXT, int ECAP, bool TRJ>
__global__ void __launch_bounds__(ECAP == 24 ? 512 : 640, 1)
    block_chebyshev_kernel(const DevSystem sys, const BlockLayout B, const BlockRun R) {
    constexpr int NT = TRJ ? kBlockTraj - 1 : 0;
    __shared__ double s_coef[kMaxCoef];
    constexpr int XN = (EXT ? 2 : 1) * kBlockRows;            // the last slot takes what no one reads
    __shared__ float2 s_x[2][XN + 1];
    __shared__ float s_norm[2][kBlockRows / 32 + 2], s_size;
    __shared__ double2 s_turn[2];
    extern __shared__ __align__(16) unsigned char smem[];
    float2 *s_b = reinterpret_cast<float2 *>(smem);          // chunk-end coefficients (b, b)
    float2 *s_mu = s_b + (R.Kmax + 2);                        // moments, one row per detection row
    float2 *s_phase = s_mu + (size_t)(R.Kmax + 2) * B.nv;
    float2 *s_rec = s_phase + (R.Mcap + 1);
    [[maybe_unused]] float2 *s_tb = s_rec + block_rec(R.Mcap, blockDim.x, kBlockPoints32);  // [step][term] inner states
    const int o = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const int role = block_role(nwarps);
    const BlockLane l = block_lane(B, role);
    const BlockSeries S = block_series(R, o);
    if (!S.ok) return;
    const int nsteps = R.nsteps, M = S.M;

    // 2 L~ = 2 (L - c) / s: the recurrence is t_{k+1} = 2 L~ t_k - t_{k-1}
    BlockEntries<ECAP> E;
    float dh = 0.f, dl = 0.f, di = 0.f;
    {
        const double scale = 2.0 / S.half;
        double v[ECAP];
        double2 dg = make_double2(0.0, 0.0);
        if (R.saved) {
            const double *save = R.saved + (size_t)o * block_saved(B.ecap, B.threads);
#pragma unroll
            for (int i = 0; i < ECAP; ++i) v[i] = i < l.ew ? save[(size_t)i * B.threads + role] : 0.0;
            save += (size_t)B.ecap * B.threads;
            dg = make_double2(save[role], save[B.threads + role]);
        } else {
            const double sign = R.adjoint ? -1.0 : 1.0;
            block_coefficients(sys, R, o, s_coef);
            block_assemble<ECAP>(sys, B, l.ew, role, s_coef, sign, v);
            if (l.state) dg = block_diagonal(sys, B.row_src[l.row], s_coef, sign);
        }
        const double sc = l.row < B.n ? scale : 1.0;          // detection rows keep their values
#pragma unroll
        for (int i = 0; i < ECAP; ++i) {
            E.set(i, v[i] * sc);
            E.col[i] = i < l.ew ? B.col[i * B.threads + role] * (int)sizeof(float2) : 0;
        }
        if (l.state) {
            split((dg.x - S.cen) * scale, dh, dl);
            di = (float)(dg.y * scale);
        }
    }
    auto coefficients = [&](int j, int Kc) {                  // of the state j steps into a chunk
        for (int k = tid; k < Kc; k += blockDim.x) {
            const float b = (float)(block_sign(k) * S.tab[k * S.ld + j]);
            s_b[k] = make_float2(b, b);
        }
        if (tid < 2) s_b[Kc + tid] = make_float2(0.f, 0.f);
    };
    coefficients(M, S.K);
    if constexpr (TRJ) {
        for (int q = tid; q < NT * (S.K + 2); q += blockDim.x) {
            const int k = q / NT, j = 1 + q % NT;
            const float b = k < S.K && j < M ? (float)(block_sign(k) * S.tab[k * S.ld + j]) : 0.f;
            s_tb[(size_t)(j - 1) * (R.Kmax + 2) + k] = make_float2(b, b);
        }
    }

    float2 st = make_float2(0.f, 0.f);
    if (l.state) {
        const double2 *r0 = R.rho0s ? R.rho0s + (size_t)block_grid_index(R, o) * R.state_stride : R.rho0;
        st = tovec(r0[B.state_pos[l.row]], float2());
    }
    // The state is carried in units of a power of two that puts the first one's
    // largest part near one, so that the squares of the norm check fit a float
    // whatever its size (in its own, states above 1.8e19 have an infinite norm
    // and a bound violated below 1e-15 goes unnoticed).  The outputs' phases turn
    // it back, so a chunk has no more work (scaling in the norm instead took 200
    // orientations of a rotor-frame system, with their short chunks, 1 % longer).
    {
        float m = fmaxf(fabsf(st.x), fabsf(st.y));
#pragma unroll
        for (int q = 16; q; q >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, q));
        if (lane == 0) s_norm[1][warp] = m;
        __syncthreads();
        for (int w = 0; w < nwarps; ++w) m = fmaxf(m, s_norm[1][w]);
        const int e = m > 0.f ? max(-100, min(100, ilogbf(m))) : 0;
        if (tid == 0) s_size = ldexpf(1.f, e);
        st.x = ldexpf(st.x, -e);
        st.y = ldexpf(st.y, -e);
        block_phases(R, S, ldexp(1.0, e), s_phase, s_turn);
    }
    const float2 *mu_row = s_mu + (size_t)(l.row >= B.n ? l.row - B.n : 0) * (R.Kmax + 2);
    float2 *fid_out = reinterpret_cast<float2 *>(R.fids) + (size_t)o * R.nchan * (nsteps + 1);
    int status = kDevOk;
    long long mv = 0;
    int par = 0;
    // squared norm of the state over the CTA (the slots alternate)
    auto norm2 = [&](float2 v) {
        float s = l.state ? v.x * v.x + v.y * v.y : 0.f;
#pragma unroll
        for (int q = 16; q; q >>= 1) s += __shfl_xor_sync(0xffffffffu, s, q);
        if (lane == 0) s_norm[par][warp] = s;
        __syncthreads();
        s = s_norm[par][0];
        for (int w = 1; w < nwarps; ++w) s += s_norm[par][w];
        par ^= 1;
        return s;
    };
    float start_n2 = norm2(st);

    const f2x DH = f2pk(dh, dh), DL = f2pk(dl, dl), DI = f2pk(-di, di);
    const f2x NEG = l.state ? f2pk(-1.f, -1.f) : 0ull;
    const char *x0 = reinterpret_cast<const char *>(&s_x[0][0]), *x1 = reinterpret_cast<const char *>(&s_x[1][0]);
    for (int a = 0; a < S.nchunks; ++a) {
        const bool last = a + 1 == S.nchunks;
        const int Kc = last ? min(S.K, S.kcut[S.j_last]) : S.K;
        mv += Kc - 1;
        if (last) coefficients(S.j_last, Kc);
        if (l.state) {
            s_x[0][l.row] = make_float2(0.5f * st.x, 0.5f * st.y);
            if (EXT) s_x[0][B.n + l.row] = make_float2(-0.5f * st.y, 0.5f * st.x);
        }
        __syncthreads();
        // Where this lane's result goes: a state row's into the other state
        // buffer, a detection row's into its moments (one further each term),
        // other lanes' nowhere.  ad[1] is for odd terms, ad[0] for even ones.
        uint32_t ad[2], inc = 0;
        if (l.state) {
            ad[1] = smem_u32(&s_x[1][l.row]);
            ad[0] = smem_u32(&s_x[0][l.row]);
        } else if (l.own) {
            ad[1] = smem_u32(mu_row);
            ad[0] = ad[1] + 8;
            inc = 16;
        } else {
            ad[0] = ad[1] = smem_u32(&s_x[0][XN]);
        }
        const uint32_t ext = l.state ? 8u * (uint32_t)B.n : 0u;
        // ntp = -t_{k-2}, so that a row's sum starts from it without another operation
        f2x tc = f2pk(st.x, st.y), ntp = 0ull;
        // chunk-end sums over even and odd terms, each with its low-order part
        f2x acc[2], accl[2] = {0ull, 0ull};
        {
            const f2x b0 = reinterpret_cast<const f2x *>(s_b)[0];
            acc[0] = mul2(b0, tc);
            accl[0] = fma2(b0, tc, sub2(0ull, acc[0]));
            acc[1] = 0ull;
        }
        [[maybe_unused]] f2x inner[NT + 1];
        if constexpr (TRJ) {
            if (l.state)
                reinterpret_cast<float2 *>(R.traj_out)[((size_t)o * (nsteps + 1) + (size_t)a * M) * B.n + l.row] =
                    make_float2(s_size * st.x, s_size * st.y);
#pragma unroll
            for (int j = 0; j < NT; ++j)
                inner[j] = mul2(reinterpret_cast<const f2x *>(s_tb + (size_t)j * (R.Kmax + 2))[0], tc);
        }
        // t_1 = L~ t_0: the first term works on t_0 / 2
        f2x neg = add2(NEG, NEG);
        tc = mul2(f2pk(0.5f, 0.5f), tc);
        auto term = [&](auto ewc, auto rnc, auto oddc, const char *src, int k) {
            constexpr int EW = decltype(ewc)::value, RND = decltype(rnc)::value;
            constexpr bool ODD = decltype(oddc)::value;
            const f2x b = reinterpret_cast<const f2x *>(s_b)[k];
            f2x Y = fma2(DH, tc, ntp);
            f2x Lw = fma2(DH, tc, sub2(ntp, Y));
            f2x P = fma2(DI, swap2(tc), mul2(DL, tc));
#pragma unroll
            for (int i0 = 0; i0 < EW; i0 += 8) {
                f2x X[8];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (i0 + i < EW) X[i] = *reinterpret_cast<const f2x *>(src + E.col[i0 + i]);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (i0 + i < EW) E.mac(i0 + i, Y, Lw, P, X[i]);
            }
            Lw = add2(Lw, P);
#pragma unroll
            for (int r = 0; r < RND; ++r) {
                f2x uy = __shfl_xor_sync(0xffffffffu, Y, 1 << r);
                f2x ul = __shfl_xor_sync(0xffffffffu, Lw, 1 << r);
                if ((l.parts >> r) <= 1) uy = ul = 0ull;
                const f2x Sm = add2(Y, uy);
                Lw = add2(add2(Lw, ul), add2(uy, sub2(Y, Sm)));
                Y = Sm;
            }
            f2x T = add2(Y, Lw);
            st_shared(ad[ODD], T);
            if (EXT && l.state) st_shared(ad[ODD] + ext, rot2(T));
            ad[ODD] += inc;
            block_sync();
            const f2x Sm = fma2(b, T, acc[ODD]);
            accl[ODD] = add2(accl[ODD], fma2(b, T, sub2(acc[ODD], Sm)));
            acc[ODD] = Sm;
            if constexpr (TRJ) {
#pragma unroll
                for (int j = 0; j < NT; ++j)
                    inner[j] = fma2(reinterpret_cast<const f2x *>(s_tb + (size_t)j * (R.Kmax + 2))[k], ODD ? turn2(T) : T, inner[j]);
            }
            ntp = mul2(neg, tc);
            tc = T;
        };
        auto terms = [&](auto ewc, auto rnc) {
            for (int k = 1; k <= Kc; k += 2) {
                term(ewc, rnc, std::true_type{}, x0, k);
                neg = NEG;
                if (k < Kc) term(ewc, rnc, std::false_type{}, x1, k + 1);
            }
        };
        block_dispatch<ECAP>(l, terms);
        if constexpr (TRJ) {
            // the states 1 .. M-1 steps into the chunk, up to the last step
            const int jn = min(M - 1, nsteps - a * M);
#pragma unroll
            for (int j = 1; j <= NT; ++j)
                if (l.state && j <= jn) {
                    const float2 f = f2up(inner[j - 1]), ph = s_phase[j];
                    reinterpret_cast<float2 *>(R.traj_out)[((size_t)o * (nsteps + 1) + (size_t)a * M + j) * B.n + l.row] =
                        make_float2(ph.x * f.x - ph.y * f.y, ph.x * f.y + ph.y * f.x);
                }
        }
        float2 fin;
        {
            // even - 1i odd, rounded once
            const f2x O = turn2(acc[1]), Sm = add2(acc[0], O);
            fin = f2up(add2(Sm, add2(add2(O, sub2(acc[0], Sm)), add2(accl[0], turn2(accl[1])))));
        }
        st = make_float2(0.f, 0.f);
        if (l.state) {
            const double2 ph = s_turn[last ? 1 : 0];
            st.x = (float)(ph.x * (double)fin.x - ph.y * (double)fin.y);
            st.y = (float)(ph.y * (double)fin.x + ph.x * (double)fin.y);
        }
        if (B.nv > 0) block_points<float2, float>(B, R, S, S.tabf, a, Kc, s_mu, s_phase, s_rec, fid_out);
        // a state that grew shows a violated spectral bound (a dissipative L
        // can only shrink it); the norm's barrier also ends this chunk's reads
        const float end_n2 = norm2(st);
        if (!isfinite(end_n2)) status = kDevNonFinite;
        else if (end_n2 > 16.f * start_n2 + 1e-30f) status = kDevDiverged;
        if (status != kDevOk) break;
        start_n2 = end_n2;
    }
    if (R.state_out && l.state)
        R.state_out[(size_t)o * R.state_stride + B.state_pos[l.row]] = tod(make_float2(s_size * st.x, s_size * st.y));
    if (tid == 0) {
        R.status[o] = status;
        R.kused[o] = S.K;
        R.mused[o] = M;
        R.matvecs[o] = mv;
    }
}

// ---------------------------------------------------------------------------
// Propagation, FP64.  An FP64 instruction takes a warp 64 cycles here (half a
// lane a cycle on each of the SM's four units), so the terms are bound by the
// FP64 instructions of a warp and nothing else: the real and imaginary parts
// of a row sit in two lanes of different warps (thread t and t + lanes), which
// halves a warp's instructions per term and spreads one orientation over the
// four units; values and columns sit in shared memory, whose loads cost
// nothing beside them, so that every warp runs just its own entries.
// ---------------------------------------------------------------------------
template <bool EXT, bool TRJ>
__global__ void __launch_bounds__(2 * kBlockRows, 1) block_chebyshev64_kernel(const DevSystem sys, const BlockLayout B,
                                                                              const BlockRun R) {
    constexpr int NT = TRJ ? kBlockTraj - 1 : 0;
    __shared__ double s_coef[kMaxCoef];
    __shared__ double s_norm[2][2 * kBlockRows / 32];
    __shared__ double2 s_turn[2];
    extern __shared__ __align__(16) unsigned char smem[];
    const int T = B.threads, n = B.n, xs = (EXT ? 2 : 1) * n + 1;
    const size_t rec = block_rec(R.Mcap, 2 * T, kBlockPoints64);
    double2 *s_rec = reinterpret_cast<double2 *>(smem);
    double2 *s_phase = s_rec + rec;
    double2 *s_mu = s_phase + (R.Mcap + 1);
    double *s_b = reinterpret_cast<double *>(s_mu + (size_t)(R.Kmax + 2) * B.nv);
    // [buffer][part]: a part of the states, with EXT also that part of 1i times
    // them, and a slot that lanes without a state row read
    double *s_x = s_b + (R.Kmax + 2);
    double *s_val = s_x + 4 * (size_t)xs;                     // [entry][lane]
    [[maybe_unused]] double *s_tb = nullptr;                  // trajectories: [step][term]
    double *s_end = s_val + (size_t)B.ecap * T;
    if constexpr (TRJ) {
        s_tb = s_end;
        s_end += NT * (size_t)(R.Kmax + 2);
    }
    uint16_t *s_col = reinterpret_cast<uint16_t *>(s_end);
    const int o = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const int part = tid >= T ? 1 : 0, t = tid - part * T;    // 0: real parts, 1: imaginary parts
    const BlockLane l = block_lane(B, t);
    const BlockSeries S = block_series(R, o);
    if (!S.ok) return;
    const int nsteps = R.nsteps, M = S.M;
    const bool damped = R.max_im_diag > 0.0;

    const double scale = 2.0 / S.half;
    block_coefficients(sys, R, o, s_coef);
    const double sc = l.row < n ? scale : 1.0, sign = R.adjoint ? -1.0 : 1.0;
    for (int i = 4 * part; i < l.ew; i += 8) {                // the two threads of a lane take turns
        double v[4];
        BlockLayout Bi = B;
        Bi.src = B.src + (size_t)i * T;
        block_assemble<4>(sys, Bi, min(4, l.ew - i), t, s_coef, sign, v);
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (i + q < l.ew) {
                s_val[(size_t)(i + q) * T + t] = v[q] * sc;
                s_col[(size_t)(i + q) * T + t] = B.col[(size_t)(i + q) * T + t];
            }
    }
    double dr = 0.0, dm = 0.0;                                // diagonal; the other part's factor
    if (l.state) {
        const double2 d = block_diagonal(sys, B.row_src[l.row], s_coef, sign);
        dr = (d.x - S.cen) * scale;
        dm = (part ? d.y : -d.y) * scale;
    }
    auto coefficients = [&](int j, int Kc) {
        for (int k = tid; k < Kc; k += blockDim.x) s_b[k] = block_sign(k) * S.tab[k * S.ld + j];
        if (tid < 2) s_b[Kc + tid] = 0.0;
    };
    block_phases(R, S, 1.0, s_phase, s_turn);
    coefficients(M, S.K);
    if constexpr (TRJ) {
        for (int q = tid; q < NT * (S.K + 2); q += blockDim.x) {
            const int k = q / NT, j = 1 + q % NT;
            s_tb[(size_t)(j - 1) * (R.Kmax + 2) + k] = k < S.K && j < M ? block_sign(k) * S.tab[k * S.ld + j] : 0.0;
        }
    }
    if (tid < 4) s_x[tid * xs + xs - 1] = 0.0;

    double st = 0.0;
    if (l.state) {
        const double2 *r0 = R.rho0s ? R.rho0s + (size_t)block_grid_index(R, o) * R.state_stride : R.rho0;
        const double2 v = r0[B.state_pos[l.row]];
        st = part ? v.y : v.x;
    }
    double *mu_row = reinterpret_cast<double *>(s_mu + (size_t)(l.row >= n ? l.row - n : 0) * (R.Kmax + 2)) + part;
    double2 *fid_out = reinterpret_cast<double2 *>(R.fids) + (size_t)o * R.nchan * (nsteps + 1);
    int status = kDevOk;
    long long mv = 0;
    int par = 0;
    auto norm2 = [&](double v) {
        double s = v * v;
#pragma unroll
        for (int q = 16; q; q >>= 1) s += __shfl_xor_sync(0xffffffffu, s, q);
        if (lane == 0) s_norm[par][warp] = s;
        __syncthreads();
        s = s_norm[par][0];
        for (int w = 1; w < nwarps; ++w) s += s_norm[par][w];
        par ^= 1;
        return s;
    };
    double start_n2 = norm2(st);

    const int own = l.state ? l.row : xs - 1;                 // where the diagonal's other part is read
    const double *val = s_val + t;
    // a state's part, and that part of 1i times it in the other part's array
    auto store = [&](int buf, double y) {
        s_x[(2 * buf + part) * xs + l.row] = y;
        if (EXT) s_x[(2 * buf + 1 - part) * xs + n + l.row] = part ? -y : y;
    };
    const uint16_t *col = s_col + t;
    for (int a = 0; a < S.nchunks; ++a) {
        const bool last = a + 1 == S.nchunks;
        const int Kc = last ? min(S.K, S.kcut[S.j_last]) : S.K;
        mv += Kc - 1;
        if (last) coefficients(S.j_last, Kc);
        if (l.state) store(0, st);
        __syncthreads();
        double tc = st, tp = 0.0, even = s_b[0] * st, odd = 0.0;
        [[maybe_unused]] double ie[NT + 1], io[NT + 1];
        if constexpr (TRJ) {
            if (l.state)
                reinterpret_cast<double *>(
                    R.traj_out)[2 * (((size_t)o * (nsteps + 1) + (size_t)a * M) * n + l.row) + part] = st;
#pragma unroll
            for (int j = 0; j < NT; ++j) { ie[j] = s_tb[(size_t)j * (R.Kmax + 2)] * st; io[j] = 0.0; }
        }
        auto term = [&](int buf, int k, double &acc, double *inner) {
            const double *x = s_x + (2 * buf + part) * xs, *xo = s_x + (2 * buf + 1 - part) * xs;
            double y = fma(dr, tc, -tp);
            if (damped) y = fma(dm, xo[own], y);
            int i = 0;
            for (; i + 4 <= l.ew; i += 4) {
                double v[4], X[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    v[q] = val[(i + q) * T];
                    X[q] = x[col[(i + q) * T]];
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) y = fma(v[q], X[q], y);
            }
            for (; i < l.ew; ++i) y = fma(val[i * T], x[col[i * T]], y);
            for (int r = 0; r < l.rounds; ++r) {
                const double u = __shfl_xor_sync(0xffffffffu, y, 1 << r);
                if ((l.parts >> r) > 1) y += u;
            }
            tp = 0.0;
            if (l.state) {
                if (k == 1) y *= 0.5;
                store(buf ^ 1, y);
                acc = fma(s_b[k], y, acc);
                if constexpr (TRJ) {
#pragma unroll
                    for (int j = 0; j < NT; ++j) inner[j] = fma(s_tb[(size_t)j * (R.Kmax + 2) + k], y, inner[j]);
                }
                tp = tc;
                tc = y;
            } else if (l.own) {
                mu_row[2 * (k - 1)] = y;
            }
            __syncthreads();
        };
        for (int k = 1; k <= Kc; k += 2) {
            term(0, k, odd, io);
            if (k + 1 <= Kc) term(1, k + 1, even, ie);
        }
        // sum of the terms: even - 1i odd, then the centre's phase; the parts
        // meet in the state buffers
        auto join = [&](double e, double d, double2 ph) {
            if (l.state) {
                s_x[part * xs + l.row] = e;
                s_x[(2 + part) * xs + l.row] = d;
            }
            __syncthreads();
            double f = 0.0;
            if (l.state) {
                const double fr = s_x[l.row] + s_x[3 * xs + l.row], fi = s_x[xs + l.row] - s_x[2 * xs + l.row];
                f = part ? fma(ph.y, fr, ph.x * fi) : fma(ph.x, fr, -ph.y * fi);
            }
            __syncthreads();
            return f;
        };
        if constexpr (TRJ) {
            const int jn = min(M - 1, nsteps - a * M);
#pragma unroll
            for (int j = 1; j <= NT; ++j)
                if (j <= jn) {
                    const double f = join(ie[j - 1], io[j - 1], s_phase[j]);
                    if (l.state)
                        reinterpret_cast<double *>(
                            R.traj_out)[2 * (((size_t)o * (nsteps + 1) + (size_t)a * M + j) * n + l.row) + part] = f;
                }
        }
        st = join(even, odd, s_turn[last ? 1 : 0]);
        if (B.nv > 0) block_points<double2, double>(B, R, S, S.tab, a, Kc, s_mu, s_phase, s_rec, fid_out);
        const double end_n2 = norm2(st);
        if (!isfinite(end_n2)) status = kDevNonFinite;
        else if (end_n2 > 16.0 * start_n2 + 1e-300) status = kDevDiverged;
        if (status != kDevOk) break;
        start_n2 = end_n2;
    }
    if (R.state_out && l.state)
        reinterpret_cast<double *>(R.state_out)[2 * ((size_t)o * R.state_stride + B.state_pos[l.row]) + part] = st;
    if (tid == 0) {
        R.status[o] = status;
        R.kused[o] = S.K;
        R.mused[o] = M;
        R.matvecs[o] = mv;
    }
}

}  // namespace spx

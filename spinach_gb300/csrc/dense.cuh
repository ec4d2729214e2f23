// Propagation of few coupled states, or of few orientations, by dense matrices
// in FP64 instead of series terms, for FP64 runs and, rounded at the end, for
// FP32 runs that are over sooner this way.
//
// An FP64 series term is a chain of instructions that hold a warp for 64
// cycles each, and a run of N steps takes thousands of terms one after another
// on one SM.  Here the N steps take about log2(N) dependent products: the
// one-step propagator U = exp(-1i L dt) from scaling, a degree-16 Taylor
// polynomial (six products, Paterson and Stockmeyer, SIAM J. Comput. 2 (1973)
// 60) and squaring, then its powers U^2, U^4, ... by squaring, the states
// U^j rho0 (j < m) and the detection rows coil' U^(a m) by doubling their
// number with each power, and every FID point as one product of a row and a
// state.  Each product is spread over the whole GPU, all orientations
// together.  The launcher (engine.cu) takes this path where its FP64 work or
// its latency is the smaller one.
//
// Matrices are stored transposed (S[c * n + r] = U(r, c)), so that a state's
// rows are neighbours.  The kernels are bound by FP64 instructions; they keep
// to 40 registers in CTAs of 64 threads, which fit beside the FP32
// propagation they run along with.
#pragma once

#include "kernels.cuh"

namespace spx {

constexpr int kDenseThreads = 64;

struct DenseSystem {
    int n;                      // coupled states
    int nent;                   // off-diagonal entries
    const int *ent;             // [nent] column * n + row
    const int *src;             // [nent] ELL entry of the system
    const int *row_src;         // [n] row of the system (sliced order)
};

static __device__ __forceinline__ int dense_grid_index(int pick, int n_orient, int o) {
    return pick ? (int)(((2 * (long long)o + 1) * pick) / (2 * (long long)n_orient)) : o;
}

// A = -1i L h (transposed) of every orientation, one CTA each; also the first
// state and detection rows, and the orientation's status words.
struct DenseStart {
    int n_orient, pick;
    const double *alpha, *beta, *gamma;
    double h;
    double2 *A;                 // [o][n][n]
    const double2 *rho0, *rho0s;
    size_t state_stride;
    double2 *V;                 // [o][m][n]
    int m;
    double2 *Y;                 // [o][nchan][rows][n]
    int nchan, rows;
    int ncoil;                  // coil entries: coupled row, channel, value
    const int *coil_row, *coil_chan;
    const double2 *coil_val;
    int *status, *kused, *mused;
    long long *matvecs;
    double *halfwidth;
    double bound;               // what halfwidth reports: a bound on |L|
    long long products;
    int *sym;                   // [o] whether A equals its transpose (null: not wanted)
};
// The CTA assembles A and sets the first state v, the first detection row of
// every channel y (apart by ystride) and the status words; ends with a barrier.
static __device__ __forceinline__ void dense_start(const DevSystem &sys, const DenseSystem &D, const DenseStart &R, int o,
                                                   double *coef, double2 *A, double2 *v, double2 *y, size_t ystride) {
    const int tid = threadIdx.x, n = D.n;
    const int g = dense_grid_index(R.pick, R.n_orient, o);
    wigner_coefficients(sys, R.alpha[g], R.beta[g], R.gamma[g], coef);
    for (int e = tid; e < n * n; e += blockDim.x) A[e] = make_double2(0.0, 0.0);
    for (int e = tid; e < R.nchan * n; e += blockDim.x) y[(size_t)(e / n) * ystride + e % n] = make_double2(0.0, 0.0);
    __syncthreads();
    for (int e = tid; e < D.nent; e += blockDim.x) {
        double re = 0.0, im = 0.0;
        for (int s = 0; s < sys.nstreams; ++s) {
            const double c = coef[sys.stream_coef[s]];
            re = fma(c, sys.ell_re[(size_t)s * sys.ell_len + D.src[e]], re);
            if (sys.ell_im) im = fma(c, sys.ell_im[(size_t)s * sys.ell_len + D.src[e]], im);
        }
        A[D.ent[e]] = make_double2(im * R.h, -re * R.h);
    }
    for (int i = tid; i < n; i += blockDim.x) {
        double re = 0.0, im = 0.0;
        for (int s = 0; s < sys.nstreams; ++s) {
            const double c = coef[sys.stream_coef[s]];
            const double2 d = sys.diag[(size_t)s * sys.n_pad + D.row_src[i]];
            re = fma(c, d.x, re);
            im = fma(c, d.y, im);
        }
        A[(size_t)i * n + i] = make_double2(im * R.h, -re * R.h);
        const double2 *r0 = R.rho0s ? R.rho0s + (size_t)g * R.state_stride : R.rho0;
        v[i] = r0[D.row_src[i]];
    }
    if (tid == 0) {
        for (int q = 0; q < R.ncoil; ++q) {
            const double2 w = R.coil_val[q];
            double2 &t = y[(size_t)R.coil_chan[q] * ystride + R.coil_row[q]];
            t = make_double2(t.x + w.x, t.y - w.y);                  // conj(coil)
        }
        R.status[o] = kDevOk;
        R.kused[o] = 16;
        R.mused[o] = R.m;
        R.matvecs[o] = R.products * n;
        R.halfwidth[o] = R.bound;
    }
    __syncthreads();
}
static __global__ void __launch_bounds__(256) dense_start_kernel(const DevSystem sys, const DenseSystem D,
                                                                 const DenseStart R) {
    __shared__ double coef[kMaxCoef];
    __shared__ int differs;
    const int o = blockIdx.x, n = D.n;
    if (threadIdx.x == 0) differs = 0;
    double2 *A = R.A + (size_t)o * n * n;
    dense_start(sys, D, R, o, coef, A, R.V + (size_t)o * R.m * n, R.Y + (size_t)o * R.nchan * R.rows * n,
                (size_t)R.rows * n);
    if (!R.sym) return;
    for (int e = threadIdx.x; e < D.nent; e += blockDim.x) {
        const double2 a = A[D.ent[e]], b = A[(size_t)(D.ent[e] % n) * n + D.ent[e] / n];
        if (a.x != b.x || a.y != b.y) differs = 1;
    }
    __syncthreads();
    if (threadIdx.x == 0) R.sym[o] = differs ? 0 : 1;
}

static __device__ __forceinline__ void dense_mac(double2 &s, const double2 a, const double2 b) {
    s.x = fma(a.x, b.x, s.x);
    s.y = fma(a.x, b.y, s.y);
    s.x = fma(-a.y, b.y, s.x);
    s.y = fma(a.y, b.x, s.y);
}

// C = A B (+ c0 + c1 M1 + c2 M2 + c3 M3 when M1), one element per thread.
struct DenseSum {
    const double2 *M1, *M2, *M3;
    double c0, c1, c2, c3;
};
// sum over k of a[k] b[k n]
static __device__ __forceinline__ double2 dense_dot(const double2 *a, const double2 *b, int n) {
    double2 s = make_double2(0.0, 0.0);
    int k = 0;
    for (; k + 2 <= n; k += 2) {
        const double2 a0 = a[k], a1 = a[k + 1], b0 = b[(size_t)k * n], b1 = b[(size_t)(k + 1) * n];
        dense_mac(s, a0, b0);
        dense_mac(s, a1, b1);
    }
    if (k < n) dense_mac(s, a[k], b[(size_t)k * n]);
    return s;
}
static __device__ __forceinline__ double2 dense_sum(const DenseSum &t, size_t at, bool diagonal, double2 s) {
    const double2 a = t.M1[at], b = t.M2[at], c = t.M3[at];
    s.x += (diagonal ? t.c0 : 0.0) + t.c1 * a.x + t.c2 * b.x + t.c3 * c.x;
    s.y += t.c1 * a.y + t.c2 * b.y + t.c3 * c.y;
    return s;
}
// Element u of the upper triangle with diagonal of an m x m matrix, rows r and
// m-1-r side by side (m+1 elements).
static __device__ __forceinline__ int2 dense_upper(int u, int m) {
    const int r = u / (m + 1), c = u - r * (m + 1);
    return c < m - r ? make_int2(r, r + c) : make_int2(m - 1 - r, c - 1);
}
// TRI: the first n (n+1) / 2 elements are the upper triangle.  An orientation
// whose A equals its transpose (real couplings; relaxation may be complex) has
// only products that do, so its lower triangles are copies: half of the FP64
// instructions that bind this kernel (two orientations of 252 states, 2048
// steps: products 5.9 -> 3.1 ms).  From kDenseTri states on: below, latency
// binds it and the longer index chain costs more (6 states: 1.5 us a product).
constexpr int kDenseTri = 32;
template <bool TRI>
static __global__ void __launch_bounds__(kDenseThreads, 24) dense_product_kernel(int64_t total, int n,
                                                                                 const int *__restrict__ sym,
                                                                                 const double2 *__restrict__ A,
                                                                                 const double2 *__restrict__ B,
                                                                                 double2 *__restrict__ C, const DenseSum t) {
    const int n2 = n * n, upper = (n2 + n) / 2;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = q / n2;
        const int e = (int)(q - o * n2);
        int r = e / n, c = e - r * n;
        bool same = false;
        if (TRI) {
            same = sym[o] != 0;
            if (e >= upper && same) continue;
            const int2 at = dense_upper(e < upper ? e : e - upper, e < upper ? n : n - 1);
            r = e < upper ? at.x : at.y + 1;
            c = e < upper ? at.y : at.x;
        }
        const double2 *a = A + o * n2 + (size_t)r * n, *b = B + o * n2 + c;
        double2 s = dense_dot(a, b, n);
        const int64_t to = o * n2 + (int64_t)r * n + c;
        if (t.M1) s = dense_sum(t, (size_t)to, r == c, s);
        C[to] = s;
        if (TRI && same && r != c) C[o * n2 + (int64_t)c * n + r] = s;
    }
}
// C = c0 + c1 M1 + c2 M2 + c3 M3 + c4 M4
static __global__ void __launch_bounds__(kDenseThreads, 24) dense_sum_kernel(int64_t total, int n, const DenseSum t,
                                                                             const double2 *M4, double c4, double2 *C) {
    const int n2 = n * n;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
        const int e = (int)(q % n2);
        const double2 d = M4[q];
        C[q] = dense_sum(t, (size_t)q, e / n == e % n, make_double2(c4 * d.x, c4 * d.y));
    }
}

// States have .. have + more - 1 from the first `more` ones and a power S (of
// the propagator, transposed): V[have + j] = U V[j].
static __global__ void __launch_bounds__(kDenseThreads, 24) dense_states_kernel(int64_t n_orient, int n, int m, int have,
                                                                                int more, const double2 *__restrict__ S,
                                                                                double2 *V) {
    const int per = more * n;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n_orient * per;
         q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = q / per;
        const int e = (int)(q - o * per), j = e / n, r = e - j * n;
        const double2 *s = S + o * n * n + r, *v = V + (o * m + j) * n;
        double2 sum = make_double2(0.0, 0.0);
        for (int k = 0; k < n; ++k) dense_mac(sum, s[(size_t)k * n], v[k]);
        V[(o * m + have + j) * n + r] = sum;
    }
}
// Detection rows alike: Y[have + j] = Y[j] U, for every channel.
static __global__ void __launch_bounds__(kDenseThreads, 24) dense_rows_kernel(int64_t n_orient, int n, int nchan, int rows,
                                                                              int have, int more,
                                                                              const double2 *__restrict__ S, double2 *Y) {
    const int per = nchan * more * n;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n_orient * per;
         q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = q / per;
        const int e = (int)(q - o * per), ch = e / (more * n), f = e - ch * more * n, j = f / n, c = f - j * n;
        double2 *base = Y + ((o * nchan + ch) * rows) * n;
        const double2 *s = S + (o * n + c) * n, *y = base + (size_t)j * n;
        double2 sum = make_double2(0.0, 0.0);
        for (int k = 0; k < n; ++k) dense_mac(sum, s[k], y[k]);
        base[(size_t)(have + j) * n + c] = sum;
    }
}
// Orientations whose points an FP32 run also keeps unrounded (its check against
// FP64): number j is orientation ((2 j + 1) of n) / (2 count).
struct DenseCheck {
    double2 *fids;              // [count][nchan][npts]
    int *status;                // [count]
    int count;
};
// fids[o][ch][a m + j] = Y[a] . V[j]
template <class Vec>
static __global__ void __launch_bounds__(kDenseThreads, 24) dense_points_kernel(int64_t n_orient, int n, int nchan, int rows,
                                                                                int m, int npts,
                                                                                const double2 *__restrict__ Y,
                                                                                const double2 *__restrict__ V, Vec *fids,
                                                                                int *status, const DenseCheck check) {
    const int64_t per = (int64_t)nchan * npts;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < n_orient * per;
         q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t o = q / per;
        const int e = (int)(q - o * per), ch = e / npts, p = e - ch * npts, a = p / m, j = p - a * m;
        const double2 *y = Y + ((o * nchan + ch) * rows + a) * n, *v = V + (o * m + j) * n;
        double2 s = make_double2(0.0, 0.0);
        for (int k = 0; k < n; ++k) dense_mac(s, y[k], v[k]);
        fids[q] = tovec(s, Vec());
        const bool finite = isfinite(s.x) && isfinite(s.y);
        if (!finite) status[o] = kDevNonFinite;
        for (int c = 0; c < check.count; ++c)
            if (((2 * (long long)c + 1) * n_orient) / (2 * (long long)check.count) == o) {
                check.fids[c * per + e] = s;
                if (!finite) check.status[c] = kDevNonFinite;
            }
    }
}

// The whole run of an orientation in one CTA, its matrices in shared memory, the
// same sums in the same order: for few states, where a product is a few
// instructions and the chain of launches took the time.  Bound by FP64 latency.
// 6 states, 1024 steps, 200 orientations: 0.17 ms in launches, 0.067 so; 8
// states 0.21 and 0.081; at 18 to 20 states no faster, with 256 threads either.
constexpr int kDenseOne = 16;            // most states
constexpr int kDenseOneThreads = 128;
struct DenseOne {
    int scale, npts;
    double f[17];                        // Taylor coefficients
};
static __host__ __device__ inline size_t dense_one_smem(int n, int m, int rows, int nchan) {
    return sizeof(double2) * (size_t)n * (6 * (size_t)n + m + (size_t)nchan * rows);
}
template <class Vec>
static __global__ void __launch_bounds__(kDenseOneThreads) dense_one_kernel(const DevSystem sys, const DenseSystem D,
                                                                            const DenseStart R, const DenseOne P, Vec *fids,
                                                                            const DenseCheck check) {
    __shared__ double coef[kMaxCoef];
    extern __shared__ __align__(16) unsigned char dense_smem[];
    const int o = blockIdx.x, tid = threadIdx.x, n = D.n, n2 = n * n;
    double2 *M[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) M[q] = reinterpret_cast<double2 *>(dense_smem) + q * n2;
    double2 *V = M[5] + n2, *Y = V + R.m * n;
    dense_start(sys, D, R, o, coef, M[0], V, Y, (size_t)R.rows * n);
    auto product = [&](const double2 *A, const double2 *B, double2 *C, const DenseSum &t) {
        for (int e = tid; e < n2; e += kDenseOneThreads) {
            const int r = e / n, c = e - r * n;
            double2 s = dense_dot(A + r * n, B + c, n);
            if (t.M1) s = dense_sum(t, e, r == c, s);
            C[e] = s;
        }
        __syncthreads();
    };
    const DenseSum none = {};
    const double *f = P.f;
    auto quarter = [&](int q, double f0) { return DenseSum{M[0], M[1], M[2], f0, f[4 * q + 1], f[4 * q + 2], f[4 * q + 3]}; };
    product(M[0], M[0], M[1], none);
    product(M[1], M[0], M[2], none);
    product(M[1], M[1], M[3], none);
    for (int e = tid; e < n2; e += kDenseOneThreads)
        M[4][e] = dense_sum(quarter(3, f[12]), e, e / n == e % n, make_double2(f[16] * M[3][e].x, f[16] * M[3][e].y));
    __syncthreads();
    product(M[3], M[4], M[5], quarter(2, f[8]));
    product(M[3], M[5], M[4], quarter(1, f[4]));
    product(M[3], M[4], M[5], quarter(0, P.scale > 0 ? 0.0 : f[0]));
    double2 *U = M[5], *W = M[4];
    auto turn = [&] { double2 *t = U; U = W; W = t; };
    for (int q = 0; q < P.scale; ++q) {
        product(U, U, W, DenseSum{U, U, U, q + 1 == P.scale ? 1.0 : 0.0, 2.0, 0.0, 0.0});
        turn();
    }
    for (int have = 1; have < R.m; have *= 2) {
        for (int e = tid; e < have * n; e += kDenseOneThreads) {
            const int j = e / n, r = e - j * n;
            double2 s = make_double2(0.0, 0.0);
            for (int k = 0; k < n; ++k) dense_mac(s, U[k * n + r], V[j * n + k]);
            V[(have + j) * n + r] = s;
        }
        __syncthreads();
        if (2 * have < R.m || R.rows > 1) {
            product(U, U, W, none);
            turn();
        }
    }
    for (int have = 1; have < R.rows; have *= 2) {
        for (int e = tid; e < R.nchan * have * n; e += kDenseOneThreads) {
            const int ch = e / (have * n), x = e - ch * have * n, j = x / n, c = x - j * n;
            double2 *y = Y + (size_t)ch * R.rows * n;
            double2 s = make_double2(0.0, 0.0);
            for (int k = 0; k < n; ++k) dense_mac(s, U[c * n + k], y[j * n + k]);
            y[(have + j) * n + c] = s;
        }
        __syncthreads();
        if (2 * have < R.rows) {
            product(U, U, W, none);
            turn();
        }
    }
    const int per = R.nchan * P.npts;
    int at = -1;                                              // of the checked orientations
    for (int c = 0; c < check.count; ++c)
        if (((2 * (long long)c + 1) * R.n_orient) / (2 * (long long)check.count) == o) at = c;
    bool finite = true;
    for (int e = tid; e < per; e += kDenseOneThreads) {
        const int ch = e / P.npts, p = e - ch * P.npts, a = p / R.m, j = p - a * R.m;
        const double2 *y = Y + ((size_t)ch * R.rows + a) * n, *v = V + (size_t)j * n;
        double2 s = make_double2(0.0, 0.0);
        for (int k = 0; k < n; ++k) dense_mac(s, y[k], v[k]);
        fids[(size_t)o * per + e] = tovec(s, Vec());
        if (at >= 0) check.fids[(size_t)at * per + e] = s;
        finite = finite && isfinite(s.x) && isfinite(s.y);
    }
    if (!finite) {
        R.status[o] = kDevNonFinite;
        if (at >= 0) check.status[at] = kDevNonFinite;
    }
}

}  // namespace spx

// Orientation surrogate for the powder FID: a small MLP over real spherical
// harmonics of the orientation (beta, gamma) that predicts the coefficients of
// an orientation's FID in an SVD basis.  Training and inference run on the GPU
// in the kernels below (split-BF16 tensor-core products with FP32 accumulation
// and BF16 weights, GELU, Adam); one training step is captured once in a CUDA
// graph and replayed.
//
// Features follow kernel/utilities/spher_harmon.m (orthonormal Y_lm with the
// Condon-Shortley phase): for each l, Re Y_l0, then Re Y_lm and Im Y_lm for
// m = 1..l, (lmax+1)^2 real numbers per orientation.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <new>
#include <random>
#include <stdexcept>
#include <string>
#include <vector>

#include "spinach_gpu.h"

namespace {

struct SurErr : std::runtime_error {
    spx_status code;
    SurErr(spx_status c, const std::string &m) : std::runtime_error(m), code(c) {}
};

#define SUR_CUDA(call)                                                                              \
    do {                                                                                            \
        cudaError_t e_ = (call);                                                                    \
        if (e_ != cudaSuccess)                                                                      \
            throw SurErr(e_ == cudaErrorMemoryAllocation ? SPX_ERR_OUT_OF_MEMORY : SPX_ERR_CUDA,    \
                         std::string(#call) + ": " + cudaGetErrorString(e_));                      \
    } while (0)

constexpr int kMaxL = 16;
constexpr int kSplitRows = 128;   // samples per split-K slab of the weight gradients (2000 samples: 27 us, 31 with 256)
constexpr int kMaxSplits = 32;

// ---------------------------------------------------------------------------
// Spherical-harmonic features: p_lm(cos beta) cos(m gamma) and sin(m gamma) with
// the orthonormal associated Legendre functions p_lm (Condon-Shortley phase
// included), by the recurrence over l at fixed m, in FP64.
//
// FP64 instructions bound it (a warp's takes 64 cycles of its FP64 unit), so
// the recurrence's coefficients come from a table (coef: a_lm, a_lm b_lm, then
// per m the factor of sin^m beta in p_mm), the sines and cosines of an
// orientation are taken once and raised to their powers by squaring, and the
// orders m of 32 orientations are spread over the warps (warp w: m = w and
// lmax - w).  Rows leave through shared memory in whole lines.  One thread per
// orientation with square roots and a sincos per feature took 402 us for 20000
// orientations at lmax 12 and 218 us for 2000; this takes 51 and 14.
// ---------------------------------------------------------------------------
constexpr int kCoefRow = kMaxL + 1;
constexpr int kCoefs = 2 * kCoefRow * kCoefRow + kCoefRow;

std::vector<double> feature_coefficients() {
    std::vector<double> c(kCoefs, 0.0);
    double pmm = 0.28209479177387814;   // sqrt(1/(4 pi))
    for (int m = 0; m <= kMaxL; ++m) {
        if (m > 0) pmm *= -std::sqrt((2.0 * m + 1.0) / (2.0 * m));
        c[2 * kCoefRow * kCoefRow + m] = pmm;
        for (int l = m + 1; l <= kMaxL; ++l) {
            const double a = std::sqrt((4.0 * l * l - 1.0) / ((double)l * l - (double)m * m));
            const double b = std::sqrt(((l - 1.0) * (l - 1.0) - (double)m * m) / (4.0 * (l - 1.0) * (l - 1.0) - 1.0));
            c[2 * (l * kCoefRow + m)] = a;
            c[2 * (l * kCoefRow + m) + 1] = l == m + 1 ? 0.0 : a * b;
        }
    }
    return c;
}

inline int feature_warps(int lmax) { return lmax / 2 + 1; }
inline size_t feature_smem(int nfeat) { return 32 * (size_t)(nfeat | 1) * sizeof(float); }

__global__ void __launch_bounds__(32 * (kMaxL / 2 + 1))
    sh_features_kernel(int64_t n, const double *__restrict__ beta, const double *__restrict__ gamma, int lmax, int nfeat,
                       int ld, const double *__restrict__ coef, float *__restrict__ X) {
    __shared__ double s_b[2][32], s_g[2][32];
    extern __shared__ float s_row[];     // [32][nfeat | 1]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int64_t i0 = blockIdx.x * (int64_t)32;
    const int rows = (int)min((int64_t)32, n - i0);
    const int64_t i = i0 + min(lane, rows - 1);
    if (warp == 0) sincos(beta[i], &s_b[1][lane], &s_b[0][lane]);
    if (warp == nwarps - 1) sincos(gamma[i], &s_g[1][lane], &s_g[0][lane]);
    __syncthreads();
    const double x = s_b[0][lane], st = s_b[1][lane];
    float *out = s_row + lane * (nfeat | 1);
    for (int m = warp; m <= lmax; m = m == warp && lmax - warp > warp ? lmax - warp : lmax + 1) {
        double pm = coef[2 * kCoefRow * kCoefRow + m], c = 1.0, s = 0.0;
        double zs = st, zc = s_g[0][lane], zi = s_g[1][lane];
        for (int q = m; q > 0; q >>= 1) {
            if (q & 1) {
                pm *= zs;
                const double t = c * zc - s * zi;
                s = c * zi + s * zc;
                c = t;
            }
            if (q > 1) {
                zs *= zs;
                const double t = zc * zc - zi * zi;
                zi = 2.0 * zc * zi;
                zc = t;
            }
        }
        double p1 = pm, p2 = 0.0;
        for (int l = m; l <= lmax; ++l) {
            if (l > m) {
                const double2 k = *reinterpret_cast<const double2 *>(coef + 2 * (l * kCoefRow + m));
                const double p = k.x * x * p1 - k.y * p2;
                p2 = p1;
                p1 = p;
            }
            // of row l: Re Y_l0, then Re and Im Y_lm of m = 1 .. l
            if (m == 0) {
                out[l * l] = (float)p1;
            } else {
                out[l * l + 2 * m - 1] = (float)(p1 * c);
                out[l * l + 2 * m] = (float)(p1 * s);
            }
        }
    }
    __syncthreads();
    for (int r = warp; r < rows; r += nwarps)
        for (int f = lane; f < nfeat; f += 32) X[(i0 + r) * ld + f] = s_row[r * (nfeat | 1) + f];
}

// ---------------------------------------------------------------------------
// C(i,j) = sum_k A(i,k) B(k,j) on the tensor cores with FP32 accumulation, and
// what follows the product in its epilogue.
//
// Operands are split into BF16 parts: an FP32 value into three (24 bits
// together, all of it), a BF16 weight is its own part.  FP32 x BF16 takes three
// mma.sync m16n8k16 products, FP32 x FP32 the six whose parts' bits reach FP32
// accuracy.  The tensor pipe's sums round towards zero, so a slab's sum starts
// from zero and joins the others in an FP32 addition (1024 features, five
// layers: predictions 1.8e-5 too small without).  32-deep slabs are loaded into
// registers while the slab before is multiplied, split once and stored as BF16
// planes in the order of global memory ([row][k] or [k][row], both padded so
// that ldmatrix, plain or transposing, reads without conflicts).  Four warps of
// 16x32 (layers) or 32x32 (weight gradients): a 32-row tile of a layer costs
// what half a 64-row one does, and 2000 rows give every SM a CTA.
//
// The products here have 100 to 4000 rows and 64 to 256 columns: latency of the
// loads and the launches bound them, not the tensor pipe.  So bias, GELU and
// its derivative and the loss are epilogues, the derivative overwrites the
// pre-activations, and all weight gradients are one launch.  20000 rows, 256 x
// 256, bias and GELU: 45 us (TF32 pairs, 16-deep slabs without prefetch and a
// separate bias pass: 78).  Loss and gradients of 2000 rows, five layers: 142 us
// (585).
// ---------------------------------------------------------------------------
constexpr int kTile = 64, kSlab = 32, kLayerRows = 32;
constexpr int kRowK = kSlab + 8, kRowMN = kTile + 8;          // 16-bit elements of a padded row
constexpr int kPlane = kTile * kRowK;                          // >= kSlab * kRowMN
static_assert(kPlane >= kSlab * kRowMN, "a plane holds either order");

template <class T> struct Operand;
template <> struct Operand<float> { using Raw = float4; static constexpr int planes = 3; };
template <> struct Operand<__nv_bfloat16> { using Raw = uint2; static constexpr int planes = 1; };

__device__ __forceinline__ uint32_t bits(__nv_bfloat162 v) { return *reinterpret_cast<uint32_t *>(&v); }
__device__ __forceinline__ uint32_t smem_at(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Four neighbouring elements (chunk c of a slab) along the contiguous index,
// zero outside the matrix.  KC: element (row, k) is P[row * ld + k], else P[k * ld + row].
template <bool KC, class T>
__device__ __forceinline__ typename Operand<T>::Raw load_chunk(const T *__restrict__ P, int ld, int r0, int rows, int k0,
                                                               int kend, int c, bool vec) {
    const int r = r0 + (KC ? c / (kSlab / 4) : c % (kTile / 4) * 4), k = k0 + (KC ? c % (kSlab / 4) * 4 : c / (kTile / 4));
    const bool in = r < rows && k < kend;
    const int left = KC ? kend - k : rows - r;
    const T *p = P + (KC ? (int64_t)r * ld + k : (int64_t)k * ld + r);
    typename Operand<T>::Raw v = {};
    if (in) {
        if (vec && left >= 4) {
            v = *reinterpret_cast<const typename Operand<T>::Raw *>(p);
        } else {
            T *e = reinterpret_cast<T *>(&v);
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (q < left) e[q] = p[q];
        }
    }
    return v;
}

template <bool KC>
__device__ __forceinline__ void put(__nv_bfloat16 *plane, int c, uint2 v) {
    const int at = KC ? c / (kSlab / 4) * kRowK + c % (kSlab / 4) * 4 : c / (kTile / 4) * kRowMN + c % (kTile / 4) * 4;
    *reinterpret_cast<uint2 *>(plane + at) = v;
}
template <bool KC>
__device__ __forceinline__ void store_chunk(__nv_bfloat16 *planes, int c, uint2 v) { put<KC>(planes, c, v); }
template <bool KC>
__device__ __forceinline__ void store_chunk(__nv_bfloat16 *planes, int c, float4 v) {
    float2 a = make_float2(v.x, v.y), b = make_float2(v.z, v.w);
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const __nv_bfloat162 ha = __float22bfloat162_rn(a), hb = __float22bfloat162_rn(b);
        put<KC>(planes + p * kPlane, c, make_uint2(bits(ha), bits(hb)));
        const float2 fa = __bfloat1622float2(ha), fb = __bfloat1622float2(hb);
        a = make_float2(a.x - fa.x, a.y - fa.y);
        b = make_float2(b.x - fb.x, b.y - fb.y);
    }
}

template <bool TRANS>
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const __nv_bfloat16 *p) {
    if constexpr (TRANS)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_at(p)) : "memory");
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_at(p)) : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// One tile's product over k in [kb, ke) (kb a multiple of 4).  AK and BK: A and
// B are contiguous in k.  asum: the calling thread's part of the sums of A over
// k, for four rows of A from 4 (threadIdx.x mod 16) on (A contiguous in rows).
template <int MT, bool AK, bool BK, class BT, bool ASUM>
__device__ __forceinline__ void tile_product(__nv_bfloat16 *sA, __nv_bfloat16 *sB, int i0, int M, int j0, int N, int kb,
                                             int ke, const float *__restrict__ A, int lda, const BT *__restrict__ B,
                                             int ldb, float (&acc)[MT][4][4], float4 &asum) {
    static_assert(AK || MT == 2, "rows in order of k: half tiles too");
    constexpr int NB = Operand<BT>::planes, Q = kTile * kSlab / 4 / 128, QA = Q * MT / 2;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = (warp >> 1) * 16 * MT, wn = (warp & 1) * 32;
    const bool va = lda % 4 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0;
    const bool vb = ldb % 4 == 0 && reinterpret_cast<uintptr_t>(B) % (4 * sizeof(BT)) == 0;
    float4 ra[QA];
    typename Operand<BT>::Raw rb[Q];
    auto load = [&](int k0) {
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            if (q < QA) ra[q < QA ? q : 0] = load_chunk<AK, float>(A, lda, i0, M, k0, ke, tid + 128 * q, va);
            rb[q] = load_chunk<BK, BT>(B, ldb, j0, N, k0, ke, tid + 128 * q, vb);
        }
    };
    if (kb < ke) load(kb);
    for (int k0 = kb; k0 < ke; k0 += kSlab) {
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            if (q < QA) store_chunk<AK>(sA, tid + 128 * q, ra[q < QA ? q : 0]);
            store_chunk<BK>(sB, tid + 128 * q, rb[q]);
            if constexpr (ASUM) {
                asum.x += ra[q].x;
                asum.y += ra[q].y;
                asum.z += ra[q].z;
                asum.w += ra[q].w;
            }
        }
        __syncthreads();
        if (k0 + kSlab < ke) load(k0 + kSlab);
        float part[MT][4][4] = {};
#pragma unroll
        for (int ks = 0; ks < kSlab; ks += 16) {
            uint32_t a[3][MT][4], b[NB][2][4];
            const int l7 = lane & 7, h1 = (lane >> 3 & 1) * 8, h2 = (lane >> 4) * 8;
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) {
                    const int r = wm + mt * 16;
                    ldmatrix4<!AK>(a[p][mt], sA + p * kPlane + (AK ? (r + l7 + h1) * kRowK + ks + h2
                                                                    : (ks + l7 + h2) * kRowMN + r + h1));
                }
#pragma unroll
            for (int p = 0; p < NB; ++p)
#pragma unroll
                for (int np = 0; np < 2; ++np) {
                    const int c = wn + np * 16;
                    ldmatrix4<!BK>(b[p][np], sB + p * kPlane + (BK ? (c + l7 + h2) * kRowK + ks + h1
                                                                    : (ks + l7 + h1) * kRowMN + c + h2));
                }
            // the smallest products first; the tiles' accumulators by turns
            auto mac = [&](int pa, int pb) {
#pragma unroll
                for (int mt = 0; mt < MT; ++mt)
#pragma unroll
                    for (int nt = 0; nt < 4; ++nt)
                        mma_bf16(part[mt][nt], a[pa][mt], b[pb][nt / 2][nt % 2 * 2], b[pb][nt / 2][nt % 2 * 2 + 1]);
            };
            mac(2, 0);
            if constexpr (NB == 3) { mac(0, 2); mac(1, 1); }
            mac(1, 0);
            if constexpr (NB == 3) mac(0, 1);
            mac(0, 0);
        }
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int nt = 0; nt < 4; ++nt)
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[mt][nt][q] += part[mt][nt][q];
        __syncthreads();
    }
}

// f(i, j, value at j, value at j + 1, whether j + 1 is a column) of the calling
// thread's part of a tile
template <int MT, class F>
__device__ __forceinline__ void for_each_pair(const float (&acc)[MT][4][4], int i0, int M, int j0, int N, F f) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wm = (warp >> 1) * 16 * MT, wn = (warp & 1) * 32;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = i0 + wm + mt * 16 + (lane >> 2) + h * 8, j = j0 + wn + nt * 8 + 2 * (lane & 3);
                if (i < M && j < N) f(i, j, acc[mt][nt][2 * h], acc[mt][nt][2 * h + 1], j + 1 < N);
            }
}
// p[0], p[1] = a, b: in one store where the address allows it
__device__ __forceinline__ void put_pair(float *p, float a, float b, bool two) {
    if (two && reinterpret_cast<uintptr_t>(p) % 8 == 0) {
        *reinterpret_cast<float2 *>(p) = make_float2(a, b);
    } else {
        p[0] = a;
        if (two) p[1] = b;
    }
}

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
    return 0.5f * (1.f + erff(z * 0.70710678118654752f)) + z * 0.3989422804014327f * expf(-0.5f * z * z);
}

// A layer: z = x W' + b.  Hidden ones: Y = gelu(z), Z = z where Z is given.  The
// last: Y = z, and with targets T also Z = d loss / d z of the mean square
// error, whose value is added to *loss.
template <bool LAST>
__global__ void __launch_bounds__(128, 5)
    layer_kernel(int n, int dd, int di, const float *__restrict__ X, int ldx, const __nv_bfloat16 *__restrict__ W,
                 int ldw, const float *__restrict__ b, float *__restrict__ Z, float *__restrict__ Y, const float *__restrict__ T,
                 float *__restrict__ loss) {
    __shared__ __align__(16) __nv_bfloat16 sA[3 * kPlane], sB[kPlane];
    __shared__ float s_e2[4];
    const int tx = (dd + kTile - 1) / kTile, i0 = blockIdx.x / tx * kLayerRows, j0 = blockIdx.x % tx * kTile;
    float acc[1][4][4] = {};
    float4 unused;
    tile_product<1, true, true, __nv_bfloat16, false>(sA, sB, i0, n, j0, dd, 0, di, X, ldx, W, ldw, acc, unused);
    float e2 = 0.f;
    const float inv = LAST ? 1.f / (float)((int64_t)n * dd) : 0.f;
    for_each_pair<1>(acc, i0, n, j0, dd, [&](int i, int j, float za, float zb, bool two) {
        const int64_t at = (int64_t)i * dd + j;
        za += b[j];
        if (two) zb += b[j + 1];
        if constexpr (!LAST) {
            if (Z) put_pair(Z + at, za, zb, two);
            put_pair(Y + at, gelu(za), gelu(zb), two);
        } else {
            put_pair(Y + at, za, zb, two);
            if (T) {
                const float da = za - T[at], db = two ? zb - T[at + 1] : 0.f;
                put_pair(Z + at, 2.f * da * inv, 2.f * db * inv, two);
                e2 += da * da * inv + db * db * inv;
            }
        }
    });
    if (LAST && T) {
#pragma unroll
        for (int q = 16; q; q >>= 1) e2 += __shfl_xor_sync(0xffffffffu, e2, q);
        if ((threadIdx.x & 31) == 0) s_e2[threadIdx.x >> 5] = e2;
        __syncthreads();
        if (threadIdx.x == 0) atomicAdd(loss, s_e2[0] + s_e2[1] + s_e2[2] + s_e2[3]);
    }
}

// Z = (dZ W) gelu'(Z): the derivative at a hidden layer's pre-activations, in
// their place, from the next layer's dZ (n x dd) and weights (dd x di)
__global__ void __launch_bounds__(128, 5)
    layer_back_kernel(int n, int dd, int di, const float *__restrict__ dZ, const __nv_bfloat16 *__restrict__ W,
                      float *__restrict__ Z) {
    __shared__ __align__(16) __nv_bfloat16 sA[3 * kPlane], sB[kPlane];
    const int tx = (di + kTile - 1) / kTile, i0 = blockIdx.x / tx * kLayerRows, j0 = blockIdx.x % tx * kTile;
    float acc[1][4][4] = {};
    float4 unused;
    tile_product<1, true, false, __nv_bfloat16, false>(sA, sB, i0, n, j0, di, 0, dd, dZ, dd, W, di, acc, unused);
    for_each_pair<1>(acc, i0, n, j0, di, [&](int i, int j, float a, float b, bool two) {
        float *z = Z + (int64_t)i * di + j;
        put_pair(z, a * gelu_grad(z[0]), two ? b * gelu_grad(z[1]) : 0.f, two);
    });
}

// dW = dZ' X (dd x di) and db = column sums of dZ of every layer, over the
// samples of slab blockIdx.y: the slabs' results lie `stride` apart, each in the
// order of the parameters.
constexpr int kMaxDense = 17;
struct GradJobs {
    const float *dZ[kMaxDense], *X[kMaxDense];
    int dd[kMaxDense], di[kMaxDense], ldx[kMaxDense], tile[kMaxDense + 1];
    int64_t off[kMaxDense];
    int layers;
};
__global__ void __launch_bounds__(128, 3)
    weight_grad_kernel(const __grid_constant__ GradJobs J, int n, float *__restrict__ out, int64_t stride) {
    __shared__ __align__(16) __nv_bfloat16 sA[3 * kPlane], sB[3 * kPlane];
    int l = 0;
    while (l + 1 < J.layers && (int)blockIdx.x >= J.tile[l + 1]) ++l;
    const int dd = J.dd[l], di = J.di[l], tx = (di + kTile - 1) / kTile, tile = blockIdx.x - J.tile[l];
    const int i0 = tile / tx * kTile, j0 = tile % tx * kTile;
    const int chunk = (((n + (int)gridDim.y - 1) / (int)gridDim.y) + kSlab - 1) / kSlab * kSlab;
    const int kb = min(n, (int)blockIdx.y * chunk), ke = min(n, kb + chunk);
    float acc[2][4][4] = {};
    float4 sum = {};
    tile_product<2, false, false, float, true>(sA, sB, i0, dd, j0, di, kb, ke, J.dZ[l], dd, J.X[l], J.ldx[l], acc, sum);
    float *dW = out + blockIdx.y * stride + J.off[l];
    for_each_pair<2>(acc, i0, dd, j0, di, [&](int i, int j, float a, float b, bool two) {
        put_pair(dW + (int64_t)i * di + j, a, b, two);
    });
    if (j0 == 0) {
        float4 *part = reinterpret_cast<float4 *>(sA);       // the product's last barrier freed it
        part[threadIdx.x] = sum;
        __syncthreads();
        if (threadIdx.x < kTile && i0 + (int)threadIdx.x < dd) {
            float t = 0.f;
            for (int r = 0; r < 128 / (kTile / 4); ++r) t += reinterpret_cast<const float *>(part + r * (kTile / 4))[threadIdx.x];
            dW[(int64_t)dd * di + i0 + threadIdx.x] = t;
        }
    }
}

// C = sum over split-K slabs (fixed order)
__global__ void split_reduce_kernel(int64_t count, int splits, const float *__restrict__ part, float *__restrict__ C) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= count) return;
    float s = 0.f;
    for (int z = 0; z < splits; ++z) s += part[(int64_t)z * count + t];
    C[t] = s;
}

// Adam with bias correction; the step counter and learning rate come from
// device memory so the whole training step can be replayed as one graph.
// Place of parameter t in the BF16 copy, where the rows of the first layer's
// weights (di features of any number) are ld = 4, 8, .. elements apart, so that
// four neighbours are one load.
struct Bf16Order {
    int64_t first;               // weights of the first layer
    int di, ld;
    __host__ __device__ int64_t at(int64_t t) const {
        return t < first ? t / di * ld + t % di : t + first / di * (ld - di);
    }
};

__global__ void adam_kernel(int64_t count, Bf16Order order, float *__restrict__ w, __nv_bfloat16 *__restrict__ wb,
                            const float *__restrict__ g, float *__restrict__ m, float *__restrict__ v,
                            const int *__restrict__ step, const float *__restrict__ lr_sched, int nsched) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= count) return;
    const int s = *step;
    const float lr = lr_sched[min(s, nsched - 1)];
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float gi = g[t];
    const float mi = b1 * m[t] + (1.f - b1) * gi;
    const float vi = b2 * v[t] + (1.f - b2) * gi * gi;
    m[t] = mi;
    v[t] = vi;
    const float c1 = 1.f - powf(b1, (float)(s + 1)), c2 = 1.f - powf(b2, (float)(s + 1));
    const float wn = w[t] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[t] = wn;
    wb[order.at(t)] = __float2bfloat16_rn(wn);
}

__global__ void step_kernel(int *step, const float *loss, float *hist, int nhist) {
    const int k = *step;
    if (k < nhist) hist[k] = *loss;
    *step = k + 1;
}

__global__ void to_bf16_kernel(int64_t count, Bf16Order order, const float *__restrict__ w, __nv_bfloat16 *__restrict__ wb) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t < count) wb[order.at(t)] = __float2bfloat16_rn(w[t]);
}

template <class T>
struct Buf {
    T *p = nullptr;
    size_t n = 0;
    ~Buf() { if (p) cudaFree(p); }
    void reserve(size_t c) {
        if (c <= n && p) return;
        if (p) cudaFree(p);
        p = nullptr;
        SUR_CUDA(cudaMalloc(&p, std::max<size_t>(c, 1) * sizeof(T)));
        n = c;
    }
};

inline unsigned blocks(int64_t count, int per = 256) { return (unsigned)((count + per - 1) / per); }

}  // namespace

struct spx_surrogate {
    int device = 0;
    cudaStream_t stream = nullptr;
    int lmax = 0, nin = 0, hidden = 0, layers = 0, nout = 0;
    std::vector<int> din, dout;          // per dense layer
    std::vector<size_t> woff, boff;      // offsets in the parameter vector
    size_t nparam = 0;
    Buf<float> w, g, m, v;               // master weights, gradients, Adam moments
    Buf<__nv_bfloat16> wb;               // BF16 weights used by every product
    Buf<float> feat, loss, lr, hist, split;
    Buf<double> coef;                    // of the features' recurrences
    Buf<int> step;
    std::vector<Buf<float>> Z, Y;        // per layer pre-activation (going back: its derivative) / output
    int64_t cap = 0;                     // rows the activation buffers hold
    cudaGraphExec_t graph = nullptr;
    int64_t graph_n = -1;
    const float *graph_targets = nullptr;
    std::string err;
    int ld(size_t l) const { return l == 0 ? (nin + 3) & ~3 : din[l]; }     // of a layer's input and BF16 weights
    Bf16Order order() const { return {(int64_t)din[0] * dout[0], din[0], ld(0)}; }
    const __nv_bfloat16 *weights(size_t l) const { return wb.p + (l == 0 ? 0 : order().at((int64_t)woff[l])); }
};

namespace {

// slabs of the samples that the weight gradients are split over
int splits_of(int64_t n) { return (int)std::min<int64_t>(kMaxSplits, std::max<int64_t>(1, n / kSplitRows)); }

size_t param_end(const spx_surrogate *s, size_t l) { return s->boff[l] + s->dout[l]; }

// layers a .. b-1 take one launch of the weight gradients: as many as leave the
// slabs' buffer at 256 MB, one at least
size_t grad_group(const spx_surrogate *s, size_t a, int splits) {
    size_t b = a + 1;
    while (b < s->din.size() && (param_end(s, b) - s->woff[a]) * splits <= (size_t)64 << 20) ++b;
    return b;
}

void ensure_rows(spx_surrogate *s, int64_t n) {
    s->feat.reserve((size_t)n * s->ld(0));
    for (size_t l = 0; l < s->Z.size(); ++l) {
        s->Z[l].reserve((size_t)n * s->dout[l]);
        s->Y[l].reserve((size_t)n * s->dout[l]);
    }
    const int splits = splits_of(n);
    for (size_t a = 0; splits > 1 && a < s->din.size();) {
        const size_t b = grad_group(s, a, splits);
        s->split.reserve((param_end(s, b - 1) - s->woff[a]) * splits);
        a = b;
    }
    s->cap = std::max(s->cap, n);
}

void features(spx_surrogate *s, int64_t n, const double *b, const double *g, float *out, int ld) {
    sh_features_kernel<<<blocks(n, 32), 32 * feature_warps(s->lmax), feature_smem(s->nin), s->stream>>>(
        n, b, g, s->lmax, s->nin, ld, s->coef.p, out);
}

unsigned tiles(int64_t rows, int cols, int height) {
    return (unsigned)((cols + kTile - 1) / kTile * ((rows + height - 1) / height));
}

// forward through every layer into out; with targets T also the derivative at
// the last layer and the loss, and the pre-activations are kept
void forward(spx_surrogate *s, int64_t n, const float *T, float *out) {
    const size_t L = s->din.size();
    if (T) SUR_CUDA(cudaMemsetAsync(s->loss.p, 0, sizeof(float), s->stream));
    for (size_t l = 0; l < L; ++l) {
        const bool last = l + 1 == L;
        const float *x = l == 0 ? s->feat.p : s->Y[l - 1].p, *b = s->w.p + s->boff[l];
        float *z = T ? s->Z[l].p : nullptr, *y = last ? out : s->Y[l].p;
        const int dd = s->dout[l], di = s->din[l], ld = s->ld(l);
        const unsigned grid = tiles(n, dd, kLayerRows);
        if (last)
            layer_kernel<true><<<grid, 128, 0, s->stream>>>((int)n, dd, di, x, ld, s->weights(l), ld, b, z, y, T, s->loss.p);
        else
            layer_kernel<false><<<grid, 128, 0, s->stream>>>((int)n, dd, di, x, ld, s->weights(l), ld, b, z, y, nullptr,
                                                             nullptr);
    }
}

// gradients of every parameter (s->g), after forward() with targets
void backward(spx_surrogate *s, int64_t n) {
    const size_t L = s->din.size();
    for (size_t l = L - 1; l > 0; --l)
        layer_back_kernel<<<tiles(n, s->din[l], kLayerRows), 128, 0, s->stream>>>(
            (int)n, s->dout[l], s->din[l], s->Z[l].p, s->weights(l), s->Z[l - 1].p);
    const int splits = splits_of(n);
    for (size_t a = 0; a < L;) {
        const size_t b = grad_group(s, a, splits), first = s->woff[a], count = param_end(s, b - 1) - first;
        GradJobs J{};
        J.layers = (int)(b - a);
        for (size_t l = a; l < b; ++l) {
            J.dZ[l - a] = s->Z[l].p;
            J.X[l - a] = l == 0 ? s->feat.p : s->Y[l - 1].p;
            J.dd[l - a] = s->dout[l];
            J.di[l - a] = s->din[l];
            J.ldx[l - a] = s->ld(l);
            J.off[l - a] = (int64_t)(s->woff[l] - first);
            J.tile[l - a + 1] = J.tile[l - a] + (int)tiles(s->dout[l], s->din[l], kTile);
        }
        weight_grad_kernel<<<dim3(J.tile[b - a], splits), 128, 0, s->stream>>>(
            J, (int)n, splits > 1 ? s->split.p : s->g.p + first, (int64_t)count);
        if (splits > 1)
            split_reduce_kernel<<<blocks((int64_t)count), 256, 0, s->stream>>>((int64_t)count, splits, s->split.p,
                                                                               s->g.p + first);
        a = b;
    }
}

void train_step(spx_surrogate *s, int64_t n, const float *T, int nsched) {
    forward(s, n, T, s->Y.back().p);
    backward(s, n);
    adam_kernel<<<blocks((int64_t)s->nparam), 256, 0, s->stream>>>((int64_t)s->nparam, s->order(), s->w.p, s->wb.p, s->g.p, s->m.p,
                                                                  s->v.p, s->step.p, s->lr.p, nsched);
    step_kernel<<<1, 1, 0, s->stream>>>(s->step.p, s->loss.p, s->hist.p, nsched);
}

template <class F>
spx_status sur_guard(spx_surrogate *s, F f) {
    try {
        f();
        if (s) s->err.clear();
        return SPX_OK;
    } catch (const SurErr &e) {
        if (s) s->err = e.what();
        return e.code;
    } catch (const std::bad_alloc &) {
        if (s) s->err = "host allocation failed";
        return SPX_ERR_OUT_OF_MEMORY;
    } catch (const std::exception &e) {
        if (s) s->err = e.what();
        return SPX_ERR_INTERNAL;
    }
}

void init_params(spx_surrogate *s, uint64_t seed) {
    std::vector<float> h(s->nparam, 0.f);
    std::mt19937_64 rng(seed);
    for (size_t l = 0; l < s->din.size(); ++l) {
        const float bound = std::sqrt(6.0f / (float)s->din[l]);     // He-uniform for GELU layers
        std::uniform_real_distribution<float> U(-bound, bound);
        for (size_t t = 0; t < (size_t)s->din[l] * s->dout[l]; ++t) h[s->woff[l] + t] = U(rng);
    }
    SUR_CUDA(cudaMemcpy(s->w.p, h.data(), s->nparam * sizeof(float), cudaMemcpyHostToDevice));
    to_bf16_kernel<<<blocks((int64_t)s->nparam), 256, 0, s->stream>>>((int64_t)s->nparam, s->order(), s->w.p, s->wb.p);
    SUR_CUDA(cudaMemsetAsync(s->m.p, 0, s->nparam * sizeof(float), s->stream));
    SUR_CUDA(cudaMemsetAsync(s->v.p, 0, s->nparam * sizeof(float), s->stream));
    SUR_CUDA(cudaStreamSynchronize(s->stream));
}

}  // namespace

extern "C" {

spx_status spx_surrogate_create(spx_surrogate **out, int device, int32_t lmax, int32_t hidden, int32_t layers,
                                int32_t n_out, uint64_t seed) {
    if (!out) return SPX_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    if (lmax < 0 || lmax > kMaxL || hidden < 1 || hidden > 4096 || layers < 1 || layers > 16 || n_out < 1 ||
        n_out > 4096)
        return SPX_ERR_INVALID_ARGUMENT;
    spx_surrogate *s = new (std::nothrow) spx_surrogate();
    if (!s) return SPX_ERR_OUT_OF_MEMORY;
    const spx_status st = sur_guard(s, [&] {
        SUR_CUDA(cudaSetDevice(device));
        s->device = device;
        SUR_CUDA(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking));
        s->lmax = lmax;
        s->nin = (lmax + 1) * (lmax + 1);
        s->hidden = hidden;
        s->layers = layers;
        s->nout = n_out;
        int prev = s->nin;
        for (int l = 0; l < layers; ++l) { s->din.push_back(prev); s->dout.push_back(hidden); prev = hidden; }
        s->din.push_back(prev);
        s->dout.push_back(n_out);
        size_t off = 0;
        for (size_t l = 0; l < s->din.size(); ++l) {
            s->woff.push_back(off);
            off += (size_t)s->din[l] * s->dout[l];
            s->boff.push_back(off);
            off += (size_t)s->dout[l];
        }
        s->nparam = off;
        s->w.reserve(off); s->g.reserve(off); s->m.reserve(off); s->v.reserve(off); s->wb.reserve((size_t)s->order().at((int64_t)off));
        s->loss.reserve(1);
        s->coef.reserve(kCoefs);
        const std::vector<double> coef = feature_coefficients();
        SUR_CUDA(cudaMemcpy(s->coef.p, coef.data(), coef.size() * sizeof(double), cudaMemcpyHostToDevice));
        s->step.reserve(1);
        s->Z.resize(s->din.size());
        s->Y.resize(s->din.size());
        init_params(s, seed);
    });
    if (st != SPX_OK) {
        spx_surrogate_destroy(s);
        return st;
    }
    *out = s;
    return SPX_OK;
}

spx_status spx_surrogate_destroy(spx_surrogate *s) {
    if (!s) return SPX_OK;
    cudaSetDevice(s->device);
    if (s->stream) cudaStreamSynchronize(s->stream);
    if (s->graph) cudaGraphExecDestroy(s->graph);
    if (s->stream) cudaStreamDestroy(s->stream);
    delete s;
    return SPX_OK;
}

int64_t spx_surrogate_num_params(const spx_surrogate *s) { return s ? (int64_t)s->nparam : 0; }

spx_status spx_surrogate_features(spx_surrogate *s, int64_t n, const double *d_beta, const double *d_gamma,
                                  float *d_features) {
    if (!s || n < 1 || !d_beta || !d_gamma || !d_features) return SPX_ERR_INVALID_ARGUMENT;
    return sur_guard(s, [&] {
        SUR_CUDA(cudaSetDevice(s->device));
        features(s, n, d_beta, d_gamma, d_features, s->nin);
        SUR_CUDA(cudaGetLastError());
        SUR_CUDA(cudaStreamSynchronize(s->stream));
    });
}

spx_status spx_surrogate_train(spx_surrogate *s, int64_t n, const double *d_beta, const double *d_gamma,
                               const float *d_targets, int32_t epochs, float lr, float *loss_out) {
    if (!s || n < 1 || !d_beta || !d_gamma || !d_targets || epochs < 1 || !(lr > 0.f)) return SPX_ERR_INVALID_ARGUMENT;
    return sur_guard(s, [&] {
        SUR_CUDA(cudaSetDevice(s->device));
        ensure_rows(s, n);
        features(s, n, d_beta, d_gamma, s->feat.p, s->ld(0));
        // cosine-decayed learning rate per step, read by the Adam kernel
        std::vector<float> sched(epochs);
        for (int e = 0; e < epochs; ++e)
            sched[e] = lr * (0.02f + 0.98f * 0.5f * (1.f + std::cos(3.14159265358979f * e / epochs)));
        s->lr.reserve(epochs);
        s->hist.reserve(epochs);
        SUR_CUDA(cudaMemcpyAsync(s->lr.p, sched.data(), epochs * sizeof(float), cudaMemcpyHostToDevice, s->stream));
        SUR_CUDA(cudaMemsetAsync(s->step.p, 0, sizeof(int), s->stream));
        SUR_CUDA(cudaStreamSynchronize(s->stream));
        // one training step as a graph, replayed every epoch
        if (s->graph) { cudaGraphExecDestroy(s->graph); s->graph = nullptr; }
        cudaGraph_t g = nullptr;
        SUR_CUDA(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
        train_step(s, n, d_targets, epochs);
        SUR_CUDA(cudaStreamEndCapture(s->stream, &g));
        const cudaError_t ie = cudaGraphInstantiate(&s->graph, g, 0);
        cudaGraphDestroy(g);
        SUR_CUDA(ie);
        for (int e = 0; e < epochs; ++e) SUR_CUDA(cudaGraphLaunch(s->graph, s->stream));
        if (loss_out)
            SUR_CUDA(cudaMemcpyAsync(loss_out, s->hist.p, epochs * sizeof(float), cudaMemcpyDeviceToHost, s->stream));
        SUR_CUDA(cudaStreamSynchronize(s->stream));
    });
}

spx_status spx_surrogate_predict(spx_surrogate *s, int64_t n, const double *d_beta, const double *d_gamma,
                                 float *d_out) {
    if (!s || n < 1 || !d_beta || !d_gamma || !d_out) return SPX_ERR_INVALID_ARGUMENT;
    return sur_guard(s, [&] {
        SUR_CUDA(cudaSetDevice(s->device));
        ensure_rows(s, n);
        features(s, n, d_beta, d_gamma, s->feat.p, s->ld(0));
        forward(s, n, nullptr, d_out);
        SUR_CUDA(cudaGetLastError());
        SUR_CUDA(cudaStreamSynchronize(s->stream));
    });
}

spx_status spx_surrogate_gradients(spx_surrogate *s, int64_t n, const double *d_beta, const double *d_gamma,
                                   const float *d_targets, float *h_grad, float *h_loss) {
    if (!s || n < 1 || !d_beta || !d_gamma || !d_targets || !h_grad) return SPX_ERR_INVALID_ARGUMENT;
    return sur_guard(s, [&] {
        SUR_CUDA(cudaSetDevice(s->device));
        ensure_rows(s, n);
        features(s, n, d_beta, d_gamma, s->feat.p, s->ld(0));
        forward(s, n, d_targets, s->Y.back().p);
        backward(s, n);
        SUR_CUDA(cudaGetLastError());
        SUR_CUDA(cudaMemcpyAsync(h_grad, s->g.p, s->nparam * sizeof(float), cudaMemcpyDeviceToHost, s->stream));
        if (h_loss) SUR_CUDA(cudaMemcpyAsync(h_loss, s->loss.p, sizeof(float), cudaMemcpyDeviceToHost, s->stream));
        SUR_CUDA(cudaStreamSynchronize(s->stream));
    });
}

spx_status spx_surrogate_get_params(spx_surrogate *s, float *h_params) {
    if (!s || !h_params) return SPX_ERR_INVALID_ARGUMENT;
    return sur_guard(s, [&] {
        SUR_CUDA(cudaSetDevice(s->device));
        SUR_CUDA(cudaMemcpy(h_params, s->w.p, s->nparam * sizeof(float), cudaMemcpyDeviceToHost));
    });
}

spx_status spx_surrogate_set_params(spx_surrogate *s, const float *h_params) {
    if (!s || !h_params) return SPX_ERR_INVALID_ARGUMENT;
    return sur_guard(s, [&] {
        SUR_CUDA(cudaSetDevice(s->device));
        SUR_CUDA(cudaMemcpy(s->w.p, h_params, s->nparam * sizeof(float), cudaMemcpyHostToDevice));
        to_bf16_kernel<<<blocks((int64_t)s->nparam), 256, 0, s->stream>>>((int64_t)s->nparam, s->order(), s->w.p, s->wb.p);
        SUR_CUDA(cudaMemsetAsync(s->m.p, 0, s->nparam * sizeof(float), s->stream));
        SUR_CUDA(cudaMemsetAsync(s->v.p, 0, s->nparam * sizeof(float), s->stream));
        SUR_CUDA(cudaStreamSynchronize(s->stream));
    });
}

const char *spx_surrogate_last_error(const spx_surrogate *s) { return s ? s->err.c_str() : "NULL surrogate"; }

}  // extern "C"

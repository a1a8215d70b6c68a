// randomized_svd (src/randomized/mod.rs:24-199) on the device.
//
//   Y = A Omega; q x [Z = A^T Y, normalise Z; Y = A Z, normalise Y];
//   Q = qr(Y).q; B^T = A^T Q; SVD(B); U = Q U_B.
//
// nalgebra's Householder qr().q() (third-party) is replaced by CholeskyQR2:
// the Gram X^T X in FP64, a one-block Cholesky, X R^-1, twice; if a Cholesky
// pivot breaks down the pass is redone with a shift (shifted CholeskyQR3).
// The column spaces are those of Householder QR; column signs may differ.
// nalgebra's svd(B) is replaced by: QR of B^T = Q_b R (CholeskyQR2), then a
// one-sided Jacobi SVD of the small R in one block, so that
// B = V_R S (Q_b U_R)^T, singular values in descending order.
//
// SVDB_MIXED runs the sparse products on FP32 matrix values and an FP32 copy
// of the dense operand (half the gathered bytes) with FP64 sums; the Gram
// products, Cholesky, both CholeskyQR passes and the small SVD stay FP64.
#include <cooperative_groups.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "dense_small.cuh"
#include "device_common.cuh"
#include "ops.cuh"
#include "svdb_internal.h"

namespace svdb {

namespace cg = cooperative_groups;

static int nb(int64_t work, int threads, int per_sm = 16) {
    int64_t b = (work + threads - 1) / threads;
    return (int)std::max<int64_t>(1, std::min<int64_t>(b, (int64_t)device_props().sms * per_sm));
}

// --------------------------------------------------------------- Omega ----
template <typename T>
__global__ void k_omega(uint64_t seed, int64_t total, T* __restrict__ out) {
    const uint64_t key = omega_key(seed);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (T)omega_value(key, i);
}

// ------------------------------------------------------ small dense ops ----
// Every kernel of a CholeskyQR pass takes `cond`: when it points to 0 the
// kernel returns at once (the conditional third pass of shifted CholeskyQR).
__global__ void __launch_bounds__(384) k_chol_inv(const double* __restrict__ G, int nparts, int c, double shift_scale,
                                                  double* __restrict__ R, double* __restrict__ Ri,
                                                  int* __restrict__ flags, int* __restrict__ shifted,
                                                  const int* __restrict__ cond, int* __restrict__ loose) {
    if (cond && *cond == 0) return;
    extern __shared__ __align__(16) double sm[];
    chol_inv_body(G, nparts, c, shift_scale, R, Ri, flags, shifted, sm, loose);
}

// CholeskyQR2 of X (rows x c, in place), the third pass included when a shift
// was used, in one cluster of kQrCluster CTAs that each own a range of rows:
// Gram partials in shared memory, summed a slice per CTA and handed round;
// every CTA factors the same G (no hand-over), and multiplies its own rows.
// One launch instead of ten to thirteen (four per pass, the third pass's
// returning at once): for few rows the launches and their gaps were most of the
// time (1,000 x 20: 40 us per factorisation against 55 and ten gaps; 5,600 x 40:
// 92 us against 105).
// Rout (may be null) = R_last ... R_first; Rw: 3 c x c of workspace.
constexpr int kQrCluster = 16, kQrThreads = 384;
struct QrLayout {
    size_t part, red, G, chol, Ri, bytes;  // doubles; red, chol and the nn factor share one region
};
__host__ __device__ inline QrLayout qr_layout(int c) {
    const TnShape h = tn_shape(1, c, c, true, 1);
    const size_t red = (size_t)(kQrThreads / 32) * h.nt * h.nt * 64;
    const size_t region = std::max(std::max(red, chol_smem(c) / 8), nn_smem(c, (c + 7) / 8) / 8);
    QrLayout L;
    L.part = 0;
    L.G = (size_t)c * c;
    L.Ri = L.G + (size_t)c * c;
    L.red = L.Ri + (size_t)c * c;
    L.chol = L.red;
    L.bytes = (L.red + region) * 8;
    return L;
}
template <int NT, int NQ>
__device__ __forceinline__ void qr_pass(double* X, int64_t rows, int c, int nb, int rg, double shift_scale, double* R,
                                        int* flags, int* shifted, int* loose, double* sm, const QrLayout& L) {
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), cc = c * c;
    tn_part_body<double, double, NT>(X, c, c, X, c, c, 0, rows, nb, nb, true, rg, sm + L.part, sm + L.red);
    cl.sync();  // every CTA's partial is there
    // a slice of G per CTA, written into all of them (tile blocks I <= J; the
    // others are never read)
    const int per = (cc + kQrCluster - 1) / kQrCluster;
    const int w = NT * 8;
    for (int e = rank * per + (int)threadIdx.x; e < min(cc, (rank + 1) * per); e += blockDim.x) {
        if ((e / c) / w > (e % c) / w) continue;
        double v[kQrCluster], t = 0.0;
#pragma unroll
        for (int b = 0; b < kQrCluster; ++b) v[b] = *cl.map_shared_rank(sm + L.part + e, b);
#pragma unroll
        for (int b = 0; b < kQrCluster; ++b) t += v[b];
#pragma unroll
        for (int b = 0; b < kQrCluster; ++b) *cl.map_shared_rank(sm + L.G + e, b) = t;
    }
    cl.sync();
    // flags and R: one CTA's stores are enough (the others' go where nobody looks)
    chol_inv_body(sm + L.G, 0, c, shift_scale, rank == 0 ? R : sm + L.part, sm + L.Ri, flags, shifted, sm + L.chol,
                  loose);
    __syncthreads();
    const NnArgs<double, double> A{X, c, rows, c, sm + L.Ri, c, nullptr, c, 1, 1.0, nullptr, 0, 0.0, nullptr, 0,
                                   nullptr, X, c, 0, nullptr, nullptr};
    nn_body<double, double, NQ, 0>(A, threadIdx.x >> 5, blockDim.x >> 5, 0, sm + L.red);
    __syncthreads();
}
template <int NT, int NQ>
__global__ void __launch_bounds__(kQrThreads, 1) k_cholqr_cluster(double* X, int64_t rows, int c, int nb, int rg,
                                                                  double shift_scale, double* Rw, double* Rout,
                                                                  int* flags, const int* cond, int* loose) {
    if (cond && *cond == 0) return;  // the same for every CTA
    extern __shared__ __align__(16) double qr_sm[];
    __shared__ int s_shifted, s_loose;
    cg::cluster_group cl = cg::this_cluster();
    const QrLayout L = qr_layout(c);
    const int rank = (int)cl.block_rank(), cc = c * c;
    const int64_t per = (rows + kQrCluster - 1) / kQrCluster;
    const int64_t r0 = min(rows, rank * per), mine = min(rows, r0 + per) - r0;
    if (threadIdx.x == 0) s_shifted = s_loose = 0;
    __syncthreads();
    X += r0 * c;
    int passes = 2;
    for (int p = 0; p < passes; ++p) {
        qr_pass<NT, NQ>(X, mine, c, nb, rg, shift_scale, Rw + p * cc, flags, &s_shifted, p == 1 ? &s_loose : nullptr,
                        qr_sm, L);
        if (p == 1 && s_shifted) passes = 3;  // every CTA factored the same matrices
    }
    if (rank == 0) {
        if (threadIdx.x == 0 && loose && (s_loose || s_shifted)) *loose = 1;
        if (Rout) {  // R_last ... R_first, this CTA's own stores
            double* acc = qr_sm + L.part;
            double* tmp = qr_sm + L.G;
            for (int t = threadIdx.x; t < cc; t += blockDim.x) acc[t] = Rw[t];
            __syncthreads();
            for (int p = 1; p < passes; ++p) {
                for (int t = threadIdx.x; t < cc; t += blockDim.x) {
                    const int i = t / c, j = t - i * c;
                    double v = 0.0;
                    for (int k = i; k <= j; ++k) v = fma(Rw[(int64_t)p * cc + i * c + k], acc[k * c + j], v);
                    tmp[t] = v;
                }
                __syncthreads();
                double* o = acc;
                acc = tmp;
                tmp = o;
            }
            for (int t = threadIdx.x; t < cc; t += blockDim.x) Rout[t] = acc[t];
        }
    }
    cl.sync();  // no CTA leaves while another may still read its shared memory
}

// C (c x c) = A (c x c) B (c x c), one thread per element
__global__ void k_small_gemm(const double* __restrict__ A, const double* __restrict__ B, int c,
                             double* __restrict__ C, const int* __restrict__ cond) {
    if (cond && *cond == 0) return;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < c * c; t += gridDim.x * blockDim.x) {
        const int i = t / c, j = t % c;
        double s = 0.0;
        for (int k = 0; k < c; ++k) s = fma(A[i * c + k], B[k * c + j], s);
        C[t] = s;
    }
}

__global__ void k_copy_cond(const double* __restrict__ src, double* __restrict__ dst, int64_t n,
                            const int* __restrict__ cond) {
    if (cond && *cond == 0) return;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dst[i] = src[i];
}

template <typename T>
__global__ void k_colnorm(T* __restrict__ X, int64_t rows, int c) {
    __shared__ double sh[32];
    __shared__ double scale;
    const int j = blockIdx.x;
    double acc = 0.0;
    for (int64_t r = threadIdx.x; r < rows; r += blockDim.x) {
        const double v = (double)X[r * c + j];
        acc = fma(v, v, acc);
    }
    const double nrm = sqrt(block_sum(acc, sh));
    if (threadIdx.x == 0) scale = nrm > 1e-10 ? 1.0 / nrm : 1.0;
    __syncthreads();
    if (nrm > 1e-10)
        for (int64_t r = threadIdx.x; r < rows; r += blockDim.x) X[r * c + j] = (T)((double)X[r * c + j] * scale);
}

// One-sided Jacobi SVD of the c x c R in one block (jacobi_svd_body).
__global__ void __launch_bounds__(960) k_jacobi_svd(const double* __restrict__ R, int trans, int c,
                                                     double* __restrict__ U, double* __restrict__ V,
                                                     double* __restrict__ sig, int* __restrict__ status) {
    extern __shared__ __align__(16) double sm[];
    jacobi_svd_body<true>(R, trans != 0, c, U, V, sig, status, sm);
}
// c <= 64: the widths of most solves, with the registers of smaller blocks
__global__ void __launch_bounds__(256) k_jacobi_svd64(const double* __restrict__ R, int trans, int c,
                                                      double* __restrict__ U, double* __restrict__ V,
                                                      double* __restrict__ sig, int* __restrict__ status) {
    extern __shared__ __align__(16) double sm[];
    jacobi_svd_body<false>(R, trans != 0, c, U, V, sig, status, sm);
}

__global__ void k_to_float(const double* __restrict__ in, float* __restrict__ out, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (float)in[i];
}

// out (rows x ldx) = in (rows x c), rounded to FP32; columns c .. ldx-1 are not written
__global__ void k_to_float_ld(const double* __restrict__ in, float* __restrict__ out, int64_t rows, int c,
                              int64_t ldx) {
    const int64_t n = rows * c;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = i < ((int64_t)1 << 32) ? (int64_t)((uint32_t)i / (uint32_t)c) : i / c;
        out[r * ldx + (i - r * c)] = (float)in[i];
    }
}
// copy the first `cout` columns of X (rows x c) into Out (rows x cout)
__global__ void k_take_cols(const double* __restrict__ X, int64_t rows, int c, int cout, double* __restrict__ Out) {
    const int64_t total = rows * cout;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x)
        Out[t] = X[(t / cout) * c + t % cout];
}

// ------------------------------------------------------------ centring ----
// Products of the centred matrix A - 1 mu^T, mu the column means
// (compute_column_means, masked.rs:240-263), as A X - 1 (mu^T X) and
// A^T Y - mu (1^T Y).  mu comes from the column-major copy, one warp per
// column with a fixed lane order.
__global__ void k_major_means(const int64_t* __restrict__ ptr, const double* __restrict__ val, int64_t nmajor,
                              double inv, double* __restrict__ mu) {
    const int lane = threadIdx.x & 31;
    const int64_t w0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t j = w0; j < nmajor; j += nw) {
        double acc = 0.0;
        for (int64_t k = ptr[j] + lane; k < ptr[j + 1]; k += 32) acc += val[k];
#pragma unroll
        for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) mu[j] = acc * inv;
    }
}
// part[b][j] = sum over the rows of chunk b of w[r] X[r][j] (w = 1 when null),
// for the c <= 128 columns of X starting at X (row stride ld).  A warp takes
// every eighth row of the chunk, its lanes the columns, four rows in flight;
// the warps' partials are added in warp order, the chunks' by k_tn_reduce.
// 256-row chunks with one row in flight and one thread per column over all
// chunks took 18 + 12 us per product of 30,011 x 40; this form 6 + 6.
constexpr int kCsCols = 128;
template <int NC>
__global__ void __launch_bounds__(256) k_wcolsum_part(const double* __restrict__ X, int64_t rows, int64_t ld, int c,
                                                      const double* __restrict__ w, int64_t chunk,
                                                      double* __restrict__ part) {
    __shared__ double sh[8][NC * 32];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int64_t r0 = blockIdx.x * chunk, r1 = std::min<int64_t>(rows, r0 + chunk);
    double acc[NC];
#pragma unroll
    for (int q = 0; q < NC; ++q) acc[q] = 0.0;
    for (int64_t r = r0 + ty; r < r1; r += 32) {
        double x[4][NC], wr[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const bool ok = r + 8 * u < r1;
            wr[u] = ok ? (w ? w[r + 8 * u] : 1.0) : 0.0;
#pragma unroll
            for (int q = 0; q < NC; ++q)
                x[u][q] = ok && tx + 32 * q < c ? X[(r + 8 * u) * ld + tx + 32 * q] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int q = 0; q < NC; ++q) acc[q] = fma(wr[u], x[u][q], acc[q]);
    }
#pragma unroll
    for (int q = 0; q < NC; ++q) sh[ty][tx + 32 * q] = acc[q];
    __syncthreads();
    for (int j = threadIdx.x; j < c; j += blockDim.x) {
        double t = 0.0;
#pragma unroll
        for (int y = 0; y < 8; ++y) t += sh[y][j];
        part[(int64_t)blockIdx.x * c + j] = t;
    }
}
// Y[r][j] -= a[r] t[j] (a = 1 when null), Y rows x c
__global__ void k_rank1_sub(double* __restrict__ Y, int64_t rows, int c, const double* __restrict__ a,
                            const double* __restrict__ t) {
    const int64_t total = rows * c;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = i < ((int64_t)1 << 32) ? (int64_t)((uint32_t)i / (uint32_t)c) : i / c;
        Y[i] -= (a ? a[r] : 1.0) * t[i - r * c];
    }
}

void column_means_dev(const DevCompressed& csc, int64_t rows, double* mu, cudaStream_t s) {
    if (csc.nmajor == 0) return;
    k_major_means<<<nb(csc.nmajor * 32, 256), 256, 0, s>>>(csc.ptr.p, csc.val.p, csc.nmajor,
                                                          rows > 0 ? 1.0 / (double)rows : 0.0, mu);
    SVDB_CHECK_LAUNCH();
}

void center_product(const double* X, int64_t xrows, int c, const double* mu, double* Out, int64_t orows,
                    bool out_is_rows, cudaStream_t s) {
    if (c <= 0 || orows <= 0) return;
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((xrows + 31) / 32, (int64_t)device_props().sms * 2));
    const int64_t chunk = (xrows + blocks - 1) / blocks;
    DevBuf<double> part((size_t)blocks * kCsCols, s), tot(c, s);
    for (int j0 = 0; j0 < c; j0 += kCsCols) {
        const int w = std::min(kCsCols, c - j0);
        const double* wt = out_is_rows ? mu : nullptr;
        if (w <= 32) k_wcolsum_part<1><<<blocks, 256, 0, s>>>(X + j0, xrows, c, w, wt, chunk, part.p);
        else if (w <= 64) k_wcolsum_part<2><<<blocks, 256, 0, s>>>(X + j0, xrows, c, w, wt, chunk, part.p);
        else k_wcolsum_part<4><<<blocks, 256, 0, s>>>(X + j0, xrows, c, w, wt, chunk, part.p);
        k_tn_reduce<<<(w + 31) / 32, 32 * kTnSlices, 0, s>>>(part.p, blocks, 1, w, 1, 0, tot.p + j0, nullptr);
        SVDB_CHECK_LAUNCH_N(2);
    }
    k_rank1_sub<<<nb(orows * c, 256), 256, 0, s>>>(Out, orows, c, out_is_rows ? nullptr : mu, tot.p);
    SVDB_CHECK_LAUNCH();
}

// ------------------------------------------------------ host helpers ----
struct RandCtx {
    cudaStream_t s;
    DevBuf<double> part, G, R1, Ri, Rtmp, T;  // R1: the passes' three factors
    DevBuf<int> flags, shifted, loose;
    int64_t part_cap = 0;
};

// G = X^T X on the tensor cores (3xTF32, FP32 accumulation; gram_tc.cu), the
// CTA partials summed in FP64 in block order
static void gram_tensor(RandCtx& cx, const double* X, int64_t rows, int c, double* G) {
    const int nblk = gram_tc_blocks(rows);
    if ((int64_t)nblk * c * c > cx.part_cap) {
        cx.part_cap = (int64_t)nblk * c * c;
        cx.part.alloc(cx.part_cap, cx.s);
    }
    gram_tc_launch(X, rows, c, cx.part.p, cx.part_cap, nullptr, cx.s);
    k_tn_reduce<<<(c * c + 31) / 32, 32 * kTnSlices, 0, cx.s>>>(cx.part.p, nblk, c, c, c, 0, G, nullptr);
    SVDB_CHECK_LAUNCH();
}

// X^T X on the FP64 matrix instruction.  Returns G, or (parts > 0) the
// partials that chol_inv adds itself: below kCholParts elements in all the
// one-block factorisation reads them faster than another launch.
constexpr int64_t kCholParts = 16384;
static const double* gram(RandCtx& cx, const double* X, int64_t rows, int c, double* G, const int* cond, int& parts) {
    if (c > 128) throw Error(SVDB_ERR_UNSUPPORTED, "randomized_svd: more than 128 sample columns");
    const TnShape h = tn_shape(rows, c, c, true, device_props().sms);
    const int64_t n = (int64_t)h.blocks * c * c;
    if (n > cx.part_cap) {
        cx.part_cap = n;
        cx.part.alloc(cx.part_cap, cx.s);
    }
    parts = n <= kCholParts ? h.blocks : 0;
    tn_launch(h, X, c, c, X, c, c, rows, cx.part.p, parts ? nullptr : G, cond, cx.s);
    return parts ? cx.part.p : G;
}

// Out (rows x cout, or cout x rows when trans) = X (rows x c) S (c x lds,
// first cout columns); upper: S is upper triangular
static void right_mul(const double* X, int64_t rows, int c, const double* S, int lds, int cout, double* Out,
                      cudaStream_t s, const int* cond = nullptr, bool upper = false, bool trans = false) {
    nn_launch<0>(NnArgs<double, double>{X, c, rows, c, S, lds, nullptr, cout, upper, 1.0, nullptr, 0, 0.0, nullptr, 0,
                                        nullptr, Out, trans ? rows : cout, trans, nullptr, cond},
                 device_props().sms, s);
}

// shifted CholeskyQR: shift = 11 (rows c + c (c + 1)) u ||X||_F^2, ||X||_F^2 = trace(G)
static double qr_shift(int64_t rows, int c) {
    return 11.0 * ((double)rows * c + (double)c * (c + 1)) * 1.1102230246251565e-16;
}

static void chol_inv(RandCtx& cx, const double* G, int parts, int c, int64_t rows, double* R, const int* cond,
                     int* loose) {
    const size_t smem = chol_smem(c);
    allow_smem(k_chol_inv, chol_smem(128));
    k_chol_inv<<<1, 384, smem, cx.s>>>(G, parts, c, qr_shift(rows, c), R, cx.Ri.p, cx.flags.p, cx.shifted.p, cond,
                                       loose);
    SVDB_CHECK_LAUNCH();
}

// The one-cluster form: c <= 64 (one column block, in place), a device that can
// hold the cluster, and few enough rows for its 16 SMs.  Whole solves (q = 2)
// with it and without: 4,000 x 60 1.33 / 1.48 ms, 8,000 x 60 1.58 / 1.56; 8,000 x
// 40 1.02 / 1.07, 16,000 x 40 1.36 / 1.17; 16,000 x 20 0.75 / 0.82.
constexpr int64_t kQrClusterSize = 320 << 10;  // rows x columns
template <int NT, int NQ>
static bool cholqr_cluster_as(RandCtx& cx, double* X, int64_t rows, int c, double* Rout, const int* cond, int* loose) {
    auto kern = k_cholqr_cluster<NT, NQ>;
    const TnShape h = tn_shape(1, c, c, true, 1);
    const size_t most = qr_layout(NQ * 8).bytes;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kQrCluster);
    cfg.blockDim = dim3(kQrThreads / (32 * h.ntb) * h.ntb * 32);
    cfg.dynamicSmemBytes = most;
    cfg.stream = cx.s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kQrCluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    // whether this device holds the kernel's widest cluster: asked once per
    // thread and device, like device_props()
    static thread_local int asked_dev = -1;
    static thread_local bool holds = false;
    int dev = 0;
    SVDB_CUDA(cudaGetDevice(&dev));
    if (dev != asked_dev) {
        int n = 0;
        holds = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) == cudaSuccess &&
                cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n >= 1;
        if (!holds) cudaGetLastError();
        asked_dev = dev;
    }
    if (!holds) return false;
    cfg.dynamicSmemBytes = qr_layout(c).bytes;
    SVDB_CUDA(cudaLaunchKernelEx(&cfg, kern, X, rows, c, h.nbp, (int)cfg.blockDim.x / (32 * h.ntb), qr_shift(rows, c),
                                 cx.R1.p, Rout, cx.flags.p, cond, loose));
    SVDB_CHECK_LAUNCH();
    return true;
}
static bool cholqr_cluster(RandCtx& cx, double* X, int64_t rows, int c, double* Rout, const int* cond, int* loose) {
    if (rows * c > kQrClusterSize || c > 64) return false;
    switch ((c + 7) / 8) {
        case 1: return cholqr_cluster_as<1, 1>(cx, X, rows, c, Rout, cond, loose);
        case 2: return cholqr_cluster_as<2, 2>(cx, X, rows, c, Rout, cond, loose);
        case 3: return cholqr_cluster_as<3, 3>(cx, X, rows, c, Rout, cond, loose);
        case 4: return cholqr_cluster_as<4, 4>(cx, X, rows, c, Rout, cond, loose);
        case 5: return cholqr_cluster_as<3, 5>(cx, X, rows, c, Rout, cond, loose);
        case 6: return cholqr_cluster_as<3, 6>(cx, X, rows, c, Rout, cond, loose);
        case 7: return cholqr_cluster_as<4, 7>(cx, X, rows, c, Rout, cond, loose);
        default: return cholqr_cluster_as<4, 8>(cx, X, rows, c, Rout, cond, loose);
    }
}

// Thin Q of X (rows x c, rows >= c) in place; Rout (c x c) = R_last ... R_first
// when requested.  CholeskyQR2; a pass whose Cholesky broke down is redone with
// a shift and a third pass follows.  Nothing here waits for the device: the
// third pass's kernels read the device flag and return when it is 0.  only_if
// (a device flag, may be null): nothing happens when it is 0.  loose: see
// chol_inv_body, for the second pass's Gram.
static void cholesky_qr(RandCtx& cx, double* X, int64_t rows, int c, double* Rout, const int* only_if = nullptr,
                        int* loose = nullptr) {
    cudaStream_t s = cx.s;
    if (cholqr_cluster(cx, X, rows, c, Rout, only_if, loose)) return;
    if ((int64_t)cx.T.n < rows * c) cx.T.alloc(rows * c, s);
    double* T = cx.T.p;
    SVDB_CUDA(cudaMemsetAsync(cx.shifted.p, 0, sizeof(int), s));
    double* R[3] = {cx.R1.p, cx.R1.p + (int64_t)c * c, cx.R1.p + 2 * (int64_t)c * c};
    auto pass = [&](const double* in, double* out, double* Rp, const int* cond, int* ls) {
        int parts = 0;
        const double* G = gram(cx, in, rows, c, cx.G.p, cond, parts);
        chol_inv(cx, G, parts, c, rows, Rp, cond, ls);
        right_mul(in, rows, c, cx.Ri.p, c, c, out, s, cond, true);
    };
    pass(X, T, R[0], only_if, nullptr);
    pass(T, X, R[1], only_if, loose);
    // pass 3 only after a shifted pass: X -> T -> X
    const int* cond = cx.shifted.p;
    pass(X, T, R[2], cond, nullptr);
    k_copy_cond<<<nb(rows * c, 256), 256, 0, s>>>(T, X, rows * c, cond);
    SVDB_CHECK_LAUNCH();
    if (Rout) {
        const int blocks = (c * c + 127) / 128;
        k_small_gemm<<<blocks, 128, 0, s>>>(R[1], R[0], c, Rout, nullptr);
        k_small_gemm<<<blocks, 128, 0, s>>>(R[2], Rout, c, cx.Rtmp.p, cond);
        k_copy_cond<<<1, 256, 0, s>>>(cx.Rtmp.p, Rout, (int64_t)c * c, cond);
        SVDB_CHECK_LAUNCH_N(3);
    }
}

// qr(X).q() for X (rows x c): returns the column count of Q; X is replaced by
// Q (rows x k, k = min(rows, c)) stored with row stride k.
static int thin_q(RandCtx& cx, DevBuf<double>& X, int64_t rows, int c, const int* only_if = nullptr,
                  int* loose = nullptr) {
    if (rows >= c) {
        cholesky_qr(cx, X.p, rows, c, nullptr, only_if, loose);
        return c;
    }
    // wide: Q spans R^rows; take the leading rows x rows block's Q
    const int k = (int)rows;
    DevBuf<double> Xk((int64_t)rows * k, cx.s);
    k_take_cols<<<nb(rows * k, 256), 256, 0, cx.s>>>(X.p, rows, c, k, Xk.p);
    SVDB_CHECK_LAUNCH();
    cholesky_qr(cx, Xk.p, rows, k, nullptr, nullptr, loose);
    X = std::move(Xk);
    return k;
}

static double ms_since(std::chrono::steady_clock::time_point t0) {
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

// svdb_gram_device: G (c x c) = X^T X for a device X (rows x c, FP64)
void gram_device(const double* X, int64_t rows, int c, double* G, int precision, cudaStream_t s) {
    if (c < 1 || c > 128) throw Error(SVDB_ERR_UNSUPPORTED, "gram: 1..128 columns");
    RandCtx cx;
    cx.s = s;
    if (precision == SVDB_MIXED) {
        if (c > 64) throw Error(SVDB_ERR_UNSUPPORTED, "gram: the tensor-core form takes at most 64 columns");
        gram_tensor(cx, X, rows, c, G);
    } else {
        const TnShape h = tn_shape(rows, c, c, true, device_props().sms);
        cx.part.alloc((int64_t)h.blocks * c * c, s);
        tn_launch(h, X, c, c, X, c, c, rows, cx.part.p, G, nullptr, s);
    }
    SVDB_CUDA(cudaStreamSynchronize(s));
    gram_tc_check();
}

void randomized(const svdb_matrix* A, uint64_t target_rank, uint64_t n_oversamples, uint64_t n_power_iters,
                int normalizer, int mean_center, int has_seed, uint64_t seed, int verbose, const svdb_options& o,
                svdb_rec* rec, bool f32) {
    cudaStream_t s = o.stream ? (cudaStream_t)o.stream : A->stream;
    // f32: the crate's T = f32 run: Omega's f64 draws rounded to f32
    // (T::from_f64, randomized/mod.rs:299-313) and FP32 operands
    const bool mixed = f32 || o.precision == SVDB_MIXED;
    const int64_t m = A->nrows, n = A->ncols;
    const int64_t rank = std::min<int64_t>((int64_t)target_rank, std::min(m, n));
    int l = (int)(rank + (int64_t)n_oversamples);
    if (l <= 0) throw Error(SVDB_ERR_SHAPE, "randomized_svd: zero sample columns");
    if (m == 0 || n == 0) throw Error(SVDB_ERR_SHAPE, "randomized_svd: the matrix has no rows or no columns");
    const DevCompressed& Acsr = csr_of(A);
    const DevCompressed& Acsc = csc_of(A);
    if (mixed) ensure_fp32(A);
    auto t0 = std::chrono::steady_clock::now();
    cudaEvent_t e0, e1;
    SVDB_CUDA(cudaEventCreate(&e0));
    SVDB_CUDA(cudaEventCreate(&e1));
    SVDB_CUDA(cudaEventRecord(e0, s));
    float spmm_ms = 0.f;

    RandCtx cx;
    cx.s = s;
    const int cmax = l;
    for (DevBuf<double>* b : {&cx.G, &cx.Ri, &cx.Rtmp}) b->alloc((size_t)cmax * cmax, s);
    cx.R1.alloc((size_t)3 * cmax * cmax, s);
    cx.flags.alloc(1, s);
    cx.shifted.alloc(1, s);
    cx.loose.alloc(1, s);
    DevBuf<int> jac_status(1, s);
    SVDB_CUDA(cudaMemsetAsync(cx.flags.p, 0, sizeof(int), s));
    SVDB_CUDA(cudaMemsetAsync(jac_status.p, 0, sizeof(int), s));

    // Omega (n x l)
    DevBuf<double> Om(std::max<int64_t>(n * l, 1), s);
    if (o.omega) {
        SVDB_CUDA(cudaMemcpyAsync(Om.p, o.omega, n * l * 8, cudaMemcpyHostToDevice, s));
    } else {
        k_omega<double><<<nb(n * l, 256), 256, 0, s>>>(has_seed ? seed : 0, n * l, Om.p);
        SVDB_CHECK_LAUNCH();
    }
    if (f32) round_f32(Om.p, n * l, s);

    // Sparse products: FP64 operands, or under SVDB_MIXED FP32 values and an
    // FP32 copy of the dense operand (half the gathered bytes), FP64 sums and output.
    DevBuf<float> f_in;
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> spmm_events;  // read once, at the end
    // SVDB_MIXED with dense columns: their share of each product on the tensor cores
    const bool split = mixed && !f32 && dense_split_usable(A, l);
    auto spmm = [&](const DevCompressed& M, const double* X, int c, double* Y) {
        cudaEvent_t a, b;
        SVDB_CUDA(cudaEventCreate(&a));
        SVDB_CUDA(cudaEventCreate(&b));
        SVDB_CUDA(cudaEventRecord(a, s));
        if (!mixed) {
            spmm_dev<double, double>(M, false, X, c, Y, s);
        } else {
            const int64_t ldp = ((int64_t)c + 31) / 32 * 32;  // rows on whole 128-byte lines
            if (!split && spmm_f32_strided_ok(M, c, ldp)) {
                if ((int64_t)f_in.n < M.nminor * ldp) f_in.alloc(M.nminor * ldp, s);
                k_to_float_ld<<<nb(M.nminor * c, 256), 256, 0, s>>>(X, f_in.p, M.nminor, c, ldp);
                SVDB_CHECK_LAUNCH();
                spmm_f32_strided(M, f_in.p, c, ldp, Y, s);
            } else {
                if ((int64_t)f_in.n < M.nminor * c) f_in.alloc(M.nminor * c, s);
                k_to_float<<<nb(M.nminor * c, 256), 256, 0, s>>>(X, f_in.p, M.nminor * c);
                SVDB_CHECK_LAUNCH();
                if (split) dense_split_spmm<double, double>(A, &M == &Acsc, X, f_in.p, c, Y, s);
                else spmm_dev<float, double>(M, true, f_in.p, c, Y, s);
            }
        }
        SVDB_CUDA(cudaEventRecord(b, s));
        spmm_events.emplace_back(a, b);
    };
    auto normalize = [&](DevBuf<double>& X, int64_t rows, int c, int* loose) -> int {
        if (normalizer == SVDB_NORM_QR) return thin_q(cx, X, rows, c, nullptr, loose);
        if (normalizer == SVDB_NORM_LU) {
            k_colnorm<double><<<c, 256, 0, s>>>(X.p, rows, c);
            SVDB_CHECK_LAUNCH();
        }
        return c;
    };

    // mean_center: the products of A - 1 mu^T
    DevBuf<double> mu;
    if (mean_center) {
        mu.alloc(std::max<int64_t>(n, 1), s);
        column_means_dev(Acsc, m, mu.p, s);
    }
    auto center = [&](const double* X, int64_t xrows, int c, double* Out, int64_t orows, bool out_is_rows) {
        if (mean_center) center_product(X, xrows, c, mu.p, Out, orows, out_is_rows, s);
    };

    if (verbose) printf("SVD | Randomized | Multiplying m with omega matrix....\n");
    DevBuf<double> Y(std::max<int64_t>(m * l, 1), s);
    spmm(Acsr, Om.p, l, Y.p);
    center(Om.p, n, l, Y.p, m, true);
    int c = l;
    if (verbose) printf("SVD | Randomized | Multiplication done, took: %.3f ms of total running time\n", ms_since(t0));
    if (verbose) printf("SVD | Randomized | Starting power iterations....\n");
    for (uint64_t it = 0; it < n_power_iters; ++it) {
        if (verbose)
            printf("SVD | Randomized | Running power-iteration: %llu, current time: %.3f ms\n",
                   (unsigned long long)it, ms_since(t0));
        DevBuf<double> Z(std::max<int64_t>(n * c, 1), s);
        spmm(Acsc, Y.p, c, Z.p);
        center(Y.p, m, c, Z.p, n, false);
        c = normalize(Z, n, c, nullptr);
        DevBuf<double> Y2(std::max<int64_t>(m * c, 1), s);
        spmm(Acsr, Z.p, c, Y2.p);
        center(Z.p, n, c, Y2.p, m, true);
        Y = std::move(Y2);
        SVDB_CUDA(cudaMemsetAsync(cx.loose.p, 0, sizeof(int), s));
        c = normalize(Y, m, c, cx.loose.p);
        if (verbose)
            printf("SVD | Randomized | Power Iteration Normalization Backward-Step %.3f ms\n", ms_since(t0));
    }
    if (verbose) printf("SVD | Randomized | Running QR-Normalization after Power-Iterations %.3f ms\n", ms_since(t0));
    // Q = qr(y).q().  After a QR-normalised iteration y is its own Q unless that
    // factorisation was a difficult one (cx.loose): nothing to do otherwise.
    const bool q_done = normalizer == SVDB_NORM_QR && n_power_iters > 0 && m >= c;
    c = thin_q(cx, Y, m, c, q_done ? cx.loose.p : nullptr);
    // B^T = A^T Q (n x c)
    DevBuf<double> Bt(std::max<int64_t>(n * c, 1), s);
    spmm(Acsc, Y.p, c, Bt.p);
    center(Y.p, m, c, Bt.p, n, false);
    if (verbose) printf("SVD | Randomized | Transposed Matrix Multiplication %.3f ms\n", ms_since(t0));

    // SVD(B), B = Bt^T (c x n).  r = min(c, n).
    // U = Q U_B (m x r) and Vt = V_B^T, of which the leading actual_rank are kept
    const int r = (int)std::min<int64_t>(c, n);
    const int64_t actual = std::min<int64_t>((int64_t)target_rank, r);
    DevBuf<double> U(std::max<int64_t>(m * actual, 1), s), Vt(std::max<int64_t>(actual * n, 1), s),
        S(std::max<int64_t>(actual, 1), s);
    {
        DevBuf<double> Ur((size_t)r * r, s), Vr((size_t)r * r, s), R((size_t)r * r, s), sig(r, s);
        if (r > 117) throw Error(SVDB_ERR_UNSUPPORTED, "randomized_svd: sample width above the Jacobi tile");
        DevBuf<double> B;  // n < c: B = Bt^T (c x n) is the tall one
        if (n < c) {
            B.alloc((size_t)c * n, s);
            transpose_dense<double>(Bt.p, B.p, n, c, s);
        }
        // tall = Q_b R;  R = U_J S V_J^T.  The one-sided Jacobi runs on
        // R^T = V_J S U_J^T, whose columns (the rows of the QR factor) are
        // graded, which takes fewer sweeps than R itself.
        double* tall = n < c ? B.p : Bt.p;
        const int64_t trows = n < c ? c : n;
        cholesky_qr(cx, tall, trows, r, R.p);
        if (r <= 64) {
            allow_smem(k_jacobi_svd64, jacobi_smem(64));
            k_jacobi_svd64<<<1, jacobi_threads(r), jacobi_smem(r), s>>>(R.p, 1, r, Vr.p, Ur.p, sig.p, jac_status.p);
        } else {
            allow_smem(k_jacobi_svd, jacobi_smem(117));
            k_jacobi_svd<<<1, jacobi_threads(r), jacobi_smem(r), s>>>(R.p, 1, r, Vr.p, Ur.p, sig.p, jac_status.p);
        }
        SVDB_CHECK_LAUNCH();
        if (actual > 0) {
            if (n >= c) {
                // B = Bt^T = V_J S (Q_b U_J)^T: U_B = V_J, V_B = Q_b U_J
                right_mul(Y.p, m, c, Vr.p, r, (int)actual, U.p, s);
                right_mul(tall, n, c, Ur.p, r, (int)actual, Vt.p, s, nullptr, false, true);
            } else {
                // B = (Q_b U_J) S V_J^T: U_B = Q_b U_J (c x r), V_B = V_J
                DevBuf<double> UB((size_t)c * r, s), VrT((size_t)r * r, s);
                right_mul(tall, c, r, Ur.p, r, r, UB.p, s);
                right_mul(Y.p, m, c, UB.p, r, (int)actual, U.p, s);
                transpose_dense<double>(Vr.p, VrT.p, r, r, s);
                SVDB_CUDA(cudaMemcpyAsync(Vt.p, VrT.p, actual * n * 8, cudaMemcpyDeviceToDevice, s));
            }
            SVDB_CUDA(cudaMemcpyAsync(S.p, sig.p, actual * 8, cudaMemcpyDeviceToDevice, s));
        }
    }
    if (verbose) printf("SVD | Randomized | Running Singular Value Decomposition, took %.3f ms\n", ms_since(t0));
    SVDB_CUDA(cudaEventRecord(e1, s));
    int hflags = 0, hjac = 0;
    SVDB_CUDA(cudaMemcpyAsync(&hflags, cx.flags.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    SVDB_CUDA(cudaMemcpyAsync(&hjac, jac_status.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    SVDB_CUDA(cudaStreamSynchronize(s));
    float tot = 0.f;
    cudaEventElapsedTime(&tot, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    for (auto& ev : spmm_events) {
        float t = 0.f;
        cudaEventElapsedTime(&t, ev.first, ev.second);
        spmm_ms += t;
        cudaEventDestroy(ev.first);
        cudaEventDestroy(ev.second);
    }
    // the opt-in product kernels' wait flags (each look is a synchronous copy)
    if (const char* e = getenv("SVDB_SPMM"); e && *e) {
        spmm_tma_check();
        spmm_panel_check();
    }
    if (split) dense_split_check();
    if (verbose) printf("SVD | Randomized | Jacobi sweeps on R: %d%s\n", hjac >> 8, (hjac & 2) ? " (limit)" : "");
    if (hflags & 2) throw Error(SVDB_ERR_LAS2, "randomized_svd: CholeskyQR broke down even with a shift");

    std::memset(rec, 0, sizeof(*rec));
    rec->d = actual;
    rec->u_rows = m; rec->u_cols = actual;
    rec->vt_rows = actual; rec->vt_cols = n;
    if (o.result_on_device) {
        rec->u = U.detach(); rec->s = S.detach(); rec->vt = Vt.detach();
        rec->on_device = 1;
    } else {
        rec->u = (double*)host_result_alloc(std::max<int64_t>(m * actual, 1) * 8);
        rec->s = (double*)host_result_alloc(std::max<int64_t>(actual, 1) * 8);
        rec->vt = (double*)host_result_alloc(std::max<int64_t>(actual * n, 1) * 8);
        if (actual) {
            SVDB_CUDA(cudaMemcpyAsync(rec->u, U.p, m * actual * 8, cudaMemcpyDeviceToHost, s));
            SVDB_CUDA(cudaMemcpyAsync(rec->s, S.p, actual * 8, cudaMemcpyDeviceToHost, s));
            SVDB_CUDA(cudaMemcpyAsync(rec->vt, Vt.p, actual * n * 8, cudaMemcpyDeviceToHost, s));
        }
        SVDB_CUDA(cudaStreamSynchronize(s));
    }
    rec->origin = SVDB_REC_RANDOMIZED;
    // create_diagnostics (mod.rs:214-237)
    svdb_diagnostics& dg = rec->diagnostics;
    dg.non_zero = A->nnz;
    dg.dimensions = target_rank;
    dg.iterations = n_power_iters;
    dg.transposed = 0;
    dg.lanczos_steps = 0;
    dg.ritz_values_stabilized = actual;
    dg.significant_values = actual;
    dg.singular_values = actual;
    dg.end_interval[0] = -1e-30;
    dg.end_interval[1] = 1e-30;
    dg.kappa = 1e-6;
    dg.random_seed = (uint32_t)(has_seed ? seed : 0);
    rec->time_ms_total = tot;
    rec->time_ms_spmv = spmm_ms;
    rec->time_ms_ortho = tot - spmm_ms;
}

}  // namespace svdb

// Adjoint of the truncated SVD with respect to A's stored values, evaluated
// only at A's nonzeros (an SDDMM), and svd_flip.  The crate has no adjoint;
// svd_flip follows src/randomized/mod.rs:332-438.
//
// For A V = U S, A^T U = V S (k leading triplets) and a loss L(U, s, V):
//   dL/dA = U M V^T + Gamma V^T + U Delta^T
//   M = diag(g_s) + (F o (J_U - J_U^T)) S + S (F o (J_V - J_V^T)),
//   J_U = U^T g_U, J_V = V^T g_V, F_ij = 1/(s_j^2 - s_i^2) off the diagonal.
// The complement parts X = (I - UU^T) dU, Y = (I - VV^T) dV satisfy
//   X S - A_p Y = (I - UU^T) dA V,   Y S - A_p^T X = (I - VV^T) dA^T U
// with A_p = A - U S V^T, so their adjoint solves, column i, the same
// symmetric system with right-hand side (a_i, b_i) = ((I-UU^T) g_U e_i,
// (I-VV^T) g_V e_i):  (s_i^2 I - A_p^T A_p) delta_i = s_i b_i + A_p^T a_i,
// gamma_i = (a_i + A_p delta_i) / s_i.  s_i above the (k+1)-th singular
// value makes the matrix SPD, so the k systems run as one block CG that
// shares its sparse products.  dL/dA is then the product of the rank-2k
// factors [U M + Gamma, U] and [V, Delta], evaluated at the nonzeros.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "dense_tall.cuh"
#include "device_common.cuh"
#include "host_scratch.h"
#include "ops.cuh"
#include "svdb_internal.h"

namespace svdb {

static int grid_for_work(int64_t work, int threads, int per_sm = 8) {
    int64_t b = (work + threads - 1) / threads;
    return (int)std::max<int64_t>(1, std::min<int64_t>(b, (int64_t)device_props().sms * per_sm));
}

// ------------------------------------------------------------------ SDDMM ----
// One warp per segment of the load-balancing plan (at most kSegNnz entries of
// one row).  H = 32 / GL groups of GL lanes take every H-th entry of a
// 32-entry chunk; a lane keeps NL 16-byte vectors of the left row, GL vectors
// apart, and reads the same columns of the right rows (dense 16-byte loads).
// A batch of U entries is reduced over the group's lanes by a butterfly
// transpose (U - 1 shuffles, then log2(GL / U) for the lanes that share an
// entry), in a fixed order; the batches run one at a time so that only U rows
// are live (unrolled, the compiler hoisted their loads and spilled).
// The gathered rows through L1 and L2 bound it.  A lane per column (4-byte
// loads, a 31-shuffle transpose with two selects each over the whole warp,
// about 20 warp instructions per entry) took 313 us for 4.3 M entries of
// rank 64 at FP32.
template <typename T, int VEC>
struct alignas(sizeof(T) * VEC) SdVec { T v[VEC]; };

template <typename T, int VEC, int GL, int NL, int U, int MINB>
__global__ void __launch_bounds__(256, MINB) k_sddmm(const int32_t* __restrict__ idx, const int32_t* __restrict__ seg_row,
                                                     const int64_t* __restrict__ seg_beg,
                                                     const int64_t* __restrict__ seg_end, int64_t nseg,
                                                     const T* __restrict__ left, const T* __restrict__ right, int rank,
                                                     T* __restrict__ out) {
    constexpr int H = 32 / GL;
    static_assert(GL % U == 0, "whole batches");
    constexpr int SH = GL / U;  // lanes that end up with one entry of a batch; batches of a chunk
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, g = lane / GL, gl = lane % GL;
    const int64_t warp0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    bool active[NL];
    int col[NL];
#pragma unroll
    for (int j = 0; j < NL; ++j) {
        const int c = (j * GL + gl) * VEC;
        active[j] = c < rank;
        col[j] = active[j] ? c : 0;
    }
    for (int64_t sg = warp0; sg < nseg; sg += nwarps) {
        int32_t r = __ldg(seg_row + sg);
        if (r < 0) r = -r - 1;
        const int64_t beg = __ldg(seg_beg + sg);
        int left_n = (int)(__ldg(seg_end + sg) - beg);
        const int32_t* ip = idx + beg + lane;
        int32_t cm = lane < left_n ? __ldg(ip) : 0;
        SdVec<T, VEC> lv[NL];
#pragma unroll
        for (int j = 0; j < NL; ++j)
            lv[j] = active[j] ? *reinterpret_cast<const SdVec<T, VEC>*>(left + (int64_t)r * rank + col[j]) : SdVec<T, VEC>{};
        for (T* op = out + beg; left_n > 0; left_n -= 32, op += 32) {
            const int cnt = left_n < 32 ? left_n : 32;
            ip += 32;
            const int32_t cnext = lane + 32 < left_n ? __ldg(ip) : 0;  // the next chunk's columns
            T res = T(0);
#pragma unroll 1
            for (int b = 0; b < SH && b * U * H < cnt; ++b) {
                SdVec<T, VEC> x[U][NL];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int q = (b * U + u) * H + g;
                    const uint32_t c = (uint32_t)__shfl_sync(full, cm, q);
                    const T* row = right + (uint64_t)c * (uint32_t)rank;
#pragma unroll
                    for (int j = 0; j < NL; ++j) {
                        if (q < cnt && active[j]) x[u][j] = *reinterpret_cast<const SdVec<T, VEC>*>(row + col[j]);
                        else x[u][j] = SdVec<T, VEC>{};
                    }
                }
                T p[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    p[u] = T(0);
#pragma unroll
                    for (int j = 0; j < NL; ++j) {
                        // four columns a vector (FP32): a chain per vector, then their sum, which
                        // rounds as often as a lane per column and a tree (one chain: 6 % further off)
                        T t = VEC > 2 ? T(0) : p[u];
#pragma unroll
                        for (int e = 0; e < VEC; ++e) t = fma(lv[j].v[e], x[u][j].v[e], t);
                        p[u] = VEC > 2 && j ? p[u] + t : t;
                    }
                }
#pragma unroll
                for (int n = U / 2, w = GL / 2; w >= 1; w >>= 1, n >>= 1) {
                    if (n >= 1) {  // transpose: the upper lanes take the later entries
                        const bool upper = (gl & w) != 0;
#pragma unroll
                        for (int i = 0; i < n; ++i) {
                            const T send = upper ? p[i] : p[i + n];
                            const T keep = upper ? p[i + n] : p[i];
                            p[i] = keep + __shfl_xor_sync(full, send, w);
                        }
                    } else {
                        p[0] += __shfl_xor_sync(full, p[0], w);
                    }
                }
                if (gl % SH == b) res = p[0];
            }
            const int mine = ((gl % SH) * U + gl / SH) * H + g;
            if (mine < cnt) op[mine] = res;
            cm = cnext;
        }
    }
}

// A lane per column (rank <= 32 SLOTS), 4- or 8-byte loads, a butterfly transpose
// over the whole warp per 32 entries: for small products at ranks above 64 that
// are no whole 16-byte vectors, where the form above has too many loads a lane.
template <typename T, int SLOTS>
__global__ void __launch_bounds__(256) k_sddmm_lane(const int32_t* __restrict__ idx, const int32_t* __restrict__ seg_row,
                                                    const int64_t* __restrict__ seg_beg,
                                                    const int64_t* __restrict__ seg_end, int64_t nseg,
                                                    const T* __restrict__ left, const T* __restrict__ right, int rank,
                                                    T* __restrict__ out) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t warp0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t sg = warp0; sg < nseg; sg += nwarps) {
        int32_t r = seg_row[sg];
        if (r < 0) r = -r - 1;
        const int64_t beg = seg_beg[sg], end = seg_end[sg];
        T lv[SLOTS];
#pragma unroll
        for (int j = 0; j < SLOTS; ++j) {
            const int t = lane + 32 * j;
            lv[j] = t < rank ? left[(int64_t)r * rank + t] : T(0);
        }
        for (int64_t p0 = beg; p0 < end; p0 += 32) {
            const int cnt = (int)min((int64_t)32, end - p0);
            const int cmine = lane < cnt ? idx[p0 + lane] : 0;
            T p[32];
#pragma unroll
            for (int q = 0; q < 32; ++q) {
                const int c = __shfl_sync(full, cmine, q);
                T acc = T(0);
                if (q < cnt) {
                    const T* rr = right + (int64_t)c * rank;
#pragma unroll
                    for (int j = 0; j < SLOTS; ++j) {
                        const int t = lane + 32 * j;
                        if (t < rank) acc = fma(lv[j], __ldg(rr + t), acc);
                    }
                }
                p[q] = acc;
            }
#pragma unroll
            for (int w = 16; w >= 1; w >>= 1) {
                const bool upper = (lane & w) != 0;
#pragma unroll
                for (int i = 0; i < w; ++i) {
                    const T send = upper ? p[i] : p[i + w];
                    const T keep = upper ? p[i + w] : p[i];
                    p[i] = keep + __shfl_xor_sync(full, send, w);
                }
            }
            if (lane < cnt) out[p0 + lane] = p[0];
        }
    }
}

// out ((rl + rr) x ldo) = the rows of l, then of r (x rank), zero past column rank
template <typename T>
__global__ void k_sddmm_pad(const T* __restrict__ l, int64_t rl, const T* __restrict__ r, int64_t rr, int rank,
                            int ldo, T* __restrict__ out) {
    const int64_t n = (rl + rr) * ldo;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t q = i / ldo;
        const int c = (int)(i - q * ldo);
        out[i] = c < rank ? (q < rl ? l[q * rank + c] : r[(q - rl) * rank + c]) : T(0);
    }
}

template <typename T>
static void sddmm_launch(const DevCompressed& m, const T* left, const T* right, int rank, T* out, cudaStream_t s) {
    if (m.nnz == 0) return;
    if (rank > 256) throw Error(SVDB_ERR_UNSUPPORTED, "sddmm: rank above 256");
    constexpr int VEC = 16 / (int)sizeof(T);
    constexpr bool f32 = sizeof(T) == 4;
    const SegPlan& pl = m.plan;
    const int blocks = grid_for_work(pl.nseg * 32, 256, 24);
    int ld = (rank + VEC - 1) / VEC * VEC;
    auto go = [&](auto kern) {
        kern<<<blocks, 256, 0, s>>>(m.idx.p, pl.seg_row.p, pl.seg_beg.p, pl.seg_end.p, pl.nseg, left, right, ld, out);
    };
    // Factors whose rows are no whole 16-byte vectors are copied to rows that are
    // (one allocation, one launch: 25-40 us of a call that runs alone) where enough
    // is gathered from them; else, and where the copy cannot be allocated, they are
    // read element by element.  20,000 x 6,000, 1.06 M, FP32, alone / on three
    // streams, element by element and copied: rank 23 (2^24.5) 49 / 28 and 61 / 25 us,
    // rank 37 (2^25.2) 80 / 49 and 79 / 29, rank 63 (2^26) 85 / 52 and 81 / 29.
    auto fits = [&](const T* x) { return ld == rank && reinterpret_cast<uintptr_t>(x) % 16 == 0; };
    const int64_t lrows = fits(left) ? 0 : m.nmajor, rrows = fits(right) ? 0 : m.nminor;
    DevBuf<T> buf;
    if (lrows + rrows) {
        bool copied = m.nnz * rank > ((int64_t)1 << 25) && m.nnz > 4 * (lrows + rrows);
        if (copied) {
            try {
                buf.alloc((lrows + rrows) * ld, s);
            } catch (const Error& e) {
                if (e.code != SVDB_ERR_OOM) throw;
                cudaGetLastError();
                copied = false;
            }
        }
        if (!copied) {
            ld = rank;
            if (rank <= 4) go(k_sddmm<T, 1, 4, 1, 4, 4>);
            else if (rank <= 8) go(k_sddmm<T, 1, 8, 1, 8, 4>);
            else if (rank <= 16) go(k_sddmm<T, 1, 8, 2, f32 ? 2 : 8, f32 ? 6 : 4>);
            else if (rank <= 32) go(k_sddmm<T, 1, 8, 4, 2, 4>);
            else if (rank <= 64) go(k_sddmm<T, 1, 16, 4, 2, 4>);
            else if (rank <= 96) go(k_sddmm_lane<T, 3>);
            else if (rank <= 128) go(k_sddmm_lane<T, 4>);
            else if (rank <= 192) go(k_sddmm_lane<T, 6>);
            else go(k_sddmm_lane<T, 8>);
            SVDB_CHECK_LAUNCH();
            return;
        }
        k_sddmm_pad<T><<<grid_for_work((lrows + rrows) * ld, 256, 16), 256, 0, s>>>(left, lrows, right, rrows, rank, ld,
                                                                                    buf.p);
        SVDB_CHECK_LAUNCH();
        if (lrows) left = buf.p;
        if (rrows) right = buf.p + lrows * ld;
    }
    // At least 64 contiguous bytes per load, two vectors per lane before the
    // group widens, and as many warps as the registers allow: warps count more
    // than entries in flight per warp (5.4 M entries, rank 64, FP32: 126 us with
    // two entries and six CTAs per SM, 144-174 with eight and two or three;
    // FP64: 240 us with four entries and four CTAs, 291 with (8, 4, 2) and three).
    const int nv = ld / VEC;  // vectors per row
    if (nv <= 4) go(k_sddmm<T, VEC, 4, 1, 4, 4>);
    else if (nv <= 8) go(k_sddmm<T, VEC, 8, 1, 8, 4>);
    else if (nv <= 16) go(k_sddmm<T, VEC, 8, 2, 2, 6>);
    else if (nv <= 24) go(k_sddmm<T, VEC, 8, 3, 2, 4>);
    else if (nv <= 32) go(k_sddmm<T, VEC, 16, 2, 4, 4>);
    else if (nv <= 64) go(k_sddmm<T, VEC, 32, 2, 4, 4>);
    else go(k_sddmm<T, VEC, 32, 4, 2, 3>);
    SVDB_CHECK_LAUNCH();
}

// The handle's own entry order: CSR handles use the CSR (rows of A, factors
// left = row side), CSC handles their CSC (rows of A^T, factors swapped).
static const DevCompressed& pattern_of(const svdb_matrix* a, bool& swapped) {
    if (a->kind == KIND_CSR) { swapped = false; return a->csr; }
    if (a->kind == KIND_CSC) { swapped = true; return a->csc; }
    throw Error(SVDB_ERR_UNSUPPORTED, "adjoint: COO handles and masked views have no stored entry order to return");
}

// ------------------------------------------------------- tall-skinny dense ----
// column of flat index t of a k-column matrix (32-bit division where it fits)
__device__ __forceinline__ int col_of(int64_t t, int k) {
    return t < ((int64_t)1 << 32) ? (int)((uint32_t)t % (uint32_t)k) : (int)(t % k);
}

// Out[r][j] = ca[j] A[r][j] + sb cb[j] B[r][j]; ca / cb null mean 1, B null
// drops the second term.  Out may alias A or B.
__global__ void k_axpby_cols(int64_t rows, int k, double* Out, int64_t ldo, const double* A, int64_t lda,
                             const double* __restrict__ ca, const double* B, int64_t ldb,
                             const double* __restrict__ cb, double sb) {
    const int64_t total = rows * k;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int j = col_of(t, k);
        const int64_t r = t < ((int64_t)1 << 32) ? (int64_t)((uint32_t)t / (uint32_t)k) : t / k;
        double v = A[r * lda + j] * (ca ? ca[j] : 1.0);
        if (B) v += sb * (cb ? cb[j] : 1.0) * B[r * ldb + j];
        Out[r * ldo + j] = v;
    }
}

// X += P diag(alpha), R -= W diag(alpha), one pass
__global__ void k_cg_step(int64_t rows, int k, double* __restrict__ X, const double* __restrict__ P,
                          double* __restrict__ R, const double* __restrict__ W, const double* __restrict__ alpha) {
    const int64_t total = rows * k;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const double al = alpha[col_of(t, k)];
        X[t] += al * P[t];
        R[t] += -1.0 * al * W[t];
    }
}

// The column sums `tot` of the CTAs' partials dots (nb x k), one warp per
// column in a fixed order, then the CG scalars of the column.  A column is
// frozen (alpha = beta = 0) once its residual norm is below freeze * ||rhs||,
// or when a denominator is not positive.
//   CG_INIT   rr = tot
//   CG_ALPHA  alpha = rr / tot (tot = p . w)
//   CG_BETA   beta = tot / rr, rr = tot (tot = r . r)
enum { CG_INIT, CG_ALPHA, CG_BETA };
template <int WHAT>
__global__ void k_cg_scalars(const double* __restrict__ dots, int nb, int k, double* __restrict__ rr,
                             const double* __restrict__ rhs_norm, double freeze, double* __restrict__ alpha,
                             double* __restrict__ beta) {
    const int lane = threadIdx.x & 31, nw = (int)((gridDim.x * blockDim.x) >> 5);
    for (int j = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); j < k; j += nw) {
        double tot = 0.0;
        for (int b = lane; b < nb; b += 32) tot += dots[(int64_t)b * k + j];
        tot = warp_sum(tot);
        if (lane) continue;
        if (WHAT == CG_INIT) {
            rr[j] = tot;
        } else if (WHAT == CG_ALPHA) {
            const bool live = rr[j] > 0.0 && tot > 0.0 && sqrt(rr[j]) > freeze * rhs_norm[j];
            alpha[j] = live ? rr[j] / tot : 0.0;
        } else {
            beta[j] = (alpha[j] != 0.0 && rr[j] > 0.0) ? tot / rr[j] : 0.0;
            rr[j] = tot;
        }
    }
}

// The tall products of an iteration go through dense_tall.cuh (FP64 matrix
// instruction).  What it measured on 50,000 x 20,000, k = 32, per launch
// before and after: X^T Y 25-37 -> 8-12 us, the sum of its partials 75 -> 5 us
// (eight blocks of one thread per element, held by load latency), X C 25 ->
// 13-18 us; the k x k Grams formed for their diagonals became column sums in
// the products' epilogues.  Adjoint 37.7 -> 22.2 ms.
struct TallCtx {
    cudaStream_t s;
    DevBuf<double> part, dots;
    int nb = 0;  // CTAs that wrote dots
};

// C (p x q) = X^T Y, X: rows x p (ld ldx), Y: rows x q (ld ldy)
static void atb(TallCtx& cx, const double* X, int64_t ldx, const double* Y, int64_t ldy, int64_t rows, int p, int q,
                double* C) {
    if (std::max(p, q) > 128) throw Error(SVDB_ERR_UNSUPPORTED, "adjoint: more than 128 triplets");
    const TnShape h = tn_shape(rows, p, q, false, device_props().sms);
    if ((int64_t)cx.part.n < (int64_t)h.blocks * p * q) cx.part.alloc((size_t)h.blocks * p * q, cx.s);
    tn_launch(h, X, ldx, p, Y, ldy, q, rows, cx.part.p, C, nullptr, cx.s);
}

// Out (rows x q, ld ldo) = beta * Y + alpha * X diag(d) C + E diag(es), X: rows x p
// (ld ldx), C: p x q row-major, d: p values or null (= 1), Y / E null: no such
// term.  Out may be Y.  DOT 1 / 2: the column sums of Out * Out / Out * E are
// left as cx.nb partials in cx.dots.
template <int DOT = 0>
static void gemm_tall(TallCtx& cx, const double* X, int64_t ldx, int64_t rows, int p, const double* C, const double* d,
                      int q, double alpha, const double* Y, int64_t ldy, double beta, double* Out, int64_t ldo,
                      const double* E = nullptr, int64_t lde = 0, const double* es = nullptr) {
    const int sms = device_props().sms;
    if (DOT) {
        cx.nb = nn_blocks(rows, sms);
        if ((int64_t)cx.dots.n < (int64_t)cx.nb * q) cx.dots.alloc((size_t)cx.nb * q, cx.s);
    }
    nn_launch<DOT>(NnArgs<double, double>{X, ldx, rows, p, C, q, d, q, 0, alpha, beta != 0.0 ? Y : nullptr, ldy, beta,
                                          E, lde, es, Out, ldo, 0, cx.dots.p, nullptr},
                   sms, cx.s);
}

template <int WHAT>
static void cg_scalars(TallCtx& cx, int k, double* rr, const double* rhs_norm, double freeze, double* alpha,
                       double* beta) {
    k_cg_scalars<WHAT><<<(k + 7) / 8, 256, 0, cx.s>>>(cx.dots.p, cx.nb, k, rr, rhs_norm, freeze, alpha, beta);
    SVDB_CHECK_LAUNCH();
}

static void axpby_cols(int64_t rows, int k, double* Out, int64_t ldo, const double* A, int64_t lda, const double* ca,
                       const double* B, int64_t ldb, const double* cb, double sb, cudaStream_t s) {
    if (rows * k == 0) return;
    k_axpby_cols<<<grid_for_work(rows * k, 256), 256, 0, s>>>(rows, k, Out, ldo, A, lda, ca, B, ldb, cb, sb);
    SVDB_CHECK_LAUNCH();
}

__global__ void k_to_f32_adj(const double* __restrict__ in, float* __restrict__ out, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (float)in[i];
}
__global__ void k_to_f64_adj(const float* __restrict__ in, double* __restrict__ out, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (double)in[i];
}

// ---------------------------------------------------------------- adjoint ----
void svd_adjoint(const svdb_matrix* A, int64_t k, const double* u, const double* s_in, const double* v,
                 const double* g_u, const double* g_s, const double* g_v, svdb_adjoint_options& o,
                 double* grad_values) {
    bool swapped = false;
    const DevCompressed& pat = pattern_of(A, swapped);
    cudaStream_t s = o.stream ? (cudaStream_t)o.stream : A->stream;
    const int64_t m = A->nrows, n = A->ncols, nnz = pat.nnz;
    const bool dev = o.inputs_on_device != 0;
    if (k < 0 || k > std::min<int64_t>(128, std::min(m, n)))
        throw Error(SVDB_ERR_UNSUPPORTED, "adjoint: k must be at most min(nrows, ncols, 128)");
    if (!grad_values || (k > 0 && (!u || !s_in || !v))) throw Error(SVDB_ERR_ARG, "null argument");
    o.cg_iterations = 0;
    o.cg_residual = 0.0;
    o.time_ms_solve = o.time_ms_sddmm = 0.0;
    if (k == 0 || nnz == 0) {
        if (dev) SVDB_CUDA(cudaMemsetAsync(grad_values, 0, std::max<int64_t>(nnz, 0) * 8, s));
        else std::memset(grad_values, 0, std::max<int64_t>(nnz, 0) * 8);
        if (dev) SVDB_CUDA(cudaStreamSynchronize(s));
        return;
    }
    const int kk = (int)k;
    // host copies of s and g_s (the k x k algebra runs on the host)
    std::vector<double> sv(k), gs(k, 0.0);
    if (dev) {
        SVDB_CUDA(cudaMemcpyAsync(sv.data(), s_in, k * 8, cudaMemcpyDeviceToHost, s));
        if (g_s) SVDB_CUDA(cudaMemcpyAsync(gs.data(), g_s, k * 8, cudaMemcpyDeviceToHost, s));
        SVDB_CUDA(cudaStreamSynchronize(s));
    } else {
        std::memcpy(sv.data(), s_in, k * 8);
        if (g_s) std::memcpy(gs.data(), g_s, k * 8);
    }
    for (int i = 0; i < kk; ++i)
        if (!(sv[i] > 0.0) || !std::isfinite(sv[i]))
            throw Error(SVDB_ERR_ARG, "adjoint: singular values must be positive and finite");

    ScopedEvent e0, e1, e2;
    SVDB_CUDA(cudaEventRecord(e0, s));

    DevBuf<double> U(m * k, s), V(n * k, s), GU(m * k, s), GV(n * k, s);
    auto load = [&](DevBuf<double>& dst, const double* src, int64_t cnt) {
        if (!src) { SVDB_CUDA(cudaMemsetAsync(dst.p, 0, cnt * 8, s)); return; }
        SVDB_CUDA(cudaMemcpyAsync(dst.p, src, cnt * 8, dev ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, s));
    };
    load(U, u, m * k);
    load(V, v, n * k);
    load(GU, g_u, m * k);
    load(GV, g_v, n * k);

    TallCtx cx;
    cx.s = s;
    DevBuf<double> kkbuf(4 * k * k, s);
    double* JU = kkbuf.p;
    double* JV = kkbuf.p + k * k;
    double* C1 = kkbuf.p + 2 * k * k;
    double* C2 = kkbuf.p + 3 * k * k;
    atb(cx, U.p, k, GU.p, k, m, kk, kk, JU);
    atb(cx, V.p, k, GV.p, k, n, kk, kk, JV);
    std::vector<double> hJ(2 * k * k);
    SVDB_CUDA(cudaMemcpyAsync(hJ.data(), JU, 2 * k * k * 8, cudaMemcpyDeviceToHost, s));

    // per-column vectors on the device: s, s^2, 1/s and CG scalars
    DevBuf<double> colv(7 * k, s);
    double* d_s = colv.p;
    double* d_s2 = colv.p + k;
    double* d_si = colv.p + 2 * k;
    double* d_rr = colv.p + 3 * k;
    double* d_al = colv.p + 4 * k;
    double* d_be = colv.p + 5 * k;
    double* d_rhsn = colv.p + 6 * k;
    std::vector<double> hcol(3 * k);
    for (int i = 0; i < kk; ++i) {
        hcol[i] = sv[i];
        hcol[k + i] = sv[i] * sv[i];
        hcol[2 * k + i] = 1.0 / sv[i];
    }
    SVDB_CUDA(cudaMemcpyAsync(colv.p, hcol.data(), 3 * k * 8, cudaMemcpyHostToDevice, s));

    // a = (I - U U^T) g_U,  b = (I - V V^T) g_V
    DevBuf<double> Aa(m * k, s), Bb(n * k, s);
    gemm_tall(cx, U.p, k, m, kk, JU, nullptr, kk, -1.0, GU.p, k, 1.0, Aa.p, k);
    gemm_tall(cx, V.p, k, n, kk, JV, nullptr, kk, -1.0, GV.p, k, 1.0, Bb.p, k);

    const DevCompressed& Ar = csr_of(A);  // rows of A
    const DevCompressed& Ac = csc_of(A);  // rows of A^T
    // rhs = b diag(s) + (I - V V^T) A^T a
    DevBuf<double> Rhs(n * k, s), Z(n * k, s), T(m * k, s);
    spmm_dev<double, double>(Ac, false, Aa.p, kk, Z.p, s);
    atb(cx, V.p, k, Z.p, k, n, kk, kk, C1);
    gemm_tall(cx, V.p, k, n, kk, C1, nullptr, kk, -1.0, Z.p, k, 1.0, Rhs.p, k, Bb.p, k, d_s);

    // block CG on S^2 - A_p^T A_p: X = 0, R = P = rhs
    DevBuf<double> X(n * k, s), R(n * k, s), P(n * k, s), W(n * k, s);
    SVDB_CUDA(cudaMemsetAsync(X.p, 0, n * k * 8, s));
    SVDB_CUDA(cudaMemcpyAsync(R.p, Rhs.p, n * k * 8, cudaMemcpyDeviceToDevice, s));
    SVDB_CUDA(cudaMemcpyAsync(P.p, Rhs.p, n * k * 8, cudaMemcpyDeviceToDevice, s));
    // page-locked: the residual's copy does not hold the host, which enqueues on
    HostScratch hrr(64 << 10, s);
    double* rr = (double*)hrr.p;
    // column norms of rhs as the dots of R with itself (C1 = 0: the product adds nothing)
    SVDB_CUDA(cudaMemsetAsync(C1, 0, k * k * 8, s));
    gemm_tall<1>(cx, V.p, k, n, kk, C1, nullptr, kk, 0.0, R.p, k, 1.0, W.p, k);
    cg_scalars<CG_INIT>(cx, kk, d_rr, nullptr, 0.0, nullptr, nullptr);
    std::vector<double> rhs_norm(k);
    SVDB_CUDA(cudaMemcpyAsync(rr, d_rr, k * 8, cudaMemcpyDeviceToHost, s));
    SVDB_CUDA(cudaStreamSynchronize(s));
    for (int j = 0; j < kk; ++j) rhs_norm[j] = std::sqrt(rr[j]);
    SVDB_CUDA(cudaMemcpyAsync(d_rhsn, rhs_norm.data(), k * 8, cudaMemcpyHostToDevice, s));
    const double tol = o.cg_tol > 0.0 ? o.cg_tol : 1e-12;
    const uint64_t max_it = o.cg_max_iters ? o.cg_max_iters : 5000;
    auto residual = [&]() {
        double worst = 0.0;
        for (int j = 0; j < kk; ++j)
            if (rhs_norm[j] > 0.0) worst = std::max(worst, std::sqrt(std::max(rr[j], 0.0)) / rhs_norm[j]);
        return worst;
    };
    double res = residual();
    uint64_t it = 0;
    ScopedEvent got(cudaEventDisableTiming);  // the residual's copy
    if (res > tol && it < max_it) spmm_dev<double, double>(Ar, false, P.p, kk, T.p, s);  // T = A P
    while (res > tol && it < max_it) {
        atb(cx, V.p, k, P.p, k, n, kk, kk, C1);                                           // C1 = V^T P
        gemm_tall(cx, U.p, k, m, kk, C1, d_s, kk, -1.0, T.p, k, 1.0, T.p, k);             // T -= U S C1
        spmm_dev<double, double>(Ac, false, T.p, kk, Z.p, s);                             // Z = A^T T
        atb(cx, U.p, k, T.p, k, m, kk, kk, C2);                                           // C2 = U^T T
        // W = P S^2 - (Z - V S C2), with the sums of P * W
        gemm_tall<2>(cx, V.p, k, n, kk, C2, d_s, kk, 1.0, Z.p, k, -1.0, W.p, k, P.p, k, d_s2);
        cg_scalars<CG_ALPHA>(cx, kk, d_rr, d_rhsn, 0.25 * tol, d_al, nullptr);
        k_cg_step<<<grid_for_work(n * k, 256), 256, 0, s>>>(n, kk, X.p, P.p, R.p, W.p, d_al);
        SVDB_CHECK_LAUNCH();
        atb(cx, V.p, k, R.p, k, n, kk, kk, C2);                                           // keep R off span(V)
        gemm_tall<1>(cx, V.p, k, n, kk, C2, nullptr, kk, -1.0, R.p, k, 1.0, R.p, k);
        cg_scalars<CG_BETA>(cx, kk, d_rr, nullptr, 0.0, d_al, d_be);
        axpby_cols(n, kk, P.p, k, R.p, k, nullptr, P.p, k, d_be, 1.0, s);                 // P = R + P beta
        SVDB_CUDA(cudaMemcpyAsync(rr, d_rr, k * 8, cudaMemcpyDeviceToHost, s));
        SVDB_CUDA(cudaEventRecord(got, s));
        // the next iteration's first product (of the last one after the end:
        // T = A X below overwrites it) runs while the host looks at the residual
        spmm_dev<double, double>(Ar, false, P.p, kk, T.p, s);
        SVDB_CUDA(cudaEventSynchronize(got));
        ++it;
        res = residual();
    }
    o.cg_iterations = it;
    o.cg_residual = res;

    // Gamma = (a + A_p Delta) diag(1/s), Delta = X
    DevBuf<double> Gm(m * k, s);
    spmm_dev<double, double>(Ar, false, X.p, kk, T.p, s);
    atb(cx, V.p, k, X.p, k, n, kk, kk, C1);
    gemm_tall(cx, U.p, k, m, kk, C1, d_s, kk, -1.0, T.p, k, 1.0, T.p, k);
    atb(cx, U.p, k, T.p, k, m, kk, kk, C2);  // A_p Delta lies off span(U): drop the rounding residue
    gemm_tall(cx, U.p, k, m, kk, C2, nullptr, kk, -1.0, T.p, k, 1.0, T.p, k);
    axpby_cols(m, kk, Gm.p, k, Aa.p, k, d_si, T.p, k, d_si, 1.0, s);

    // M on the host
    std::vector<double> M(k * k, 0.0);
    {
        const double* hJU = hJ.data();
        const double* hJV = hJ.data() + k * k;
        for (int i = 0; i < kk; ++i)
            for (int j = 0; j < kk; ++j) {
                if (i == j) { M[i * k + j] = gs[i]; continue; }
                const double den = sv[j] * sv[j] - sv[i] * sv[i];
                const double f = std::fabs(den) > 1e-300 ? 1.0 / den : 0.0;
                const double au = hJU[i * k + j] - hJU[j * k + i];
                const double avv = hJV[i * k + j] - hJV[j * k + i];
                M[i * k + j] = f * au * sv[j] + sv[i] * f * avv;
            }
    }
    DevBuf<double> dM(k * k, s);
    SVDB_CUDA(cudaMemcpyAsync(dM.p, M.data(), k * k * 8, cudaMemcpyHostToDevice, s));

    // factors: Lf = [U M + Gamma | U] (m x 2k), Rf = [V | Delta] (n x 2k)
    const int rank = 2 * kk;
    DevBuf<double> Lf(m * rank, s), Rf(n * rank, s);
    gemm_tall(cx, U.p, k, m, kk, dM.p, nullptr, kk, 1.0, Gm.p, k, 1.0, Lf.p, rank);
    axpby_cols(m, kk, Lf.p + k, rank, U.p, k, nullptr, nullptr, 0, nullptr, 0.0, s);
    axpby_cols(n, kk, Rf.p, rank, V.p, k, nullptr, nullptr, 0, nullptr, 0.0, s);
    axpby_cols(n, kk, Rf.p + k, rank, X.p, k, nullptr, nullptr, 0, nullptr, 0.0, s);
    SVDB_CUDA(cudaEventRecord(e1, s));

    const double* left = swapped ? Rf.p : Lf.p;
    const double* right = swapped ? Lf.p : Rf.p;
    DevBuf<double> out_dev;
    double* out = grad_values;
    if (!dev) {
        out_dev.alloc(nnz, s);
        out = out_dev.p;
    }
    if (o.precision == SVDB_MIXED) {
        const int64_t nl = (swapped ? n : m) * rank, nr = (swapped ? m : n) * rank;
        DevBuf<float> l32(nl, s), r32(nr, s), o32(nnz, s);
        k_to_f32_adj<<<grid_for_work(nl, 256), 256, 0, s>>>(left, l32.p, nl);
        k_to_f32_adj<<<grid_for_work(nr, 256), 256, 0, s>>>(right, r32.p, nr);
        SVDB_CHECK_LAUNCH_N(2);
        sddmm_launch<float>(pat, l32.p, r32.p, rank, o32.p, s);
        k_to_f64_adj<<<grid_for_work(nnz, 256), 256, 0, s>>>(o32.p, out, nnz);
        SVDB_CHECK_LAUNCH();
    } else {
        sddmm_launch<double>(pat, left, right, rank, out, s);
    }
    SVDB_CUDA(cudaEventRecord(e2, s));
    if (!dev) SVDB_CUDA(cudaMemcpyAsync(grad_values, out, nnz * 8, cudaMemcpyDeviceToHost, s));
    SVDB_CUDA(cudaStreamSynchronize(s));
    float t1 = 0.f, t2 = 0.f;
    cudaEventElapsedTime(&t1, e0, e1);
    cudaEventElapsedTime(&t2, e1, e2);
    o.time_ms_solve = t1;
    o.time_ms_sddmm = t2;
    if (res > tol)
        throw Error(SVDB_ERR_NOCONV, "adjoint: block CG stopped at relative residual " + std::to_string(res) +
                                         " after " + std::to_string(it) + " iterations");
}

void sddmm_device(const svdb_matrix* A, const void* left, const void* right, int64_t rank, void* out, int precision,
                  cudaStream_t s) {
    bool swapped = false;
    const DevCompressed& pat = pattern_of(A, swapped);
    if (rank <= 0 || rank > 256) throw Error(SVDB_ERR_UNSUPPORTED, "sddmm: rank must be in 1..256");
    const void* l = swapped ? right : left;
    const void* r = swapped ? left : right;
    if (precision == SVDB_MIXED)
        sddmm_launch<float>(pat, (const float*)l, (const float*)r, (int)rank, (float*)out, s);
    else
        sddmm_launch<double>(pat, (const double*)l, (const double*)r, (int)rank, (double*)out, s);
}

// --------------------------------------------------------------- svd_flip ----
// sign[v] for vector v of X (rows x cols row-major): column v (by_row = 0) or
// row v (by_row = 1).  The deciding entry is the first one of largest
// magnitude (a strict > scan, as mod.rs:357-365 / :405-413); an all-zero
// vector decides by its entry 0.
__global__ void k_flip_signs(const double* __restrict__ X, int64_t rows, int64_t cols, int by_row,
                             double* __restrict__ sign) {
    __shared__ double sa[256];
    __shared__ int64_t si[256];
    const int64_t v = blockIdx.x;
    const int64_t len = by_row ? cols : rows;
    double best = 0.0;
    int64_t bi = INT64_MAX;
    for (int64_t i = threadIdx.x; i < len; i += blockDim.x) {
        const double a = fabs(by_row ? X[v * cols + i] : X[i * cols + v]);
        if (a > best) { best = a; bi = i; }
    }
    sa[threadIdx.x] = best;
    si[threadIdx.x] = bi;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            const double a2 = sa[threadIdx.x + w];
            const int64_t i2 = si[threadIdx.x + w];
            if (a2 > sa[threadIdx.x] || (a2 == sa[threadIdx.x] && i2 < si[threadIdx.x])) {
                sa[threadIdx.x] = a2;
                si[threadIdx.x] = i2;
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const int64_t i = si[0] == INT64_MAX ? 0 : si[0];
        const double x = len ? (by_row ? X[v * cols + i] : X[i * cols + v]) : 0.0;
        sign[v] = x < 0.0 ? -1.0 : 1.0;
    }
}
// X (rows x cols): by_row = 0 scales column j by sign[j] (j < nsign), 1 scales row i.
__global__ void k_apply_signs(double* __restrict__ X, int64_t rows, int64_t cols, int by_row,
                              const double* __restrict__ sign, int64_t nsign) {
    const int64_t total = rows * cols;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t which = by_row ? t / cols : t % cols;
        if (which < nsign) X[t] *= sign[which];
    }
}

void svd_flip(double* u, int64_t u_rows, int64_t u_cols, double* v, int64_t v_rows, int64_t v_cols, bool u_based,
              bool on_device) {
    if (!u && !v) throw Error(SVDB_ERR_LAS2, "Both u and v cannot be None");
    if (u_based && !u) throw Error(SVDB_ERR_LAS2, "u cannot be None when u_based_decision is true");
    if (!u_based && !v) throw Error(SVDB_ERR_LAS2, "v cannot be None when u_based_decision is false");
    cudaStream_t s = 0;
    const int64_t nu = u ? u_rows * u_cols : 0, nv = v ? v_rows * v_cols : 0;
    DevBuf<double> du, dv;
    double* pu = u;
    double* pv = v;
    if (!on_device) {
        if (u) {
            du.alloc(std::max<int64_t>(nu, 1), s);
            if (nu) SVDB_CUDA(cudaMemcpyAsync(du.p, u, nu * 8, cudaMemcpyHostToDevice, s));
            pu = du.p;
        }
        if (v) {
            dv.alloc(std::max<int64_t>(nv, 1), s);
            if (nv) SVDB_CUDA(cudaMemcpyAsync(dv.p, v, nv * 8, cudaMemcpyHostToDevice, s));
            pv = dv.p;
        }
    }
    const int64_t nsign = u_based ? u_cols : v_rows;
    DevBuf<double> sign(std::max<int64_t>(nsign, 1), s);
    if (nsign > 0) {
        if (u_based) k_flip_signs<<<(unsigned)nsign, 256, 0, s>>>(pu, u_rows, u_cols, 0, sign.p);
        else k_flip_signs<<<(unsigned)nsign, 256, 0, s>>>(pv, v_rows, v_cols, 1, sign.p);
        SVDB_CHECK_LAUNCH();
        if (pu && nu) {
            k_apply_signs<<<grid_for_work(nu, 256), 256, 0, s>>>(pu, u_rows, u_cols, 0, sign.p,
                                                                 u_based ? u_cols : std::min(u_cols, v_rows));
            SVDB_CHECK_LAUNCH();
        }
        if (pv && nv) {
            k_apply_signs<<<grid_for_work(nv, 256), 256, 0, s>>>(pv, v_rows, v_cols, 1, sign.p,
                                                                 u_based ? std::min(v_rows, u_cols) : v_rows);
            SVDB_CHECK_LAUNCH();
        }
    }
    if (!on_device) {
        if (u && nu) SVDB_CUDA(cudaMemcpyAsync(u, du.p, nu * 8, cudaMemcpyDeviceToHost, s));
        if (v && nv) SVDB_CUDA(cudaMemcpyAsync(v, dv.p, nv * 8, cudaMemcpyDeviceToHost, s));
    }
    SVDB_CUDA(cudaStreamSynchronize(s));
}

}  // namespace svdb

// Tall-skinny FP64 products on the FP64 matrix instruction (mma.sync
// m8n8k4.f64): C = X^T Y (k_tn_part + k_tn_reduce) and Out = alpha X C + ...
// (k_nn).  X and Y have many rows and at most 128 columns.
//
// Why this instruction: one m8n8k4 is 256 fused multiply-adds whose operands
// are one double per lane, so a warp with a 32 x 32 tile of C issues 8 loads
// for 16 of them.  A 4 x 4 register tile per thread (DFMA) reads 8 shared
// doubles for 16 FMAs and is held by shared memory and issue slots instead of
// the FP64 units.  Measured on B200: 18.5 T FMA/s with eight warps per SM
// (DFMA: 17.0), 27 cycles of latency.  Sums stay FP64.
// Against register-tile kernels staged through shared memory, c = 60:
// X^T X of 100,000 rows 90 -> 35 us, of 30,000 rows 38 -> 20 us; X R^-1 72 ->
// 44 us and 36 -> 25 us (ncu, cold caches).
//
// Fragments (lane l): A (8 x 4) holds [l / 4][l % 4], B (4 x 8) holds
// [l % 4][l / 4], C (8 x 8) holds [l / 4][2 (l % 4) + {0, 1}].  For X^T Y both
// fragments are X[r + l % 4][col0 + l / 4]: four rows of 64 contiguous bytes,
// read straight from global memory with no staging.
#pragma once

#include <algorithm>
#include <cstdint>

#include "svdb_internal.h"

namespace svdb {

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// ------------------------------------------------------------- X^T Y ----
// A warp owns one tile block of C, NT x NT fragments (NT <= 4: 32 accumulator
// doubles per lane), and every rg-th group of four rows of its CTA's chunk;
// the rg copies are added in order in shared memory, the CTAs' partials by
// k_tn_reduce, also in order.  sym (X = Y): only tile blocks I <= J.
struct TnShape {
    int nt = 1, nbp = 1, nbq = 1, ntb = 1, rg = 1, blocks = 1;
    bool sym = false;
    int64_t chunk = 0;
    int threads() const { return 32 * ntb * rg; }
    size_t smem() const { return (size_t)ntb * rg * nt * nt * 64 * sizeof(double); }
};
inline size_t tn_smem_max(int nt) { return (size_t)16 * nt * nt * 64 * sizeof(double); }  // sixteen warps
// `ctas` CTAs at most.  One CTA of up to 16 warps per SM: 148 partials to add
// instead of the 296 of two smaller CTAs.
__host__ __device__ inline TnShape tn_shape(int64_t rows, int p, int q, bool sym, int ctas) {
    TnShape h;
    h.sym = sym;
    const int tiles = (std::max(p, q) + 7) / 8;
    const int nb = (tiles + 3) / 4;
    h.nt = (tiles + nb - 1) / nb;
    h.nbp = ((p + 7) / 8 + h.nt - 1) / h.nt;
    h.nbq = ((q + 7) / 8 + h.nt - 1) / h.nt;
    h.ntb = sym ? h.nbp * (h.nbp + 1) / 2 : h.nbp * h.nbq;
    h.rg = std::max(1, 16 / h.ntb);
    const int64_t step = 4 * h.rg;  // rows per round of the CTA's warps
    h.chunk = std::max<int64_t>(1, (rows + ctas * step - 1) / (ctas * step)) * step;
    h.blocks = (int)std::max<int64_t>(1, (rows + h.chunk - 1) / h.chunk);
    return h;
}

__device__ __forceinline__ void tn_block_of(int tb, int nbp, int nbq, bool sym, int& I, int& J) {
    if (!sym) {
        I = tb / nbq;
        J = tb - I * nbq;
        return;
    }
    I = 0;
    while (tb >= nbp - I) { tb -= nbp - I; ++I; }
    J = I + tb;
}

// One CTA's partial of X^T Y over rows [r0, r1) into out (p x q row-major;
// sym: only its tile blocks I <= J).  sm: TnShape::smem() bytes.
template <typename TX, typename TY, int NT>
__device__ __forceinline__ void tn_part_body(const TX* __restrict__ X, int64_t ldx, int p, const TY* __restrict__ Y,
                                             int64_t ldy, int q, int64_t r0, int64_t r1, int nbp, int nbq, bool sym,
                                             int rg, double* __restrict__ out, double* sm) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ntb = (blockDim.x >> 5) / rg;
    const int tb = warp % ntb, g = warp / ntb;
    int I, J;
    tn_block_of(tb, nbp, nbq, sym, I, J);
    const bool diag = sym && I == J;
    const int kl = lane & 3, il = lane >> 2;
    const int ca = I * NT * 8 + il, cb = J * NT * 8 + il;
    double acc[NT][NT][2];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    // KS groups of four rows per step; the next step's loads are in flight during
    // this one's products (NT = 4: the accumulators leave registers for one group)
    constexpr int KS = NT <= 3 ? 2 : 1;
    TX a[KS][NT];  // converted when used: a conversion beside its load would wait for it
    TY b[KS][NT];
    auto load = [&](int64_t r, TX (&fa)[KS][NT], TY (&fb)[KS][NT]) {
#pragma unroll
        for (int k = 0; k < KS; ++k) {
            const int64_t row = r + (int64_t)k * 4 * rg + kl;
            const bool rok = row < r1;
            const TX* px = X + row * ldx + ca;
            const TY* py = Y + row * ldy + cb;
#pragma unroll
            for (int t = 0; t < NT; ++t) fa[k][t] = (rok && ca + 8 * t < p) ? px[8 * t] : TX(0);
            if (!diag) {
#pragma unroll
                for (int t = 0; t < NT; ++t) fb[k][t] = (rok && cb + 8 * t < q) ? py[8 * t] : TY(0);
            }
        }
    };
    int64_t r = r0 + 4 * g;
    if (r < r1) load(r, a, b);
    for (; r < r1; r += (int64_t)KS * 4 * rg) {
        TX na[KS][NT];
        TY nb[KS][NT];
        if (r + (int64_t)KS * 4 * rg < r1) load(r + (int64_t)KS * 4 * rg, na, nb);
#pragma unroll
        for (int k = 0; k < KS; ++k) {
            double da[NT], db[NT];
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                da[t] = (double)a[k][t];
                db[t] = diag ? da[t] : (double)b[k][t];
            }
#pragma unroll
            for (int i = 0; i < NT; ++i)
#pragma unroll
                for (int j = 0; j < NT; ++j) dmma(acc[i][j], da[i], db[j]);
        }
#pragma unroll
        for (int k = 0; k < KS; ++k)
#pragma unroll
            for (int t = 0; t < NT; ++t) { a[k][t] = na[k][t]; b[k][t] = nb[k][t]; }
    }
    constexpr int W = NT * 8;
    double* mine = sm + (size_t)warp * W * W;
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            double* o = mine + (i * 8 + il) * W + j * 8 + 2 * kl;
            o[0] = acc[i][j][0];
            o[1] = acc[i][j][1];
        }
    __syncthreads();
    for (int t = threadIdx.x; t < ntb * W * W; t += blockDim.x) {
        const int bq = t / (W * W), e = t - bq * W * W;
        double s = 0.0;
        for (int gg = 0; gg < rg; ++gg) s += sm[(size_t)(gg * ntb + bq) * W * W + e];
        int bi, bj;
        tn_block_of(bq, nbp, nbq, sym, bi, bj);
        const int row = bi * W + e / W, col = bj * W + e % W;
        if (row < p && col < q) out[(int64_t)row * q + col] = s;
    }
}

template <typename TX, typename TY, int NT>
__global__ void __launch_bounds__(512, 1) k_tn_part(const TX* __restrict__ X, int64_t ldx, int p,
                                                    const TY* __restrict__ Y, int64_t ldy, int q, int64_t rows,
                                                    int64_t chunk, int nbp, int nbq, int sym, int rg,
                                                    double* __restrict__ part, const int* __restrict__ cond) {
    if (cond && *cond == 0) return;
    extern __shared__ __align__(16) double tn_sm[];
    const int64_t r0 = blockIdx.x * chunk;
    tn_part_body<TX, TY, NT>(X, ldx, p, Y, ldy, q, r0, std::min<int64_t>(rows, r0 + chunk), nbp, nbq, sym != 0, rg,
                             part + (int64_t)blockIdx.x * p * q, tn_sm);
}

// C = the sum of the CTAs' partials.  32 elements per block, kTnSlices warps
// sum fixed slices of the partials and the slices are added in order (one
// thread per element over 148 partials took 75 us in eight blocks, held by
// load latency).  sym: an element of a tile block I > J is its transpose's.
constexpr int kTnSlices = 16;
static __global__ void __launch_bounds__(32 * kTnSlices) k_tn_reduce(const double* __restrict__ part, int nblocks,
                                                                     int p, int q, int w, int sym,
                                                                     double* __restrict__ C,
                                                                     const int* __restrict__ cond) {
    if (cond && *cond == 0) return;
    __shared__ double sh[kTnSlices][32];
    const int pq = p * q, lane = threadIdx.x & 31, sl = threadIdx.x >> 5;
    const int e = blockIdx.x * 32 + lane;
    double acc = 0.0;
    if (e < pq) {
        const int i = e / q, j = e - i * q;
        const int src = (sym && i / w > j / w) ? j * q + i : e;
        const int per = (nblocks + kTnSlices - 1) / kTnSlices;
        const int b0 = sl * per, b1 = min(nblocks, b0 + per);
#pragma unroll 4
        for (int b = b0; b < b1; ++b) acc += part[(int64_t)b * pq + src];
    }
    sh[sl][lane] = acc;
    __syncthreads();
    if (sl == 0 && e < pq) {
        double t = 0.0;
#pragma unroll
        for (int k = 0; k < kTnSlices; ++k) t += sh[k][lane];
        C[e] = t;
    }
}

// host: C (p x q) = X^T Y.  part: at least tn_shape(...).blocks * p * q doubles.
// C null: the partials are left as they are (sym: their tile blocks I <= J).
template <typename TX, typename TY>
inline void tn_launch(const TnShape& h, const TX* X, int64_t ldx, int p, const TY* Y, int64_t ldy, int q, int64_t rows,
                      double* part, double* C, const int* cond, cudaStream_t s) {
    auto go = [&](auto kern) {
        allow_smem(kern, tn_smem_max(h.nt));
        kern<<<h.blocks, h.threads(), h.smem(), s>>>(X, ldx, p, Y, ldy, q, rows, h.chunk, h.nbp, h.nbq, (int)h.sym, h.rg,
                                                 part, cond);
    };
    switch (h.nt) {
        case 1: go(k_tn_part<TX, TY, 1>); break;
        case 2: go(k_tn_part<TX, TY, 2>); break;
        case 3: go(k_tn_part<TX, TY, 3>); break;
        default: go(k_tn_part<TX, TY, 4>); break;
    }
    SVDB_CHECK_LAUNCH();
    if (!C) return;
    k_tn_reduce<<<(p * q + 31) / 32, 32 * kTnSlices, 0, s>>>(part, h.blocks, p, q, h.nt * 8, (int)h.sym, C, cond);
    SVDB_CHECK_LAUNCH();
}

// -------------------------------------------------------------- X C ----
// Out[r][j] = alpha sum_k X[r][k] d[k] C[k][j] + beta Y[r][j] + es[j] E[r][j]
// for up to NQ * 8 columns j from blockIdx.y * NQ * 8.  C sits in shared
// memory (rows padded to a multiple of four with zeros, row stride NQ * 8 + 4
// doubles: conflict-free fragment reads); a warp takes 16 rows, whose
// fragments come straight from global memory four k-steps ahead.  tri: C is
// upper triangular, and the fragments of C below its diagonal are skipped.
// Out may be X (q <= NQ * 8) or Y: a warp has read all of a row before it
// writes it.  trans: Out is stored q x rows.  DOT 1 / 2: the column sums of
// Out * Out / Out * E over the CTA's rows go to dots[blockIdx.x * q + j].
template <typename TX, typename TO>
struct NnArgs {
    const TX* X;
    int64_t ldx, rows;
    int p;
    const double* C;
    int ldc;
    const double* d;  // null: 1
    int q, tri;
    double alpha;
    const double* Y;  // null: no beta term
    int64_t ldy;
    double beta;
    const double* E;  // null: no third term
    int64_t lde;
    const double* es;
    TO* Out;
    int64_t ldo;
    int trans;
    double* dots;
    const int* cond;
};

constexpr int kNnWarps = 8, kNnMT = 2, kNnKU = 4;
__host__ __device__ inline size_t nn_smem(int p, int nq) { return (size_t)((p + 3) / 4 * 4) * (nq * 8 + 4) * sizeof(double); }

// the warps of the calling CTA walk row groups g0, g0 + gstep, ... (16 rows each)
template <typename TX, typename TO, int NQ, int DOT>
__device__ __forceinline__ void nn_body(const NnArgs<TX, TO>& A, int64_t g0, int64_t gstep, int col0, double* cs) {
    constexpr int LD = NQ * 8 + 4;
    const int lane = threadIdx.x & 31;
    const int kl = lane & 3, il = lane >> 2;
    const int p4 = (A.p + 3) / 4 * 4;
    for (int t = threadIdx.x; t < p4 * NQ * 8; t += blockDim.x) {
        const int k = t / (NQ * 8), j = t - k * (NQ * 8);
        double v = 0.0;
        if (k < A.p && col0 + j < A.q) {
            v = A.C[(int64_t)k * A.ldc + col0 + j];
            if (A.d) v *= A.d[k];
        }
        cs[k * LD + j] = v;
    }
    __syncthreads();
    double dacc[DOT ? NQ : 1][2];
    if constexpr (DOT != 0) {
#pragma unroll
        for (int n = 0; n < NQ; ++n) dacc[n][0] = dacc[n][1] = 0.0;
    }
    const int nk = p4 / 4;
    TX a[kNnKU][kNnMT];
    auto load = [&](int64_t grp, int k0, TX (&f)[kNnKU][kNnMT]) {
#pragma unroll
        for (int u = 0; u < kNnKU; ++u)
#pragma unroll
            for (int i = 0; i < kNnMT; ++i) {
                const int64_t row = (grp * kNnMT + i) * 8 + il;
                const int col = 4 * (k0 + u) + kl;
                f[u][i] = (row < A.rows && col < A.p) ? A.X[row * A.ldx + col] : TX(0);
            }
    };
    load(g0, 0, a);
    for (int64_t g = g0; g * (8 * kNnMT) < A.rows; g += gstep) {
        const int64_t row0 = g * (8 * kNnMT);
        double acc[kNnMT][NQ][2];
#pragma unroll
        for (int i = 0; i < kNnMT; ++i)
#pragma unroll
            for (int n = 0; n < NQ; ++n) acc[i][n][0] = acc[i][n][1] = 0.0;
        for (int k0 = 0; k0 < nk; k0 += kNnKU) {
            TX na[kNnKU][kNnMT];  // in flight meanwhile: this group's next k-steps, or the next group's first
            if (k0 + kNnKU < nk) load(g, k0 + kNnKU, na);
            else load(g + gstep, 0, na);
#pragma unroll
            for (int u = 0; u < kNnKU; ++u) {
                if (k0 + u >= nk) break;
                const double* cr = cs + (4 * (k0 + u) + kl) * LD + il;
                const int nlow = A.tri ? ((k0 + u) >> 1) - (col0 >> 3) : 0;  // tiles left of it hold zeros only
#pragma unroll
                for (int n = 0; n < NQ; ++n) {
                    if (n < nlow) continue;
                    const double bf = cr[8 * n];
#pragma unroll
                    for (int i = 0; i < kNnMT; ++i) dmma(acc[i][n], (double)a[u][i], bf);
                }
            }
#pragma unroll
            for (int u = 0; u < kNnKU; ++u)
#pragma unroll
                for (int i = 0; i < kNnMT; ++i) a[u][i] = na[u][i];
        }
        const bool pair = !A.trans && (A.ldo & 1) == 0 && (reinterpret_cast<uintptr_t>(A.Out) % (2 * sizeof(TO))) == 0;
#pragma unroll
        for (int i = 0; i < kNnMT; ++i) {
            const int64_t row = row0 + 8 * i + il;
            if (row >= A.rows) continue;
#pragma unroll
            for (int n = 0; n < NQ; ++n) {
                const int j = col0 + 8 * n + 2 * kl;
                double v[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    v[h] = A.alpha * acc[i][n][h];
                    if (j + h < A.q) {
                        if (A.Y) v[h] += A.beta * A.Y[row * A.ldy + j + h];
                        if (A.E) {
                            const double e = A.E[row * A.lde + j + h];
                            v[h] += A.es[j + h] * e;
                            if constexpr (DOT == 2) dacc[n][h] = fma(v[h], e, dacc[n][h]);
                        }
                        if constexpr (DOT == 1) dacc[n][h] = fma(v[h], v[h], dacc[n][h]);
                    }
                }
                if (pair && j + 1 < A.q) {
                    struct alignas(2 * sizeof(TO)) Two { TO x, y; };
                    *reinterpret_cast<Two*>(A.Out + row * A.ldo + j) = Two{(TO)v[0], (TO)v[1]};
                } else {
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        if (j + h < A.q) {
                            if (A.trans) A.Out[(int64_t)(j + h) * A.ldo + row] = (TO)v[h];
                            else A.Out[row * A.ldo + j + h] = (TO)v[h];
                        }
                }
            }
        }
    }
    if constexpr (DOT != 0) {  // lanes of one column, then the warps in order
        const int warp = threadIdx.x >> 5;
        __syncthreads();  // cs is read; it holds the warps' sums now (kNnWarps * NQ * 8 doubles fit: see nn_launch)
#pragma unroll
        for (int n = 0; n < NQ; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                double t = dacc[n][h];
                t += __shfl_xor_sync(0xffffffffu, t, 4);
                t += __shfl_xor_sync(0xffffffffu, t, 8);
                t += __shfl_xor_sync(0xffffffffu, t, 16);
                if (il == 0) cs[warp * (NQ * 8) + 8 * n + 2 * kl + h] = t;
            }
        __syncthreads();
        for (int j = threadIdx.x; j < NQ * 8; j += blockDim.x) {
            double t = 0.0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += cs[w * (NQ * 8) + j];
            if (col0 + j < A.q) A.dots[(int64_t)blockIdx.x * A.q + col0 + j] = t;
        }
    }
}

template <typename TX, typename TO, int NQ, int DOT>
__global__ void __launch_bounds__(32 * kNnWarps, 2) k_nn(const __grid_constant__ NnArgs<TX, TO> A) {
    if (A.cond && *A.cond == 0) return;
    extern __shared__ __align__(16) double nn_sm[];
    nn_body<TX, TO, NQ, DOT>(A, (int64_t)blockIdx.x * kNnWarps + (threadIdx.x >> 5), (int64_t)gridDim.x * kNnWarps,
                             (int)blockIdx.y * NQ * 8, nn_sm);
}

// CTAs of one column block: one wave of two per SM
inline int nn_blocks(int64_t rows, int sms) {
    const int64_t per = 8 * kNnMT * kNnWarps;
    return (int)std::max<int64_t>(1, std::min<int64_t>((rows + per - 1) / per, (int64_t)sms * 2));
}

template <int DOT, typename TX, typename TO>
inline void nn_launch(const NnArgs<TX, TO>& A, int sms, cudaStream_t s) {
    if (A.rows <= 0 || A.q <= 0) return;
    // 64 columns per CTA; 32 where the column sums take another 2 NQ registers pairs (64 spilled 956 bytes)
    constexpr int kMaxQ = DOT ? 4 : 8;
    const int tiles = (A.q + 7) / 8, ny = (tiles + kMaxQ - 1) / kMaxQ, nq = (tiles + ny - 1) / ny;
    size_t smem = nn_smem(A.p, nq);
    if (DOT) smem = std::max(smem, (size_t)kNnWarps * nq * 8 * sizeof(double));
    const dim3 grid(nn_blocks(A.rows, sms), ny);
    auto go = [&](auto kern) {
        allow_smem(kern, nn_smem(128, nq));
        kern<<<grid, 32 * kNnWarps, smem, s>>>(A);
    };
    switch (nq) {
        case 1: go(k_nn<TX, TO, 1, DOT>); break;
        case 2: go(k_nn<TX, TO, 2, DOT>); break;
        case 3: go(k_nn<TX, TO, 3, DOT>); break;
        case 4: go(k_nn<TX, TO, 4, DOT>); break;
        default:
            if constexpr (DOT == 0) {
                if (nq == 5) go(k_nn<TX, TO, 5, 0>);
                else if (nq == 6) go(k_nn<TX, TO, 6, 0>);
                else if (nq == 7) go(k_nn<TX, TO, 7, 0>);
                else go(k_nn<TX, TO, 8, 0>);
            }
    }
    SVDB_CHECK_LAUNCH();
}

}  // namespace svdb

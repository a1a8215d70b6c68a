// Cooperative Lanczos-block kernel: runs lanczos_step for j in [first, last)
// (src/lanczos/mod.rs:674-758) entirely on the device, including the
// ortbnd recurrence (mod.rs:815-838) and purge (mod.rs:760-813), with one
// launch per lanso block.  All blocks advance in lockstep through bounded grid
// barriers; scalar results of reductions are recomputed identically by every
// block from the same partials, so no extra broadcast round is needed.
//
// Arithmetic: sparse products and dot products use FMA and a fixed-order
// tree; the element-wise updates (datx, dscal, daxpy) use unfused IEEE
// multiply-then-add, which is what the crate's `y += a * x` computes.
#include <cooperative_groups.h>

#include <mutex>
#include <type_traits>

#include "lanczos_kernel.cuh"
#include "spmv.cuh"
#include "svdb_internal.h"

namespace svdb {

constexpr double kEps = 2.220446049250313e-16;
constexpr int kThreads = 512;
constexpr int kClSlots = 16 * (kThreads / 32);  // cluster sums: blocks x warps

__device__ __forceinline__ bool cmp_eq(double a, double b) { return fabs(b - a) < kEps; }

// Row-gather SpMV over the rows of `op`: rows of more than kSegNnz entries
// (the first of op.bins.rows) one block each, the others through the length bins
// (spmv_binned, spmv.cuh).  SCALE: x is read as x * rinv (the dscal
// of w3 folded in).  EPI: y = acc + (-rnm) * w2, and returns this thread's
// share of dot(y, w3).  Only the matrix arrays are read through the
// non-coherent path: the vectors change between phases of the same launch.
template <bool FP32, bool SCALE, bool EPI, bool SL>
__device__ __forceinline__ double spmv_rows(const LzOperand& op, const double* x, double rinv, double* y,
                                            double neg_rnm, const double* w2, const double* w3, double* sh,
                                            double* dyn) {
    auto xl = [&](int32_t c) {
        double xv = x[c];
        if (SCALE) xv = mul_rn(xv, rinv);
        return xv;
    };
    double dotacc = 0.0;
    auto finish = [&](int64_t r, double acc) {
        if (EPI) {
            const double w0 = add_rn(acc, mul_rn(neg_rnm, w2[r]));
            y[r] = w0;
            dotacc = fma(w0, w3[r], dotacc);
        } else {
            y[r] = acc;
        }
    };
    if constexpr (SL) {  // x slices in shared memory (spmv.cuh)
        if (FP32) sliced_rows<float, SCALE>(op.sl, op.svf, x, rinv, dyn, finish);
        else sliced_rows<double, SCALE>(op.sl, op.sv, x, rinv, dyn, finish);
        return dotacc;
    }
    spmv_deal(blockIdx.x, gridDim.x, op.bins.off[0], [&](int64_t i) {  // uniform over the block
        const int64_t r = __ldg(op.bins.rows + i);
        const int64_t s = __ldg(op.rp + r), e = __ldg(op.rp + r + 1);
        double acc = FP32 ? row_dot(op.ci, op.vf, s, e, (int)threadIdx.x, (int)blockDim.x, xl)
                          : row_dot(op.ci, op.v, s, e, (int)threadIdx.x, (int)blockDim.x, xl);
        acc = block_sum(acc, sh);
        if (threadIdx.x == 0) finish(r, acc);
    });
    const int64_t gwarp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    if (FP32) spmv_binned(op.rp, op.ci, op.vf, op.bins, gwarp, nwarps, xl, finish);
    else spmv_binned(op.rp, op.ci, op.v, op.bins, gwarp, nwarps, xl, finish);
    return dotacc;
}

namespace cg = cooperative_groups;

// Barrier over all blocks: the bounded grid barrier of a cooperative launch,
// or (CL) the hardware barrier of a thread-block cluster that holds the whole
// grid.  Cluster mode needs control flow uniform over the blocks, which holds
// here: every branch depends on values all blocks compute identically.
template <bool CL>
__device__ __forceinline__ bool lz_sync(GridBarrier* bar) {
    if constexpr (CL) {
        cg::this_cluster().sync();
        return true;
    } else {
        return grid_sync(bar);
    }
}

// Sum over all blocks of one value per thread: block partial -> barrier ->
// every block adds the partials in the same order.  `par` alternates between
// two sets of partial slots, so a block that starts the next sum never
// overwrites a partial another block is still reading.  Cluster mode: each of
// the `nwa` warps that have a share (the same number in every block) writes its
// partial into all blocks' shared memory (cl_slot, blocks x nwa), and after the
// one cluster barrier every warp adds them all in the same order, so no block
// barrier is needed on either side.  Block sums around the cluster barrier
// (six block barriers per sum) took 2.7 us; all sixteen warps writing 1.2-1.3,
// four 1.1: the barrier waits for the remote stores.
template <bool CL>
__device__ __forceinline__ bool lz_sum(double v, double* part, GridBarrier* bar, double* sh, double* cl_slot, int nwa,
                                       int& par, double& out) {
    const int p = par;
    par ^= 1;
    if constexpr (CL) {
        cg::cluster_group cl = cg::this_cluster();
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const int nb = (int)cl.num_blocks();
        if (warp < nwa) {
            double* mine = cl_slot + p * kClSlots + (int)cl.block_rank() * nwa + warp;
            v = warp_sum(v);
            if (lane < nb) *cl.map_shared_rank(mine, lane) = v;
        }
        cl.sync();
        double t = 0.0;
        for (int k = lane; k < nb * nwa; k += 32) t += cl_slot[p * kClSlots + k];
        out = warp_sum(t);
        return true;
    } else {
        const double b = block_sum(v, sh);
        double* pp = part + (size_t)p * gridDim.x;
        if (threadIdx.x == 0) pp[blockIdx.x] = b;
        if (!grid_sync(bar)) return false;
        out = reduce_partials(pp, gridDim.x, sh);
        return true;
    }
}

// Rows of this CTA's slice of an operand in shared memory, into y: g lanes per
// row, eight entries of each lane in flight (four warps per scheduler do not
// hide a chain of shared reads: with two in flight a product of 6,200 entries
// per CTA took 3.8-4.1 us, with eight 2.2-2.7, near what the random 8-byte
// reads of x cost in bank conflicts); rows of more than 32 g entries by whole
// warps.
template <typename VT>
__device__ __forceinline__ void res_rows(const int* rp, const uint16_t* ci, const VT* v, int rows, int g,
                                         bool has_long, const double* x, double* y) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int sub = lane & (g - 1), per = 32 / g;
    auto dot = [&](int s, int e, int step) {  // first entry s + (this lane's place)
        double a0 = 0.0, a1 = 0.0;
        for (int k = s; k < e; k += 8 * step) {
            double vv[8], xv[8];
            int c[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) c[u] = k + u * step < e ? (int)ci[k + u * step] : -1;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                vv[u] = c[u] >= 0 ? (double)v[k + u * step] : 0.0;
                xv[u] = c[u] >= 0 ? x[c[u]] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < 8; u += 2) {
                a0 = fma(vv[u], xv[u], a0);
                a1 = fma(vv[u + 1], xv[u + 1], a1);
            }
        }
        return a0 + a1;
    };
    for (int base = warp * per; base < rows; base += nw * per) {
        const int r = base + lane / g;
        int s = 0, e = 0;
        if (r < rows) { s = rp[r]; e = rp[r + 1]; }
        const bool mine = r < rows && e - s <= 32 * g;
        double acc = mine ? dot(s + sub, e, g) : 0.0;
        for (int o = g >> 1; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (mine && sub == 0) y[r] = acc;
    }
    if (!has_long) return;
    for (int r = warp; r < rows; r += nw) {
        const int s = rp[r], e = rp[r + 1];
        if (e - s <= 32 * g) continue;
        const double acc = warp_sum(dot(s + lane, e, 32));
        if (lane == 0) y[r] = acc;
    }
}

// RES (cluster launches on small operators): both operands' slices, the
// gathered vector and the step's own elements live in shared memory and
// registers (a thread owns one element of every vector); the copies in global
// memory are kept for the purge and the host.  The gathered vectors (w3, temp)
// are written by their owners into every CTA's shared memory ahead of a
// cluster barrier that the step has anyway.  A step on the 5000 x 2000
// workload takes 18 us, against 27 with the operands in L2: six sums 6.9, the
// products 4.9, gathering temp 2.5, eta and the purge test 1.7.
template <bool FP32, bool CL, bool SL = false, bool RES = false>
__global__ void __launch_bounds__(kThreads, (CL || SL) ? 1 : 2) k_lanczos_block(const __grid_constant__ LzArgs a) {
    extern __shared__ __align__(16) double lz_dyn[];  // SL: the x slice and the row accumulators; RES: lz_res_layout
    __shared__ double sh[32];
    __shared__ double cl_slot[CL ? 2 * kClSlots : 1];
    __shared__ int cl_flag;
    int par = 0;
    const int64_t n = a.n;
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t nth = (int64_t)gridDim.x * blockDim.x;
    const bool leader = (blockIdx.x == 0 && threadIdx.x == 0);

    // Every block starts from the state the host wrote.
    double rnm = a.st->rnm, tol = a.st->tol;
    int64_t ll = a.st->ll;
    int perm[7];
#pragma unroll
    for (int k = 0; k < 7; ++k) perm[k] = a.st->perm[k];
    int eta_sel = a.st->eta_sel;
    int64_t npurge = a.st->npurge;
    bool resume = a.resume != 0;
    int64_t j = a.first;
    const double eps1 = a.eps1;
    const double sqrt_eps = a.sqrt_eps;  // of the run's scalar T

#define WV(k) (a.W[perm[k]])

    using VT = typename std::conditional<FP32, float, double>::type;
    double* xa = nullptr;  // w3, unscaled when `fresh`
    double* xb = nullptr;  // temp
    double* ys = nullptr;
    bool fresh = false;    // the owners have written w3 into every xa
    const int* rrp[2] = {nullptr, nullptr};
    const uint16_t* rci[2] = {nullptr, nullptr};
    const VT* rv[2] = {nullptr, nullptr};
    int rrows[2] = {0, 0};
    int64_t rfirst[2] = {0, 0};
    bool rlong[2] = {false, false};
    if constexpr (RES) {  // this CTA's rows of both operands
        char* base = reinterpret_cast<char*>(lz_dyn);
        const LzResLayout L = lz_res_layout(a.res, (int)sizeof(VT));
        xa = reinterpret_cast<double*>(base + L.xa);
        xb = reinterpret_cast<double*>(base + L.xb);
        ys = reinterpret_cast<double*>(base + L.y);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const LzOperand& op = k ? a.op2 : a.op1;
            int* lrp = reinterpret_cast<int*>(base + L.rp[k]);
            VT* lv = reinterpret_cast<VT*>(base + L.v[k]);
            uint16_t* lci = reinterpret_cast<uint16_t*>(base + L.ci[k]);
            const int64_t r0 = min(op.rows, (int64_t)blockIdx.x * a.res.rows_c[k]);
            const int64_t r1 = min(op.rows, r0 + a.res.rows_c[k]);
            const int64_t e0 = op.rp[r0], e1 = op.rp[r1];
            rfirst[k] = r0;
            rrows[k] = (int)(r1 - r0);
            int any_long = 0;
            for (int64_t r = r0 + threadIdx.x; r <= r1; r += blockDim.x) {
                lrp[r - r0] = (int)(op.rp[r] - e0);
                any_long |= r < r1 && op.rp[r + 1] - op.rp[r] > 32 * a.res.g[k];
            }
            rlong[k] = __syncthreads_or(any_long) != 0;
            for (int64_t e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
                lci[e - e0] = (uint16_t)op.ci[e];
                if constexpr (FP32) lv[e - e0] = op.vf[e];
                else lv[e - e0] = op.v[e];
            }
            rrp[k] = lrp;
            rci[k] = lci;
            rv[k] = lv;
        }
        __syncthreads();
    }
    const int nwa = RES ? (a.res.rows_c[1] + 31) / 32 : kThreads / 32;  // warps with a share in the step's sums
    // RES: this thread's element of the vectors
    const bool own = RES && (int)threadIdx.x < rrows[1];
    const int64_t oe = rfirst[1] + threadIdx.x;
    double w0e = 0.0, w1e = 0.0, w2e = 0.0, w3e = 0.0, w4e = 0.0;
    double p0e = 0.0, p1e = 0.0, q0e = 0.0, q1e = 0.0;  // of p_0, p_1, q_0, q_1
    if constexpr (RES) {
        const int64_t have = resume ? j : j - 1;  // rows stored before this launch
        if (own && have > 0) { p0e = a.P[oe]; q0e = a.Q[oe]; }
        if (own && have > 1) { p1e = a.P[n + oe]; q1e = a.Q[n + oe]; }
    }
    // alpha, beta and eta in block 0's shared memory while the kernel runs (its
    // threads alone read them); copied back at the end
    double* const g_alf = a.alf;
    double* const g_bet = a.bet;
    double* l_alf = a.alf;
    double* l_bet = a.bet;
    double* l_etaA = a.etaA;
    double* l_etaB = a.etaB;
    double alf_prev = a.alf[j - 1];
    if constexpr (RES) {
        if (blockIdx.x == 0 && a.res.coef > 0) {
            double* c = reinterpret_cast<double*>(reinterpret_cast<char*>(lz_dyn) +
                                                  lz_res_layout(a.res, (int)sizeof(VT)).coef);
            const int64_t len = a.last + 1;
            for (int64_t i = threadIdx.x; i < len; i += blockDim.x) {
                c[i] = a.alf[i];
                c[a.res.coef + i] = a.bet[i];
                c[2 * a.res.coef + i] = a.etaA[i];
                c[3 * a.res.coef + i] = a.etaB[i];
            }
            l_alf = c;
            l_bet = c + a.res.coef;
            l_etaA = c + 2 * a.res.coef;
            l_etaB = c + 3 * a.res.coef;
        }
        // the copies above, and every CTA has started: the first step stores into all of them
        cg::this_cluster().sync();
    }
    auto put_back = [&] {
        if constexpr (RES) {
            __syncthreads();
            if (l_alf != g_alf) {
                for (int64_t i = threadIdx.x; i <= a.last; i += blockDim.x) {
                    a.alf[i] = l_alf[i];
                    a.bet[i] = l_bet[i];
                    a.etaA[i] = l_etaA[i];
                    a.etaB[i] = l_etaB[i];
                }
            }
        }
    };

    while (j < a.last) {
        double bet_j;
        if (!resume) {
            // mem::swap(w1, w2); mem::swap(w3, w4)
            int t = perm[1]; perm[1] = perm[2]; perm[2] = t;
            t = perm[3]; perm[3] = perm[4]; perm[4] = t;
            bet_j = rnm;  // wrk.bet[j] = rnm
            if (leader) l_bet[j] = bet_j;
            if (cmp_eq(rnm, 0.0)) {
                // invariant subspace: store q_{j-1}, p_{j-1} and hand over to the host's startv
                double* w2 = WV(2);
                double* w4 = WV(4);
                for (int64_t e = tid; e < n; e += nth) {
                    a.Q[(j - 1) * n + e] = w2[e];
                    if (j - 1 < 2) a.P[(j - 1) * n + e] = w4[e];
                }
                if (leader) {
                    a.st->status = 1;
                    a.st->j = j;
                    for (int k = 0; k < 7; ++k) a.st->perm[k] = perm[k];
                    a.st->rnm = rnm; a.st->tol = tol; a.st->ll = ll;
                    a.st->eta_sel = eta_sel; a.st->npurge = npurge;
                }
                put_back();
                if constexpr (CL) cg::this_cluster().sync();  // no block leaves while others may read its slots
                return;
            }
        } else {
            bet_j = g_bet[j];  // set before the host restart
        }

        // ---- phase 1: temp = op1 (w3 / rnm); w1 = w0 / rnm; w3' = w3 / rnm; store copies
        const double rinv = 1.0 / rnm;
        {
            const double* w0 = WV(0);
            const double* w2 = WV(2);
            const double* w3 = WV(3);
            const double* w4 = WV(4);
            double* w1 = WV(1);
            double* w3s = WV(6);
            if constexpr (RES) {
                if (own) {
                    if (fresh) {  // the swaps above, on the last step's values
                        w2e = w1e;
                        const double t = w3e;
                        w3e = w4e;
                        w4e = t;
                    } else {
                        w0e = w0[oe];
                        w2e = w2[oe];
                        w3e = w3[oe];
                        w4e = w4[oe];
                    }
                }
                for (int k = threadIdx.x; k < (int)n; k += kThreads) xa[k] = mul_rn(fresh ? xa[k] : w3[k], rinv);
                __syncthreads();
                res_rows(rrp[0], rci[0], rv[0], rrows[0], a.res.g[0], rlong[0], xa, ys);
                __syncthreads();
                // rows_c is even: two rows per store (the pad of an odd last row stays in its slot's pad)
                for (int r = 2 * threadIdx.x; r < rrows[0]; r += 2 * kThreads) {
                    const double2 t = make_double2(ys[r], ys[r + 1]);
                    double2* dst = reinterpret_cast<double2*>(xb + rfirst[0] + r);
#pragma unroll
                    for (int c = 0; c < kLzResCluster; ++c) *cg::this_cluster().map_shared_rank(dst, c) = t;
                }
                if (own) {
                    w1e = mul_rn(rinv, w0e);
                    w3e = mul_rn(w3e, rinv);
                    w1[oe] = w1e;
                    w3s[oe] = w3e;
                    if (!resume) {
                        a.Q[(j - 1) * n + oe] = w2e;
                        if (j - 1 < 2) a.P[(j - 1) * n + oe] = w4e;
                        if (j == 1) { p0e = w4e; q0e = w2e; }
                        if (j == 2) { p1e = w4e; q1e = w2e; }
                    }
                }
            } else {
            spmv_rows<FP32, true, false, SL>(a.op1, w3, rinv, a.temp, 0.0, nullptr, nullptr, sh, lz_dyn);
            for (int64_t e = tid; e < n; e += nth) {
                w1[e] = mul_rn(rinv, w0[e]);
                w3s[e] = mul_rn(w3[e], rinv);
                if (!resume) {
                    a.Q[(j - 1) * n + e] = w2[e];
                    if (j - 1 < 2) a.P[(j - 1) * n + e] = w4[e];
                }
            }
            }
            int t = perm[3]; perm[3] = perm[6]; perm[6] = t;
        }
        resume = false;
        if (!lz_sync<CL>(a.bar)) return;

        // ---- phase 2: w0 = op2 temp - rnm w2; alf[j] = w0 . w3
        double alf_j;
        {
            double part = 0.0;
            if constexpr (RES) {
                res_rows(rrp[1], rci[1], rv[1], rrows[1], a.res.g[1], rlong[1], xb, ys);
                __syncthreads();
                if (own) {
                    w0e = add_rn(ys[threadIdx.x], mul_rn(-rnm, w2e));
                    part = mul_rn(w0e, w3e);
                }
            } else {
                part = spmv_rows<FP32, false, true, SL>(a.op2, a.temp, 1.0, WV(0), -rnm, WV(2), WV(3), sh, lz_dyn);
            }
            if (!lz_sum<CL>(part, a.part, a.bar, sh, cl_slot, nwa, par, alf_j)) return;
        }

        // orthogonalise against the initial Lanczos vectors (mod.rs:722-731)
        if (j <= 2 && fabs(alf_prev) > 4.0 * fabs(alf_j)) ll = j;
        const int64_t nloc = (j - 1 < ll) ? (j - 1) : ll;
        double* etaC = eta_sel ? l_etaB : l_etaA;  // eta
        double* etaO = eta_sel ? l_etaA : l_etaB;  // oldeta

        // ---- chain of (t = dot(w0, d); w0 -= t * u), fused pairwise
        double coef = alf_j, axe = w1e;
        const double* axv = WV(1);
        for (int64_t step = 0; step < nloc + 2; ++step) {
            const double* dv = (step < nloc) ? (a.P + step * n) : (step == nloc ? WV(4) : WV(3));
            double* w0 = WV(0);
            double acc = 0.0;
            if constexpr (RES) {
                if (own) {
                    const double dve = step < nloc ? (step ? p1e : p0e) : (step == nloc ? w4e : w3e);  // nloc <= 2
                    w0e = add_rn(w0e, mul_rn(-coef, axe));
                    acc = mul_rn(w0e, dve);
                    axe = step < nloc ? (step ? q1e : q0e) : (step == nloc ? w2e : w1e);
                }
            } else {
            for (int64_t e = tid; e < n; e += nth) {
                const double v = add_rn(w0[e], mul_rn(-coef, axv[e]));
                w0[e] = v;
                acc = fma(v, dv[e], acc);
            }
            }
            double t;
            if (!lz_sum<CL>(acc, a.part, a.bar, sh, cl_slot, nwa, par, t)) return;
            if (step < nloc) {
                if (leader) { etaC[step] = eps1; etaO[step] = eps1; }
                axv = a.Q + step * n;
            } else if (step == nloc) {
                if (bet_j > 0.0) bet_j += t;
                axv = WV(2);
            } else {
                alf_j += t;
                axv = WV(1);
            }
            coef = t;
        }
        {
            double* w0 = WV(0);
            double* w4 = WV(4);
            double acc = 0.0;
            if constexpr (RES) {
                if (own) {
                    const double v = add_rn(w0e, mul_rn(-coef, axe));
                    w0[oe] = w0e = v;
                    w4[oe] = w4e = v;
                    acc = mul_rn(v, v);
                    // the next step's w3 (the sum's barrier orders these stores)
#pragma unroll
                    for (int c = 0; c < kLzResCluster; ++c) *cg::this_cluster().map_shared_rank(xa + oe, c) = v;
                }
                fresh = true;
            } else {
            for (int64_t e = tid; e < n; e += nth) {
                const double v = add_rn(w0[e], mul_rn(-coef, axv[e]));
                w0[e] = v;
                w4[e] = v;
                acc = fma(v, v, acc);
            }
            }
            double s2;
            if (!lz_sum<CL>(acc, a.part, a.bar, sh, cl_slot, nwa, par, s2)) return;
            rnm = sqrt(s2);
        }
        if (leader) { l_alf[j] = alf_j; l_bet[j] = bet_j; }
        alf_prev = alf_j;
        tol = sqrt_eps * (bet_j + fabs(alf_j) + rnm);

        // ---- ortbnd (mod.rs:815-838) and the purge test (mod.rs:768-770) in block 0.
        // A thread keeps the largest of the |eta| it computes for the test's
        // idamax; alf[j] and bet[j] are alf_j and bet_j (the leader's stores
        // need not be waited for).
        if (blockIdx.x == 0) {
            // k = svd_idamax(step - (ll + 1), eta) + ll; purge if |eta[k]| > sqrt(eps).
            // idamax keeps the first index of the largest |eta[i]|, i in [0, cnt).
            const int64_t cnt = j >= ll + 2 ? j - ll - 1 : 0;
            const bool rec = !cmp_eq(rnm, 0.0) && j > 1;
            double best = -1.0;
            int64_t bi = 0;
            for (int64_t i = threadIdx.x; i <= j - 2; i += blockDim.x) {
                double v;
                if (rec) {
                    if (i == 0) {
                        v = sub_rn(add_rn(mul_rn(l_bet[1], etaC[1]), mul_rn(sub_rn(l_alf[0], alf_j), etaC[0])),
                                   mul_rn(bet_j, etaO[0]));
                    } else {
                        v = sub_rn(add_rn(add_rn(mul_rn(l_bet[i + 1], etaC[i + 1]),
                                                 mul_rn(sub_rn(l_alf[i], alf_j), etaC[i])),
                                          mul_rn(l_bet[i], etaC[i - 1])),
                                   mul_rn(bet_j, etaO[i]));
                    }
                    v = add_rn(__ddiv_rn(v, rnm), eps1);
                    etaO[i] = v;
                } else {
                    v = etaO[i];
                }
                if (i < cnt && fabs(v) > best) { best = fabs(v); bi = i; }
            }
            if (threadIdx.x == 0) etaO[j - 1] = eps1;
            // swap(oldeta, eta); eta[j] = eps1
            double* t = etaC; etaC = etaO; etaO = t;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double ob = __shfl_xor_sync(0xffffffffu, best, o);
                const int64_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
            }
            __shared__ double shb[32];
            __shared__ int64_t shi[32];
            if ((threadIdx.x & 31) == 0) { shb[threadIdx.x >> 5] = best; shi[threadIdx.x >> 5] = bi; }
            __syncthreads();  // every eta is stored, and nobody reads the other array any more
            if (threadIdx.x == 0) etaC[j] = eps1;
            if (threadIdx.x < 32) {
                const int nw = (int)(blockDim.x >> 5);
                best = (int)threadIdx.x < nw ? shb[threadIdx.x] : -2.0;
                bi = (int)threadIdx.x < nw ? shi[threadIdx.x] : 0;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const double ob = __shfl_xor_sync(0xffffffffu, best, o);
                    const int64_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
                    if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
                }
                const int flag = cnt > 0 && fabs(etaC[bi + ll]) > sqrt_eps;
                if constexpr (CL) {
                    cg::cluster_group cl = cg::this_cluster();
                    if (threadIdx.x < cl.num_blocks()) *cl.map_shared_rank(&cl_flag, threadIdx.x) = flag;
                } else if (threadIdx.x == 0) {
                    a.st->purge_flag = flag;
                }
            }
        } else {
            double* t = etaC; etaC = etaO; etaO = t;
        }
        eta_sel ^= 1;
        if (!lz_sync<CL>(a.bar)) return;
        const int do_purge = CL ? cl_flag : *(volatile int*)&a.st->purge_flag;

        if (do_purge) {
            fresh = false;  // w3 and w4 change in global memory
            // ---- purge (mod.rs:760-813): <= 2 sweeps of classical Gram-Schmidt
            // of q (w1, via w3) and r (w0, via w4) against q_ll .. q_{j-1}.
            ++npurge;
            const double reps1 = eps1 / sqrt_eps;
            const int64_t cnt = j - ll;
            int64_t nsplit = (n + 2047) / 2048;
            int64_t maxsplit = a.part_cap / (2 * cnt);
            if (nsplit > maxsplit) nsplit = maxsplit < 1 ? 1 : maxsplit;
            const int64_t chunk = (n + nsplit - 1) / nsplit;
            const int lane = threadIdx.x & 31;
            const int64_t gwarp = tid >> 5, nwarps = nth >> 5;
            for (int it = 0; it < 2; ++it) {
                if (!(rnm > tol)) continue;
                const double* w3 = WV(3);
                const double* w4 = WV(4);
                // dots Q[i] . w3 and Q[i] . w4 (the crate computes them before each
                // axpy, but w3 and w4 are not modified inside the loop)
                for (int64_t task = gwarp; task < cnt * nsplit; task += nwarps) {
                    const int64_t i = ll + task / nsplit, c = task % nsplit;
                    const int64_t e0 = c * chunk, e1 = (e0 + chunk < n) ? e0 + chunk : n;
                    const double* q = a.Q + i * n;
                    double sq = 0.0, sr = 0.0;
#pragma unroll 4
                    for (int64_t e = e0 + lane; e < e1; e += 32) {
                        const double qv = q[e];
                        sq = fma(qv, w3[e], sq);
                        sr = fma(qv, w4[e], sr);
                    }
                    sq = warp_sum(sq);
                    sr = warp_sum(sr);
                    if (lane == 0) { a.part[2 * task] = sq; a.part[2 * task + 1] = sr; }
                }
                if (!lz_sync<CL>(a.bar)) return;
                for (int64_t i = gwarp; i < cnt; i += nwarps) {
                    double sq = 0.0, sr = 0.0;
                    for (int64_t c = lane; c < nsplit; c += 32) {
                        sq += a.part[2 * (i * nsplit + c)];
                        sr += a.part[2 * (i * nsplit + c) + 1];
                    }
                    sq = warp_sum(sq);
                    sr = warp_sum(sr);
                    if (lane == 0) { a.tq[ll + i] = sq; a.tr[ll + i] = sr; }
                }
                if (!lz_sync<CL>(a.bar)) return;
                // tq = sum |t_q|, tr = sum |t_r|
                double aq = 0.0, ar = 0.0;
                for (int64_t i = threadIdx.x; i < cnt; i += blockDim.x) {
                    aq += fabs(a.tq[ll + i]);
                    ar += fabs(a.tr[ll + i]);
                }
                const double tq_sum = block_sum(aq, sh);
                double tr_sum = block_sum(ar, sh);
                // w1 -= sum_i tq_i q_i ; w0 -= sum_i tr_i q_i (in i order); w3 = w1
                double* w1 = WV(1);
                double* w0 = WV(0);
                double* w3w = WV(3);
                double acc = 0.0;
                for (int64_t e = tid; e < n; e += nth) {
                    double v1 = w1[e], v0 = w0[e];
                    // the crate's order over i (unfused multiply, then add); the
                    // loads of eight vectors are issued before their updates
                    int64_t i = ll;
                    for (; i + 8 <= j; i += 8) {
                        double qv[8], t1[8], t0[8];
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            qv[u] = a.Q[(i + u) * n + e];
                            t1[u] = a.tq[i + u];
                            t0[u] = a.tr[i + u];
                        }
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            v1 = add_rn(v1, mul_rn(-t1[u], qv[u]));
                            v0 = add_rn(v0, mul_rn(-t0[u], qv[u]));
                        }
                    }
                    for (; i < j; ++i) {
                        const double qv = a.Q[i * n + e];
                        v1 = add_rn(v1, mul_rn(-a.tq[i], qv));
                        v0 = add_rn(v0, mul_rn(-a.tr[i], qv));
                    }
                    w1[e] = v1;
                    w3w[e] = v1;
                    w0[e] = v0;
                    acc = fma(v0, v1, acc);
                }
                double t;
                if (!lz_sum<CL>(acc, a.part, a.bar, sh, cl_slot, kThreads / 32, par, t)) return;
                tr_sum += fabs(t);
                double* w4w = WV(4);
                double acc2 = 0.0;
                for (int64_t e = tid; e < n; e += nth) {
                    const double v = add_rn(w0[e], mul_rn(-t, w1[e]));
                    w0[e] = v;
                    w4w[e] = v;
                    acc2 = fma(v, v, acc2);
                }
                double s2;
                if (!lz_sum<CL>(acc2, a.part, a.bar, sh, cl_slot, kThreads / 32, par, s2)) return;
                rnm = sqrt(s2);
                if (tq_sum <= reps1 && tr_sum <= rnm * reps1) break;
            }
            if (blockIdx.x == 0) {
                for (int64_t i = ll + threadIdx.x; i <= j; i += blockDim.x) { etaC[i] = eps1; etaO[i] = eps1; }
            }
        }
        if (rnm <= tol) rnm = 0.0;
        ++j;
    }
    put_back();
    if (leader) {
        a.st->status = 0;
        a.st->j = j;
        for (int k = 0; k < 7; ++k) a.st->perm[k] = perm[k];
        a.st->rnm = rnm; a.st->tol = tol; a.st->ll = ll;
        a.st->eta_sel = eta_sel; a.st->npurge = npurge;
    }
    if constexpr (CL) cg::this_cluster().sync();  // no block leaves while others may read its slots
#undef WV
}

int lanczos_max_blocks(int threads) {
    int per_sm = 0;
    SVDB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_lanczos_block<false, false>, threads, 0));
    int per_sm32 = 0;
    SVDB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm32, k_lanczos_block<true, false>, threads, 0));
    per_sm = per_sm < per_sm32 ? per_sm : per_sm32;
    if (per_sm < 1) per_sm = 1;
    return per_sm * device_props().sms;
}

// Blocks of the sliced cooperative grid: one per SM (the x slice takes most
// of the SM's shared memory).
int lanczos_sliced_blocks(int threads) {
    static std::once_flag attr;
    std::call_once(attr, [] {
        SVDB_CUDA(cudaFuncSetAttribute(k_lanczos_block<false, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kSlSmem));
        SVDB_CUDA(cudaFuncSetAttribute(k_lanczos_block<true, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kSlSmem));
    });
    int per_sm = 0, per_sm32 = 0;
    SVDB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_lanczos_block<false, false, true>, threads,
                                                            kSlSmem));
    SVDB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm32, k_lanczos_block<true, false, true>, threads,
                                                            kSlSmem));
    per_sm = per_sm < per_sm32 ? per_sm : per_sm32;
    return per_sm >= 1 ? per_sm * device_props().sms : 0;
}

void launch_lanczos_block(const LzArgs& a, int blocks, int threads, int cluster, cudaStream_t s, bool sliced) {
    const bool fp32 = a.op1.vf != nullptr;
    if (a.res.on) {  // one cluster with the operands in its shared memory
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kLzResCluster);
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = lz_res_layout(a.res, fp32 ? 4 : 8).bytes;
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kLzResCluster;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (fp32) SVDB_CUDA(cudaLaunchKernelEx(&cfg, k_lanczos_block<true, true, false, true>, a));
        else SVDB_CUDA(cudaLaunchKernelEx(&cfg, k_lanczos_block<false, true, false, true>, a));
        count_launches(1);
        return;
    }
    if (sliced) {
        void* args[] = {(void*)&a};
        const void* fn = fp32 ? (const void*)k_lanczos_block<true, false, true>
                              : (const void*)k_lanczos_block<false, false, true>;
        SVDB_CUDA(cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(threads), args, kSlSmem, s));
        count_launches(1);
        return;
    }
    if (cluster > 0) {  // the whole grid is one cluster of `cluster` blocks
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(cluster);
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = 0;
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = cluster;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (fp32) SVDB_CUDA(cudaLaunchKernelEx(&cfg, k_lanczos_block<true, true>, a));
        else SVDB_CUDA(cudaLaunchKernelEx(&cfg, k_lanczos_block<false, true>, a));
    } else {
        void* args[] = {(void*)&a};
        const void* fn = fp32 ? (const void*)k_lanczos_block<true, false> : (const void*)k_lanczos_block<false, false>;
        SVDB_CUDA(cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(threads), args, 0, s));
    }
    count_launches(1);
}

// Whether a cluster of `cluster` blocks of `threads` threads can be resident
// (sizes above 8 are opted into per kernel).
bool lanczos_cluster_ok(int cluster, int threads) {
    if (cluster > 8) {
        if (cudaFuncSetAttribute(k_lanczos_block<false, true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
                cudaSuccess ||
            cudaFuncSetAttribute(k_lanczos_block<true, true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
                cudaSuccess) {
            cudaGetLastError();
            return false;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cluster);
    cfg.blockDim = dim3(threads);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0, n32 = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_lanczos_block<false, true>, &cfg) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n32, k_lanczos_block<true, true>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return n >= 1 && n32 >= 1;
}

// (the kernels' static shared memory is below 8 KB)
size_t lanczos_resident_smem() { return device_props().smem_optin > 8192 ? device_props().smem_optin - 8192 : 0; }

bool lanczos_resident_ok(int threads) {
    const size_t smem = lanczos_resident_smem();  // what a launch may grow to with its coefficients
    auto fits = [&](auto kern) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kLzResCluster);
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kLzResCluster;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return n >= 1;
    };
    return fits(k_lanczos_block<false, true, false, true>) && fits(k_lanczos_block<true, true, false, true>);
}

}  // namespace svdb

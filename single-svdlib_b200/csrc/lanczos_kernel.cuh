// Shared declarations of the cooperative Lanczos-block kernel.
#pragma once

#include <cstdint>

#include "device_common.cuh"
#include "spmv.cuh"
#include "svdb_internal.h"

namespace svdb {

// Scalar state of a Lanczos run, shared by the host driver and the kernel.
struct LzState {
    double rnm, tol;
    int64_t j;        // on exit: the step the loop stopped at
    int64_t ll;
    int32_t perm[8];  // work vector k lives in buffer W[perm[k]] (k = 0..6)
    int32_t eta_sel;  // 0: eta = etaA / oldeta = etaB, 1: swapped
    int32_t status;   // 0: reached `last`; 1: restart (startv) needed at step j
    int32_t purge_flag;
    int32_t pad;
    int64_t npurge;
};

struct LzOperand {
    const int64_t* rp;
    const int32_t* ci;
    const double* v;
    const float* vf;  // FP32 values (mixed precision) or null
    int64_t rows;
    SpmvBins bins;             // all rows, longest first
    // the column-sliced copy (sliced launches only, spmv.cuh): its values
    SlicedOp sl;
    const double* sv;
    const float* svf;
};

// Cluster launches on small operators keep both matrices in the CTAs' shared
// memory: CTA c owns rows [c rows_c, (c + 1) rows_c) of each operand, with
// 16-bit column indices, at most max_nnz entries; g lanes take a row.
constexpr int kLzResCluster = 16;
struct LzResident {
    int on;
    int rows_c[2], max_nnz[2], g[2];
    int n, m;  // doubles of the two gathered vectors' copies (w3, temp)
    int coef;  // doubles of each of alpha, beta and the two eta in block 0 (0: they stay in global memory)
};
// offsets (bytes) of the shared arrays; `bytes` in all
struct LzResLayout {
    size_t xa, xb, y, coef, rp[2], v[2], ci[2], bytes;
};
__host__ __device__ inline LzResLayout lz_res_layout(const LzResident& r, int value_bytes) {
    LzResLayout L;
    size_t o = 0;
    L.xa = o; o += (size_t)(r.n + 1) / 2 * 16;
    L.xb = o; o += (size_t)(r.m + 1) / 2 * 16;
    L.coef = o; o += (size_t)r.coef * 32;
    L.y = o; o += (size_t)(r.rows_c[0] > r.rows_c[1] ? r.rows_c[0] : r.rows_c[1]) * 8;
    for (int k = 0; k < 2; ++k) { L.v[k] = o; o += ((size_t)r.max_nnz[k] * value_bytes + 7) / 8 * 8; }
    for (int k = 0; k < 2; ++k) { L.rp[k] = o; o += (size_t)(r.rows_c[k] + 2) / 2 * 8; }
    for (int k = 0; k < 2; ++k) { L.ci[k] = o; o += ((size_t)r.max_nnz[k] * 2 + 7) / 8 * 8; }
    L.bytes = o;
    return L;
}

struct LzArgs {
    LzOperand op1;     // temp = op1 x  (rows: internal nrows)
    LzOperand op2;     // y = op2 temp  (rows: n)
    int64_t n;
    double* W[7];
    double* temp;
    double* Q;         // store: q_i = Q + i * n
    double* P;         // p_0, p_1
    double* alf;
    double* bet;
    double* etaA;
    double* etaB;
    double* part;      // per-block / per-task partial sums
    int64_t part_cap;  // doubles available in part
    double* tq;        // purge coefficients (step-indexed)
    double* tr;
    LzState* st;
    GridBarrier* bar;
    int64_t first, last;
    int32_t resume;    // 1: the host performed startv for step `first`
    double eps1;       // eps * sqrt(n), lanczos_step / purge (mod.rs:685,774)
    double sqrt_eps;   // sqrt(eps): lanczos_step's tol and purge's reps (mod.rs:745,773)
    LzResident res;
};

// blocks: a cooperative grid; cluster > 0: one thread-block cluster of that many blocks instead.
// sliced: both operands carry their column-sliced copy (op.sl), and the grid
// (one block per SM) stages x slices in kSlSmem bytes of dynamic shared memory.
void launch_lanczos_block(const LzArgs& a, int blocks, int threads, int cluster, cudaStream_t s, bool sliced = false);
int lanczos_sliced_blocks(int threads);
// The column-sliced copy of m (spmv_sliced.cu): built on first use, and its
// FP32 values when fp32; false when m gets none.  sliced_view: its arrays.
bool sliced_prepare(const DevCompressed& m, bool fp32, cudaStream_t s);
SlicedOp sliced_view(const DevCompressed& m);
int lanczos_max_blocks(int threads);
bool lanczos_cluster_ok(int cluster, int threads);
// Whether a resident cluster launch (a.res) with `smem` bytes of shared memory per CTA can run.
bool lanczos_resident_ok(size_t smem, int threads);
size_t lanczos_resident_smem();  // most dynamic shared memory of such a CTA

}  // namespace svdb

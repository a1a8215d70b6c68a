// Which operators the Lanczos cluster keeps in its shared memory, and where.
// Host code and layout only (no kernels), so that the decision can be checked
// without a GPU.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace svdb {

// Lanczos blocks on operators of at most this many nonzeros run as one cluster;
// a structure's slice16_nnz is counted up to here (inclusive) and is
// kSlice16Unknown above.
constexpr int64_t kLzClusterNnz = 1 << 20;
constexpr int64_t kSlice16Unknown = -1;
inline bool slice16_counted(int64_t nnz) { return nnz <= kLzClusterNnz; }

// Rows of one of the 16 equal ranges slice16_nnz is counted over (even).
__host__ __device__ inline int64_t slice16_rows(int64_t rows) { return ((rows + 15) / 16 + 1) / 2 * 2; }

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

struct LzResOperand {
    int64_t nmajor, nnz;
    int64_t slice16_nnz;  // most entries in one of the 16 ranges, or kSlice16Unknown
};

// Whether a cluster of kLzResCluster CTAs of `threads` threads with `smem`
// bytes each can hold op[0] (op1, its rows) and op[1] (op2, n rows), and the
// layout if so: one element of every vector per thread, 16-bit column indices
// and entry offsets, and each CTA's slices beside the gathered vectors.  A
// count that was not taken, or that cannot be the most of 16 ranges, holds
// nothing.
inline bool lz_resident_plan(const LzResOperand (&op)[2], int64_t n, int threads, int value_bytes, size_t smem,
                             LzResident& out) {
    out = LzResident{};
    if (n <= 0 || n > (int64_t)kLzResCluster * threads || op[0].nmajor > 65535) return false;
    for (const LzResOperand& p : op)
        if (p.slice16_nnz < 0 || p.slice16_nnz > 65535 || p.slice16_nnz * 16 < p.nnz) return false;
    if (op[0].slice16_nnz + op[1].slice16_nnz >= 65536) return false;
    LzResident r{};
    for (int k = 0; k < 2; ++k) {
        r.rows_c[k] = (int)slice16_rows(op[k].nmajor);
        r.max_nnz[k] = (int)op[k].slice16_nnz;
        r.g[k] = 2;  // lanes per row: about six entries each, eight in flight
        const double avg = op[k].nmajor ? (double)op[k].nnz / (double)op[k].nmajor : 0.0;
        while (r.g[k] < 32 && 6.5 * r.g[k] < avg) r.g[k] *= 2;
    }
    r.n = (int)n;
    r.m = (int)op[0].nmajor;
    if (lz_res_layout(r, value_bytes).bytes > smem) return false;
    r.on = 1;
    out = r;
    return true;
}

}  // namespace svdb

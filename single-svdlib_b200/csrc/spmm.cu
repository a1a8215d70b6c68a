// SpMM row gather: Y (rows x l) = M X, X (minor x l), both row-major, for the
// dense products of randomized_svd (masked.rs:265-733) and the sigma/u step
// of ritvec (mod.rs:1197-1210).
//
// Work unit: a row segment (SegPlan, at most kSegNnz entries), so rows of
// any length spread over warps evenly; rows cut into several segments write
// per-segment partials that a second kernel adds in segment order, keeping
// the result deterministic.  Inside a warp, H groups of 32/H lanes each take
// every H-th entry of the segment; a lane owns CPL consecutive columns and
// reads them with one vector load, and each group keeps U gathers in flight.
// Accumulation is FP64 (for FP32 operands: FP32 within a 32-entry chunk,
// FP64 across chunks).  Register caps: 64 per thread for FP32 operands, 85 for
// FP64 operands (no spills at 4 gathers in flight per group).
#include <cub/cub.cuh>
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <string>
#include <type_traits>

#include "device_common.cuh"
#include "lean.cuh"
#include "ops.cuh"
#include "svdb_internal.h"

namespace svdb {

namespace {

template <typename T, int N>
struct Vec;
template <>
struct alignas(8) Vec<float, 2> { float v[2]; };
template <>
struct alignas(16) Vec<float, 4> { float v[4]; };
template <>
struct alignas(16) Vec<double, 2> { double v[2]; };
template <>
struct alignas(16) Vec<double, 4> { double v[4]; };  // two 16-byte loads
template <typename T>
struct alignas(sizeof(T)) Vec<T, 1> { T v[1]; };

template <typename T, int N>
__device__ __forceinline__ void load_cols(const T* __restrict__ p, bool vec, int ncols_here, double (&out)[N]) {
    if (vec && ncols_here == N) {
        if constexpr (sizeof(T) * N <= 16) {
            Vec<T, N> t = *reinterpret_cast<const Vec<T, N>*>(p);
#pragma unroll
            for (int j = 0; j < N; ++j) out[j] = (double)t.v[j];
        } else {
            const Vec<T, 2>* q = reinterpret_cast<const Vec<T, 2>*>(p);
#pragma unroll
            for (int h = 0; h < N / 2; ++h) {
                Vec<T, 2> t = q[h];
                out[2 * h] = (double)t.v[0];
                out[2 * h + 1] = (double)t.v[1];
            }
        }
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j) out[j] = j < ncols_here ? (double)p[j] : 0.0;
    }
}

template <typename T, int N>
__device__ __forceinline__ void store_cols(T* __restrict__ p, int ncols_here, const double (&a)[N]) {
#pragma unroll
    for (int j = 0; j < N; ++j)
        if (j < ncols_here) p[j] = (T)a[j];
}

}  // namespace

// Work per lane group and round: U gathers are issued before any of them is
// used.  The (index, value) pairs of the next 32 entries are loaded while the
// current ones are consumed.  With FP32 operands the products of one 32-entry
// chunk are summed in FP32 and the chunk sum is added to an FP64 accumulator.
template <typename VT, typename XT, typename OT, int CPL, int H, int U>
__global__ void __launch_bounds__(256, sizeof(XT) == 4 ? 4 : 3) k_spmm_seg(const int32_t* __restrict__ ci, const VT* __restrict__ val,
                                                     const int32_t* __restrict__ seg_row,
                                                     const int64_t* __restrict__ seg_beg,
                                                     const int64_t* __restrict__ seg_end, int64_t nseg,
                                                     const XT* __restrict__ X, int64_t ldx, int l, bool vec,
                                                     OT* __restrict__ Y, int64_t ldy, double* __restrict__ part) {
    using CT = typename AccOf<XT>::type;  // chunk accumulator: FP32 for FP32 operands
    constexpr int GL = 32 / H;
    const int lane = threadIdx.x & 31;
    const int g = lane / GL, gl = lane % GL;
    const int col0 = gl * CPL;
    const int ncols_here = (l - col0) < CPL ? (l - col0) : CPL;
    const bool active = ncols_here > 0;
    const bool full = vec && ncols_here == CPL;
    const int64_t gwarp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t s = gwarp; s < nseg; s += nwarps) {
        const int32_t rr = __ldg(seg_row + s);
        const int64_t a = __ldg(seg_beg + s), b = __ldg(seg_end + s);
        double acc[CPL];
#pragma unroll
        for (int j = 0; j < CPL; ++j) acc[j] = 0.0;
        int32_t myc = 0;
        VT myv = VT(0);
        if (a + lane < b) { myc = __ldg(ci + a + lane); myv = __ldg(val + a + lane); }
        for (int64_t k0 = a; k0 < b; k0 += 32) {
            const int cnt = (b - k0) < 32 ? (int)(b - k0) : 32;
            // prefetch the next 32 pairs
            int32_t nc = 0;
            VT nv = VT(0);
            if (k0 + 32 + lane < b) { nc = __ldg(ci + k0 + 32 + lane); nv = __ldg(val + k0 + 32 + lane); }
            CT cacc[CPL];
#pragma unroll
            for (int j = 0; j < CPL; ++j) cacc[j] = CT(0);
            for (int qb = 0; qb < cnt; qb += H * U) {
                XT xv[U][CPL];
                CT vq[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int q = qb + u * H + g;
                    const int32_t c = __shfl_sync(0xffffffffu, myc, q & 31);
                    const VT v = __shfl_sync(0xffffffffu, myv, q & 31);
                    const bool ok = q < cnt && active;
                    vq[u] = ok ? (CT)v : CT(0);
                    const XT* p = X + (int64_t)c * ldx + col0;
                    if (ok && full) {
                        if constexpr (sizeof(XT) * CPL <= 16) {
                            const Vec<XT, CPL> t = *reinterpret_cast<const Vec<XT, CPL>*>(p);
#pragma unroll
                            for (int j = 0; j < CPL; ++j) xv[u][j] = t.v[j];
                        } else {
#pragma unroll
                            for (int h = 0; h < CPL / 2; ++h) {
                                const Vec<XT, 2> t = reinterpret_cast<const Vec<XT, 2>*>(p)[h];
                                xv[u][2 * h] = t.v[0];
                                xv[u][2 * h + 1] = t.v[1];
                            }
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < CPL; ++j) xv[u][j] = (ok && j < ncols_here) ? p[j] : XT(0);
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int j = 0; j < CPL; ++j) cacc[j] = fma(vq[u], (CT)xv[u][j], cacc[j]);
            }
#pragma unroll
            for (int j = 0; j < CPL; ++j) acc[j] += (double)cacc[j];
            myc = nc;
            myv = nv;
        }
        if (H == 2) {
#pragma unroll
            for (int j = 0; j < CPL; ++j) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], 16);
        }
        if (g == 0 && active) {
            if (rr >= 0) store_cols<OT, CPL>(Y + (int64_t)rr * ldy + col0, ncols_here, acc);
            else store_cols<double, CPL>(part + s * (int64_t)l + col0, ncols_here, acc);
        }
    }
}

// Lean gather kernel: values and dense operand of one type T (float or
// double), rows of X 16-byte aligned and a multiple of 16 bytes apart.  A warp
// takes a segment; its H groups of GL = 32 / H lanes take entries g, g + H, ...
// of each 32-entry chunk, and a lane owns NL vectors of VEC = 16 / sizeof(T)
// columns, GL * VEC columns apart, so that every gather instruction reads
// contiguous bytes of a row.  FP32 sums within a chunk and FP64 across chunks
// for float, FP64 throughout for double: the summation order of k_spmm_seg.
//
// What bounds it: the gathered rows, through L1 and L2 (15-17 TB/s of rows).
// At FP64 a lane that owned four neighbouring columns read them as two 16-byte
// loads at a 32-byte stride, so each load touched every sector of the row: L1
// at 97 % of its peak, half of it for bytes already read.  With the vectors
// GL * VEC apart the same loads are dense: 1,133 -> 914 us for A X of
// 50,000 x 30,000, 28 M nonzeros, l = 60.
//
// A chunk's row offsets and values are written once to per-warp shared
// buffers, a group's entries side by side, and read back four at a time by
// broadcast (a 16-byte struct per entry took an LDS.128 each, 914 -> 812 us).
// Offsets are 32-bit byte offsets from X where X is below 4 GB (BYTES: one add
// per gather), else element offsets.  A chunk runs U gathers per lane at a
// time, all issued before they are used; the last chunk of a segment runs
// masked batches of four (one entry after another, a short last chunk cost
// as much as a full one).  Tried and not kept: loading the next segment's
// bounds and first chunk ahead (928 us), and segments ordered by length with a
// CTA's warps starting together, which raised the L1 hits from 7 to 26 % and
// gained 3 % on long rows but lost 10 % on A^T X.
constexpr int kLeanWarps = 8;
template <typename T, typename OT, int H, int NL, int U, int MINB, bool BYTES>
__global__ void __launch_bounds__(kLeanWarps * 32, MINB)
    k_spmm_lean(const int32_t* __restrict__ ci, const T* __restrict__ val, const int32_t* __restrict__ seg_row,
                const int64_t* __restrict__ seg_beg, const int64_t* __restrict__ seg_end, int64_t nseg,
                const T* __restrict__ X, uint32_t ldx, int l, OT* __restrict__ Y, int64_t ldy, int yvec,
                double* __restrict__ part) {
    using CT = typename AccOf<T>::type;  // chunk sums: FP32 for float, FP64 for double
    constexpr int VEC = 16 / (int)sizeof(T);
    constexpr int GL = 32 / H;   // lanes per group
    using Slots = LeanSlots<T, H>;
    __shared__ __align__(16) uint32_t s_off[kLeanWarps][32];
    __shared__ __align__(16) T s_val[kLeanWarps][H * Slots::VS];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int g = lane / GL, gl = lane % GL;
    bool active[NL];
    uint32_t col[NL];
#pragma unroll
    for (int j = 0; j < NL; ++j) {
        const int c = (j * GL + gl) * VEC;
        active[j] = c < l;
        col[j] = active[j] ? (uint32_t)c : 0u;
    }
    const uint32_t scale = BYTES ? ldx * (uint32_t)sizeof(T) : ldx;
    uint32_t* const oput = s_off[w] + Slots::off(lane);
    T* const vput = s_val[w] + Slots::val(lane);
    const uint32_t* const og = s_off[w] + g * Slots::PER;
    const T* const vg = s_val[w] + g * Slots::VS;
    const int64_t gwarp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t sg = gwarp; sg < nseg; sg += nwarps) {
        const int32_t rr = __ldg(seg_row + sg);
        const int64_t a = __ldg(seg_beg + sg);
        int left = (int)(__ldg(seg_end + sg) - a);
        const int32_t* cp = ci + a + lane;
        const T* vp = val + a + lane;
        double acc[NL][VEC];
#pragma unroll
        for (int j = 0; j < NL; ++j)
#pragma unroll
            for (int e = 0; e < VEC; ++e) acc[j][e] = 0.0;
        int32_t myc = 0;
        T myv = T(0);
        if (lane < left) { myc = __ldg(cp); myv = __ldg(vp); }
        for (; left > 0; left -= 32) {
            __syncwarp();  // the previous chunk's entries have been read
            *oput = (uint32_t)myc * scale;
            *vput = myv;
            __syncwarp();
            cp += 32;
            vp += 32;
            if (lane + 32 < left) { myc = __ldg(cp); myv = __ldg(vp); }  // the next chunk's, while this one is used
            CT cs[NL][VEC];
#pragma unroll
            for (int j = 0; j < NL; ++j)
#pragma unroll
                for (int e = 0; e < VEC; ++e) cs[j][e] = CT(0);
            lean_chunk<T, H, NL, U, BYTES>(og, vg, left, g, X, col, active, cs);
#pragma unroll
            for (int j = 0; j < NL; ++j)
#pragma unroll
                for (int e = 0; e < VEC; ++e) acc[j][e] += (double)cs[j][e];
        }
#pragma unroll
        for (int o = GL; o < 32; o <<= 1)
#pragma unroll
            for (int j = 0; j < NL; ++j)
#pragma unroll
                for (int e = 0; e < VEC; ++e) acc[j][e] += __shfl_xor_sync(0xffffffffu, acc[j][e], o);
        if (g != 0) continue;
#pragma unroll
        for (int j = 0; j < NL; ++j) {
            if (!active[j]) continue;
            const int here = l - (int)col[j];
            if (rr >= 0) {
                OT* o = Y + (int64_t)rr * ldy + col[j];
                if (yvec && here >= VEC) {
                    struct alignas(sizeof(OT) * VEC > 16 ? 16 : sizeof(OT) * VEC) Row { OT v[VEC]; };
                    Row t;
#pragma unroll
                    for (int e = 0; e < VEC; ++e) t.v[e] = (OT)acc[j][e];
                    *reinterpret_cast<Row*>(o) = t;
                } else {
                    store_cols<OT, VEC>(o, here, acc[j]);
                }
            } else {
                store_cols<double, VEC>(part + sg * (int64_t)l + col[j], here, acc[j]);
            }
        }
    }
}

// A block of cut rows: 8 >> cls warps per row, 1 << cls rows from cut.rows[p0];
// class 0 walks one row of any length in rounds, the others' rows fit their warps.
// Not inlined: the rest of k_spmm_cut then compiles as k_spmm_lean does (in one
// loop with it, or inlined beside it, it cost the FP64 products 10-20 %).
template <typename T, typename OT, int VEC, int H, int NL, int U, bool BYTES>
__device__ __noinline__ void cut_block(const int32_t* __restrict__ ci, const T* __restrict__ val,
                                       const int64_t* __restrict__ ptr, const CutRows* cut, const T* __restrict__ X,
                                       uint32_t ldx, int l, OT* __restrict__ Y, int ldy) {
    using CT = typename AccOf<T>::type;  // chunk sums: FP32 for float, FP64 for double
    constexpr int GL = 32 / H;  // lanes per group
    constexpr int COLS = GL * NL * VEC;
    using Slots = LeanSlots<T, H>;
    extern __shared__ __align__(16) double cut_sums[];
    __shared__ __align__(16) uint32_t s_off[kLeanWarps][32];
    __shared__ __align__(16) T s_val[kLeanWarps][H * Slots::VS];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int g = lane / GL, gl = lane % GL;
    bool active[NL];
    uint32_t col[NL];
#pragma unroll
    for (int j = 0; j < NL; ++j) {
        const int c = (j * GL + gl) * VEC;
        active[j] = c < l;
        col[j] = active[j] ? (uint32_t)c : 0u;
    }
    const uint32_t scale = BYTES ? ldx * (uint32_t)sizeof(T) : ldx;
    uint32_t* const oput = s_off[w] + Slots::off(lane);
    T* const vput = s_val[w] + Slots::val(lane);
    const uint32_t* const og = s_off[w] + g * Slots::PER;
    const T* const vg = s_val[w] + g * Slots::VS;
    int cls = 0, p0 = blockIdx.x;
    for (; p0 >= cut->items(cls); ++cls) p0 -= cut->items(cls);
    p0 = cut->first[cls] + (p0 << cls);
    const int pend = cut->first[cls + 1], width = kLeanWarps >> cls, p = p0 + w / width;
    int64_t beg = 0, n = 0;
    if (p < pend) {
        const int32_t r = __ldg(cut->rows + p);
        beg = __ldg(ptr + r);
        n = __ldg(ptr + r + 1) - beg;
    }
    const int rounds = cls == 0 ? (int)((n + cut->len * kLeanWarps - 1) / (cut->len * kLeanWarps)) : 1;
    double carry = 0.0;
    for (int q = 0; q < rounds; ++q) {
        const int64_t at = (int64_t)(q * kLeanWarps + w % width) * cut->len, a = beg + at;
        int left = (int)max((int64_t)0, min((int64_t)cut->len, n - at));
        const int32_t* cp = ci + a + lane;
        const T* vp = val + a + lane;
        double acc[NL][VEC];
#pragma unroll
        for (int j = 0; j < NL; ++j)
#pragma unroll
            for (int e = 0; e < VEC; ++e) acc[j][e] = 0.0;
        int32_t myc = 0;
        T myv = T(0);
        if (lane < left) { myc = __ldg(cp); myv = __ldg(vp); }
        for (; left > 0; left -= 32) {
            __syncwarp();  // the previous chunk's entries have been read
            *oput = (uint32_t)myc * scale;
            *vput = myv;
            __syncwarp();
            cp += 32;
            vp += 32;
            if (lane + 32 < left) { myc = __ldg(cp); myv = __ldg(vp); }  // the next chunk's, while this one is used
            CT cs[NL][VEC];
#pragma unroll
            for (int j = 0; j < NL; ++j)
#pragma unroll
                for (int e = 0; e < VEC; ++e) cs[j][e] = CT(0);
            lean_chunk<T, H, NL, U, BYTES, VEC>(og, vg, left, g, X, col, active, cs);
#pragma unroll
            for (int j = 0; j < NL; ++j)
#pragma unroll
                for (int e = 0; e < VEC; ++e) acc[j][e] += (double)cs[j][e];
        }
#pragma unroll
        for (int o = GL; o < 32; o <<= 1)
#pragma unroll
            for (int j = 0; j < NL; ++j)
#pragma unroll
                for (int e = 0; e < VEC; ++e) acc[j][e] += __shfl_xor_sync(0xffffffffu, acc[j][e], o);
        if (g == 0) {
#pragma unroll
            for (int j = 0; j < NL; ++j)
#pragma unroll
                for (int e = 0; e < VEC; ++e) cut_sums[w * COLS + (j * GL + gl) * VEC + e] = acc[j][e];
        }
        __syncthreads();
        for (int t = threadIdx.x; t < (l << cls); t += kLeanWarps * 32) {  // at most once a thread in class 0
            const int slot = t / l, c = t - slot * l;
            double tot = carry;
            for (int u = 0; u < width; ++u) tot += cut_sums[(slot * width + u) * COLS + c];
            if (q + 1 < rounds) carry = tot;
            else if (p0 + slot < pend) Y[(int64_t)__ldg(cut->rows + p0 + slot) * ldy + c] = (OT)tot;
        }
        __syncthreads();
    }
}

// The same products where some rows are cut: rows of more than cut.len entries
// are the first blocks' work, longest first: 8, 4 or 2 warps take a row's
// segments, and the block adds their sums in segment order through shared memory
// (dynamic, 8 x GL NL VEC doubles); the other blocks' warps take the other rows.
// Written out as partials and added by a second kernel, a product of 10^5 to 10^6
// nonzeros took an allocation and a launch more, which outlast its one kernel
// (3,000 x 1,200, 0.26 M, l = 20, FP64, A X alone: 45 us a call, here 18).
template <typename T, typename OT, int VEC, int H, int NL, int U, int MINB, bool BYTES>
__global__ void __launch_bounds__(kLeanWarps * 32, MINB)
    k_spmm_cut(const int32_t* __restrict__ ci, const T* __restrict__ val, const int64_t* __restrict__ ptr, int64_t rows,
               const __grid_constant__ CutRows cut, const T* __restrict__ X, uint32_t ldx, int l, OT* __restrict__ Y,
               int ldy, int yvec) {
    if ((int)blockIdx.x < cut.blocks) {
        cut_block<T, OT, VEC, H, NL, U, BYTES>(ci, val, ptr, &cut, X, ldx, l, Y, ldy);
        return;
    }
    using CT = typename AccOf<T>::type;  // chunk sums: FP32 for float, FP64 for double
    constexpr int GL = 32 / H;   // lanes per group
    using Slots = LeanSlots<T, H>;
    __shared__ __align__(16) uint32_t s_off[kLeanWarps][32];
    __shared__ __align__(16) T s_val[kLeanWarps][H * Slots::VS];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int g = lane / GL, gl = lane % GL;
    bool active[NL];
    uint32_t col[NL];
#pragma unroll
    for (int j = 0; j < NL; ++j) {
        const int c = (j * GL + gl) * VEC;
        active[j] = c < l;
        col[j] = active[j] ? (uint32_t)c : 0u;
    }
    const uint32_t scale = BYTES ? ldx * (uint32_t)sizeof(T) : ldx;
    uint32_t* const oput = s_off[w] + Slots::off(lane);
    T* const vput = s_val[w] + Slots::val(lane);
    const uint32_t* const og = s_off[w] + g * Slots::PER;
    const T* const vg = s_val[w] + g * Slots::VS;
    const int64_t gwarp = (int64_t)(blockIdx.x - cut.blocks) * kLeanWarps + w;
    const int64_t nwarps = (int64_t)(gridDim.x - cut.blocks) * kLeanWarps;
    for (int64_t rr = gwarp; rr < rows; rr += nwarps) {
        const int64_t a = __ldg(ptr + rr);
        const int64_t len = __ldg(ptr + rr + 1) - a;
        if (len > cut.len) continue;  // a block's
        int left = (int)len;
        const int32_t* cp = ci + a + lane;
        const T* vp = val + a + lane;
        double acc[NL][VEC];
#pragma unroll
        for (int j = 0; j < NL; ++j)
#pragma unroll
            for (int e = 0; e < VEC; ++e) acc[j][e] = 0.0;
        int32_t myc = 0;
        T myv = T(0);
        if (lane < left) { myc = __ldg(cp); myv = __ldg(vp); }
        for (; left > 0; left -= 32) {
            __syncwarp();  // the previous chunk's entries have been read
            *oput = (uint32_t)myc * scale;
            *vput = myv;
            __syncwarp();
            cp += 32;
            vp += 32;
            if (lane + 32 < left) { myc = __ldg(cp); myv = __ldg(vp); }  // the next chunk's, while this one is used
            CT cs[NL][VEC];
#pragma unroll
            for (int j = 0; j < NL; ++j)
#pragma unroll
                for (int e = 0; e < VEC; ++e) cs[j][e] = CT(0);
            lean_chunk<T, H, NL, U, BYTES, VEC>(og, vg, left, g, X, col, active, cs);
#pragma unroll
            for (int j = 0; j < NL; ++j)
#pragma unroll
                for (int e = 0; e < VEC; ++e) acc[j][e] += (double)cs[j][e];
        }
#pragma unroll
        for (int o = GL; o < 32; o <<= 1)
#pragma unroll
            for (int j = 0; j < NL; ++j)
#pragma unroll
                for (int e = 0; e < VEC; ++e) acc[j][e] += __shfl_xor_sync(0xffffffffu, acc[j][e], o);
        if (g != 0) continue;
#pragma unroll
        for (int j = 0; j < NL; ++j) {
            if (!active[j]) continue;
            const int here = l - (int)col[j];
            OT* o = Y + rr * ldy + col[j];
            if (yvec && here >= VEC) {
                struct alignas(sizeof(OT) * VEC > 16 ? 16 : sizeof(OT) * VEC) Row { OT v[VEC]; };
                Row t;
#pragma unroll
                for (int e = 0; e < VEC; ++e) t.v[e] = (OT)acc[j][e];
                *reinterpret_cast<Row*>(o) = t;
            } else {
                store_cols<OT, VEC>(o, here, acc[j]);
            }
        }
    }
}

// rows split into several segments: add their partials in segment order
template <typename OT>
__global__ void k_spmm_merge(const int64_t* __restrict__ seg_first, const int32_t* __restrict__ multi_rows,
                             int64_t nmulti, const double* __restrict__ part, int l, OT* __restrict__ Y,
                             int64_t ldy) {
    const int lane = threadIdx.x & 31;
    const int64_t gwarp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t t = gwarp; t < nmulti; t += nwarps) {
        const int64_t r = multi_rows[t];
        const int64_t f = seg_first[r], f1 = seg_first[r + 1];
        for (int c = lane; c < l; c += 32) {
            double acc = 0.0;
            for (int64_t s = f; s < f1; ++s) acc += part[s * (int64_t)l + c];
            Y[r * ldy + c] = (OT)acc;
        }
    }
}

// ------------------------------------------------------------- the plan --
// SpMM segment length of a structure, a power of two.  Rows longer than it are
// cut, so that one long row does not outlast the rest of the product.
//  - Up to kCutNnz entries a cut row is one block's (k_spmm_cut): the length at
//    which the resident warps (24 an SM) get two segments' worth of entries each,
//    and no less than the mean row, or most rows would be cut (unless there are
//    too few rows to fill the warps).  At half of it the
//    blocks' idle warps cost more than the shorter chains give (40,000 x 9,000,
//    1.1 M, A^T X, l = 60, FP64, three streams: 42 us a call against 36), at twice
//    the mean the chains are back (2,000 x 2,000, 0.47 M: 39 us against 25).
//  - Above, cut rows are merged from partials (k_spmm_merge), whose allocation and
//    launch no longer outweigh the balance: four segments a warp (but where the
//    rows are even enough: cut_in_blocks).  At 2,048 throughout, A^T X of a
//    30,011 x 8,009 matrix (3.1 M, columns up to a few thousand entries, l = 40)
//    took 196 us, at 256 85.
// kCutNnz: A^T X, l = 60, FP64, alone / on three streams, by blocks and merged: at
// 1.1 M 54 / 35 and 62 / 32 us, at 2.2 M 92 / 70 and 92 / 64, at 4.2 M 163 / 127
// and 151 / 116.
constexpr int64_t kCutNnz = 1 << 21;
static int64_t seg_len_for(int64_t nnz) {
    int64_t len = 128;
    while (len < kSegNnz && len * 4 * device_props().sms * 24 < nnz) len *= 2;
    return len;
}
static int64_t cut_len_for(int64_t nnz, int64_t rows) {
    const int64_t warps = (int64_t)device_props().sms * 24;
    int64_t len = 128;
    while (len < kSegNnz && (len * 2 * warps < nnz || (rows * 4 >= warps && len * rows < nnz))) len *= 2;
    return len;
}
__global__ void k_seg_count(const int64_t* __restrict__ rp, int64_t rows, int64_t seg, int64_t* __restrict__ cnt) {
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r <= rows; r += (int64_t)gridDim.x * blockDim.x) {
        if (r == rows) { cnt[r] = 0; continue; }
        const int64_t len = rp[r + 1] - rp[r];
        cnt[r] = len <= seg ? 1 : (len + seg - 1) / seg;
    }
}
__global__ void k_seg_fill(const int64_t* __restrict__ rp, const int64_t* __restrict__ first, int64_t rows,
                           int64_t seg, int32_t* __restrict__ seg_row, int64_t* __restrict__ seg_beg,
                           int64_t* __restrict__ seg_end, int32_t* __restrict__ multi_rows,
                           unsigned long long* __restrict__ counts) {
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < rows; r += (int64_t)gridDim.x * blockDim.x) {
        const int64_t f = first[r], f1 = first[r + 1], e = rp[r + 1];
        const bool multi = f1 - f > 1;
        for (int64_t s = f; s < f1; ++s) {
            const int64_t a = rp[r] + (s - f) * seg;
            seg_row[s] = multi ? -(int32_t)r - 1 : (int32_t)r;
            seg_beg[s] = a;
            seg_end[s] = (a + seg < e) ? a + seg : e;
        }
        // the list's order is irrelevant to the sums
        if (multi) multi_rows[atomicAdd(counts, 1ull)] = (int32_t)r;
    }
}

// counts[1] = the most entries in one of 16 equal row ranges
__global__ void k_slice16(const int64_t* __restrict__ rp, int64_t rows, unsigned long long* __restrict__ counts) {
    const int64_t per = slice16_rows(rows);
    const int64_t r0 = min(rows, threadIdx.x * per), r1 = min(rows, r0 + per);
    if (threadIdx.x < 16) atomicMax(counts + 1, (unsigned long long)(rp[r1] - rp[r0]));
}

// Sort key of a row's SpMV class, longest first, and counts[2 ..]: the rows
// of more than kSegNnz entries, then those of each bin.  Above 64 entries a
// class is a quarter octave of the length (by octaves A x of the Zipf operator
// in k_spmv's comment took 136 us, against 130); below, one bin, so that rows
// next to each other in memory, which share cache lines, stay together.  A class
// ends at its upper length (2^e + q 2^(e-2), inclusive), so no class holds rows on
// both sides of a bin's or the long rows' bound.
constexpr int kSpmvKeyBits = 7;
constexpr int kKeyCounts = kSpmvBins + 1 + 4;  // and the rows of more than kCutMax, 4, 2 and 1 cut_len entries
__global__ void k_spmv_keys(const int64_t* __restrict__ rp, int64_t rows, int64_t cut_len, uint8_t* __restrict__ key,
                            int32_t* __restrict__ ids, unsigned long long* __restrict__ counts) {
    __shared__ unsigned int sc[kKeyCounts];
    if (threadIdx.x < kKeyCounts) sc[threadIdx.x] = 0;
    __syncthreads();
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < rows; r += (int64_t)gridDim.x * blockDim.x) {
        const int64_t len = rp[r + 1] - rp[r];
        int c = 0;  // 0: one block, c: bin c - 1
        while (c < kSpmvBins && len <= spmv_bin_len(c)) ++c;
        if (c < 2) {
            const int64_t k = len - 1;
            const int e = min(63 - __clzll(k), 31);
            key[r] = (uint8_t)(127 - 4 * e - (int)((k >> (e - 2)) & 3));
        } else {
            key[r] = (uint8_t)(104 + c);  // 65 entries: 103
        }
        ids[r] = (int32_t)r;
        atomicAdd(sc + c, 1u);
        if (len > cut_len) {
            unsigned int* cut = sc + kSpmvBins + 1;
            atomicAdd(cut + 3, 1u);
            if (len > 2 * cut_len) atomicAdd(cut + 2, 1u);
            if (len > 4 * cut_len) atomicAdd(cut + 1, 1u);
            if (len > kCutMax) atomicAdd(cut, 1u);
        }
    }
    __syncthreads();
    if (threadIdx.x < kKeyCounts && sc[threadIdx.x])
        atomicAdd(counts + 2 + threadIdx.x, (unsigned long long)sc[threadIdx.x]);
}

static int nblk(int64_t work, int threads, int per_sm) {
    int64_t b = (work + threads - 1) / threads;
    return (int)std::max<int64_t>(1, std::min<int64_t>(b, (int64_t)device_props().sms * per_sm));
}

void build_seg_plan(DevCompressed& m, cudaStream_t s) {
    SegPlan& p = m.plan;
    const int64_t rows = m.nmajor;
    p.seg_first.alloc(rows + 1, s);
    if (rows == 0) {
        SVDB_CUDA(cudaMemsetAsync(p.seg_first.p, 0, sizeof(int64_t), s));
        p.nseg = p.nmulti = p.nlong = 0;
        return;
    }
    const int64_t seg = seg_len_for(m.nnz), cut = cut_len_for(m.nnz, rows);
    p.multi_rows.alloc(rows, s);
    p.bin_rows.alloc(rows, s);
    // One scratch allocation for all temporaries: an allocation takes 10-25 us
    // where the pool's free blocks belong to other streams.
    constexpr int kCounts = 2 + kKeyCounts;
    size_t tb = 0, tb2 = 0;
    SVDB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, (int64_t*)nullptr, p.seg_first.p, rows + 1, s));
    SVDB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb2, (uint8_t*)nullptr, (uint8_t*)nullptr, (int32_t*)nullptr,
                                              p.bin_rows.p, rows, 0, kSpmvKeyBits, s));
    size_t bytes = 0;
    auto piece = [&](size_t n) {
        const size_t at = bytes;
        bytes += (n + 255) / 256 * 256;
        return at;
    };
    const size_t o_cnt = piece((rows + 1) * sizeof(int64_t)), o_nm = piece(kCounts * sizeof(unsigned long long)),
                 o_key = piece(rows), o_skey = piece(rows), o_ids = piece(rows * sizeof(int32_t)),
                 o_cub = piece(std::max(tb, tb2));
    DevBuf<uint8_t> scratch(bytes, s);
    int64_t* cnt = reinterpret_cast<int64_t*>(scratch.p + o_cnt);
    unsigned long long* nm = reinterpret_cast<unsigned long long*>(scratch.p + o_nm);
    uint8_t *key = scratch.p + o_key, *skey = scratch.p + o_skey, *cub_tmp = scratch.p + o_cub;
    int32_t* ids = reinterpret_cast<int32_t*>(scratch.p + o_ids);

    k_seg_count<<<nblk(rows + 1, 256, 16), 256, 0, s>>>(m.ptr.p, rows, seg, cnt);
    SVDB_CHECK_LAUNCH();
    SVDB_CUDA(cub::DeviceScan::ExclusiveSum(cub_tmp, tb, cnt, p.seg_first.p, rows + 1, s));
    int64_t nseg = 0;
    SVDB_CUDA(cudaMemcpyAsync(&nseg, p.seg_first.p + rows, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    SVDB_CUDA(cudaStreamSynchronize(s));
    p.nseg = nseg;
    p.seg_row.alloc(std::max<int64_t>(nseg, 1), s);
    p.seg_beg.alloc(std::max<int64_t>(nseg, 1), s);
    p.seg_end.alloc(std::max<int64_t>(nseg, 1), s);
    SVDB_CUDA(cudaMemsetAsync(nm, 0, kCounts * sizeof(unsigned long long), s));
    k_seg_fill<<<nblk(rows, 256, 16), 256, 0, s>>>(m.ptr.p, p.seg_first.p, rows, seg, p.seg_row.p, p.seg_beg.p,
                                                   p.seg_end.p, p.multi_rows.p, nm);
    SVDB_CHECK_LAUNCH();
    const bool slices = slice16_counted(m.nnz);
    if (slices) {
        k_slice16<<<1, 32, 0, s>>>(m.ptr.p, rows, nm);
        SVDB_CHECK_LAUNCH();
    }
    // SpMV order: the rows' length classes, longest first, by one stable sort
    k_spmv_keys<<<nblk(rows, 256, 16), 256, 0, s>>>(m.ptr.p, rows, cut, key, ids, nm);
    SVDB_CHECK_LAUNCH();
    SVDB_CUDA(cub::DeviceRadixSort::SortPairs(cub_tmp, tb2, key, skey, ids, p.bin_rows.p, rows, 0, kSpmvKeyBits, s));
    unsigned long long hm[kCounts];
    SVDB_CUDA(cudaMemcpyAsync(hm, nm, sizeof(hm), cudaMemcpyDeviceToHost, s));
    SVDB_CUDA(cudaStreamSynchronize(s));
    p.nmulti = (int64_t)hm[0];
    p.slice16_nnz = slices ? (int64_t)hm[1] : kSlice16Unknown;
    p.nlong = (int64_t)hm[2];
    int64_t off = p.nlong, items = 0;
    for (int b = 0; b < kSpmvBins; ++b) {
        const int64_t cnt = (int64_t)hm[3 + b], rpw = (int64_t)1 << b;
        p.bins.off[b] = (int32_t)off;
        p.bins.items[b] = (int32_t)items;
        off += cnt;
        items += (cnt + rpw - 1) / rpw;
    }
    p.bins.off[kSpmvBins] = (int32_t)off;
    p.bins.items[kSpmvBins] = (int32_t)items;
    p.bins.rows = p.bin_rows.p;
    // the cut rows head the same order (its length and kCutMax are class bounds)
    p.cut.rows = p.bin_rows.p;
    p.cut.len = (int)cut;
    for (int k = 0; k < 4; ++k) p.cut.first[k] = (int)hm[3 + kSpmvBins + k];
    p.cut.blocks = m.nnz < 2 * kCutNnz ? p.cut.items(0) + p.cut.items(1) + p.cut.items(2) : 0;
}

// ------------------------------------------------------------- launcher --
template <typename VT, typename XT, typename OT, int CPL, int H>
static void launch_seg(const DevCompressed& m, const VT* v, const XT* X, int64_t ldx, int lc, OT* Y, int64_t ldy,
                       double* part, cudaStream_t s, int64_t lo = 0, int64_t hi = -1) {
    if (hi < 0) hi = m.plan.nseg;
    if (hi <= lo) return;
    const uintptr_t align = std::min<uintptr_t>(16, sizeof(XT) * CPL);
    const bool vec = (CPL > 1) && (ldx % CPL == 0) && ((reinterpret_cast<uintptr_t>(X) % align) == 0);
    const int blocks = nblk((hi - lo) * 32, 256, 16);
    constexpr int U = 4;
    // segment s of the range is segment lo + s of the plan; its partial row lives at part[(lo + s) * lc]
    k_spmm_seg<VT, XT, OT, CPL, H, U><<<blocks, 256, 0, s>>>(m.idx.p, v, m.plan.seg_row.p + lo, m.plan.seg_beg.p + lo,
                                                             m.plan.seg_end.p + lo, hi - lo, X, ldx, lc, vec, Y,
                                                             ldy, part ? part + lo * (int64_t)lc : nullptr);
    SVDB_CHECK_LAUNCH();
}

// SVDB_SPMM=seg keeps k_spmm_seg, for comparisons
static bool lean_off() {
    const char* e = getenv("SVDB_SPMM");
    return e && std::string(e) == "seg";
}

// k_spmm_lean takes X as it is: rows 16-byte aligned, 32-bit element offsets
template <typename T>
static bool lean_aligned(const DevCompressed& m, const T* X, int64_t ldx) {
    return (ldx * (int64_t)sizeof(T)) % 16 == 0 && (reinterpret_cast<uintptr_t>(X) % 16) == 0 &&
           m.nminor * ldx < ((int64_t)1 << 31);
}

// Of the structures that have rows of several segments, those whose products of l
// columns k_spmm_cut does in one kernel, without partials and their merge:
//  - below kCutNnz, where no row is longer than kCutMax;
//  - up to 64 columns to twice that, where no row is longer than 4 cut.len;
//  - above, where no row is longer than cut.len: every row is then one warp's.
//    Above 64 columns only up to 512 entries: there a warp has one row of X in
//    flight per vector, and the longer chains show.
// In one kernel and merged, A X, alone / on one stream in turn: 45,477 x 21,986
// (2.8 M, rows of up to 374) at l = 24, FP64, 67 / 60 and 88 / 64 us; 32,169 x 10,970
// (3.9 M, up to 540) at l = 60, FP32, 82 / 74 and 96 / 80; 8,465 x 6,126 (2.3 M, up
// to 910) at l = 44, FP32, 55 / 47 and 66 / 50; and where it is merged, 23,109 x
// 11,277 (3.9 M, up to 964) at l = 120, FP32, 166 / 158 and 153 / 137; A^T X of
// 12,889 x 6,080 (2.4 M, up to 3,705) at l = 64, FP32, 61 / 53 and 65 / 49.
static bool cut_in_blocks(const DevCompressed& m, int l) {
    const CutRows& cut = m.plan.cut;
    if (m.plan.nmulti == 0 || cut.first[0] > 0) return false;
    if (m.nnz < kCutNnz || (m.nnz < 2 * kCutNnz && l <= 64 && cut.first[1] == 0)) return true;
    return cut.first[3] == 0 && (l <= 64 || cut.len <= 512);
}

// How launch_lean's kernels go over the rows
enum class Rows {
    kSegments,  // k_spmm_lean, a segment a warp; rows of several leave partials
    kWhole,     // k_spmm_cut
    kNarrow     // k_spmm_cut, X read element by element
};

template <typename T, typename OT, int H, int NL, int U, int MINB>
static void lean_go(const DevCompressed& m, const T* v, const T* X, int l, int64_t ldx, Rows form, OT* Y,
                    int64_t ldy, double* part, cudaStream_t s) {
    constexpr int VEC = 16 / (int)sizeof(T);
    // 8x the resident blocks: timed against the resident blocks only, 1.10
    // against 1.20 ms for A X of the 100k x 30k workload
    const int work = nblk(m.plan.nseg * 32, kLeanWarps * 32, MINB * 8);
    const int yvec = ldy % VEC == 0 && reinterpret_cast<uintptr_t>(Y) % 16 == 0;
    const bool bytes = m.nminor * ldx * (int64_t)sizeof(T) < ((int64_t)1 << 32);
    if (form != Rows::kSegments) {
        const CutRows& cut = m.plan.cut;
        auto go = [&](auto kern) {
            kern<<<cut.blocks + work, kLeanWarps * 32, (size_t)kLeanWarps * (32 / H) * NL * 16 / sizeof(T) * 8, s>>>(
                m.idx.p, v, m.ptr.p, m.nmajor, cut, X, (uint32_t)ldx, l, Y, (int)ldy, yvec);
        };
        if (form == Rows::kNarrow) go(k_spmm_cut<T, OT, 1, H, NL * VEC, 4, MINB, true>);  // four rows in flight: more spill
        else if (bytes) go(k_spmm_cut<T, OT, VEC, H, NL, U, MINB, true>);
        else go(k_spmm_cut<T, OT, VEC, H, NL, U, MINB, false>);
    } else {
        auto go = [&](auto kern) {
            kern<<<work, kLeanWarps * 32, 0, s>>>(m.idx.p, v, m.plan.seg_row.p, m.plan.seg_beg.p, m.plan.seg_end.p,
                                                  m.plan.nseg, X, (uint32_t)ldx, l, Y, ldy, yvec, part);
        };
        if (bytes) go(k_spmm_lean<T, OT, H, NL, U, MINB, true>);
        else go(k_spmm_lean<T, OT, H, NL, U, MINB, false>);
    }
    SVDB_CHECK_LAUNCH();
}

// l <= 128 columns of X (ldx apart) into Y (ldy apart).  Lane groups as narrow
// as the columns allow, so that few lanes idle.  kNarrow has VEC times the vectors
// a lane in the same groups.
template <typename T, typename OT>
static void launch_lean(const DevCompressed& m, const T* v, const T* X, int l, int64_t ldx, Rows form, OT* Y,
                        int64_t ldy, double* part, cudaStream_t s) {
    if (m.plan.nseg <= 0) return;
    if constexpr (std::is_same<T, float>::value) {
        if (l <= 16) lean_go<T, OT, 8, 1, 4, 4>(m, v, X, l, ldx, form, Y, ldy, part, s);
        else if (l <= 32) lean_go<T, OT, 4, 1, 8, 4>(m, v, X, l, ldx, form, Y, ldy, part, s);
        else if (l <= 64) lean_go<T, OT, 2, 1, 8, 4>(m, v, X, l, ldx, form, Y, ldy, part, s);
        else lean_go<T, OT, 1, 1, 8, 4>(m, v, X, l, ldx, form, Y, ldy, part, s);
    } else {
        if (l <= 8) lean_go<T, OT, 8, 1, 4, 3>(m, v, X, l, ldx, form, Y, ldy, part, s);
        else if (l <= 16) lean_go<T, OT, 4, 1, 8, 3>(m, v, X, l, ldx, form, Y, ldy, part, s);
        else if (l <= 32) lean_go<T, OT, 4, 2, 4, 3>(m, v, X, l, ldx, form, Y, ldy, part, s);
        else if (l <= 48) lean_go<T, OT, 4, 3, 4, 2>(m, v, X, l, ldx, form, Y, ldy, part, s);
        else if (l <= 64) lean_go<T, OT, 2, 2, 4, 3>(m, v, X, l, ldx, form, Y, ldy, part, s);
        else lean_go<T, OT, 1, 2, 4, 3>(m, v, X, l, ldx, form, Y, ldy, part, s);
    }
}

// out (rows x ldx) = in (rows x l), zero past column l; rows * ldx < 2^31
template <typename T>
__global__ void k_pad_rows(const T* __restrict__ in, T* __restrict__ out, uint32_t n, uint32_t l, uint32_t ldx) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t r = i / ldx, c = i - r * ldx;
        out[i] = c < l ? in[r * l + c] : T(0);
    }
}

template <typename OT>
static void merge_rows(const DevCompressed& m, const double* part, int l, OT* Y, int64_t ldy, cudaStream_t s) {
    k_spmm_merge<OT><<<nblk(m.plan.nmulti * 32, 256, 16), 256, 0, s>>>(m.plan.seg_first.p, m.plan.multi_rows.p,
                                                                      m.plan.nmulti, part, l, Y, ldy);
    SVDB_CHECK_LAUNCH();
}

// The operand the lean kernels read: X itself, or a copy in `buf` where its rows
// are no whole 16-byte vectors (odd l, unaligned X).  A copy is an allocation and
// a launch, 10-17 us of a call that runs alone, so small products read X as it is,
// element by element (narrow: k_spmm_cut in the same lane groups, the same bits):
// up to 2^24 gathered elements, 2^25 above 64 columns, and at FP64 above 64 columns
// always.  A X of 20,000 x 6,000, 1.07 M, alone / on three streams, narrow and
// copied, us: l = 7 (2^23) FP32 27 / 13 and 37 / 13; l = 23 (2^24.5) FP32 39 / 22
// and 42 / 17, FP64 43 / 27 and 54 / 26; l = 63 (2^26) FP32 50 / 31 and 51 / 24, FP64
// 83 / 56 and 68 / 38; l = 101 (2^26.7) FP32 85 / 54 and 70 / 36, FP64 91 / 65 and
// 107 / 66.  A copy that cannot be allocated is done without.  Null: k_spmm_seg
// takes X as it is (also fewer entries than rows of X, and 2^31 elements or more).
// Rows padded further, to whole 128-byte lines, were no faster (50,000 x 30,000,
// 28 M nonzeros, l = 60: 805 against 812 us FP64, 865 against 870 FP32 at 100,000
// rows): the gathers run at 15-17 TB/s of rows, near what L2 delivers.
template <typename T>
static const T* lean_operand(const DevCompressed& m, const T* X, int l, int64_t& ldx, bool& narrow, DevBuf<T>& buf,
                             cudaStream_t s) {
    constexpr bool f32 = sizeof(T) == 4;
    narrow = false;
    ldx = l;
    if (lean_off()) return nullptr;
    if (lean_aligned(m, X, ldx)) return X;
    const int64_t gathered = m.nnz * l;
    const bool can = m.nnz < kCutNnz && m.plan.cut.first[0] == 0 &&
                     m.nminor * ldx * (int64_t)sizeof(T) < ((int64_t)1 << 32);
    if (can && ((!f32 && l > 64) || gathered <= ((int64_t)1 << (l > 64 ? 25 : 24)) || m.nnz < m.nminor)) {
        narrow = true;
        return X;
    }
    constexpr int64_t VEC = 16 / (int64_t)sizeof(T);
    const int64_t ldc = (l + VEC - 1) / VEC * VEC;
    if (m.nnz < m.nminor || m.nminor * ldc >= ((int64_t)1 << 31)) return nullptr;
    try {
        buf.alloc(std::max<int64_t>(m.nminor * ldc, 1), s);
    } catch (const Error& e) {
        if (e.code != SVDB_ERR_OOM) throw;
        cudaGetLastError();
        narrow = can;
        return can ? X : nullptr;
    }
    ldx = ldc;
    k_pad_rows<T><<<nblk(m.nminor * ldx, 256, 16), 256, 0, s>>>(X, buf.p, (uint32_t)(m.nminor * ldx), (uint32_t)l,
                                                               (uint32_t)ldx);
    SVDB_CHECK_LAUNCH();
    return buf.p;
}

template <typename T, typename OT>
static void lean_product(const DevCompressed& m, const T* v, const T* X, int l, int64_t ldx, bool narrow, OT* Y,
                         int64_t ldy, cudaStream_t s) {
    const Rows form = narrow ? Rows::kNarrow : cut_in_blocks(m, l) ? Rows::kWhole : Rows::kSegments;
    const int64_t merged = form == Rows::kSegments ? m.plan.nmulti : 0;
    DevBuf<double> part;
    if (merged) part.alloc(m.plan.nseg * (int64_t)std::min(l, 128), s);
    for (int c0 = 0; c0 < l; c0 += 128) {
        const int lc = std::min(128, l - c0);
        launch_lean<T, OT>(m, v, X + c0, lc, ldx, form, Y + c0, ldy, part.p, s);
        if (merged) merge_rows(m, part.p, lc, Y + c0, ldy, s);
    }
}

template <typename VT, typename XT, typename OT>
static void spmm_impl(const DevCompressed& m, const VT* v, const XT* X, int l, OT* Y, cudaStream_t s) {
    if constexpr (std::is_same<VT, XT>::value) {
        DevBuf<XT> buf;
        int64_t ldx = 0;
        bool narrow = false;
        const XT* Xa = lean_operand(m, X, l, ldx, narrow, buf, s);
        if (Xa) {
            lean_product<VT, OT>(m, v, Xa, l, ldx, narrow, Y, l, s);
            return;
        }
    }
    DevBuf<double> part;
    if (m.plan.nmulti) part.alloc(m.plan.nseg * (int64_t)std::min(l, 128), s);
    for (int c0 = 0; c0 < l; c0 += 128) {
        const int lc = std::min(128, l - c0);
        const XT* Xc = X + c0;
        OT* Yc = Y + c0;
        if (lc <= 32) launch_seg<VT, XT, OT, 2, 2>(m, v, Xc, l, lc, Yc, l, part.p, s);
        else if (lc <= 64) launch_seg<VT, XT, OT, 4, 2>(m, v, Xc, l, lc, Yc, l, part.p, s);
        else launch_seg<VT, XT, OT, 4, 1>(m, v, Xc, l, lc, Yc, l, part.p, s);
        if (part.p) merge_rows(m, part.p, lc, Yc, l, s);
    }
}


// ------------------------------------------------------ TMA row gathers --
// FP32 dense operand, FP32 matrix values: the rows X[c] of a chunk of 32
// entries are fetched by the tensor memory accelerator (tile::gather4: four
// rows of one box each, the box one row high and BOXW columns wide; columns
// past l read as zero) into a per-warp shared-memory ring of kTS chunks, so
// the bytes in flight cost no registers.  Each warp owns whole segments of
// the plan; a chunk's sums are FP32, chunks are added in FP64 as in
// k_spmm_seg.  Waits on the ring's mbarriers give up after 2 s of
// %globaltimer and raise g_tma_err (read by spmm_tma_check).
constexpr int kTW = 8;   // warps per CTA
constexpr int kTS = 3;   // chunks in flight per warp
constexpr int kTE = 32;  // entries per chunk
__device__ int g_tma_err;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint64_t gtimer() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, uint64_t limit_ns) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = gtimer();
    while (!mbar_try_wait(bar, parity))
        if (gtimer() - t0 > limit_ns) return false;
    return true;
}

template <typename OT, int BOXW>
__global__ void __launch_bounds__(kTW * 32, 1) k_spmm_tma(const __grid_constant__ CUtensorMap xmap,
                                                           const int32_t* __restrict__ ci,
                                                           const float* __restrict__ val,
                                                           const int32_t* __restrict__ seg_row,
                                                           const int64_t* __restrict__ seg_beg,
                                                           const int64_t* __restrict__ seg_end, int64_t nseg, int l,
                                                           OT* __restrict__ Y, int64_t ldy,
                                                           double* __restrict__ part) {
    constexpr int ROWB = BOXW * 4;            // bytes of one gathered row
    constexpr int CHUNKB = kTE * ROWB;        // bytes of one chunk
    constexpr int CPL = BOXW / 32;            // columns per lane
    const unsigned full = 0xffffffffu;
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t bars[kTW][kTS];
    __shared__ float svals[kTW][kTS][kTE];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (smem_u32(smem) & 127) {  // TMA destinations need 128-byte alignment
        if (threadIdx.x == 0) atomicOr(&g_tma_err, 2);
        return;
    }
    unsigned char* ring = smem + (size_t)w * kTS * CHUNKB;
    if (lane == 0) {
        for (int st = 0; st < kTS; ++st)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bars[w][st])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    const int64_t nw = (int64_t)gridDim.x * kTW;
    int64_t i_sg = blockIdx.x * (int64_t)kTW + w, i_k0 = i_sg < nseg ? seg_beg[i_sg] : 0;
    int64_t c_sg = i_sg, c_k0 = i_k0;
    int issued = 0, consumed = 0;

    auto issue = [&]() {
        if (i_sg >= nseg) return;
        const int64_t e = seg_end[i_sg];
        const int cnt = (int)min((int64_t)kTE, e - i_k0);
        const int st = issued % kTS;
        const int32_t cm = lane < cnt ? __ldg(ci + i_k0 + lane) : 0;
        svals[w][st][lane] = lane < cnt ? __ldg(val + i_k0 + lane) : 0.f;
        const int ng = (cnt + 3) >> 2;
        int32_t r[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int32_t cu = __shfl_sync(full, cm, (4 * lane + u) & 31);
            const int32_t cb = __shfl_sync(full, cm, (4 * lane) & 31);
            r[u] = (4 * lane + u < cnt) ? cu : cb;  // pad a short group with its first row
        }
        const uint32_t bar = smem_u32(&bars[w][st]);
        if (lane == 0)
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(ng * 4 * ROWB)
                         : "memory");
        __syncwarp();
        if (lane < ng) {
            const uint32_t dst = smem_u32(ring + st * CHUNKB + lane * 4 * ROWB);
            asm volatile(
                "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes"
                " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
                "l"(reinterpret_cast<uint64_t>(&xmap)), "r"(0), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(bar)
                : "memory");
        }
        ++issued;
        i_k0 += kTE;
        if (i_k0 >= e) {
            i_sg += nw;
            if (i_sg < nseg) i_k0 = seg_beg[i_sg];
        }
    };

#pragma unroll
    for (int p = 0; p < kTS; ++p) issue();
    double acc[CPL];
#pragma unroll
    for (int u = 0; u < CPL; ++u) acc[u] = 0.0;
    bool failed = false;
    while (consumed < issued) {
        const int st = consumed % kTS;
        if (!mbar_wait_bounded(smem_u32(&bars[w][st]), (uint32_t)((consumed / kTS) & 1), 2000000000ull)) {
            failed = true;
            break;
        }
        const int64_t e = seg_end[c_sg];
        const int cnt = (int)min((int64_t)kTE, e - c_k0);
        const float v = svals[w][st][lane];
        const float* xs = reinterpret_cast<const float*>(ring + st * CHUNKB) + CPL * lane;
        float sum[CPL];
#pragma unroll
        for (int u = 0; u < CPL; ++u) sum[u] = 0.f;
#pragma unroll 4
        for (int q = 0; q < cnt; ++q) {
            const float vq = __shfl_sync(full, v, q);
            if (CPL == 2) {
                const float2 x = *reinterpret_cast<const float2*>(xs + q * BOXW);
                sum[0] = fmaf(vq, x.x, sum[0]);
                sum[CPL - 1] = fmaf(vq, x.y, sum[CPL - 1]);
            } else {
                sum[0] = fmaf(vq, xs[q * BOXW], sum[0]);
            }
        }
#pragma unroll
        for (int u = 0; u < CPL; ++u) acc[u] += (double)sum[u];
        __syncwarp();
        ++consumed;
        c_k0 += kTE;
        if (c_k0 >= e) {
            const int32_t rr = seg_row[c_sg];
#pragma unroll
            for (int u = 0; u < CPL; ++u) {
                const int col = CPL * lane + u;
                if (col < l) {
                    if (rr >= 0) Y[(int64_t)rr * ldy + col] = (OT)acc[u];
                    else part[c_sg * (int64_t)l + col] = acc[u];
                }
                acc[u] = 0.0;
            }
            c_sg += nw;
            if (c_sg < nseg) c_k0 = seg_beg[c_sg];
        }
        issue();
    }
    if (failed) {
        if (lane == 0) atomicOr(&g_tma_err, 1);
        // let the copies already issued land before the ring goes away (bounded)
        for (; consumed < issued; ++consumed)
            mbar_wait_bounded(smem_u32(&bars[w][consumed % kTS]), (uint32_t)((consumed / kTS) & 1), 100000000ull);
    }
}

static PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        cudaDriverEntryPointQueryResult q;
        void* p = nullptr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

// TMA path (opt-in, SVDB_SPMM=tma): FP32 operand with contiguous rows of l
// (a multiple of 4, at most 64) on a 16-byte aligned base.  On B200 it moved
// about 4.9 TB/s of 256-byte rows against 7.4 TB/s for the register gathers
// of k_spmm_seg (100,000 x 30,000, 65 M nonzeros, l = 60), and splitting the
// segments between the two kernels on two streams was no faster than
// k_spmm_seg alone: both are held by the same L2 gather traffic.  So it is
// not the default; the variable is read on every call.
static bool tma_eligible(const void* X, int l, int64_t ldx) {
    const char* e = getenv("SVDB_SPMM");
    const bool on = e && std::string(e) == "tma";
    return on && ldx == l && l % 4 == 0 && l <= 64 && (reinterpret_cast<uintptr_t>(X) % 16) == 0 && encode_fn();
}

template <typename OT>
static void launch_tma(const DevCompressed& m, const float* v, const float* X, int l, OT* Y, double* part,
                       cudaStream_t s, int64_t lo = 0, int64_t hi = -1, bool merge = true) {
    if (hi < 0) hi = m.plan.nseg;
    const int boxw = l <= 32 ? 32 : 64;
    CUtensorMap map;
    cuuint64_t gdim[2] = {(cuuint64_t)l, (cuuint64_t)m.nminor};
    cuuint64_t gstr[1] = {(cuuint64_t)l * 4};
    cuuint32_t box[2] = {(cuuint32_t)boxw, 1};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = encode_fn()(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(X), gdim, gstr, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw Error(SVDB_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
    const size_t smem = (size_t)kTW * kTS * kTE * boxw * 4;
    const int64_t ns = hi - lo;
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((ns + kTW - 1) / kTW, (int64_t)device_props().sms));
    double* pp = part ? part + lo * (int64_t)l : nullptr;
    if (ns > 0) {
        if (boxw == 32) {
            SVDB_CUDA(cudaFuncSetAttribute(k_spmm_tma<OT, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            k_spmm_tma<OT, 32><<<blocks, kTW * 32, smem, s>>>(map, m.idx.p, v, m.plan.seg_row.p + lo,
                                                              m.plan.seg_beg.p + lo, m.plan.seg_end.p + lo, ns, l, Y,
                                                              l, pp);
        } else {
            SVDB_CUDA(cudaFuncSetAttribute(k_spmm_tma<OT, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            k_spmm_tma<OT, 64><<<blocks, kTW * 32, smem, s>>>(map, m.idx.p, v, m.plan.seg_row.p + lo,
                                                              m.plan.seg_beg.p + lo, m.plan.seg_end.p + lo, ns, l, Y,
                                                              l, pp);
        }
        SVDB_CHECK_LAUNCH();
    }
    if (merge && m.plan.nmulti) {
        k_spmm_merge<OT><<<nblk(m.plan.nmulti * 32, 256, 16), 256, 0, s>>>(m.plan.seg_first.p, m.plan.multi_rows.p,
                                                                          m.plan.nmulti, part, l, Y, l);
        SVDB_CHECK_LAUNCH();
    }
}

void spmm_tma_check() {
    int e = 0;
    SVDB_CUDA(cudaMemcpyFromSymbol(&e, g_tma_err, sizeof(int)));
    if (e) {
        const int z = 0;
        SVDB_CUDA(cudaMemcpyToSymbol(g_tma_err, &z, sizeof(int)));
        if (e & 2) throw Error(SVDB_ERR_CUDA, "SpMM: shared-memory ring not 128-byte aligned; no gather was issued");
        throw Error(SVDB_ERR_TIMEOUT, "SpMM: a tensor-memory gather did not complete within 2 s");
    }
}

// The rows the panel kernel leaves to the segment kernel: an explicit list
// of segments (row < 0: partial k of the list, at part[k * l]).
static void heavy_segments_f32(const DevCompressed& m, const int32_t* row, const int64_t* beg, const int64_t* end,
                               int64_t n, const float* X, int l, double* Y, double* part, cudaStream_t s) {
    if (n <= 0) return;
    const uintptr_t align = 16;
    const bool vec = (l % 4 == 0) && ((reinterpret_cast<uintptr_t>(X) % align) == 0);
    const int blocks = nblk(n * 32, 256, 16);
    if (l <= 32)
        k_spmm_seg<float, float, double, 2, 2, 4><<<blocks, 256, 0, s>>>(m.idx.p, m.val32.p, row, beg, end, n, X, l,
                                                                         l, vec, Y, l, part);
    else
        k_spmm_seg<float, float, double, 4, 2, 4><<<blocks, 256, 0, s>>>(m.idx.p, m.val32.p, row, beg, end, n, X, l,
                                                                         l, vec, Y, l, part);
    SVDB_CHECK_LAUNCH();
}

// FP32 products with the dense operand's rows ldx floats apart (ldx >= l, a
// multiple of 32: every row starts on a 128-byte line, so a gathered row of
// l <= 64 floats touches whole lines only).  False when k_spmm_lean does not
// apply (the caller then keeps the unpadded path).
bool spmm_f32_strided_ok(const DevCompressed& m, int l, int64_t ldx) {
    const char* e = getenv("SVDB_SPMM");
    if (e && *e) return false;  // an explicit kernel choice keeps the unpadded path
    return m.val32.p && m.nnz > 0 && l >= 1 && l <= 64 && l % 4 == 0 && ldx >= l && ldx % 32 == 0 &&
           m.nminor * ldx < ((int64_t)1 << 31);
}

void spmm_f32_strided(const DevCompressed& m, const float* X, int l, int64_t ldx, double* Y, cudaStream_t s) {
    if (m.nmajor == 0) return;
    if (!spmm_f32_strided_ok(m, l, ldx) || (reinterpret_cast<uintptr_t>(X) % 16))
        throw Error(SVDB_ERR_ARG, "spmm_f32_strided: operand layout not supported");
    lean_product<float, double>(m, m.val32.p, X, l, ldx, false, Y, l, s);
}

template <typename XT, typename OT>
void spmm_dev(const DevCompressed& m, bool fp32, const XT* X, int l, OT* Y, cudaStream_t s) {
    if (m.nmajor == 0 || l == 0) return;
    if constexpr (std::is_same<XT, float>::value && std::is_same<OT, double>::value) {
        if (fp32 && spmm_panel_eligible(m, l, X) &&
            spmm_panel(const_cast<DevCompressed&>(m), X, l, Y, s, heavy_segments_f32))
            return;
    }
    if constexpr (std::is_same<XT, float>::value) {
        if (fp32 && m.val32.p && m.nnz > 0 && tma_eligible(X, l, l)) {
            DevBuf<double> part;
            if (m.plan.nmulti) part.alloc(m.plan.nseg * (int64_t)l, s);
            launch_tma<OT>(m, m.val32.p, X, l, Y, part.p, s);
            return;
        }
    }
    if (fp32 && m.val32.p) spmm_impl<float, XT, OT>(m, m.val32.p, X, l, Y, s);
    else spmm_impl<double, XT, OT>(m, m.val.p, X, l, Y, s);
}

template void spmm_dev<double, double>(const DevCompressed&, bool, const double*, int, double*, cudaStream_t);
template void spmm_dev<float, float>(const DevCompressed&, bool, const float*, int, float*, cudaStream_t);
template void spmm_dev<float, double>(const DevCompressed&, bool, const float*, int, double*, cudaStream_t);

}  // namespace svdb

// Device bodies of the small dense steps of randomized_svd, shared by the
// single-problem kernels (randomized.cu) and the batched kernels (batch.cu):
// the Omega generator, the one-block Cholesky with R^-1, and the one-block
// one-sided Jacobi SVD.
#pragma once

#include <cstdint>
#include <type_traits>

#include "dense_tall.cuh"
#include "device_common.cuh"
#include "qr_loose.h"

namespace svdb {

// --------------------------------------------------------------- Omega ----
// N(0,1) entries from a counter-based generator: splitmix64 (Steele, Lea and
// Flood 2014) of (seed, index) gives two uniforms, Box-Muller gives the
// normal.  rand_distr's ziggurat stream is not reproduced.
__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}
__device__ __forceinline__ uint64_t omega_key(uint64_t seed) { return splitmix64(seed ^ 0x5DEECE66Dull); }
// entry i of the row-major Omega stream of `key`
__device__ __forceinline__ double omega_value(uint64_t key, int64_t i) {
    const uint64_t a = splitmix64(key + 2 * (uint64_t)i), b = splitmix64(key + 2 * (uint64_t)i + 1);
    const double u1 = ((double)(a >> 11) + 0.5) * (1.0 / 9007199254740992.0);  // (0,1)
    const double u2 = (double)(b >> 11) * (1.0 / 9007199254740992.0);          // [0,1)
    return sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
}

// One block: G = R^T R (upper R), and R^-1, in one sweep over panels of eight
// rows.  The forward elimination of [G | I] leaves [R | R^-T], so R^-1 has no
// dependent chain of its own.  Per panel K:
//   - every warp that owns columns factors the 8 x 8 diagonal block in
//     registers (redundantly: no broadcast, no barrier) and eliminates one
//     column per thread;
//   - the trailing tiles of G are updated by FMAs, those of R^-T by the FP64
//     matrix instruction.
// What bounds it is the chain of c pivots (a division, a multiplication and a
// multiply-add each, about 135 cycles) and two barriers per eight of them.  A
// barrier per pivot, then a forward substitution per row of R^-1, took 70 us
// at c = 60, 36 at 40 and 15 at 20; this form, with twelve warps, 24, 15 and
// 11 (ncu, cold caches; eight warps 29, 17 and 13: the FMA tiles' latency).
//
// Every element sees one fixed sequence of operations, whatever the panels:
//   a_ij = fma(-(a_ki a_kj), 1 / a_kk, a_ij), k ascending, unscaled rows;
//   R_kj = a_kj (1 / sqrt(a_kk)), R_kk = sqrt(a_kk);
//   y_e = fma(-y_k, R_ke, y_e), k ascending, then y_e (1 / R_ee)   (R^-1 = y^T)
// (m8n8k4.f64 is the same ascending chain of FMAs).  Mixed batches store
// X R^-1 in FP32, so a factor that differed in its last FP64 bit would now and
// then flip an FP32 rounding; this keeps their results reproducible.
//
// Layout: rows of 8 x 8 tiles, row tile I: tiles 0 .. I hold R^-T (I, 0 .. I)
// (the identity before panel I), tiles I + 1 .. nt hold G's unscaled rows
// (I, I .. nt - 1); padded to whole tiles with the identity.  The factored
// diagonal tiles go to a buffer of their own, since other warps may still be
// reading the unfactored one.
//
// A pivot that is not positive and finite restarts the factorisation on
// G + shift I with shift = shift_scale * trace(G) (shifted CholeskyQR); that
// sets bit 1 of *flags and *shifted (which enables the third pass).  A second
// breakdown sets bit 2 and leaves R = R^-1 = I.
// G: c x c, or with nparts > 0 the sum of nparts such matrices, in order (only
// the tiles on and above the diagonal are read).  c <= 128; blockDim.x a
// multiple of 32, at least 160.  sm: chol_smem(c) bytes.  loose (may be null) is
// set when ||G - I||_F > 0.5 (qr_loose.h), or on a shift.
__host__ __device__ inline int chol_ld(int c) { return ((c + 7) / 8 + 1) * 8 + 4; }  // = 4 or 12 mod 16: no conflicts
__host__ __device__ inline size_t chol_smem(int c) {
    const int nt = (c + 7) / 8;
    return ((size_t)(nt + 1) * 8 * chol_ld(c) + (size_t)nt * (64 + 8)) * sizeof(double);
}
__device__ __forceinline__ void chol_inv_body(const double* __restrict__ G, int nparts, int c, double shift_scale,
                                              double* __restrict__ R, double* __restrict__ Ri,
                                              int* __restrict__ flags, int* __restrict__ shifted, double* sm,
                                              int* __restrict__ loose = nullptr) {
    __shared__ int s_fail;
    __shared__ double s_inv[8], s_shift, s_dev[32];
    const int nt = (c + 7) / 8, c8 = nt * 8, ld = chol_ld(c), cc = c * c;
    double* const rp = sm + (size_t)c8 * ld;  // the panel's rows of R (8 x ld)
    double* const dg = rp + 8 * ld;           // the factored diagonal tiles, unscaled
    double* const rs = dg + nt * 64;          // 1 / sqrt of the pivots
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    if (blockDim.x < 160 || c > 128) {  // one thread per column of the widest row
        if (threadIdx.x == 0) atomicOr(flags, 2);
        for (int t = threadIdx.x; t < cc; t += blockDim.x) R[t] = Ri[t] = (t / c == t % c) ? 1.0 : 0.0;
        return;
    }
    auto g_at = [&](int i, int j) {
        if (nparts <= 0) return G[i * c + j];
        double v = 0.0;
#pragma unroll 8
        for (int b = 0; b < nparts; ++b) v += G[(int64_t)b * cc + i * c + j];
        return v;
    };
    double shift = 0.0;
    for (int attempt = 0;; ++attempt) {
        double dev = 0.0;  // this thread's share of ||G - I||_F^2
        for (int i = warp; i < c8; i += nw) {
            const int i8 = i & ~7;
            for (int j = lane; j < i8; j += 32) sm[i * ld + j] = 0.0;
            for (int j = i8 + lane; j < c8; j += 32) {
                double v = i == j ? 1.0 : 0.0;
                if (i < c && j < c) {
                    const double g = g_at(i, j);
                    dev += loose_term(g, i, j);
                    v = g + (i == j ? shift : 0.0);
                }
                sm[i * ld + 8 + j] = v;
            }
        }
        if (loose && attempt == 0) {
            dev = warp_sum(dev);
            if (lane == 0) s_dev[warp] = dev;
        }
        if (threadIdx.x == 0) s_fail = 0;
        __syncthreads();
        if (loose && attempt == 0 && threadIdx.x == 0) {
            double t = 0.0;
            for (int w = 0; w < nw; ++w) t += s_dev[w];
            if (is_loose(t)) *loose = 1;
        }
        bool failed = false;
        for (int K = 0; K < nt; ++K) {
            if (warp * 32 < c8 + 8) {
                double d[8][8], inv[8];
                const double* blk = sm + 8 * K * ld + 8 * (K + 1);
#pragma unroll
                for (int k = 0; k < 8; ++k)
#pragma unroll
                    for (int i = k; i < 8; ++i) d[k][i] = blk[k * ld + i];
                bool ok = true;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    ok = ok && d[k][k] > 0.0 && isfinite(d[k][k]);
                    inv[k] = 1.0 / d[k][k];
#pragma unroll
                    for (int i = k + 1; i < 8; ++i)
#pragma unroll
                        for (int j = i; j < 8; ++j) d[i][j] = fma(-(d[k][i] * d[k][j]), inv[k], d[i][j]);
                }
                if (!ok && lane == 0) s_fail = 1;
                // 1 / sqrt and 1 / R_kk = 1 / (sqrt) of pivot k in lane k, read from there: once per
                // warp, off the chain of the factorisation
                double piv = d[0][0];
#pragma unroll
                for (int k = 1; k < 8; ++k)
                    if (lane == k) piv = d[k][k];
                const double rq = 1.0 / sqrt(piv);
                if (warp == 0 && lane < 8) {
                    s_inv[lane] = 1.0 / piv;
                    rs[8 * K + lane] = rq;
                }
                const int j = threadIdx.x, tile = j >> 3;
                double a[8];
                if (j < c8 + 8) {
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        a[k] = tile == K ? ((j & 7) == k ? 1.0 : 0.0) : sm[(8 * K + k) * ld + j];
                    if (tile > K) {  // a column of G
#pragma unroll
                        for (int k = 0; k < 8; ++k)
#pragma unroll
                            for (int i = k + 1; i < 8; ++i) a[i] = fma(-(d[k][i] * a[k]), inv[k], a[i]);
                    }
                }
                double r[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) r[k] = __shfl_sync(0xffffffffu, rq, k);
                if (j < c8 + 8) {
                    if (tile <= K) {  // a column of R^-T
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            a[k] *= r[k];
#pragma unroll
                            for (int i = k + 1; i < 8; ++i) a[i] = fma(-a[k], d[k][i] * r[k], a[i]);
                            sm[(8 * K + k) * ld + j] = a[k];
                        }
                    } else if (tile == K + 1) {
#pragma unroll
                        for (int k = 0; k < 8; ++k) dg[(8 * K + k) * 8 + (j & 7)] = a[k];
                    } else {
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            sm[(8 * K + k) * ld + j] = a[k];
                            rp[k * ld + j] = a[k] * r[k];
                        }
                    }
                }
            }
            __syncthreads();
            if (s_fail) {  // the same value for every thread
                failed = true;
                break;
            }
            // row tiles I > K: tiles 0 .. K of R^-T and I .. nt - 1 of G
            const int kl = lane & 3, il = lane >> 2;
            for (int qq = warp; qq < (nt - 1 - K) * (nt + 1); qq += nw) {
                const int I = K + 1 + qq / (nt + 1), t = qq % (nt + 1);
                if (t > K && t <= I) continue;
                double* cp = sm + (8 * I + il) * ld + 8 * t + 2 * kl;
                double acc[2] = {cp[0], cp[1]};
                if (t <= K) {
                    const double* pa = rp + kl * ld + 8 * (I + 1) + il;
                    const double* pb = sm + (8 * K + kl) * ld + 8 * t + il;
                    dmma(acc, -pa[0], pb[0]);
                    dmma(acc, -pa[4 * ld], pb[4 * ld]);
                } else {
                    const double* pa = sm + 8 * K * ld + 8 * (I + 1) + il;
                    const double* pb = sm + 8 * K * ld + 8 * t + 2 * kl;
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const double x = pa[k * ld];
                        acc[0] = fma(-(x * pb[k * ld]), s_inv[k], acc[0]);
                        acc[1] = fma(-(x * pb[k * ld + 1]), s_inv[k], acc[1]);
                    }
                }
                cp[0] = acc[0];
                cp[1] = acc[1];
            }
            __syncthreads();
        }
        if (!failed || attempt == 1) break;
        if (threadIdx.x == 0) {
            double tr = 0.0;
            for (int i = 0; i < c; ++i) tr += g_at(i, i);
            s_shift = shift_scale * tr > 0.0 ? shift_scale * tr : 1e-300;
            atomicOr(flags, 1);
            *shifted = 1;
            if (loose) *loose = 1;
        }
        __syncthreads();  // also orders this attempt's reads before the next one's writes
        shift = s_shift;
    }
    if (s_fail) {
        if (threadIdx.x == 0) atomicOr(flags, 2);
        for (int t = threadIdx.x; t < cc; t += blockDim.x) R[t] = Ri[t] = (t / c == t % c) ? 1.0 : 0.0;
        return;
    }
    for (int i = warp; i < c; i += nw)
        for (int j = lane; j < c; j += 32) {
            const double v = (j >> 3) == (i >> 3) ? dg[i * 8 + (j & 7)] : sm[i * ld + 8 + j];
            R[i * c + j] = j > i ? v * rs[i] : j == i ? sqrt(v) : 0.0;
            Ri[i * c + j] = j >= i ? sm[j * ld + i] : 0.0;
        }
}

// Lanes per column pair in jacobi_svd_body (at most four 16-byte vectors of a
// column per lane), and the block size that gives every pair of the padded
// columns its lanes.  c <= 128.
__host__ __device__ inline int jacobi_group(int c) { return c <= 32 ? 4 : (c <= 64 ? 8 : 16); }
__host__ __device__ inline int jacobi_threads(int c) {
    const int cp = c + (c & 1);
    const int t = ((cp / 2) * jacobi_group(c) + 31) / 32 * 32;
    return t < 32 ? 32 : t;
}
__host__ __device__ inline size_t jacobi_smem(int c) {
    const size_t cp = c + (c & 1);
    return (2 * cp * cp + cp) * sizeof(double) + cp * sizeof(int);
}

// One round: every pair of columns (p, q) of the round-robin is made
// orthogonal.  G lanes per pair, E double2 of each column per lane, all held
// in registers between the sums and the update, and the columns of Vs read
// while the rotation is computed.  Returns whether this thread's pair rotated.
template <int G, int E>
__device__ __forceinline__ bool jacobi_round(double* W, double* Vs, int cp, int round, double tol2) {
    const int lane = threadIdx.x & 31, sub = lane & (G - 1);
    const int pr = (int)threadIdx.x / G, half = cp / 2, ring = cp - 1;
    // round-robin: position 0 fixed, the others rotate
    int p = pr - 1 + round, q = cp - 2 - pr + round;
    p = pr == 0 ? 0 : 1 + (p >= ring ? p - ring : p);
    q = 1 + (q >= ring ? q - ring : q);
    const bool valid = pr < half;
    if (p > q) { const int t = p; p = q; q = t; }
    if (!valid) p = q = 0;
    double2* wp = reinterpret_cast<double2*>(W + p * cp) + sub;
    double2* wq = reinterpret_cast<double2*>(W + q * cp) + sub;
    double2* vp = reinterpret_cast<double2*>(Vs + p * cp) + sub;
    double2* vq = reinterpret_cast<double2*>(Vs + q * cp) + sub;
    constexpr bool AHEAD = G < 16;  // registers: wide blocks (c > 64) read Vs after the rotation
    double2 x[E], y[E], vx[AHEAD ? E : 1], vy[AHEAD ? E : 1];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const bool in = valid && sub + G * e < half;
        x[e] = in ? wp[G * e] : make_double2(0.0, 0.0);
        y[e] = in ? wq[G * e] : make_double2(0.0, 0.0);
    }
    if constexpr (AHEAD) {
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const bool in = valid && sub + G * e < half;
            vx[e] = in ? vp[G * e] : make_double2(0.0, 0.0);
            vy[e] = in ? vq[G * e] : make_double2(0.0, 0.0);
        }
    }
    double al = 0, be = 0, ga = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        al = fma(x[e].y, x[e].y, fma(x[e].x, x[e].x, al));
        be = fma(y[e].y, y[e].y, fma(y[e].x, y[e].x, be));
        ga = fma(x[e].y, y[e].y, fma(x[e].x, y[e].x, ga));
    }
#pragma unroll
    for (int o = G >> 1; o > 0; o >>= 1) {
        al += __shfl_xor_sync(0xffffffffu, al, o);
        be += __shfl_xor_sync(0xffffffffu, be, o);
        ga += __shfl_xor_sync(0xffffffffu, ga, o);
    }
    // |ga| > tol sqrt(al be), compared in squares.  The rotation of the
    // usual zeta = (be - al) / (2 ga), t = sign(zeta) / (|zeta| +
    // sqrt(1 + zeta^2)), cs = 1 / sqrt(1 + t^2), with numerator and
    // denominator of t scaled by |2 ga|: one sqrt, one division, one
    // reciprocal square root on the dependent path.
    if (!(valid && ga != 0.0 && ga * ga > tol2 * (al * be))) return false;
    const double d = be - al, g2 = 2.0 * ga;
    const bool pos = (d >= 0.0) == (ga > 0.0) || d == 0.0;  // sign(zeta) >= 0
    const double t = (pos ? fabs(g2) : -fabs(g2)) / (fabs(d) + sqrt(fma(d, d, g2 * g2)));
    const double cs = rsqrt(fma(t, t, 1.0)), sn = cs * t;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        if (sub + G * e >= half) continue;
        wp[G * e] = make_double2(cs * x[e].x - sn * y[e].x, cs * x[e].y - sn * y[e].y);
        wq[G * e] = make_double2(sn * x[e].x + cs * y[e].x, sn * x[e].y + cs * y[e].y);
        const double2 a = AHEAD ? vx[AHEAD ? e : 0] : vp[G * e], b = AHEAD ? vy[AHEAD ? e : 0] : vq[G * e];
        vp[G * e] = make_double2(cs * a.x - sn * b.x, cs * a.y - sn * b.y);
        vq[G * e] = make_double2(sn * a.x + cs * b.x, sn * a.y + cs * b.y);
    }
    return true;
}

// One-sided Jacobi SVD of R (c x c, row-major; its transpose when `trans`) in
// one block: W = R V with orthogonal columns, sigma_j = |W_j|, U_j = W_j /
// sigma_j.  Round-robin pair ordering.  Outputs sorted by descending sigma: U
// (c x c), V (c x c), sig (c).  *status = sweeps << 8, | 2 if the sweep limit
// is reached.  sm: jacobi_smem(c) bytes; jacobi_threads(c) threads; c <= 64, or
// 65 to 128 when WIDE.
// A round is a chain (reads, three sums over the pair's lanes, square root,
// division and reciprocal square root, update, barrier) and, at c = 60, 115 KB
// through shared memory.  With every element read again for the update, 8-byte
// accesses and Vs read after the rotation one solve took 750 us at c = 60, 388
// at 40 and 136 at 20; this form 417, 228 and 79.
template <bool WIDE>
__device__ __forceinline__ void jacobi_svd_body(const double* __restrict__ R, bool trans, int c,
                                                double* __restrict__ U, double* __restrict__ V,
                                                double* __restrict__ sig, int* __restrict__ status, double* sm) {
    // W (cp x cp) | Vs (cp x cp) | norms (cp) | ranks (cp) ; column-major, an
    // odd c padded with a zero row and column
    const int cp = c + (c & 1);
    double* W = sm;
    double* Vs = sm + (size_t)cp * cp;
    double* nr = Vs + (size_t)cp * cp;
    int* rank = reinterpret_cast<int*>(nr + cp);
    for (int t = threadIdx.x; t < cp * cp; t += blockDim.x) {
        const int j = t / cp, i = t - j * cp;
        W[t] = (i < c && j < c) ? (trans ? R[j * c + i] : R[i * c + j]) : 0.0;
        Vs[t] = i == j ? 1.0 : 0.0;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const double tol = 2.220446049250313e-16 * (double)(c > 4 ? c : 4), tol2 = tol * tol;
    auto sweeps = [&](auto g, auto e) {
        int sweep = 0;
        for (; sweep < 60; ++sweep) {
            int rot = 0;
            for (int round = 0; round < cp - 1; ++round) {
                rot |= jacobi_round<decltype(g)::value, decltype(e)::value>(W, Vs, cp, round, tol2);
                __syncthreads();
            }
            if (!__syncthreads_or(rot)) break;
        }
        return sweep;
    };
    int sweep;
    using std::integral_constant;
#define SVDB_JACOBI(G, E) sweep = sweeps(integral_constant<int, G>(), integral_constant<int, E>())
    if constexpr (WIDE) {
        if (c <= 96) SVDB_JACOBI(16, 3);
        else SVDB_JACOBI(16, 4);
    } else {
        if (c <= 16) SVDB_JACOBI(4, 2);
        else if (c <= 24) SVDB_JACOBI(4, 3);
        else if (c <= 32) SVDB_JACOBI(4, 4);
        else if (c <= 48) SVDB_JACOBI(8, 3);
        else SVDB_JACOBI(8, 4);
    }
#undef SVDB_JACOBI
    if (threadIdx.x == 0) *status = (sweep << 8) | (sweep == 60 ? 2 : 0);  // sweeps, limit flag
    for (int j = warp; j < cp; j += nwarps) {
        double s = 0.0;
        for (int i = lane; i < c; i += 32) s = fma(W[j * cp + i], W[j * cp + i], s);
        s = warp_sum(s);
        if (lane == 0) nr[j] = sqrt(s);
    }
    __syncthreads();
    // rank of each column by descending norm (ties by index) -> output position
    for (int j = threadIdx.x; j < c; j += blockDim.x) {
        int pos = 0;
        for (int k = 0; k < c; ++k)
            if (nr[k] > nr[j] || (nr[k] == nr[j] && k < j)) ++pos;
        rank[j] = pos;
        sig[pos] = nr[j];
    }
    __syncthreads();
    for (int t = threadIdx.x; t < c * c; t += blockDim.x) {
        const int j = t / c, i = t - j * c, pos = rank[j];
        U[i * c + pos] = nr[j] > 0.0 ? W[j * cp + i] / nr[j] : (i == pos ? 1.0 : 0.0);
        V[i * c + pos] = Vs[j * cp + i];
    }
}

}  // namespace svdb

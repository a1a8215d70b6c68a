// Device bodies of the small dense steps of randomized_svd, shared by the
// single-problem kernels (randomized.cu) and the batched kernels (batch.cu):
// the Omega generator, the one-block Cholesky with R^-1, and the one-block
// one-sided Jacobi SVD.
#pragma once

#include <cstdint>

#include "dense_tall.cuh"
#include "device_common.cuh"

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
// multiple of 32, at least 160.  sm: chol_smem(c) bytes.
__host__ __device__ inline int chol_ld(int c) { return ((c + 7) / 8 + 1) * 8 + 4; }  // = 4 or 12 mod 16: no conflicts
__host__ __device__ inline size_t chol_smem(int c) {
    const int nt = (c + 7) / 8;
    return ((size_t)(nt + 1) * 8 * chol_ld(c) + (size_t)nt * (64 + 8)) * sizeof(double);
}
__device__ __forceinline__ void chol_inv_body(const double* __restrict__ G, int nparts, int c, double shift_scale,
                                              double* __restrict__ R, double* __restrict__ Ri,
                                              int* __restrict__ flags, int* __restrict__ shifted, double* sm) {
    __shared__ int s_fail;
    __shared__ double s_inv[8], s_shift;
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
        for (int i = warp; i < c8; i += nw) {
            const int i8 = i & ~7;
            for (int j = lane; j < i8; j += 32) sm[i * ld + j] = 0.0;
            for (int j = i8 + lane; j < c8; j += 32) {
                double v = i == j ? 1.0 : 0.0;
                if (i < c && j < c) v = g_at(i, j) + (i == j ? shift : 0.0);
                sm[i * ld + 8 + j] = v;
            }
        }
        if (threadIdx.x == 0) s_fail = 0;
        __syncthreads();
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

// Lanes per column pair in jacobi_svd_body (about eight elements of a column
// per lane), and the block size that gives every pair of the padded columns
// its lanes, capped at `cap` threads.
__host__ __device__ inline int jacobi_group(int c) { return c <= 64 ? 8 : (c <= 128 ? 16 : 32); }
__host__ __device__ inline int jacobi_threads(int c, int cap) {
    const int cp = c + (c & 1);
    const int t = ((cp / 2) * jacobi_group(c) + 31) / 32 * 32;
    return t < 32 ? 32 : (t > cap ? cap : t);
}

// One-sided Jacobi SVD of R (c x c, row-major) in one block: W = R V with
// orthogonal columns, sigma_j = |W_j|, U_j = W_j / sigma_j.  Round-robin pair
// ordering, jacobi_group(c) lanes per pair.  Outputs sorted by descending sigma:
// U (c x c), V (c x c), sig (c).  *status = sweeps << 8, | 2 if the sweep limit is reached.
// sm: (c * cp + cp * cp + cp) doubles, cp = c rounded up to even.  Any
// block size that is a multiple of 32.
__device__ __forceinline__ void jacobi_svd_body(const double* __restrict__ R, int c, double* __restrict__ U,
                                                double* __restrict__ V, double* __restrict__ sig,
                                                int* __restrict__ status, double* sm) {
    // W (c x cp) | Vs (c x cp) | norms (cp) ; column-major
    const int cp = c + (c & 1);     // even number of columns (zero padding column)
    double* W = sm;
    double* Vs = sm + (size_t)c * cp;
    double* nr = Vs + (size_t)cp * cp;
    __shared__ int s_rot;
    for (int t = threadIdx.x; t < c * cp; t += blockDim.x) {
        const int i = t % c, j = t / c;
        W[j * c + i] = (j < c) ? R[i * c + j] : 0.0;
    }
    for (int t = threadIdx.x; t < cp * cp; t += blockDim.x) Vs[t] = ((t % cp) == (t / cp)) ? 1.0 : 0.0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int half = cp / 2;
    // G lanes per column pair, 32 / G pairs per warp: the pair's scalar work
    // (three sums, the rotation's sqrt, division and rsqrt) is issued once
    // per warp for 32 / G pairs.  Pairs are walked warp by warp so that the
    // shuffles see the whole warp.
    const int G = jacobi_group(c), gpw = 32 / G, sub = lane & (G - 1), gw = lane / G;
    const double tol = 2.220446049250313e-16 * (double)(c > 4 ? c : 4);
    int sweep = 0;
    for (; sweep < 60; ++sweep) {
        if (threadIdx.x == 0) s_rot = 0;
        __syncthreads();
        for (int round = 0; round < cp - 1; ++round) {
            for (int base = warp * gpw; base < half; base += nwarps * gpw) {
                const int pr = base + gw;
                const bool valid = pr < half;
                // round-robin: position 0 fixed, others rotate
                auto at = [&](int pos) { return pos == 0 ? 0 : 1 + (pos - 1 + round) % (cp - 1); };
                int p = 0, q = 0;
                if (valid) {
                    p = at(pr);
                    q = at(cp - 1 - pr);
                    if (p > q) { int t = p; p = q; q = t; }
                }
                double al = 0, be = 0, ga = 0;
                if (valid)
                    for (int i = sub; i < c; i += G) {
                        const double x = W[p * c + i], y = W[q * c + i];
                        al = fma(x, x, al);
                        be = fma(y, y, be);
                        ga = fma(x, y, ga);
                    }
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
                if (valid && ga != 0.0 && ga * ga > (tol * tol) * (al * be)) {
                    const double d = be - al, g2 = 2.0 * ga;
                    const bool pos = (d >= 0.0) == (ga > 0.0) || d == 0.0;  // sign(zeta) >= 0
                    const double t = (pos ? fabs(g2) : -fabs(g2)) / (fabs(d) + sqrt(fma(d, d, g2 * g2)));
                    const double cs = rsqrt(fma(t, t, 1.0)), sn = cs * t;
                    for (int i = sub; i < c; i += G) {
                        const double x = W[p * c + i], y = W[q * c + i];
                        W[p * c + i] = cs * x - sn * y;
                        W[q * c + i] = sn * x + cs * y;
                    }
                    for (int i = sub; i < cp; i += G) {
                        const double x = Vs[p * cp + i], y = Vs[q * cp + i];
                        Vs[p * cp + i] = cs * x - sn * y;
                        Vs[q * cp + i] = sn * x + cs * y;
                    }
                    if (sub == 0) s_rot = 1;
                }
            }
            __syncthreads();
        }
        if (!s_rot) break;
        __syncthreads();
    }
    if (threadIdx.x == 0) *status = (sweep << 8) | (sweep == 60 ? 2 : 0);  // sweeps, limit flag
    for (int j = warp; j < cp; j += nwarps) {
        double s = 0.0;
        for (int i = lane; i < c; i += 32) s = fma(W[j * c + i], W[j * c + i], s);
        s = warp_sum(s);
        if (lane == 0) nr[j] = sqrt(s);
    }
    __syncthreads();
    // rank of each column by descending norm (ties by index) -> output position
    for (int j = threadIdx.x; j < c; j += blockDim.x) {
        int pos = 0;
        for (int k = 0; k < c; ++k)
            if (nr[k] > nr[j] || (nr[k] == nr[j] && k < j)) ++pos;
        sig[pos] = nr[j];
        for (int i = 0; i < c; ++i) {
            U[i * c + pos] = nr[j] > 0.0 ? W[j * c + i] / nr[j] : (i == pos ? 1.0 : 0.0);
            V[i * c + pos] = Vs[j * cp + i];
        }
    }
}

}  // namespace svdb

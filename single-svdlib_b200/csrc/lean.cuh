// The gather of up to 32 staged entries shared by the SpMM kernels (spmm.cu)
// and the FP64 batch products (batch.cu).
#pragma once

#include <cstdint>

namespace svdb {

// Products of one 32-entry chunk are summed in FP32 for FP32 operands (the
// chunk sum is then added to an FP64 accumulator), in FP64 otherwise.
template <typename T>
struct AccOf { using type = double; };
template <>
struct AccOf<float> { using type = float; };

// VEC elements of a row read at once: 16 bytes, or single elements of rows that
// are no whole 16-byte vectors
template <typename T, int VEC = 16 / (int)sizeof(T)>
struct alignas(sizeof(T) * VEC) LeanVec { T v[VEC]; };

// Shared-memory slots of a chunk: its H groups' entries side by side, the
// FP64 values' groups two slots apart so that they sit on different banks.
template <typename T, int H>
struct LeanSlots {
    static constexpr int PER = 32 / H;                                    // entries of a chunk per group
    static constexpr int VS = PER + (sizeof(T) == 8 && H > 1 ? 2 : 0);    // value slots per group
    static __device__ __forceinline__ int off(int q) { return (q % H) * PER + q / H; }
    static __device__ __forceinline__ int val(int q) { return (q % H) * VS + q / H; }
};

template <typename T>
__device__ __forceinline__ void lean_values4(const T* p, T (&v)[4]) {  // four consecutive shared values
    constexpr int VEC = 16 / (int)sizeof(T);
#pragma unroll
    for (int i = 0; i < 4 / VEC; ++i) {
        const LeanVec<T> t = reinterpret_cast<const LeanVec<T>*>(p)[i];
#pragma unroll
        for (int e = 0; e < VEC; ++e) v[i * VEC + e] = t.v[e];
    }
}

// cs[j] += sum over this group's entries (og, vg: its slots) of the first
// `cnt` staged ones of v X[off + col[j] ..].  A full chunk runs U gathers per
// lane at a time, a shorter one masked batches of four.  BYTES: offsets are
// bytes from X, else elements.
template <typename T, int H, int NL, int U, bool BYTES, int VEC = 16 / (int)sizeof(T)>
__device__ __forceinline__ void lean_chunk(const uint32_t* og, const T* vg, int cnt, int g, const T* __restrict__ X,
                                           const uint32_t (&col)[NL], const bool (&active)[NL],
                                           typename AccOf<T>::type (&cs)[NL][VEC]) {
    using CT = typename AccOf<T>::type;
    using Vec = LeanVec<T, VEC>;
    constexpr int PER = LeanSlots<T, H>::PER;
    static_assert(U % 4 == 0 && U <= PER, "batches of whole quads");
    auto gather = [&](uint32_t off, int j) {
        if constexpr (BYTES)
            return *reinterpret_cast<const Vec*>(reinterpret_cast<const char*>(X) +
                                                        (off + col[j] * (uint32_t)sizeof(T)));
        else
            return *reinterpret_cast<const Vec*>(X + (off + col[j]));
    };
    if (cnt >= 32) {
#pragma unroll 1
        for (int qb = 0; qb < PER; qb += U) {  // one batch live at a time
            Vec xv[U][NL];
            T vv[U];
#pragma unroll
            for (int q = 0; q < U; q += 4) {
                const uint4 o = *reinterpret_cast<const uint4*>(og + qb + q);
                T v4[4];
                lean_values4(vg + qb + q, v4);
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    vv[q + u] = v4[u];
                    const uint32_t off = u == 0 ? o.x : u == 1 ? o.y : u == 2 ? o.z : o.w;
#pragma unroll
                    for (int j = 0; j < NL; ++j) {
                        if (active[j]) xv[q + u][j] = gather(off, j);
                        else xv[q + u][j] = Vec{};
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int j = 0; j < NL; ++j)
#pragma unroll
                    for (int e = 0; e < VEC; ++e) cs[j][e] = fma((CT)vv[u], (CT)xv[u][j].v[e], cs[j][e]);
        }
    } else {
        const int mine = (cnt - g + H - 1) / H;  // entries of this group
#pragma unroll 1
        for (int qb = 0; qb * H < cnt; qb += 4) {
            Vec xv[4][NL];
            T vv[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const bool ok = qb + u < mine;
                vv[u] = ok ? vg[qb + u] : T(0);
                const uint32_t off = og[qb + u];
#pragma unroll
                for (int j = 0; j < NL; ++j) {
                    if (ok && active[j]) xv[u][j] = gather(off, j);
                    else xv[u][j] = Vec{};
                }
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int j = 0; j < NL; ++j)
#pragma unroll
                    for (int e = 0; e < VEC; ++e) cs[j][e] = fma((CT)vv[u], (CT)xv[u][j].v[e], cs[j][e]);
        }
    }
}

}  // namespace svdb

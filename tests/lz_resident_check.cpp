// Checks lz_resident_plan (single-svdlib_b200/csrc/lz_resident.h): which
// operators the Lanczos cluster may hold in shared memory.
//  - around kLzClusterNnz: counted up to it, and an uncounted structure, or a
//    count too small to be the most of 16 ranges, is never held;
//  - n, the row count, the entry count and the shared memory at their limits;
//  - every accepted layout has room for what the CTAs copy: sizes, alignment
//    and order of the arrays.
// Prints "ok" or the first failure.  Built and run by test_lz_resident.py.
#include <cstdio>
#include <cstdlib>
#include <random>
#include <algorithm>

#include "lz_resident.h"

using namespace svdb;

#define CHECK(x)                                              \
    do {                                                      \
        if (!(x)) {                                           \
            std::printf("line %d: %s\n", __LINE__, #x);       \
            std::exit(1);                                     \
        }                                                     \
    } while (0)

static const size_t kSmem = 232448 - 1024 - 8192;

// what creation would store for a structure of `nnz` entries whose fullest range has `most`
static LzResOperand operand(int64_t rows, int64_t nnz, int64_t most) {
    return {rows, nnz, slice16_counted(nnz) ? most : kSlice16Unknown};
}
static bool plan(LzResOperand a, LzResOperand b, int64_t n, LzResident& r, int vb = 8, size_t smem = kSmem) {
    const LzResOperand ops[2] = {a, b};
    return lz_resident_plan(ops, n, 512, vb, smem, r);
}
static bool even(int64_t m, int64_t n, int64_t nnz, LzResident& r, int vb = 8, size_t smem = kSmem) {
    return plan(operand(m, nnz, (nnz + 15) / 16), operand(n, nnz, (nnz + 15) / 16), n, r, vb, smem);
}

int main() {
    LzResident r;
    // the cluster's bound on the nonzeros, inclusive on both sides
    CHECK(slice16_counted(kLzClusterNnz - 1) && slice16_counted(kLzClusterNnz) && !slice16_counted(kLzClusterNnz + 1));
    for (int64_t nnz : {kLzClusterNnz - 1, kLzClusterNnz, kLzClusterNnz + 1, 40 * kLzClusterNnz}) {
        CHECK(!even(16384, 4096, nnz, r) && !r.on);   // too many entries for the shared memory
        CHECK(!even(4096, 4096, nnz, r, 4));
        CHECK(!plan({16384, nnz, 0}, {4096, nnz, 0}, 4096, r));                            // counts of nothing
        CHECK(!plan({16384, nnz, kSlice16Unknown}, {4096, nnz, kSlice16Unknown}, 4096, r));  // not counted
        CHECK(!plan({16384, nnz, nnz / 16 - 1}, {4096, nnz, nnz / 16 - 1}, 4096, r));
    }
    const LzResOperand some = operand(3000, 60000, 3750);
    CHECK(plan(some, some, 3000, r) && r.on);
    CHECK(!plan({3000, 60000, kSlice16Unknown}, some, 3000, r));
    CHECK(!plan(some, {3000, 60000, kSlice16Unknown}, 3000, r));
    CHECK(!plan(some, {3000, 60000, 3749}, 3000, r));
    CHECK(plan(some, {3000, 60000, 3750}, 3000, r));
    // n: one element of every vector per thread
    CHECK(even(8000, 8192, 9000, r) && !even(8000, 8193, 9000, r) && !even(8000, 0, 0, r));
    // rows: 16-bit column indices of the second operand, if the vectors fit at all
    const size_t huge = size_t(1) << 24;
    CHECK(even(65535, 64, 9000, r, 8, huge) && !even(65536, 64, 9000, r, 8, huge));
    // entries: 16-bit offsets inside a slice pair
    CHECK(plan(operand(64, 300000, 32767), operand(64, 300000, 32768), 64, r, 8, huge));
    CHECK(!plan(operand(64, 300000, 32768), operand(64, 300000, 32768), 64, r, 8, huge));
    // shared memory: held at exactly the layout's bytes, not below
    CHECK(even(3000, 2000, 90000, r));
    const size_t need = lz_res_layout(r, 8).bytes;
    CHECK(even(3000, 2000, 90000, r, 8, need) && !even(3000, 2000, 90000, r, 8, need - 1));
    // every accepted layout holds its arrays
    std::mt19937_64 g(1);
    int held = 0;
    for (int t = 0; t < 20000; ++t) {
        const int64_t m = 1 + g() % 20000, n = 1 + g() % 9000, nnz = g() % (kLzClusterNnz + 1000);
        const int64_t most = std::min<int64_t>(nnz, nnz / 16 + g() % 500);
        const int vb = g() % 2 ? 8 : 4;
        if (!plan(operand(m, nnz, most), operand(n, nnz, most), n, r, vb)) continue;
        ++held;
        r.coef = (int)(g() % 64);
        const LzResLayout L = lz_res_layout(r, vb);
        CHECK(L.bytes - (size_t)r.coef * 32 <= kSmem && nnz <= kLzClusterNnz && 16 * (int64_t)r.max_nnz[0] >= nnz);
        const int64_t rows[2] = {m, n};
        CHECK(L.xa % 16 == 0 && L.xb % 16 == 0 && L.coef % 8 == 0 && L.y % 8 == 0);
        CHECK(L.xb >= L.xa + 8 * (size_t)n && L.coef >= L.xb + 8 * (size_t)(m + m % 2) && L.y >= L.coef + 32 * (size_t)r.coef);
        for (int k = 0; k < 2; ++k) {
            CHECK(16 * (int64_t)r.rows_c[k] >= rows[k] && r.rows_c[k] % 2 == 0);
            CHECK(L.v[0] >= L.y + 8 * (size_t)r.rows_c[k]);
            CHECK(L.v[k] % 8 == 0 && L.rp[k] % 4 == 0 && L.ci[k] % 2 == 0);
        }
        CHECK(r.rows_c[1] <= 512);
        CHECK(L.v[1] >= L.v[0] + (size_t)vb * r.max_nnz[0] && L.rp[0] >= L.v[1] + (size_t)vb * r.max_nnz[1]);
        CHECK(L.rp[1] >= L.rp[0] + 4 * (size_t)(r.rows_c[0] + 1) && L.ci[0] >= L.rp[1] + 4 * (size_t)(r.rows_c[1] + 1));
        CHECK(L.ci[1] >= L.ci[0] + 2 * (size_t)r.max_nnz[0] && L.bytes >= L.ci[1] + 2 * (size_t)r.max_nnz[1]);
    }
    CHECK(held > 500);
    std::printf("ok\n");
    return 0;
}

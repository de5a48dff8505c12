// logup-GKR fraction trees: all instances of a batch level by level, two levels per launch.
//
// A level holds a numerator and a denominator array.  The next level adds the
// fraction at index i to the one at i + half (the split is on the top
// variable): (n1/d1) + (n2/d2) = (n1*d2 + n2*d1) / (d1*d2), following
// LogUpLayer::next_layer (zkml/src/lookup/logup_gkr/circuit.rs:88-184) and
// Fraction's add (zkml/src/lookup/logup_gkr/structs.rs:48-58).
//
// The large levels are bound by their products and by HBM, the many small ones by launches.  So blockIdx.y is the
// instance, a thread makes two entries of one level and, from registers, the entry of the next that they add up to
// (the first of the two levels is written, never read back), and one block per instance finishes once a level has at
// most kLogupSmall entries.  Where registers for two levels cost more than reading a level back, a launch makes one
// (logup_leaf_level, logup_one_level).  A BN254 denominator  c + col_0 + s col_1 + ..  over integer columns is one sum of
// rows (8 multiply-adds per column) with one reduction, where every column was widened and multiplied mod r.
// 36 instances of 2^16 rows, Goldilocks: 780 us in 216 launches of one instance's level each, 64 us in 5; three
// instances of 2^21 rows, 5 integer columns, BN254: 560 us in 33 launches, 416 us two levels at a time, about 20 us less
// since large levels are made alone.
#pragma once
#include "family.cuh"
#include "lazy_sum.cuh"
#include "sumcheck_kernels.cuh"

namespace dpb {

constexpr int kMaxLogupCols = 8;
constexpr uint32_t kLogupSmall = 512;  // entries of a level from which one block makes the rest of its tree

template <class F>
struct LogupTree {
    const void* col[kMaxLogupCols];
    typename F::E sep_pow[kMaxLogupCols];  // sep^j, j = 0..
    typename F::E constant;
    typename F::E int_constant;            // constant - 2^31 sum_j sep^j
    uint32_t rows[kMaxLogupCols][2][8];    // BN254, integer columns: rows of sep^j and of 2^32 sep^j (fr_fixed_row 8, 9)
    const void* mult;                      // tables: the multiplicities
    typename F::E* slab;                   // levels 1, 2, ..: numerators, then denominators
    int32_t dtype[kMaxLogupCols];
    int32_t mult_dtype;
    uint32_t n_cols, m;
    uint32_t is_table, int_rows;           // int_rows: BN254, every column holds integers (rows above)
};

// entries before level l of a tree over 2^m rows (level l has 2^(m-l) fractions)
__host__ __device__ __forceinline__ uint64_t logup_level_offset(uint32_t m, uint32_t l) { return (2ull << m) - (2ull << (m - l + 1)); }

__device__ __forceinline__ Fr logup_int_denominator(const LogupTree<FrFam>& t, uint64_t i) {
    // An entry x enters as the unsigned word x + 2^31, which int_constant takes back.  The constant stands at word
    // positions 2..9 (times 2^64), the upper two words in O, whose carry word its top word cannot overflow.
    frw::RowAcc acc = frw::rowacc_zero();
    const frw::F8 c = frw::from_fr(t.int_constant);
#pragma unroll
    for (int w = 0; w < 6; w++) acc.E[2 + w] = c.w[w];
    acc.O[8] = c.w[6];
    acc.O[9] = c.w[7];
    for (uint32_t j = 0; j < t.n_cols; j++) {
        uint32_t lo, hi = 0;
        bool neg = false;
        if (t.dtype[j] == DPB_FR_I32) {
            lo = (uint32_t)((const int32_t*)t.col[j])[i] ^ 0x80000000u;
        } else {
            const int64_t x = ((const int64_t*)t.col[j])[i];
            const uint64_t y = (uint64_t)x + 0x80000000ull;  // hi 2^32 + lo, hi of x's sign and zero for 32-bit integers
            lo = (uint32_t)y;
            hi = (uint32_t)(y >> 32);
            neg = x < 0;
        }
        frw::rowacc_mac(acc, t.rows[j][0], lo);
        if (hi) {
            frw::F8 row;
#pragma unroll
            for (int w = 0; w < 8; w++) row.w[w] = t.rows[j][1][w];
            if (neg) row = frw::from_fr(fr_neg(frw::to_fr(row)));
            frw::rowacc_mac(acc, row.w, neg ? (uint32_t)0 - hi : hi);
        }
    }
    // below c + r (1 + 2^-27): one subtraction leaves it below r but for a sliver above r, which its top word gives away
    frw::F8 v = frw::reduce_rows(acc.E, acc.O);
    if (v.w[7] >= DPB_FRW_P7) v = frw::reduce_once(v);
    return frw::to_fr(v);
}
__device__ __forceinline__ Gl2 logup_int_denominator(const LogupTree<GlFam>&, uint64_t) { return gl2_zero(); }

template <class F>
struct LogupFrac {
    typename F::E n, d;
};
template <class F>
__device__ __forceinline__ LogupFrac<F> logup_add(const LogupFrac<F>& a, const LogupFrac<F>& b) {
    LogupFrac<F> r;
    r.n = TwoProducts<F>::sum(a.n, b.d, b.n, a.d);
    r.d = F::mul(a.d, b.d);
    return r;
}
template <class F>
__device__ __forceinline__ void logup_store(const LogupTree<F>& t, uint32_t l, uint64_t i, const LogupFrac<F>& f) {
    typename F::E* num = t.slab + logup_level_offset(t.m, l);
    F::store(num, i, f.n);
    F::store(num, (1ull << (t.m - l)) + i, f.d);
}
template <class F>
__device__ __forceinline__ LogupFrac<F> logup_load(const LogupTree<F>& t, uint32_t l, uint64_t i) {
    const typename F::E* num = t.slab + logup_level_offset(t.m, l);
    LogupFrac<F> f;
    f.n = F::load(num, F::kChalDtype, i);
    f.d = F::load(num, F::kChalDtype, (1ull << (t.m - l)) + i);
    return f;
}

// Denominators of K rows, column by column, so that K loads and products are under way at once (Goldilocks, 2^24 rows, two
// columns: 411 us one row at a time, 348 by four).
// A launch of logup_leaf_level never meets integer columns' rows: ROWS = false keeps their registers out of it.
template <class F, bool ROWS, int K>
__device__ __forceinline__ void logup_denominators(const LogupTree<F>& t, const uint64_t (&row)[K], typename F::E (&d)[K]) {
    if (ROWS && sizeof(typename F::E) == 32 && t.int_rows) {
#pragma unroll
        for (int k = 0; k < K; k++) d[k] = logup_int_denominator(t, row[k]);
        return;
    }
#pragma unroll
    for (int k = 0; k < K; k++) d[k] = t.constant;
    for (uint32_t j = 0; j < t.n_cols; j++) {
        typename F::E v[K];
#pragma unroll
        for (int k = 0; k < K; k++) v[k] = F::load(t.col[j], t.dtype[j], row[k]);
        // sep^0 = 1: the first column is added as is (circuit.rs:162-171)
#pragma unroll
        for (int k = 0; k < K; k++) d[k] = F::add(d[k], j == 0 ? v[k] : F::mul(t.sep_pow[j], v[k]));
    }
}
// entry i of level 1: the rows i and i + 2^(m-1) with denominators d1 and d2.  A lookup's numerators are -1
// (circuit.rs:151-182), a table's its multiplicities (circuit.rs:117-150).
template <class F, bool ROWS>
__device__ __forceinline__ LogupFrac<F> logup_leaf(const LogupTree<F>& t, uint64_t i, const typename F::E& d1, const typename F::E& d2) {
    const uint64_t half = 1ull << (t.m - 1);
    LogupFrac<F> r;
    if (!t.is_table) r.n = F::neg(F::add(d1, d2));
    else if (ROWS) r.n = TwoProducts<F>::sum(F::load(t.mult, t.mult_dtype, i), d2, d1, F::load(t.mult, t.mult_dtype, i + half));
    else r.n = F::add(F::mul(F::load(t.mult, t.mult_dtype, i), d2), F::mul(d1, F::load(t.mult, t.mult_dtype, i + half)));
    r.d = F::mul(d1, d2);
    return r;
}

// ONE: a launch over one tree takes it as a parameter.  That saves the upload (10 us of a tree of 2^10 rows) and a trip
// to memory for every column's address.
template <class F, bool ONE>
__device__ __forceinline__ const LogupTree<F>& logup_tree(const LogupTree<F>* trees, const LogupTree<F>& one, uint32_t i) {
    return ONE ? one : trees[i];
}

// Levels 1 and 2 from the columns; with rows_only the trees over integer columns alone (BN254, rows).
template <class F, bool ONE>
__global__ void __launch_bounds__(kThreads, 2)
    logup_leaf_levels(const LogupTree<F>* __restrict__ trees, const __grid_constant__ LogupTree<F> one, bool rows_only) {
    const LogupTree<F>& t = logup_tree<F, ONE>(trees, one, blockIdx.y);
    if (rows_only && !t.int_rows) return;
    const uint64_t q = 1ull << (t.m - 2), stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < q; i += stride) {
        LogupFrac<F> a, b;
        if (sizeof(typename F::E) == 32) {  // 128 registers hold two rows of BN254 columns
            typename F::E d[2];
            logup_denominators<F, true>(t, {i, i + 2 * q}, d);
            a = logup_leaf<F, true>(t, i, d[0], d[1]);
            logup_store<F>(t, 1, i, a);
            logup_denominators<F, true>(t, {i + q, i + 3 * q}, d);
            b = logup_leaf<F, true>(t, i + q, d[0], d[1]);
        } else {
            typename F::E d[4];
            logup_denominators<F, true>(t, {i, i + 2 * q, i + q, i + 3 * q}, d);
            a = logup_leaf<F, true>(t, i, d[0], d[1]);
            logup_store<F>(t, 1, i, a);
            b = logup_leaf<F, true>(t, i + q, d[2], d[3]);
        }
        logup_store<F>(t, 1, i + q, b);
        if (t.m > 2) logup_store<F>(t, 2, i, logup_add<F>(a, b));
    }
}

// Level 1 alone, for the trees logup_leaf_levels leaves out with rows_only, and one later level: large BN254 levels are
// bound by loads and products that want four blocks per SM (64 registers, a reduction per product), where two levels
// together take 104 or 128 registers and a sum of two products 76.  Trees of 2^24 rows, 1 / 2 / 4 field columns: 898 /
// 1305 / 2108 us in launches of two levels, 745 / 1036 / 1620 here.
template <class F, bool ONE>
__global__ void __launch_bounds__(kThreads, 4)
    logup_leaf_level(const LogupTree<F>* __restrict__ trees, const __grid_constant__ LogupTree<F> one) {
    const LogupTree<F>& t = logup_tree<F, ONE>(trees, one, blockIdx.y);
    if (t.int_rows) return;
    const uint64_t half = 1ull << (t.m - 1), stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < half; i += stride) {
        typename F::E d[2];
        logup_denominators<F, false>(t, {i, i + half}, d);
        logup_store<F>(t, 1, i, logup_leaf<F, false>(t, i, d[0], d[1]));
    }
}
// Level l + 1 from level l.  l = 1: for the trees of logup_leaf_level; later: in pairs with an even l first, for the
// trees whose level at that even l is still too large for one block.
template <class F, bool ONE>
__global__ void __launch_bounds__(kThreads, 4)
    logup_one_level(const LogupTree<F>* __restrict__ trees, const __grid_constant__ LogupTree<F> one, uint32_t l) {
    const LogupTree<F>& t = logup_tree<F, ONE>(trees, one, blockIdx.y);
    if (l == 1 ? t.int_rows || t.m <= 2 : t.m < (l & ~1u) + 2 || (1ull << (t.m - (l & ~1u))) <= kLogupSmall) return;
    const uint64_t half = 1ull << (t.m - l - 1), stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < half; i += stride) {
        const LogupFrac<F> a = logup_load<F>(t, l, i), b = logup_load<F>(t, l, i + half);
        LogupFrac<F> r;
        r.n = F::add(F::mul(a.n, b.d), F::mul(b.n, a.d));
        r.d = F::mul(a.d, b.d);
        logup_store<F>(t, l + 1, i, r);
    }
}

// Levels l + 1 and l + 2 from level l, for the trees whose level l is still too large for one block.
template <class F, bool ONE>
__global__ void __launch_bounds__(kThreads, 2)
    logup_two_levels(const LogupTree<F>* __restrict__ trees, const __grid_constant__ LogupTree<F> one, uint32_t l) {
    const LogupTree<F>& t = logup_tree<F, ONE>(trees, one, blockIdx.y);
    if (t.m < l + 2 || (1ull << (t.m - l)) <= kLogupSmall) return;
    const uint64_t q = 1ull << (t.m - l - 2), stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < q; i += stride) {
        const LogupFrac<F> a = logup_add<F>(logup_load<F>(t, l, i), logup_load<F>(t, l, i + 2 * q));
        logup_store<F>(t, l + 1, i, a);
        const LogupFrac<F> b = logup_add<F>(logup_load<F>(t, l, i + q), logup_load<F>(t, l, i + 3 * q));
        logup_store<F>(t, l + 1, i + q, b);
        logup_store<F>(t, l + 2, i, logup_add<F>(a, b));
    }
}

// The rest of every tree, one block each, and the top level's four values per tree side by side in `outputs` (when
// given).
template <class F, bool ONE>
__global__ void __launch_bounds__(kThreads)
    logup_small_levels(const LogupTree<F>* __restrict__ trees, const __grid_constant__ LogupTree<F> one,
                       typename F::E* __restrict__ outputs) {
    const LogupTree<F>& t = logup_tree<F, ONE>(trees, one, blockIdx.x);
    uint32_t l = t.m > 2 ? 2 : 1;  // the last level there is
    while ((1ull << (t.m - l)) > kLogupSmall) l += 2;
    for (; l + 1 < t.m; l++) {
        const uint32_t half = 1u << (t.m - l - 1);
        for (uint32_t i = threadIdx.x; i < half; i += blockDim.x)
            logup_store<F>(t, l + 1, i, logup_add<F>(logup_load<F>(t, l, i), logup_load<F>(t, l, i + half)));
        __syncthreads();  // this level is complete (and visible to the block) before the next one reads it
    }
    if (outputs && threadIdx.x < 4) {
        const typename F::E* top = t.slab + logup_level_offset(t.m, t.m - 1);
        outputs[4 * blockIdx.x + threadIdx.x] = top[threadIdx.x];
    }
}

}  // namespace dpb

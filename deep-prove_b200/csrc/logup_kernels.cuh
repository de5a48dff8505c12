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
// most kLogupSmall entries.  A BN254 denominator  c + col_0 + s col_1 + ..  over integer columns is one sum of rows
// (8 multiply-adds per column) with one reduction, where every column was widened and multiplied mod r.
// Three instances of 2^21 rows, 5 integer columns, BN254: 560 us in 33 launches before, 416 us in 7; 36 instances of
// 2^16 rows, Goldilocks: 780 us in 216 launches and 64 us in 5.
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
    uint32_t is_table, int_cols;           // int_cols: every column holds integers
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

template <class F>
__device__ __forceinline__ typename F::E logup_denominator(const LogupTree<F>& t, uint64_t i) {
    if (sizeof(typename F::E) == 32 && t.int_cols) return logup_int_denominator(t, i);
    typename F::E d = t.constant;
    for (uint32_t j = 0; j < t.n_cols; j++) {
        const typename F::E v = F::load(t.col[j], t.dtype[j], i);
        // sep^0 = 1: the first column is added as is (circuit.rs:162-171)
        d = F::add(d, j == 0 ? v : F::mul(t.sep_pow[j], v));
    }
    return d;
}
// entry i of level 1: the rows i and i + 2^(m-1).  A lookup's numerators are -1 (circuit.rs:151-182), a table's its
// multiplicities (circuit.rs:117-150).
template <class F>
__device__ __forceinline__ LogupFrac<F> logup_leaf(const LogupTree<F>& t, uint64_t i) {
    const uint64_t half = 1ull << (t.m - 1);
    const typename F::E d1 = logup_denominator<F>(t, i), d2 = logup_denominator<F>(t, i + half);
    LogupFrac<F> r;
    r.n = t.is_table ? TwoProducts<F>::sum(F::load(t.mult, t.mult_dtype, i), d2, d1, F::load(t.mult, t.mult_dtype, i + half))
                     : F::neg(F::add(d1, d2));
    r.d = F::mul(d1, d2);
    return r;
}

// Levels 1 and 2 from the columns.
template <class F>
__global__ void __launch_bounds__(kThreads, 2)
    logup_leaf_levels(const LogupTree<F>* __restrict__ trees) {
    const LogupTree<F>& t = trees[blockIdx.y];
    const uint64_t q = 1ull << (t.m - 2), stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < q; i += stride) {
        const LogupFrac<F> a = logup_leaf<F>(t, i);
        logup_store<F>(t, 1, i, a);
        const LogupFrac<F> b = logup_leaf<F>(t, i + q);
        logup_store<F>(t, 1, i + q, b);
        if (t.m > 2) logup_store<F>(t, 2, i, logup_add<F>(a, b));
    }
}

// Levels l + 1 and l + 2 from level l, for the trees whose level l is still too large for one block.
template <class F>
__global__ void __launch_bounds__(kThreads, 2)
    logup_two_levels(const LogupTree<F>* __restrict__ trees, uint32_t l) {
    const LogupTree<F>& t = trees[blockIdx.y];
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

// The rest of every tree, one block each, and the top level's four values per tree side by side in `outputs`.
template <class F>
__global__ void __launch_bounds__(kThreads)
    logup_small_levels(const LogupTree<F>* __restrict__ trees, typename F::E* __restrict__ outputs) {
    const LogupTree<F>& t = trees[blockIdx.x];
    uint32_t l = t.m > 2 ? 2 : 1;  // the last level there is
    while ((1ull << (t.m - l)) > kLogupSmall) l += 2;
    for (; l + 1 < t.m; l++) {
        const uint32_t half = 1u << (t.m - l - 1);
        for (uint32_t i = threadIdx.x; i < half; i += blockDim.x)
            logup_store<F>(t, l + 1, i, logup_add<F>(logup_load<F>(t, l, i), logup_load<F>(t, l, i + half)));
        __syncthreads();  // this level is complete (and visible to the block) before the next one reads it
    }
    if (threadIdx.x < 4) {
        const typename F::E* top = t.slab + logup_level_offset(t.m, t.m - 1);
        outputs[4 * blockIdx.x + threadIdx.x] = top[threadIdx.x];
    }
}

}  // namespace dpb

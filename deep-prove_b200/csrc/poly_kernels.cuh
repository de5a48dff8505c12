// Multilinear-table kernels outside the sumcheck loop: layout conversion, eq
// tables, partial evaluation of the top / bottom variables.
#pragma once
#include "family.cuh"
#include "lazy_sum.cuh"

namespace dpb {

// ---- layout conversion ---------------------------------------------------
// in and out may be the same array
__global__ void fr_canonical_to_mont(const Fr* in, Fr* out, uint64_t n) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        FrFam::store(out, i, fr_to_mont(FrFam::load(in, DPB_FR, i)));
}
__global__ void fr_mont_to_canonical(const Fr* in, Fr* out, uint64_t n) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        FrFam::store(out, i, fr_from_mont(FrFam::load(in, DPB_FR, i)));
}
__global__ void fr_from_i64_kernel(const int64_t* __restrict__ in, Fr* __restrict__ out,
                                   uint64_t n) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        FrFam::store(out, i, fr_from_i64(in[i]));
}
__global__ void gl_from_i64_kernel(const int64_t* __restrict__ in, uint64_t* __restrict__ out,
                                   uint64_t n) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const int64_t x = in[i];
        // |x| < 2^63 < p, so the magnitude is already canonical
        out[i] = x < 0 ? GL_P - ((uint64_t)0 - (uint64_t)x) : (uint64_t)x;
    }
}

// ---- eq tables -------------------------------------------------------------
// prod_j (bit_j(i) ? pt[j] : 1 - pt[j]) over bits coordinates
template <class F>
__device__ __forceinline__ typename F::E eq_entry(const typename F::E* __restrict__ pt, uint32_t bits, uint32_t i) {
    typedef typename F::E E;
    E acc = F::one();
    for (uint32_t j = 0; j < bits; j++) {
        const E r = pt[j], f = ((i >> j) & 1) ? r : F::sub(F::one(), r);
        acc = j ? F::mul(acc, f) : f;
    }
    return acc;
}
// The eq tables of two short points in one launch (m0, m1 <= kEqSmallBits; blocks0 blocks work on the first, the rest
// on the second).  What such a table waits for is one thread's chain of products (about half a microsecond each), so
// a block makes the tables of four parts of the point (at most three coordinates each: two products), of its two
// halves (one more) and then its entries (one more), where one thread per entry multiplied all coordinates: a table of
// 2^10 entries 6.9 us, 4.3 us since (BN254).
constexpr uint32_t kEqSmallBits = 12, kEqSmallThreads = 128;
template <class F>
__global__ void __launch_bounds__(kEqSmallThreads)
    eq_small(const typename F::E* __restrict__ pt0, uint32_t m0, typename F::E* __restrict__ out0, uint32_t blocks0,
             const typename F::E* __restrict__ pt1, uint32_t m1, typename F::E* __restrict__ out1) {
    typedef typename F::E E;
    __shared__ E part[4][8], half[2][64];
    const bool second = blockIdx.x >= blocks0;
    const E* pt = second ? pt1 : pt0;
    E* out = second ? out1 : out0;
    const uint32_t m = second ? m1 : m0;
    const uint32_t block = second ? blockIdx.x - blocks0 : blockIdx.x, blocks = second ? gridDim.x - blocks0 : blocks0;
    const uint32_t h0 = (m + 1) / 2, h1 = m - h0;  // coordinates of the halves
    const uint32_t lo0 = (h0 + 1) / 2, lo1 = (h1 + 1) / 2;
    if (threadIdx.x < 32) {
        const uint32_t q = threadIdx.x >> 3, i = threadIdx.x & 7;
        const uint32_t bits = q == 0 ? lo0 : q == 1 ? h0 - lo0 : q == 2 ? lo1 : h1 - lo1;
        const uint32_t first = q == 0 ? 0 : q == 1 ? lo0 : q == 2 ? h0 : h0 + lo1;
        if (i < (1u << bits)) part[q][i] = eq_entry<F>(pt + first, bits, i);
    }
    __syncthreads();
    {
        const uint32_t q = threadIdx.x >> 6, i = threadIdx.x & 63, bits = q ? h1 : h0, lo = q ? lo1 : lo0;
        if (i < (1u << bits)) half[q][i] = F::mul(part[2 * q][i & ((1u << lo) - 1)], part[2 * q + 1][i >> lo]);
    }
    __syncthreads();
    for (uint32_t i = block * blockDim.x + threadIdx.x; i < (1u << m); i += blocks * blockDim.x)
        F::store(out, i, F::mul(half[0][i & ((1u << h0) - 1)], half[1][i >> h0]));
}
// out[i] = hi[i >> lo_bits] * lo[i & (2^lo_bits - 1)]
template <class F>
__global__ void eq_combine(const typename F::E* __restrict__ lo, uint32_t lo_bits,
                           const typename F::E* __restrict__ hi, uint64_t n,
                           typename F::E* __restrict__ out) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t mask = (1ull << lo_bits) - 1;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        F::store(out, i,
                 F::mul(F::load(hi, F::kChalDtype, i >> lo_bits), F::load(lo, F::kChalDtype, i & mask)));
}

// ---- many eq tables at once -----------------------------------------------------
// Table t has m_t variables and its point at pts[pt_off[t] ..].  Its table is
// the outer product of a "low" part over the first h_t = ceil(m_t / 2) variables
// and a "high" part over the rest, each computed directly (at most m_t / 2 + 1
// multiplies per entry of tables of about sqrt(2^m_t) entries), then one
// multiply per output entry.  Work items of all tables are laid end to end;
// `prefix` holds the first item of every table (n + 1 entries) and a thread
// finds its table by binary search.
struct EqBatchDesc {
    uint32_t m;        // variables
    uint32_t pt_off;   // first coordinate in the points array
    uint64_t part_off; // low part at parts[part_off], high part right after it
    uint64_t out_off;  // table at out[out_off]
};

__device__ __forceinline__ uint32_t find_segment(const uint64_t* __restrict__ prefix, uint32_t n, uint64_t item) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (prefix[mid] <= item) lo = mid;
        else hi = mid;
    }
    return lo;
}

template <class F>
__global__ void __launch_bounds__(kThreads)
    eq_batch_parts(const EqBatchDesc* __restrict__ desc, const uint64_t* __restrict__ prefix, uint32_t n,
                   const typename F::E* __restrict__ pts, typename F::E* __restrict__ parts) {
    typedef typename F::E E;
    const uint64_t total = prefix[n];
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += stride) {
        const uint32_t t = find_segment(prefix, n, w);
        const EqBatchDesc d = desc[t];
        const uint32_t h = (d.m + 1) / 2;
        uint64_t i = w - prefix[t];
        uint32_t first = 0, bits = h;  // low part: coordinates [0, h)
        if (i >= (1ull << h)) {        // high part: coordinates [h, m)
            i -= 1ull << h;
            first = h;
            bits = d.m - h;
        }
        F::store(parts, d.part_off + (w - prefix[t]), eq_entry<F>(pts + d.pt_off + first, bits, (uint32_t)i));
    }
}

template <class F>
__global__ void __launch_bounds__(kThreads)
    eq_batch_combine(const EqBatchDesc* __restrict__ desc, const uint64_t* __restrict__ prefix, uint32_t n,
                     const typename F::E* __restrict__ parts, typename F::E* __restrict__ out) {
    const uint64_t total = prefix[n];
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += stride) {
        const uint32_t t = find_segment(prefix, n, w);
        const EqBatchDesc d = desc[t];
        const uint32_t h = (d.m + 1) / 2;
        const uint64_t i = w - prefix[t];
        const uint64_t lo = i & ((1ull << h) - 1), hi = i >> h;
        F::store(out, d.out_off + i,
                 F::mul(F::load(parts, F::kChalDtype, d.part_off + lo),
                        F::load(parts, F::kChalDtype, d.part_off + (1ull << h) + hi)));
    }
}

// Many tables evaluated at one point: table t (2^m_t entries, any layout of its family) against the eq table of the
// point's first m_t coordinates.  Every block sums one piece of `piece` entries of one table (pieces of all tables are
// laid end to end, `first[t]` the first piece of table t), so a long table among many short ones still fills the GPU.
// The sums stay unreduced (EntrySum).  128 BN254 int32 tables, 16 of them of 2^20 entries: 918 us with a reduction per
// product and the same number of blocks for every table, 116 us since.
struct EvalManySrc {
    const void* ptr;
    const void* eq;  // eq table over this table's variables (challenge elements)
    uint64_t len;
    int32_t dtype;
    uint32_t first;
};
template <class F, bool INT>
__device__ __forceinline__ typename F::E evaluate_piece(const EvalManySrc& t, uint64_t begin, uint64_t end) {
    EntrySum<F, INT> acc;
    acc.zero();
    for (uint64_t x = begin + threadIdx.x; x < end; x += blockDim.x)
        acc.mac(F::load(t.eq, F::kChalDtype, x), t.ptr, t.dtype, x);
    return acc.finish();
}
template <class F>
__global__ void __launch_bounds__(kThreads)
    evaluate_many_kernel(const EvalManySrc* __restrict__ src, uint32_t n, uint64_t piece, typename F::E* __restrict__ partial) {
    typedef typename F::E E;
    uint32_t lo = 0, hi = n;  // the table with first <= this block's piece < the next table's first
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (src[mid].first <= blockIdx.x) lo = mid;
        else hi = mid;
    }
    const EvalManySrc t = src[lo];
    const uint64_t begin = (uint64_t)(blockIdx.x - t.first) * piece;
    const uint64_t end = begin + piece < t.len ? begin + piece : t.len;
    const bool ints = t.dtype >= DPB_GL_I64;
    E acc[1] = {ints ? evaluate_piece<F, true>(t, begin, end) : evaluate_piece<F, false>(t, begin, end)};
    block_sum<F, 1>(acc);
    if (threadIdx.x == 0) partial[blockIdx.x] = acc[0];
}
// out[t] = scale[t] * (sum of the table's pieces, less 2^31 where EntrySum added it: a whole eq table sums to one);
// one warp per table
template <class F>
__global__ void __launch_bounds__(kThreads)
    evaluate_many_finish(const typename F::E* __restrict__ partial, const EvalManySrc* __restrict__ src, uint64_t piece,
                         const typename F::E* __restrict__ scale, uint32_t n, typename F::E* __restrict__ out) {
    typedef typename F::E E;
    const uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (t >= n) return;
    const EvalManySrc d = src[t];
    const uint32_t pieces = (uint32_t)((d.len + piece - 1) / piece);
    E acc = F::zero();
    for (uint32_t s = lane; s < pieces; s += 32) acc = F::add(acc, partial[d.first + s]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc = F::add(acc, F::shfl_down(acc, off));
    if (lane == 0) {
        if (EntrySum<F, true>::kPlus31 && d.dtype >= DPB_GL_I64) acc = F::sub(acc, F::from_u64(0x80000000ull));
        out[t] = F::mul(acc, scale[t]);
    }
}

// One source table of a linear combination.
struct LinCombSrc {
    const void* ptr;
    uint64_t len;
    int32_t dtype;
    int32_t pad;
};

// The eq table of a rotary layer with its entries moved and negated the way the rotation pairs them
// (RopeLayout::permuted_eq_poly, zkml/src/layers/transformer/positional/rope.rs:238-258).
// layout 0 (adjacent pairs): out[i] = eq[i + 1] for even i, -eq[i - 1] for odd i.
// layout 1 (rotate half, rows of `row` entries): out[i] = eq[i + row/2] in a row's first half, -eq[i - row/2] in its second.
template <class F>
__global__ void __launch_bounds__(kThreads)
    rope_permuted_eq_kernel(const typename F::E* __restrict__ eq, uint64_t len, int layout, uint64_t row,
                            typename F::E* __restrict__ out) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += stride) {
        bool first;
        uint64_t src;
        if (layout == 0) {
            first = (i & 1) == 0;
            src = i ^ 1;
        } else {
            const uint64_t half = row >> 1, c = i % row;
            first = c < half;
            src = first ? i + half : i - half;
        }
        const typename F::E v = eq[src];
        out[i] = first ? v : F::neg(v);
    }
}

// out[i] = sum_j coeff[j] * table_j[i], tables shorter than the output read as zero beyond their length.
// Consecutive threads read consecutive entries of each table in turn.  BN254: the coefficients are laid out as rows
// first (lincomb_rows_kernel), so that a term is 8 multiply-adds for an int32 entry (the row of the coefficient or of
// its negative), 16 for a 64-bit one that needs its upper word and 64 for a field entry, and the sum is reduced once
// (twice every kRowTerms terms).  119 int32 tables, 15 of 2^20 entries: 641 us with a field product per
// term, 208 us since.
constexpr uint32_t kLinRows = 8;        // rows per table: a field table's eight, or an integer table's c, -c, 2^32 c, -2^32 c
constexpr uint32_t kRowTerms = 1024;    // row products a RowAcc may hold
__global__ void __launch_bounds__(kThreads)
    lincomb_rows_kernel(const LinCombSrc* __restrict__ src, const Fr* __restrict__ coeff, uint32_t n, uint32_t* __restrict__ rows) {
    const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x, j = w / kLinRows, q = w % kLinRows;
    if (j >= n) return;
    uint32_t row[8];
    if (src[j].dtype == DPB_FR) {
        fr_fixed_row(coeff[j], (int)q, row);
    } else {
        if (q >= 4) return;
        fr_fixed_row((q & 1) ? fr_neg(coeff[j]) : coeff[j], 8 + (int)(q >> 1), row);
    }
#pragma unroll
    for (int i = 0; i < 8; i++) rows[(size_t)w * 8 + i] = row[i];
}
__device__ __forceinline__ void lincomb_row_mac(frw::RowAcc& acc, const uint32_t* __restrict__ row, uint32_t x) {
    const uint4 a = ((const uint4*)row)[0], b = ((const uint4*)row)[1];
    const uint32_t r[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    frw::rowacc_mac(acc, r, x);
}
__global__ void __launch_bounds__(kThreads, 4)  // four blocks per SM: 64 registers
    linear_combination_fr(const LinCombSrc* __restrict__ src, const uint32_t* __restrict__ rows, uint32_t n, uint64_t len,
                          Fr* __restrict__ out) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += stride) {
        Fr total = fr_zero();
        frw::RowAcc acc = frw::rowacc_zero();
        uint32_t terms = 0;
        for (uint32_t j = 0; j < n; j++) {
            const LinCombSrc s = src[j];
            if (i >= s.len) continue;
            if (terms + 8 > kRowTerms) {
                total = fr_add(total, frw::to_fr(frw::reduce_rows(acc.E, acc.O)));
                acc = frw::rowacc_zero();
                terms = 0;
            }
            const uint32_t* row = rows + (size_t)j * kLinRows * 8;
            if (s.dtype == DPB_FR) {
                const frw::F8 v = frw::from_fr(FrFam::load(s.ptr, DPB_FR, i));
#pragma unroll
                for (int w = 0; w < 8; w++) lincomb_row_mac(acc, row + 8 * w, v.w[w]);
                terms += 8;
            } else {
                const int64_t x = s.dtype == DPB_FR_I32 ? (int64_t)((const int32_t*)s.ptr)[i] : ((const int64_t*)s.ptr)[i];
                const uint64_t mag = x < 0 ? (uint64_t)0 - (uint64_t)x : (uint64_t)x;
                if (x < 0) row += 8;
                lincomb_row_mac(acc, row, (uint32_t)mag);
                if (mag >> 32) lincomb_row_mac(acc, row + 16, (uint32_t)(mag >> 32));
                terms += 2;
            }
        }
        FrFam::store(out, i, fr_add(total, frw::to_fr(frw::reduce_rows(acc.E, acc.O))));
    }
}
// Goldilocks: the products are added up unreduced
__global__ void __launch_bounds__(kThreads)
    linear_combination_gl(const LinCombSrc* __restrict__ src, const Gl2* __restrict__ coeff, uint32_t n, uint64_t len,
                          Gl2* __restrict__ out) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += stride) {
        EntrySum<GlFam, false> acc;
        acc.zero();
        for (uint32_t j = 0; j < n; j++) {
            const LinCombSrc s = src[j];
            if (i < s.len) acc.mac(coeff[j], s.ptr, s.dtype, i);
        }
        GlFam::store(out, i, acc.finish());
    }
}

}  // namespace dpb

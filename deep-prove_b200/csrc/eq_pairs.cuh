// Rounds of a sumcheck over  sum_t c_t * table_t * eq_t  with zero-padded tables: the claim batching of the opening
// (zkml/src/poly_commit/prover.rs:140-255), one term per claim, every claim with an eq table over its own point.
//
// What bounds these rounds is the number of field products, and most of them are not needed:
//  * With the first i variables of eq_t bound, its entries 2p, 2p + 1 are S ((1 - q_i), q_i) W[p], S = prod eq(q_k, r_k)
//    and W the eq table over the variables after i.  W of the next round is the sum of W's neighbouring entries: no
//    product, and the challenges never enter it.  So a round needs  A0 = sum f[2p] W[p]  and  A1 = sum f[2p + 1] W[p]
//    per term, and three scalar products turn them into the samples  c S (1 - q) A0,  c S q A1  and
//    c S (1 - 2q) (A0 - A1).
//  * A0 and A1 are sums: their products stay unreduced until a thread's part of them ends (frw::Wide, RowAcc).
//  * Integer entries multiply W as integers (8 multiply-adds instead of a conversion and a product) and fold through
//    two rows.
//  * The fold and the sums are one pass over the tables.
// Per pair of a later round: four folds' two products by the challenge (160 multiply-adds) and two unreduced products
// (128), where fold and evaluation over the general term list took 960 (folds of both tables, the coefficient, three
// points).  Claims on 12 polynomials of 2^20 (one in four chunks), 40 of 2^16 and 64 of 2^12, int32, BN254: the rounds
// took 3140 us in 39 launches before, 1477 us in 20 launches since.
#pragma once
#include "common.cuh"
#include "fused_int.cuh"
#include "lazy_sum.cuh"

namespace dpb {

constexpr uint32_t kEqPairsPerThread = 8;  // pairs a thread takes of one tile at most (RowAcc has room for 1024)

struct EqPairTerm {
    const void* f;   // the table
    const void* eq;  // the eq table (challenge elements)
    void* fb[2];     // the table bound to 1, 2, 3, .. challenges, in turn
    void* wb[2];     // W after rounds 0, 1, 2, .., in turn
    uint32_t q_off;  // the eq table's point in the points array
    uint16_t nv;     // variables of both tables
    uint16_t dtype;  // of f
    uint32_t f_id, eq_id;  // places of the two tables in the sumcheck's list
    uint32_t pad[2];
    alignas(16) uint8_t coeff[32];
};

// The sums A0, A1 of one thread over field entries.
template <class F>
struct PairSum;
template <>
struct PairSum<FrFam> {
    frw::Wide a0, a1;
    __device__ __forceinline__ void zero() { a0 = a1 = frw::wide_zero(); }
    __device__ __forceinline__ void mac(const Fr& f0, const Fr& f1, const Fr& w) {
        const frw::F8 ww = frw::from_fr(w);
        frw::wide_mac(a0, frw::from_fr(f0), ww);
        frw::wide_mac(a1, frw::from_fr(f1), ww);
    }
    __device__ __forceinline__ void finish(Fr (&a)[2]) const {
        a[0] = fr_wide_finish(a0);
        a[1] = fr_wide_finish(a1);
    }
};
template <>
struct PairSum<GlFam> {
    glw::A8 s00, s01, s10, s11;
    __device__ __forceinline__ void zero() { s00 = s01 = s10 = s11 = glw::acc_zero(); }
    __device__ __forceinline__ void mac(const Gl2& f0, const Gl2& f1, const Gl2& w) {
        const glw::W2 x = gl2_words(f0), y = gl2_words(f1), ww = gl2_words(w);
        const glw::W w7 = glw::mul7(ww.c1);
        glw::acc_mac(s00, x.c0, ww.c0);
        glw::acc_mac(s00, x.c1, w7);
        glw::acc_mac(s01, x.c0, ww.c1);
        glw::acc_mac(s01, x.c1, ww.c0);
        glw::acc_mac(s10, y.c0, ww.c0);
        glw::acc_mac(s10, y.c1, w7);
        glw::acc_mac(s11, y.c0, ww.c1);
        glw::acc_mac(s11, y.c1, ww.c0);
    }
    __device__ __forceinline__ static Gl2 one(const glw::A8& c0, const glw::A8& c1) {
        return gl2_make(glw::to_u64(glw::canon(glw::acc_reduce(c0))), glw::to_u64(glw::canon(glw::acc_reduce(c1))));
    }
    __device__ __forceinline__ void finish(Gl2 (&a)[2]) const {
        a[0] = one(s00, s01);
        a[1] = one(s10, s11);
    }
};

// The same over integer entries of round 0.  BN254: RowAcc sums of magnitude * (W or r - W), which its two reduction
// words divide by 2^64 (kScaled: the caller multiplies the tile's sums by 2^64); the rare magnitude of more than
// 32 bits takes a full product, divided by 2^64 to match.
template <class F>
struct IntPairSum;
template <>
struct IntPairSum<FrFam> {
    static constexpr bool kScaled = true;
    frw::RowAcc a0, a1;
    Fr rare0, rare1;
    __device__ __forceinline__ void zero() {
        a0 = a1 = frw::rowacc_zero();
        rare0 = rare1 = fr_zero();
    }
    __device__ __forceinline__ static void add(frw::RowAcc& a, Fr& rare, const frw::F8& w, const frw::F8& nw, int64_t x) {
        const uint64_t mag = x < 0 ? (uint64_t)0 - (uint64_t)x : (uint64_t)x;
        if (mag >> 32) {
            Fr two_m64;  // 2^-64 in Montgomery form: 2^192
            two_m64.l[0] = two_m64.l[1] = two_m64.l[2] = 0;
            two_m64.l[3] = 1;
            rare = fr_add(rare, fr_mul(fr_mul(frw::to_fr(w), fr_from_int_rows(x)), two_m64));
            return;
        }
        frw::F8 v;
#pragma unroll
        for (int i = 0; i < 8; i++) v.w[i] = x < 0 ? nw.w[i] : w.w[i];
        frw::rowacc_mac(a, v.w, (uint32_t)mag);
    }
    __device__ __forceinline__ void mac(int64_t x0, int64_t x1, const Fr& w) {
        const frw::F8 ww = frw::from_fr(w), nw = frw::from_fr(fr_neg(w));
        add(a0, rare0, ww, nw, x0);
        add(a1, rare1, ww, nw, x1);
    }
    __device__ __forceinline__ void finish(Fr (&a)[2]) {
        a[0] = fr_add(frw::to_fr(frw::reduce_rows(a0.E, a0.O)), rare0);
        a[1] = fr_add(frw::to_fr(frw::reduce_rows(a1.E, a1.O)), rare1);
    }
};
template <>
struct IntPairSum<GlFam> {
    static constexpr bool kScaled = false;
    glw::A8 s00, s01, s10, s11;
    __device__ __forceinline__ void zero() { s00 = s01 = s10 = s11 = glw::acc_zero(); }
    __device__ __forceinline__ void mac(int64_t x0, int64_t x1, const Gl2& w) {
        const uint64_t u0 = GlFam::base_from_int(x0), u1 = GlFam::base_from_int(x1);
        const glw::W a = glw::make_w((uint32_t)u0, (uint32_t)(u0 >> 32)), b = glw::make_w((uint32_t)u1, (uint32_t)(u1 >> 32));
        const glw::W2 ww = gl2_words(w);
        glw::acc_mac(s00, a, ww.c0);
        glw::acc_mac(s01, a, ww.c1);
        glw::acc_mac(s10, b, ww.c0);
        glw::acc_mac(s11, b, ww.c1);
    }
    __device__ __forceinline__ void finish(Gl2 (&a)[2]) const {
        a[0] = PairSum<GlFam>::one(s00, s01);
        a[1] = PairSum<GlFam>::one(s10, s11);
    }
};

// What the folds of a round multiply by.
template <class F>
struct EqPairKey;
template <>
struct EqPairKey<FrFam> {
    frw::FixedMul r;
    IntFoldKey ints;
    static EqPairKey make(const Fr& c) {
        EqPairKey k;
        fr_fixed_table(c, k.r);
        int_fold_key(c, k.ints);
        return k;
    }
    // entry p of the bound table of `in`
    __device__ __forceinline__ Fr fold(const void* in, int dtype, uint64_t p) const {
        if (dtype == DPB_FR_I32) {
            const int2 v = ((const int2*)in)[p];
            return fold_i32(ints, v.x, v.y);
        }
        if (dtype == DPB_FR_I64) {
            const longlong2 v = ((const longlong2*)in)[p];
            if (v.x == (int32_t)v.x && v.y == (int32_t)v.y) return fold_i32(ints, (int32_t)v.x, (int32_t)v.y);
        }
        Fr a, b;
        FrFam::load_pair(in, dtype, p, a, b);
        return fr_add(a, fr_mul_fixed(r, fr_sub(b, a)));
    }
};
template <>
struct EqPairKey<GlFam> {
    Gl2 r;
    static EqPairKey make(const Gl2& c) {
        EqPairKey k;
        k.r = c;
        return k;
    }
    __device__ __forceinline__ Gl2 fold(const void* in, int dtype, uint64_t p) const {
        Gl2 a, b;
        GlFam::load_pair(in, dtype, p, a, b);
        return GlFam::add(a, GlFam::mul(r, GlFam::sub(b, a)));
    }
};

// One round.  A tile is kThreads * per_thread pairs of one term (one item once a term's variables are all bound);
// tile_prefix[t] is term t's first tile.  s_in[t] holds prod eq(q_k, r_k) up to two rounds ago, s_out[t] gets one more.
// Publishes the samples P(0), P(1) and prod (f(0) - f(1)) of the round polynomial.
template <class F>
__global__ void __launch_bounds__(kThreads, 2)
    eq_pairs_round(const EqPairTerm* __restrict__ terms, uint32_t n_terms, const typename F::E* __restrict__ points,
                   const uint32_t* __restrict__ tile_prefix, uint32_t per_thread, uint32_t round, typename F::E r,
                   EqPairKey<F> key_g, const typename F::E* __restrict__ s_in, typename F::E* __restrict__ s_out,
                   ReduceScratch<F> rs, typename F::E* out) {
    typedef typename F::E E;
    __shared__ EqPairKey<F> key;
    __shared__ E sh_s;
    for (uint32_t i = threadIdx.x; i < sizeof(key) / 4; i += blockDim.x) ((uint32_t*)&key)[i] = ((const uint32_t*)&key_g)[i];
    __syncthreads();
    E acc[3] = {F::zero(), F::zero(), F::zero()};
    const uint32_t total_tiles = tile_prefix[n_terms];
    for (uint32_t tile = blockIdx.x; tile < total_tiles; tile += gridDim.x) {
        uint32_t lo = 0, hi = n_terms;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (tile_prefix[mid] <= tile) lo = mid;
            else hi = mid;
        }
        const EqPairTerm& t = terms[lo];
        const uint32_t nv = t.nv;
        const bool first = tile == tile_prefix[lo];
        // the scalar of the term, by a thread of the last warp while the others start on the pairs
        if (threadIdx.x == kThreads - 1) {
            E s = F::one();
            if (round > 0) {
                E e = F::sub(F::one(), r);  // a padded variable: 1 - r
                if (round - 1 < nv) {       // eq(q, r) = 1 - q - r + 2 q r
                    const E q = points[t.q_off + round - 1], qr = F::mul(q, r);
                    e = F::add(F::sub(e, q), F::add(qr, qr));
                }
                s = F::mul(s_in[lo], e);
            }
            if (first) s_out[lo] = s;
            sh_s = F::mul(s, *(const E*)t.coeff);
        }
        E a[2] = {F::zero(), F::zero()};
        const void* prev = round <= 1 ? t.f : t.fb[(round - 2) & 1];
        const int prev_dtype = round <= 1 ? (int)t.dtype : F::kChalDtype;
        const bool scaled = IntPairSum<F>::kScaled && round == 0 && t.dtype >= DPB_GL_I64;
        if (round >= nv) {
            if (threadIdx.x == 0) {  // one entry left (round 0 never gets here: every table has a variable)
                if (round == nv) a[0] = key.fold(prev, prev_dtype, 0);
                else a[0] = F::mul(F::load(prev, F::kChalDtype, 0), F::sub(F::one(), r));
                F::store(t.fb[(round - 1) & 1], 0, a[0]);
            }
        } else {
            const uint64_t n_pairs = 1ull << (nv - round - 1);
            const uint64_t p0 = (uint64_t)(tile - tile_prefix[lo]) * kThreads * per_thread + threadIdx.x;
            const void* w_in = round == 0 ? t.eq : t.wb[(round - 1) & 1];
            void* w_out = t.wb[round & 1];
            auto weight = [&](uint64_t p) {
                E x, y;
                F::load_pair(w_in, F::kChalDtype, p, x, y);
                const E w = F::add(x, y);
                F::store(w_out, p, w);
                return w;
            };
            if (round == 0 && t.dtype >= DPB_GL_I64) {
                IntPairSum<F> sum;
                sum.zero();
                for (uint32_t i = 0; i < per_thread; i++) {
                    const uint64_t p = p0 + (uint64_t)i * kThreads;
                    if (p >= n_pairs) break;
                    int64_t x0, x1;
                    if (t.dtype == DPB_FR_I32 || t.dtype == DPB_GL_I32) {
                        const int2 v = ((const int2*)t.f)[p];
                        x0 = v.x;
                        x1 = v.y;
                    } else {
                        const longlong2 v = ((const longlong2*)t.f)[p];
                        x0 = v.x;
                        x1 = v.y;
                    }
                    sum.mac(x0, x1, weight(p));
                }
                sum.finish(a);
            } else {
                PairSum<F> sum;
                sum.zero();
                for (uint32_t i = 0; i < per_thread; i++) {
                    const uint64_t p = p0 + (uint64_t)i * kThreads;
                    if (p >= n_pairs) break;
                    E f0, f1;
                    if (round == 0) {
                        F::load_pair(t.f, t.dtype, p, f0, f1);
                    } else {
                        f0 = key.fold(prev, prev_dtype, 2 * p);
                        f1 = key.fold(prev, prev_dtype, 2 * p + 1);
                        F::store(t.fb[(round - 1) & 1], 2 * p, f0);
                        F::store(t.fb[(round - 1) & 1], 2 * p + 1, f1);
                    }
                    sum.mac(f0, f1, weight(p));
                }
                sum.finish(a);
            }
        }
        block_sum<F, 2>(a);  // also orders sh_s before thread 0's read
        if (threadIdx.x == 0) {
            const E s = sh_s;
            if (scaled) {  // times 2^64 (2^320 is its Montgomery form)
                const E two64 = F::from_u64_pow64();
                a[0] = F::mul(a[0], two64);
                a[1] = F::mul(a[1], two64);
            }
            if (round >= nv) {
                const E v = F::mul(s, a[0]);
                acc[0] = F::add(acc[0], v);
                acc[2] = F::add(acc[2], v);
            } else {
                const E sq = F::mul(s, points[t.q_off + round]), s1 = F::sub(s, sq);  // S q, S (1 - q)
                acc[0] = F::add(acc[0], F::mul(s1, a[0]));
                acc[1] = F::add(acc[1], F::mul(sq, a[1]));
                acc[2] = F::add(acc[2], F::mul(F::sub(s1, sq), F::sub(a[0], a[1])));
            }
        }
        __syncthreads();  // sh_s is free again
    }
    grid_sum_publish<F, 3>(acc, rs, out);
}

// Every table's value at the point, r the last challenge and `round` the last round.
template <class F>
__global__ void __launch_bounds__(kThreads)
    eq_pairs_finals(const EqPairTerm* __restrict__ terms, uint32_t n_terms, const typename F::E* __restrict__ points,
                    uint32_t round, typename F::E r, const typename F::E* __restrict__ s_in, typename F::E* __restrict__ out) {
    typedef typename F::E E;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_terms) return;
    const EqPairTerm& t = terms[i];
    const void* last = round == 0 ? t.f : t.fb[(round - 1) & 1];
    const int dtype = round == 0 ? (int)t.dtype : F::kChalDtype;
    E e = F::sub(F::one(), r);
    if (round < t.nv) {  // the table has this variable (nv = round + 1)
        E a, b;
        F::load_pair(last, dtype, 0, a, b);
        out[t.f_id] = F::add(a, F::mul(r, F::sub(b, a)));
        const E q = points[t.q_off + round], qr = F::mul(q, r);
        e = F::add(F::sub(e, q), F::add(qr, qr));
    } else {
        out[t.f_id] = F::mul(F::load(last, dtype, 0), e);
    }
    out[t.eq_id] = F::mul(s_in[i], e);
}

}  // namespace dpb

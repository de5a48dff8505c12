// The sumcheck of a logup-GKR layer, from the layer's own formula (zkml/src/lookup/logup_gkr/circuit.rs:231-412).
//
// Per instance j the layer sums  alpha_j eq (n_lo d_hi + n_hi d_lo + lambda d_lo d_hi),  where in an instance's input
// layer d = c + column_0 + s column_1, a lookup's numerators are -1 and a table's its multiplicities.  An instance is kept
// as the tables C = d_lo, D = d_hi, U = n_hi + lambda D and A = n_lo of  g = C U + A D  (a lookup's input layer as C and D
// alone: g = lambda C D - C - D).  They are linear in the original tables, so they are bound like them; C, D and U
// take the place of the originals from round 1 on, and the originals are read off at the end (columns of an input layer
// that are not linear in C and D are evaluated at the point once).  A round is sampled at 0, 1 (round 0 only: later the
// host knows s(0) + s(1)) and infinity, without the factor of eq's bound and current variables, which is the host's;
// a pair's weight is the eq table's original entry at the stride of the round: nothing of it is bound or stored.
//
// Two kernels run the rounds.  logup_layer_round takes the large ones, bound by their products: one thread per pair and
// slice of the instances, products of two tables summed before they are reduced, the sum over the instances kept as
// unreduced rows of alpha_j.  sc_tail_logup takes the rest in one launch.
#pragma once
#include <cooperative_groups.h>

#include "generic_round.cuh"
#include "lazy_sum.cuh"

namespace dpb {

namespace cg = cooperative_groups;

constexpr int kLogupInner = 0, kLogupLookup = 1, kLogupTable = 2;
constexpr uint32_t kLogupMaxInst = 128;

// One instance on the device.  Tables ("slots"): 0 C, 1 D, 2 U, 3 A; a lookup's input layer has the first two.
struct LgInst {
    const void* orig[6];  // inner: n_lo, n_hi, d_lo, d_hi; otherwise (multiplicities' halves,) columns' low, high halves
    void* buf[4][2];      // the slots bound to 1, 2, 3, .. challenges, in turn
    int8_t dtype[6];
    uint16_t kind, ncol;
    uint16_t first;       // place of its first original table in the sumcheck's list
    uint16_t tab0;        // first of its tables in the resident kernel's shared memory
    uint16_t pad;
};
__host__ __device__ __forceinline__ uint32_t lg_slots(const LgInst& in) { return in.kind == kLogupLookup ? 2u : 4u; }

template <class F>
struct LgConst {
    typename F::E alpha, sep, c;
};

// Where a round's tables come from.
constexpr int kLgOriginal = 0;  // round 0: the originals
constexpr int kLgBind = 1;      // round 1: the originals, bound to the first challenge
constexpr int kLgSlots = 2;     // later: the slots of the round before, bound

// Rows for the integer columns of an input layer (BN254): a column entry enters as the unsigned word x + 2^31.
// Round 0: c' + x + s y with rows of 1 and s; round 1: c' + (1 - r) x_0 + r x_1 + s (..) with rows of 1 - r, r,
// s (1 - r), s r; c' = c - 2^31 (1 + s) takes the 2^31 back in both (without the second column: c - 2^31).
struct LgRows {
    uint32_t row[4][8];
    uint32_t c[8];
};
__device__ __forceinline__ bool lg_fits32(int64_t x) { return x == (int64_t)(int32_t)x; }
__device__ __forceinline__ int64_t lg_int(const void* p, int dtype, uint64_t i) {
    return dtype == DPB_FR_I32 ? (int64_t)((const int32_t*)p)[i] : ((const int64_t*)p)[i];
}

// original table q at entry e, bound to r in round 1
template <class F, int MODE>
__device__ __forceinline__ typename F::E lg_entry(const LgInst& in, uint32_t q, uint64_t e, const typename F::FoldKey& rk) {
    if (MODE == kLgOriginal) return F::load(in.orig[q], in.dtype[q], e);
    typename F::E a, b;
    F::load_pair(in.orig[q], in.dtype[q], e, a, b);
    return F::add(a, F::mul_key(rk, F::sub(b, a)));
}

// The denominator of an input layer's low (half 0) or high columns.
template <class F, int MODE>
__device__ __forceinline__ typename F::E lg_columns(const LgInst& in, const LgConst<F>& k, const LgRows*, uint32_t half, uint64_t e,
                                                    const typename F::FoldKey& rk) {
    typedef typename F::E E;
    const uint32_t q = (in.kind == kLogupTable ? 2u : 0u) + half * in.ncol;
    E v = F::add(k.c, lg_entry<F, MODE>(in, q, e, rk));
    if (in.ncol == 2) v = F::add(v, F::mul(k.sep, lg_entry<F, MODE>(in, q + 1, e, rk)));
    return v;
}
template <int MODE>
__device__ __forceinline__ Fr lg_columns_fr(const LgInst& in, const LgConst<FrFam>& k, const LgRows* rows, uint32_t half, uint64_t e,
                                            const frw::FixedMul& rk) {
    const uint32_t q = (in.kind == kLogupTable ? 2u : 0u) + half * in.ncol;
    if (rows) {
        int64_t x[4];
        bool fits = true;
#pragma unroll
        for (uint32_t j = 0; j < 2; j++) {
            if (j >= in.ncol) {
                x[2 * j] = x[2 * j + 1] = 0;
                continue;
            }
            if (MODE == kLgOriginal) {
                x[2 * j] = lg_int(in.orig[q + j], in.dtype[q + j], e);
                x[2 * j + 1] = 0;
            } else {
                x[2 * j] = lg_int(in.orig[q + j], in.dtype[q + j], 2 * e);
                x[2 * j + 1] = lg_int(in.orig[q + j], in.dtype[q + j], 2 * e + 1);
            }
            fits = fits && lg_fits32(x[2 * j]) && lg_fits32(x[2 * j + 1]);
        }
        if (fits) {
            frw::RowAcc acc = frw::rowacc_zero();
            // c' * 2^64 at word positions 2..9, the upper two words in O, whose carry word cannot overflow
#pragma unroll
            for (int w = 0; w < 6; w++) acc.E[2 + w] = rows->c[w];
            acc.O[8] = rows->c[6];
            acc.O[9] = rows->c[7];
            auto word = [](int64_t y) { return (uint32_t)y ^ 0x80000000u; };
            frw::rowacc_mac(acc, rows->row[0], word(x[0]));
            if (MODE == kLgBind) frw::rowacc_mac(acc, rows->row[1], word(x[1]));
            if (in.ncol == 2) {
                frw::rowacc_mac(acc, rows->row[2], word(x[2]));
                if (MODE == kLgBind) frw::rowacc_mac(acc, rows->row[3], word(x[3]));
            }
            // below c' + r (1 + 2^-29): one subtraction leaves a sliver above r, which the top word gives away
            frw::F8 v = frw::reduce_rows(acc.E, acc.O);
            if (v.w[7] >= DPB_FRW_P7) v = frw::reduce_once(v);
            return frw::to_fr(v);
        }
    }
    return lg_columns<FrFam, MODE>(in, k, nullptr, half, e, rk);
}
template <class F, int MODE>
struct LgColumns {
    __device__ __forceinline__ static typename F::E get(const LgInst& in, const LgConst<F>& k, const LgRows* rows, uint32_t half,
                                                        uint64_t e, const typename F::FoldKey& rk) {
        return lg_columns<F, MODE>(in, k, rows, half, e, rk);
    }
};
template <int MODE>
struct LgColumns<FrFam, MODE> {
    __device__ __forceinline__ static Fr get(const LgInst& in, const LgConst<FrFam>& k, const LgRows* rows, uint32_t half, uint64_t e,
                                             const frw::FixedMul& rk) {
        return lg_columns_fr<MODE>(in, k, rows, half, e, rk);
    }
};

// Entry e of a slot in the round's tables.  `prev`: which of the slots' buffers holds the round before (kLgSlots).
template <class F, int MODE>
__device__ __forceinline__ typename F::E lg_slot(const LgInst& in, const LgConst<F>& k, uint32_t slot, uint64_t e,
                                                 const typename F::FoldKey& rk, const typename F::FoldKey& lamk, uint32_t prev) {
    typedef typename F::E E;
    if (MODE == kLgSlots) {
        E a, b;
        F::load_pair(in.buf[slot][prev], F::kChalDtype, e, a, b);
        return F::add(a, F::mul_key(rk, F::sub(b, a)));
    }
    const bool inner = in.kind == kLogupInner;
    if (slot == 0) return inner ? lg_entry<F, MODE>(in, 2, e, rk) : LgColumns<F, MODE>::get(in, k, nullptr, 0, e, rk);
    if (slot == 3) return lg_entry<F, MODE>(in, 0, e, rk);
    const E d = inner ? lg_entry<F, MODE>(in, 3, e, rk) : LgColumns<F, MODE>::get(in, k, nullptr, 1, e, rk);
    if (slot == 1) return d;
    return F::add(lg_entry<F, MODE>(in, 1, e, rk), F::mul_key(lamk, d));
}

// Sums over instances of alpha_j t_j as unreduced rows.
template <class F>
struct AlphaSum;
template <>
struct AlphaSum<FrFam> {
    typedef frw::FixedMul Key;
    frw::RowAcc s;
    __device__ __forceinline__ void zero() { s = frw::rowacc_zero(); }
    __device__ __forceinline__ void mac(const Key& k, const Fr& t) {  // 8 rows a time: kLogupMaxInst of them stay below 2^296
        const frw::F8 v = frw::from_fr(t);
#pragma unroll
        for (int w = 0; w < 8; w++) frw::rowacc_mac(s, k.c[w], v.w[w]);
    }
    __device__ __forceinline__ Fr finish() { return frw::to_fr(frw::reduce_rows(s.E, s.O)); }
};
template <>
struct AlphaSum<GlFam> {
    typedef Gl2 Key;
    glw::A8 s0, s1;
    __device__ __forceinline__ void zero() { s0 = s1 = glw::acc_zero(); }
    __device__ __forceinline__ void mac(const Key& k, const Gl2& t) {
        const glw::W2 a = gl2_words(k), v = gl2_words(t);
        glw::acc_mac(s0, a.c0, v.c0);
        glw::acc_mac(s0, glw::mul7(a.c1), v.c1);
        glw::acc_mac(s1, a.c0, v.c1);
        glw::acc_mac(s1, a.c1, v.c0);
    }
    __device__ __forceinline__ Gl2 finish() {
        return gl2_make(glw::to_u64(glw::canon(glw::acc_reduce(s0))), glw::to_u64(glw::canon(glw::acc_reduce(s1))));
    }
};

// One round of a layer whose instances are all of one kind, one thread per pair and slice of inst_per_slice instances (a
// round with few pairs still fills the GPU).
// Publishes the sums at 0, 1 (round 0 only) and infinity.  Three instances, BN254: layer of 2^19, rounds 0 / 1 / 2 305 /
// 227 / 145 us, top layer (integer columns) 557 / 412 / 203 us with every term reduced, the columns widened and all of
// them bound; 236 / 208 / 104 and 430 / 211 / 99 us since (three blocks of 128 threads per SM once the slots are bound,
// two before: 524 / 269 us in rounds 0 / 1 of the top layer at three).
template <class F, int MODE, int KIND>
__global__ void __launch_bounds__(128, sizeof(typename F::E) == 16 ? 4 : MODE == kLgSlots ? 3 : 2)
    logup_layer_round(const LgInst* __restrict__ inst_g, const LgConst<F>* __restrict__ consts_g,
                      const typename AlphaSum<F>::Key* __restrict__ alphas_g, const LgRows* __restrict__ rows_g, uint32_t n_inst,
                      const __grid_constant__ typename F::FoldKey rk_g, const __grid_constant__ typename F::FoldKey lamk_g,
                      const typename F::E* __restrict__ eq, uint32_t eq_stride_log2, uint64_t n_pairs, uint32_t prev,
                      uint32_t blocks_x, uint32_t inst_per_slice, ReduceScratch<F> rs, typename F::E* out) {
    typedef typename F::E E;
    typedef typename AlphaSum<F>::Key Key;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ typename F::FoldKey rk, lamk;
    for (uint32_t i = threadIdx.x; i < sizeof(rk) / 4; i += blockDim.x) {
        ((uint32_t*)&rk)[i] = ((const uint32_t*)&rk_g)[i];
        ((uint32_t*)&lamk)[i] = ((const uint32_t*)&lamk_g)[i];
    }
    const uint32_t slice = blockIdx.x / blocks_x, bx = blockIdx.x % blocks_x;
    const uint32_t i_begin = slice * inst_per_slice, i_end = min(n_inst, i_begin + inst_per_slice);
    // this slice's instances and keys on chip
    Key* keys = (Key*)smem_raw;
    LgInst* inst = (LgInst*)(keys + inst_per_slice);
    {
        const uint32_t n = i_end - i_begin;
        for (uint32_t i = threadIdx.x; i < n * (uint32_t)(sizeof(Key) / 4); i += blockDim.x)
            ((uint32_t*)keys)[i] = ((const uint32_t*)(alphas_g + i_begin))[i];
        for (uint32_t i = threadIdx.x; i < n * (uint32_t)(sizeof(LgInst) / 4); i += blockDim.x)
            ((uint32_t*)inst)[i] = ((const uint32_t*)(inst_g + i_begin))[i];
    }
    __syncthreads();
    E acc[3] = {F::zero(), F::zero(), F::zero()};
    const uint64_t stride = (uint64_t)blocks_x * blockDim.x;
    for (uint64_t p = (uint64_t)bx * blockDim.x + threadIdx.x; p < n_pairs; p += stride) {
        AlphaSum<F> s0, s1, si;
        s0.zero();
        s1.zero();
        si.zero();
        for (uint32_t i = i_begin; i < i_end; i++) {
            const LgInst& in = inst[i - i_begin];
            const LgConst<F>& k = consts_g[i];
            const LgRows* rows = rows_g ? rows_g + i : nullptr;
            auto value = [&](uint32_t slot, uint64_t e) -> E {
                if (MODE == kLgSlots) return lg_slot<F, kLgSlots>(in, k, slot, e, rk, lamk, prev);
                constexpr int M = MODE == kLgSlots ? kLgOriginal : MODE;
                if (slot == 3) return lg_entry<F, M>(in, 0, e, rk);
                if (KIND == kLogupInner) return lg_entry<F, M>(in, slot == 0 ? 2 : 3, e, rk);
                return LgColumns<F, M>::get(in, k, rows, slot, e, rk);
            };
            auto pair = [&](uint32_t slot, E& f0, E& f1) {
                f0 = value(slot, 2 * p);
                f1 = value(slot, 2 * p + 1);
                if (MODE != kLgOriginal) {
                    E* o = (E*)in.buf[slot][MODE == kLgBind ? 0 : prev ^ 1];
                    F::store(o, 2 * p, f0);
                    F::store(o, 2 * p + 1, f1);
                }
            };
            E c0, c1, d0, d1;
            pair(0, c0, c1);
            pair(1, d0, d1);
            const Key& al = keys[i - i_begin];
            if (KIND == kLogupLookup) {
                // lambda C D - C - D; the last two do not reach infinity
                s0.mac(al, F::sub(F::mul_key(lamk, F::mul(c0, d0)), F::add(c0, d0)));
                if (MODE == kLgOriginal) s1.mac(al, F::sub(F::mul_key(lamk, F::mul(c1, d1)), F::add(c1, d1)));
                si.mac(al, F::mul_key(lamk, F::mul(F::sub(c1, c0), F::sub(d1, d0))));
                continue;
            }
            E a0, a1;
            pair(3, a0, a1);
            E u0, u1;
            if (MODE == kLgSlots) {
                pair(2, u0, u1);
            } else {  // D is at hand: no second look at the tables it comes from
                u0 = F::add(lg_entry<F, MODE == kLgSlots ? kLgOriginal : MODE>(in, 1, 2 * p, rk), F::mul_key(lamk, d0));
                u1 = F::add(lg_entry<F, MODE == kLgSlots ? kLgOriginal : MODE>(in, 1, 2 * p + 1, rk), F::mul_key(lamk, d1));
                if (MODE == kLgBind) {
                    F::store(in.buf[2][0], 2 * p, u0);
                    F::store(in.buf[2][0], 2 * p + 1, u1);
                }
            }
            s0.mac(al, TwoProducts<F>::sum(c0, u0, a0, d0));
            if (MODE == kLgOriginal) s1.mac(al, TwoProducts<F>::sum(c1, u1, a1, d1));
            si.mac(al, TwoProducts<F>::sum(F::sub(c1, c0), F::sub(u1, u0), F::sub(a1, a0), F::sub(d1, d0)));
        }
        const E w = F::load(eq, F::kChalDtype, p << eq_stride_log2);
        acc[0] = F::add(acc[0], F::mul(w, s0.finish()));
        if (MODE == kLgOriginal) acc[1] = F::add(acc[1], F::mul(w, s1.finish()));
        acc[2] = F::add(acc[2], F::mul(w, si.finish()));
    }
    grid_sum_publish<F, 3>(acc, rs, out);
}

// The slots' values at the point, 4 per instance (C, D, U, A), when the resident kernel did not run.
template <class F>
__global__ void __launch_bounds__(128)
    logup_layer_finals(const LgInst* __restrict__ inst, const LgConst<F>* __restrict__ consts, uint32_t n_inst, typename F::FoldKey rk,
                       typename F::FoldKey lamk, uint32_t last_round, typename F::E* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_inst) return;
    const LgInst& in = inst[i];
    for (uint32_t s = 0; s < lg_slots(in); s++)
        out[4 * i + s] = last_round == 0 ? lg_slot<F, kLgBind>(in, consts[i], s, 0, rk, lamk, 0)
                                         : lg_slot<F, kLgSlots>(in, consts[i], s, 0, rk, lamk, (last_round - 1) & 1);
}

// ---- the resident kernel ----------------------------------------------------------
//
// Most of a batched logup proof is rounds of a few hundred pairs or fewer, and there the latency of one thread's chain
// of products, of barriers and of trips to memory is what the proof waits for (the generic resident kernel walks the
// layer's term list: 16 dependent products per pair and point).  Here
//  * the slots live in shared memory for all rounds; nothing is written back: when the host was held up beyond the
//    kernel's limit, the rounds so far are played again from the tables the first of them read;
//  * items are (instance, pair) over the threads; a pair is weighted by the eq table, an instance by its alpha once per
//    round;
//  * a cluster of eight blocks runs the rounds that are too large for one: every block holds a contiguous eighth of the
//    pairs, partial sums and the challenge travel through distributed shared memory, and one block goes on alone once
//    32 pairs (BN254; 256 Goldilocks, fewer with many tables) are left.  Blocks of a cluster are resident together, so
//    their barriers end; the one wait for the host is bounded and its outcome is handed to all.
// Measured, BN254, three instances of 2^21 rows: 144 rounds of up to 256 pairs took 3460 us in sc_tail_generic and 32
// rounds of up to 2048 pairs 1100 us as fold + evaluation launches and the gaps between them; 176 rounds take 2730 us
// here (15.5 us each, of which the host's transcript and the bus take 6).  A lookup of 2^10 rows: 1100 us and 680 us.
constexpr uint32_t kLogupTailBlocks = 8;     // the cluster (the portable size)

// Bound tables in shared memory: entry e of table t, n entries each; word planes keep neighbouring entries apart.
template <class F>
struct TailTabs {
    typedef typename F::E E;
    static constexpr int W = sizeof(E) / 16;
    uint4* base;
    uint32_t n;
    __device__ __forceinline__ E get(uint32_t t, uint32_t e) const {
        E v;
        uint4* q = (uint4*)&v;
#pragma unroll
        for (int w = 0; w < W; w++) q[w] = base[((size_t)t * W + w) * n + e];
        return v;
    }
    __device__ __forceinline__ void put(uint32_t t, uint32_t e, const E& v) const {
        const uint4* q = (const uint4*)&v;
#pragma unroll
        for (int w = 0; w < W; w++) base[((size_t)t * W + w) * n + e] = q[w];
    }
};

// Entries per table of the two sets of tables (even rounds, odd rounds), nb pairs of a block in the first round: a
// cluster's first block needs room for all that is left when it goes on alone, in whichever set that falls.
__host__ __device__ __forceinline__ size_t logup_tail_set_entries(size_t nb, uint32_t blocks, uint32_t alone, int set) {
    const size_t own = set ? (nb > 1 ? nb : 1) : 2 * nb, gathered = blocks > 1 ? 2 * (size_t)alone : 0;
    return own > gathered ? own : gathered;
}

__host__ __device__ __forceinline__ size_t logup_tail_weights(size_t nb, uint32_t blocks, uint32_t alone) {
    return blocks > 1 && alone > nb ? alone : nb;
}

// `extra`: the second columns of input layers are bound too (the kernel starts from the originals), and every original
// table can be read off at the end.  MODE: where the first round's tables come from; prev: see lg_slot.
template <class F, int MODE>
__global__ void __launch_bounds__(kTailThreads)
    sc_tail_logup(const LgInst* __restrict__ inst_g, const LgConst<F>* __restrict__ consts_g, uint32_t n_inst, uint32_t n_tabs,
                  uint32_t extra, typename F::E lambda, const typename F::E* __restrict__ eq, uint32_t eq_stride_log2,
                  typename F::E r, uint32_t prev, uint32_t first_round, uint32_t n_rounds, uint32_t alone, TailBox* box,
                  unsigned long long wait_ns) {
    typedef typename F::E E;
    constexpr int W8 = sizeof(E) / 8;
    cg::cluster_group cluster = cg::this_cluster();
    uint32_t blocks = cluster.num_blocks();
    const uint32_t rank = cluster.block_rank();
    // [constants per instance | W of the first round | tables of even rounds | of odd rounds | instances]
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(16) E sh_r;
    __shared__ int sh_stop;
    __shared__ typename F::FoldKey sh_key, sh_lam;
    __shared__ __align__(16) E sh_part[3][kLogupTailBlocks];
    __shared__ __align__(16) E sh_sum[3][kLogupMaxInst];
    const uint32_t first_pairs = (1u << (n_rounds - first_round - 1)) / blocks;  // of this block
    LgConst<F>* consts = (LgConst<F>*)smem_raw;
    E* weights = (E*)(consts + n_inst);
    uint4* const tab_mem = (uint4*)(weights + logup_tail_weights(first_pairs, blocks, alone));
    const size_t set_words = (size_t)n_tabs * TailTabs<F>::W * logup_tail_set_entries(first_pairs, blocks, alone, 0);
    LgInst* inst = (LgInst*)(tab_mem + set_words +
                             (size_t)n_tabs * TailTabs<F>::W * logup_tail_set_entries(first_pairs, blocks, alone, 1));
    for (uint32_t i = threadIdx.x; i < n_inst * (uint32_t)(sizeof(LgConst<F>) / 4); i += blockDim.x)
        ((uint32_t*)consts)[i] = ((const uint32_t*)consts_g)[i];
    for (uint32_t i = threadIdx.x; i < n_inst * (uint32_t)(sizeof(LgInst) / 4); i += blockDim.x)
        ((uint32_t*)inst)[i] = ((const uint32_t*)inst_g)[i];
    for (uint32_t p = threadIdx.x; p < first_pairs; p += blockDim.x)
        weights[p] = F::load(eq, F::kChalDtype, ((uint64_t)rank * first_pairs + p) << eq_stride_log2);
    F::fold_key_block(r, &sh_key);
    F::fold_key_block(lambda, &sh_lam);
    if (blocks > 1) cluster.sync();  // every block has started: its shared memory may be written
    if (threadIdx.x == 0) {
        if (rank == 0) {
            const int stop = tail_hello(box, kTailHelloNs) ? 0 : 1;
            for (uint32_t b = 0; b < blocks; b++) *cluster.map_shared_rank(&sh_stop, b) = stop;
        }
    }
    if (blocks > 1) cluster.sync();
    else __syncthreads();
    if (sh_stop) return;

    TailTabs<F> cur, old;
    cur.base = old.base = tab_mem;
    cur.n = 2 * first_pairs;
    // first round: the instances' tables from the originals, this block's entries
    {
        const uint64_t e0 = (uint64_t)rank * 2 * first_pairs;
        for (uint32_t w = threadIdx.x; w < n_tabs * cur.n; w += blockDim.x) {
            const uint32_t t = w / cur.n, e = w % cur.n;
            uint32_t i = 0, hi = n_inst;  // the instance of table t: tables are laid out instance by instance
            while (hi - i > 1) {
                const uint32_t mid = (i + hi) >> 1;
                if (inst[mid].tab0 <= t) i = mid;
                else hi = mid;
            }
            const LgInst& in = inst[i];
            const uint32_t slot = t - in.tab0, slots = lg_slots(in);
            E v;
            if (slot < slots) {
                v = lg_slot<F, MODE>(in, consts[i], slot, e0 + e, sh_key, sh_lam, prev);
            } else {  // the second column's halves, for the end (only from the originals: MODE is not kLgSlots then)
                const uint32_t q = (in.kind == kLogupTable ? 2u : 0u) + (slot - slots) * 2 + 1;
                v = lg_entry<F, MODE == kLgSlots ? kLgOriginal : MODE>(in, q, e0 + e, sh_key);
            }
            cur.put(t, e, v);
        }
        __syncthreads();
    }
    uint32_t nb = first_pairs;  // pairs of this block
    for (uint32_t round = first_round; round < n_rounds; round++) {
        if (round > first_round) {
            // bind the previous challenge
            const bool gather = blocks > 1 && nb * blocks <= 2 * alone;  // block 0 goes on alone
            old = cur;
            nb = gather ? nb * blocks / 2 : nb / 2;
            cur.n = 2 * nb;
            cur.base = tab_mem + (((round - first_round) & 1) ? set_words : 0);
            const E rr = sh_r;
            const uint32_t items = n_tabs * cur.n;
            const bool use_key = items > 2 * blockDim.x;  // rows pay once a thread has several products to make
            if (use_key) {
                F::fold_key_block(rr, &sh_key);
                __syncthreads();
            }
            if (!gather || rank == 0) {
                for (uint32_t w = threadIdx.x; w < items; w += blockDim.x) {
                    const uint32_t t = w / cur.n, e = w % cur.n;
                    E a, b;
                    if (gather) {
                        TailTabs<F> src = old;
                        src.base = cluster.map_shared_rank(old.base, (2 * e) / old.n);
                        a = src.get(t, (2 * e) % old.n);
                        b = src.get(t, (2 * e) % old.n + 1);
                    } else {
                        a = old.get(t, 2 * e);
                        b = old.get(t, 2 * e + 1);
                    }
                    const E d = F::sub(b, a);
                    cur.put(t, e, F::add(a, use_key ? F::mul_key(sh_key, d) : F::mul(rr, d)));
                }
            }
            if (gather) {
                // the weights come along (through the sums' space); then the other blocks are done
                static_assert(kTailAloneGl <= 3 * kLogupMaxInst, "the weights pass through sh_sum");
                if (rank == 0) {
                    const uint32_t stride = first_pairs * blocks / nb;  // in the first round's weights
                    for (uint32_t p = threadIdx.x; p < nb; p += blockDim.x) {
                        const uint32_t at = p * stride;
                        (&sh_sum[0][0])[p] = cluster.map_shared_rank(weights, at / first_pairs)[at % first_pairs];
                    }
                }
                cluster.sync();
                if (rank != 0) return;
                for (uint32_t p = threadIdx.x; p < nb; p += blockDim.x) weights[p] = (&sh_sum[0][0])[p];
                blocks = 1;
            }
            __syncthreads();
        }
        const uint32_t n_all = 1u << (n_rounds - round - 1);  // pairs of the round, over all blocks
        // stride of the round in `weights`
        const uint32_t wstride = (blocks == 1 && cluster.num_blocks() > 1) ? alone / n_all : first_pairs / nb;
        const bool with_one = round == 0;
        const uint32_t items = n_inst * nb, parts = nb > 32 ? nb / 32 : 1;
        for (uint32_t w0 = 0; w0 < items; w0 += blockDim.x) {
            const uint32_t w = w0 + threadIdx.x;
            if ((w & ~31u) >= items) continue;  // whole warps: the sums below shuffle
            const uint32_t i = w / nb, p = w % nb;
            E g0 = F::zero(), g1 = F::zero(), gi = F::zero();
            if (w < items) {
                const LgInst& in = inst[i];
                const E wt = weights[p * wstride];
                const E c0 = cur.get(in.tab0, 2 * p), d0 = cur.get(in.tab0 + 1, 2 * p);
                const E c1 = cur.get(in.tab0, 2 * p + 1), d1 = cur.get(in.tab0 + 1, 2 * p + 1);
                const E dc = F::sub(c1, c0), dd = F::sub(d1, d0);
                if (in.kind == kLogupLookup) {
                    g0 = F::sub(F::mul(c0, F::sub(F::mul(lambda, d0), F::one())), d0);
                    gi = F::mul(dc, F::mul(lambda, dd));
                    if (with_one) g1 = F::sub(F::mul(c1, F::sub(F::mul(lambda, d1), F::one())), d1);
                } else {
                    const E u0 = cur.get(in.tab0 + 2, 2 * p), a0 = cur.get(in.tab0 + 3, 2 * p);
                    const E u1 = cur.get(in.tab0 + 2, 2 * p + 1), a1 = cur.get(in.tab0 + 3, 2 * p + 1);
                    g0 = TwoProducts<F>::sum(c0, u0, a0, d0);
                    gi = TwoProducts<F>::sum(dc, F::sub(u1, u0), F::sub(a1, a0), dd);
                    if (with_one) g1 = TwoProducts<F>::sum(c1, u1, a1, d1);
                }
                g0 = F::mul(g0, wt);
                gi = F::mul(gi, wt);
                if (with_one) g1 = F::mul(g1, wt);
            }
            g0 = segment_sum<F>(g0, nb);
            gi = segment_sum<F>(gi, nb);
            if (with_one) g1 = segment_sum<F>(g1, nb);
            if (w < items && (p & 31) == 0) {
                sh_sum[0][i * parts + p / 32] = g0;
                sh_sum[1][i * parts + p / 32] = g1;
                sh_sum[2][i * parts + p / 32] = gi;
            }
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            const uint32_t lane = threadIdx.x;
            E v0 = F::zero(), v1 = F::zero(), vi = F::zero();
            for (uint32_t s = lane; s < n_inst * parts; s += 32) {
                const E al = consts[s / parts].alpha;
                v0 = F::add(v0, F::mul(al, sh_sum[0][s]));
                vi = F::add(vi, F::mul(al, sh_sum[2][s]));
                if (with_one) v1 = F::add(v1, F::mul(al, sh_sum[1][s]));
            }
            uint32_t span = 1;
            while (span < 32 && span < n_inst * parts) span *= 2;
            v0 = segment_sum<F>(v0, span);
            vi = segment_sum<F>(vi, span);
            if (with_one) v1 = segment_sum<F>(v1, span);
            if (lane == 0) {
                E* dst = blocks > 1 ? cluster.map_shared_rank(&sh_part[0][0], 0) : &sh_part[0][0];
                const uint32_t at = blocks > 1 ? rank : 0;
                dst[at] = v0;
                dst[kLogupTailBlocks + at] = v1;
                dst[2 * kLogupTailBlocks + at] = vi;
            }
            __syncwarp();
        }
        if (blocks > 1) cluster.sync();
        if (rank == 0 && threadIdx.x < 32) {
            const uint32_t lane = threadIdx.x;
            // lanes 0..7: the blocks' sums at 0; 8..15: at 1; 16..23: at infinity
            const uint32_t pt = lane / kLogupTailBlocks, b = lane % kLogupTailBlocks;
            E v = (pt < 3 && b < blocks) ? sh_part[pt][b] : F::zero();
            v = segment_sum<F>(v, blocks > 1 ? kLogupTailBlocks : 1);
            if (pt < 3 && b == 0 && (pt != 1 || with_one)) chunks_store<E>(&box->evals[pt * W8], v, round + 1);
            uint64_t word = 0;
            const int stop = tail_wait<E>(box, round + 1, wait_ns, word);
            for (uint32_t q = 0; q < blocks; q++) {
                if (lane < W8) ((uint64_t*)cluster.map_shared_rank(&sh_r, q))[lane] = word;
                if (lane == 0) *cluster.map_shared_rank(&sh_stop, q) = stop;
            }
            __syncwarp();
        }
        if (blocks > 1) cluster.sync();
        else __syncthreads();
        if (sh_stop) return;
    }
    // one pair per table left: bind the last challenge and read the original tables off
    for (uint32_t i = threadIdx.x; i < n_inst; i += blockDim.x) {
        const LgInst& in = inst[i];
        const E rr = sh_r;
        auto final_of = [&](uint32_t slot) {
            const E a = cur.get(in.tab0 + slot, 0), b = cur.get(in.tab0 + slot, 1);
            return F::add(a, F::mul(rr, F::sub(b, a)));
        };
        auto post = [&](uint32_t table, const E& v) { chunks_store<E>(&box->finals[table * W8], v, n_rounds + 1); };
        const E c = final_of(0), d = final_of(1);
        uint32_t col = in.first;
        if (in.kind != kLogupLookup) {
            post(in.first, final_of(3));
            post(in.first + 1, F::sub(final_of(2), F::mul(lambda, d)));
            col += 2;
        }
        if (in.kind == kLogupInner) {
            post(col, c);
            post(col + 1, d);
            continue;
        }
        if (!extra) continue;  // the host evaluates the columns
        for (uint32_t half = 0; half < 2; half++) {
            E x = F::sub(half ? d : c, consts[i].c);
            if (in.ncol == 2) {
                const E y = final_of(lg_slots(in) + half);
                post(col + half * 2 + 1, y);
                x = F::sub(x, F::mul(consts[i].sep, y));
            }
            post(col + half * in.ncol, x);
        }
    }
}

}  // namespace dpb

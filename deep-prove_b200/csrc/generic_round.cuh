// One-pass sumcheck round for any list of product terms.
//
// A round of the generic prover used to be two launches: bind the previous
// challenge into every table (read 2^v, write 2^(v-1)), then evaluate the terms
// (read 2^(v-1) again).  Here one kernel does both: a thread that owns pair p
// of this round reads the four previous-round entries 4p..4p+3 of every table,
// binds the challenge, stores the two new entries and evaluates the terms on
// them while they are still on chip.
//
// Three things cut the multiplies per pair:
//  * every table is loaded and bound once per pair, whatever the number of
//    terms that use it: the pair (value at 0, difference) of each table sits in
//    a per-thread slot of shared memory, and moving to the next evaluation point
//    is one addition per table;
//  * after round 0 the value at 1 is not computed: the host gets it from the
//    previous round polynomial (s(0) + s(1) = previous s(r));
//  * terms that share a table are grouped on the host, and that table
//    multiplies the group's sum once per point instead of once per term.
// Results are exact field sums, so they equal the two-pass kernels' bit for bit.
#pragma once
#include <cooperative_groups.h>

#include <algorithm>
#include <vector>

#include "sumcheck_kernels.cuh"

namespace dpb {

// A table as one round's kernel sees it.
struct RoundTab {
    const void* in;    // fold mode: the table of the previous round; otherwise this round's table
    void* out;         // fold mode: where the bound table goes (2 entries per pair); else nullptr
    int32_t dtype_in;  // layout of `in`
    int32_t shift;     // < 0: entries 2p, 2p+1 (4p..4p+3 in fold mode); >= 0: constant this round, entry p >> shift
};

constexpr uint16_t kNoOuter = 0xFFFF;
constexpr int kMaxAccTail = 8;  // sums a round publishes (degree <= 7)

// Terms [term_begin, term_end) multiplied by table `outer` (kNoOuter: by nothing).
struct ProgGroup {
    uint16_t outer, term_begin, term_end, pad;
};

// One step of a group's inner sum (the group's outer table is not listed), which is evaluated as a Horner chain:
//   kOpTerm  adds coeff * product of idx[0..n_factors).  Terms with the same coefficient are stored next to each
//            other and the coefficient multiplies their sum, at the term with run_last set (neg: the coefficient
//            is -1 and the sum is subtracted);
//   kOpConst adds coeff;
//   kOpFold  multiplies everything added so far by the tables idx[0..n_factors).
// z*(z*(a - v) + b) + v is thus: const a, term -v, fold z, const b, fold z, term v: two products instead of the
// four (and three coefficient products) of its monomials.
constexpr uint8_t kOpTerm = 0, kOpConst = 1, kOpFold = 2;
template <class F>
struct ProgTerm {
    typename F::E coeff;
    uint16_t n_factors;
    uint8_t coeff_is_one;
    uint8_t run_last;
    uint8_t op;
    uint8_t neg;
    uint16_t idx[DPB_MAX_FACTORS];
};

// Per-thread slots in shared memory: slot s (= 2 * table + {0: value, 1: difference}) is W 16-byte words,
// word w of thread t at ((s * W + w) * blockDim + t): consecutive threads touch consecutive words.
template <class F>
struct Slots {
    typedef typename F::E E;
    static constexpr int W = sizeof(E) / 16;
    uint4* base;
    __device__ __forceinline__ E get(uint32_t s) const {
        E v;
        uint4* q = (uint4*)&v;
#pragma unroll
        for (int w = 0; w < W; w++) q[w] = base[((size_t)s * W + w) * blockDim.x + threadIdx.x];
        return v;
    }
    __device__ __forceinline__ void put(uint32_t s, const E& v) const {
        const uint4* q = (const uint4*)&v;
#pragma unroll
        for (int w = 0; w < W; w++) base[((size_t)s * W + w) * blockDim.x + threadIdx.x] = q[w];
    }
};

// sum over groups of outer * sum over terms of coeff * product, at the tables' current values
// (only the groups g with bit g of `mask` equal to `want`; mask = want = 0 takes all)
template <class F>
__device__ __noinline__ typename F::E eval_program(const Slots<F>& sl, const ProgGroup* __restrict__ groups,
                                                   uint32_t n_groups, const ProgTerm<F>* __restrict__ terms,
                                                   uint32_t mask = 0, uint32_t want = 0) {
    typedef typename F::E E;
    E total = F::zero();
    for (uint32_t g = 0; g < n_groups; g++) {
        if (((mask >> (g & 31)) & 1u) != want) continue;
        const ProgGroup pg = groups[g];
        E inner = F::zero(), run = F::zero();
        for (uint32_t t = pg.term_begin; t < pg.term_end; t++) {
            const ProgTerm<F>& tm = terms[t];
            const uint32_t nf = tm.n_factors;
            if (tm.op == kOpFold) {
                for (uint32_t j = 0; j < nf; j++) inner = F::mul(inner, sl.get(2 * tm.idx[j]));
                continue;
            }
            if (tm.op == kOpConst) {
                inner = F::add(inner, tm.coeff);
                continue;
            }
            E prod;
            if (nf == 0) {
                prod = F::one();
            } else {
                prod = sl.get(2 * tm.idx[0]);
                for (uint32_t j = 1; j < nf; j++) prod = F::mul(prod, sl.get(2 * tm.idx[j]));
            }
            run = F::add(run, prod);
            if (tm.run_last) {
                if (tm.neg) inner = F::sub(inner, run);
                else inner = F::add(inner, tm.coeff_is_one ? run : F::mul(run, tm.coeff));
                run = F::zero();
            }
        }
        if (pg.outer != kNoOuter) inner = F::mul(inner, sl.get(2 * pg.outer));
        total = F::add(total, inner);
    }
    return total;
}

// every table's current value moves one evaluation point on
template <class F>
__device__ __noinline__ void advance_point(const Slots<F>& sl, const RoundTab* __restrict__ tabs, uint32_t k) {
    for (uint32_t j = 0; j < k; j++) {
        if (tabs[j].shift >= 0) continue;  // constant in this round
        sl.put(2 * j, F::add(sl.get(2 * j), sl.get(2 * j + 1)));
    }
}

// acc[x] = sum over pairs of the program at point x, for x = 0..D; with SKIP_ONE, x = 1 is left at zero.
template <class F, int D, bool SKIP_ONE>
__global__ void __launch_bounds__(kThreads)
    sc_round_generic(const RoundTab* __restrict__ tabs, uint32_t k, const ProgGroup* __restrict__ groups,
                     uint32_t n_groups, const ProgTerm<F>* __restrict__ terms, typename F::FoldKey rk, uint64_t n_pairs,
                     ReduceScratch<F> rs, typename F::E* out) {
    typedef typename F::E E;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Slots<F> sl;
    sl.base = (uint4*)smem_raw;
    E acc[D + 1];
#pragma unroll
    for (int x = 0; x <= D; x++) acc[x] = F::zero();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n_pairs; p += stride) {
        for (uint32_t j = 0; j < k; j++) {
            const RoundTab t = tabs[j];
            E f0, f1;
            if (t.out) {
                E a0, a1, b0, b1;
                F::load_pair(t.in, t.dtype_in, 2 * p, a0, a1);
                F::load_pair(t.in, t.dtype_in, 2 * p + 1, b0, b1);
                f0 = F::add(a0, F::mul_key(rk, F::sub(a1, a0)));
                f1 = F::add(b0, F::mul_key(rk, F::sub(b1, b0)));
                F::store(t.out, 2 * p, f0);
                F::store(t.out, 2 * p + 1, f1);
            } else if (t.shift < 0) {
                F::load_pair(t.in, t.dtype_in, p, f0, f1);
            } else {
                f0 = F::load(t.in, t.dtype_in, p >> t.shift);
                f1 = f0;
            }
            sl.put(2 * j, f0);
            sl.put(2 * j + 1, F::sub(f1, f0));
        }
#pragma unroll
        for (int x = 0; x <= D; x++) {
            if (!(SKIP_ONE && x == 1)) acc[x] = F::add(acc[x], eval_program<F>(sl, groups, n_groups, terms));
            if (x < D) advance_point<F>(sl, tabs, k);
        }
    }
    grid_sum_publish<F, D + 1>(acc, rs, out);
}

// ---- rounds in split-eq form -----------------------------------------------------
//
// When every group of the program is "an eq table times a sum of products", the
// round polynomial factors.  After the first i' variables of an eq table over the
// point q are bound to challenges c, its pair p is S * W[p] * ((1 - q_i'), q_i') with
// S = prod_k eq(q_k, c_k) and W the eq table of the remaining coordinates, and W[p] is
// the ORIGINAL table's entry p << (i' + 1) divided by prod_{k <= i'} (1 - q_k).  So
//     s(X) = ((1 - q) + (2 q - 1) X) * H(X) + C,    H(X) = sum_p kappa * eq[p << (i' + 1)] * G(X, p),
// with G the group's sum of products (one degree less than s), kappa a host-side scalar,
// and C the groups whose tables do not move in this round.  The kernel accumulates H at
// 0, 1, .., D - 1 (without 1 after round 0: the host gets H(1) from s(0) + s(1)) and C
// once per pair; the eq tables are neither bound nor stored.  One evaluation point and
// the eq table's folds less than the direct form; results are the same field elements.
constexpr int kMaxSplitEq = 4;
template <class F>
struct SplitEqArgs {
    uint32_t n_eq;                         // eq tables read in strided form this round
    uint32_t const_groups;                 // bit g: group g does not depend on this round's variable
    uint32_t table[kMaxSplitEq];           // their table ids
    uint32_t stride_log2[kMaxSplitEq];     // pair p reads entry p << stride_log2 of the original table
    typename F::E scale[kMaxSplitEq];      // kappa
};

// acc[x] = H(x) for x = 0..D-1 (x = 1 left at zero with SKIP_ONE), acc[D] = C.
template <class F, int D, bool SKIP_ONE>
__global__ void __launch_bounds__(kThreads)
    sc_round_spliteq(const RoundTab* __restrict__ tabs, uint32_t k, const ProgGroup* __restrict__ groups,
                     uint32_t n_groups, const ProgTerm<F>* __restrict__ terms, typename F::FoldKey rk,
                     SplitEqArgs<F> eq, uint64_t n_pairs, ReduceScratch<F> rs, typename F::E* out) {
    typedef typename F::E E;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Slots<F> sl;
    sl.base = (uint4*)smem_raw;
    E acc[D + 1];
#pragma unroll
    for (int x = 0; x <= D; x++) acc[x] = F::zero();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n_pairs; p += stride) {
        for (uint32_t j = 0; j < k; j++) {
            const RoundTab t = tabs[j];
            E f0, f1;
            int e = -1;
            for (uint32_t q = 0; q < eq.n_eq; q++)
                if (eq.table[q] == j) e = (int)q;
            if (e >= 0) {
                // descriptors mark these tables constant (shift >= 0), so advance_point leaves them alone
                f0 = F::mul(eq.scale[e], F::load(t.in, t.dtype_in, p << eq.stride_log2[e]));
                f1 = f0;
            } else if (t.out) {
                E a0, a1, b0, b1;
                F::load_pair(t.in, t.dtype_in, 2 * p, a0, a1);
                F::load_pair(t.in, t.dtype_in, 2 * p + 1, b0, b1);
                f0 = F::add(a0, F::mul_key(rk, F::sub(a1, a0)));
                f1 = F::add(b0, F::mul_key(rk, F::sub(b1, b0)));
                F::store(t.out, 2 * p, f0);
                F::store(t.out, 2 * p + 1, f1);
            } else if (t.shift < 0) {
                F::load_pair(t.in, t.dtype_in, p, f0, f1);
            } else {
                f0 = F::load(t.in, t.dtype_in, p >> t.shift);
                f1 = f0;
            }
            sl.put(2 * j, f0);
            sl.put(2 * j + 1, F::sub(f1, f0));
        }
        if (eq.const_groups) acc[D] = F::add(acc[D], eval_program<F>(sl, groups, n_groups, terms, eq.const_groups, 1u));
#pragma unroll
        for (int x = 0; x < D; x++) {
            if (!(SKIP_ONE && x == 1))
                acc[x] = F::add(acc[x], eval_program<F>(sl, groups, n_groups, terms, eq.const_groups, 0u));
            if (x < D - 1) advance_point<F>(sl, tabs, k);
        }
    }
    grid_sum_publish<F, D + 1>(acc, rs, out);
}

// out[i] = scale * in[i << stride_log2]: an eq table in the bound form the direct kernels expect, made from the
// original when a sumcheck leaves the split-eq form (the resident last-rounds kernel takes over).
template <class F>
__global__ void __launch_bounds__(kThreads)
    eq_materialize(const void* __restrict__ in, int dtype_in, uint32_t stride_log2, typename F::E scale, uint64_t n,
                   typename F::E* __restrict__ out) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
        F::store(out, i, F::mul(scale, F::load(in, dtype_in, i << stride_log2)));
}

// ---- one-pass rounds over a program cut into segments ------------------------------
//
// The kernels above keep (value, difference) of EVERY table in a thread's shared-memory slots, so a program over
// many tables leaves room for few threads per SM (13 BN254 tables: one block of 128), and one thread's chain of
// dependent products is then what the round waits for.  Most long programs are sums of independent parts, though:
// the instances of a logup batch, the heads of a stacked einsum.  Inside a group (terms sharing an outer table) the
// host finds the connected components of "terms that share a table"; each becomes a segment with its own few
// tables and its own Horner-chained term list over local table numbers.  A thread then walks the segments one
// after the other, reusing the same few slots: load (bind, store) the segment's tables, evaluate its terms at
// every point into the group's running sums, and multiply by the outer table once per group and point.  Same
// field sums as the unsegmented kernels, so the same messages.
constexpr int kSegTables = 6;
struct SegDesc {
    uint16_t group;                 // program group (bit of SplitEqArgs::const_groups)
    uint16_t outer;                 // the group's outer table, or kNoOuter
    uint16_t n_tabs;
    uint16_t term_begin, term_end;  // steps in the segmented program; their idx[] number the segment's tables
    uint8_t first, last;            // first / last segment of its group
    uint16_t tab[kSegTables];
};

// a group's inner sum over the steps [begin, end) at the slots' current values
template <class F>
__device__ __noinline__ typename F::E eval_steps(const Slots<F>& sl, const ProgTerm<F>* __restrict__ terms,
                                                 uint32_t begin, uint32_t end) {
    typedef typename F::E E;
    E inner = F::zero(), run = F::zero();
    for (uint32_t t = begin; t < end; t++) {
        const ProgTerm<F>& tm = terms[t];
        const uint32_t nf = tm.n_factors;
        if (tm.op == kOpFold) {
            for (uint32_t j = 0; j < nf; j++) inner = F::mul(inner, sl.get(2 * tm.idx[j]));
            continue;
        }
        if (tm.op == kOpConst) {
            inner = F::add(inner, tm.coeff);
            continue;
        }
        E prod;
        if (nf == 0) {
            prod = F::one();
        } else {
            prod = sl.get(2 * tm.idx[0]);
            for (uint32_t j = 1; j < nf; j++) prod = F::mul(prod, sl.get(2 * tm.idx[j]));
        }
        run = F::add(run, prod);
        if (tm.run_last) {
            if (tm.neg) inner = F::sub(inner, run);
            else inner = F::add(inner, tm.coeff_is_one ? run : F::mul(run, tm.coeff));
            run = F::zero();
        }
    }
    return inner;
}

// (value at 0, difference) of table t for pair p; binds the previous challenge and stores when the round folds
template <class F>
__device__ __forceinline__ void seg_load(const RoundTab& t, uint64_t p, const typename F::FoldKey& rk,
                                         typename F::E& f0, typename F::E& df) {
    typedef typename F::E E;
    E f1;
    if (t.out) {
        E a0, a1, b0, b1;
        F::load_pair(t.in, t.dtype_in, 2 * p, a0, a1);
        F::load_pair(t.in, t.dtype_in, 2 * p + 1, b0, b1);
        f0 = F::add(a0, F::mul_key(rk, F::sub(a1, a0)));
        f1 = F::add(b0, F::mul_key(rk, F::sub(b1, b0)));
        F::store(t.out, 2 * p, f0);
        F::store(t.out, 2 * p + 1, f1);
    } else if (t.shift < 0) {
        F::load_pair(t.in, t.dtype_in, p, f0, f1);
    } else {
        f0 = F::load(t.in, t.dtype_in, p >> t.shift);
        df = F::zero();
        return;
    }
    df = F::sub(f1, f0);
}

// SPLIT: the sums of sc_round_spliteq (H at 0..D-1, then C); otherwise those of sc_round_generic (0..D).
template <class F, int D, bool SKIP_ONE, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 2)
    sc_round_seg(const RoundTab* __restrict__ tabs, const SegDesc* __restrict__ segs, uint32_t n_segs,
                 const ProgTerm<F>* __restrict__ terms, typename F::FoldKey rk, SplitEqArgs<F> eq, uint64_t n_pairs,
                 uint32_t inner_slot, ReduceScratch<F> rs, typename F::E* out) {
    typedef typename F::E E;
    constexpr int NP = SPLIT ? D : D + 1;  // evaluation points per pair; the group's running sums live in the
                                           // slots inner_slot .. inner_slot + NP - 1 (registers are for the products)
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Slots<F> sl;
    sl.base = (uint4*)smem_raw;
    E acc[D + 1];
#pragma unroll
    for (int x = 0; x <= D; x++) acc[x] = F::zero();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n_pairs; p += stride) {
        for (uint32_t s = 0; s < n_segs; s++) {
            const SegDesc sd = segs[s];
            for (uint32_t j = 0; j < sd.n_tabs; j++) {
                E f0, df;
                seg_load<F>(tabs[sd.tab[j]], p, rk, f0, df);
                sl.put(2 * j, f0);
                sl.put(2 * j + 1, df);
            }
            if (sd.term_begin == sd.term_end && sd.outer == kNoOuter) continue;  // tables no term uses: bound, stored
            const bool cg = SPLIT && ((eq.const_groups >> (sd.group & 31)) & 1u);  // the group does not move this round
            if (sd.first) {
#pragma unroll
                for (int x = 0; x < NP; x++) sl.put(inner_slot + x, F::zero());
            }
            if (sd.term_begin != sd.term_end) {
#pragma unroll
                for (int x = 0; x < NP; x++) {
                    if (cg && x > 0) break;
                    if (!(SKIP_ONE && x == 1))
                        sl.put(inner_slot + x, F::add(sl.get(inner_slot + x), eval_steps<F>(sl, terms, sd.term_begin, sd.term_end)));
                    if (x < NP - 1 && !cg)
                        for (uint32_t j = 0; j < sd.n_tabs; j++) sl.put(2 * j, F::add(sl.get(2 * j), sl.get(2 * j + 1)));
                }
            }
            if (!sd.last) continue;
            if (sd.outer == kNoOuter) {
                if (cg) {
                    acc[D] = F::add(acc[D], sl.get(inner_slot));
                } else {
#pragma unroll
                    for (int x = 0; x < NP; x++) acc[x] = F::add(acc[x], sl.get(inner_slot + x));
                }
                continue;
            }
            E o, od;
            int e = -1;
            if (SPLIT)
                for (uint32_t q = 0; q < eq.n_eq; q++)
                    if (eq.table[q] == sd.outer) e = (int)q;
            if (e >= 0) {
                const RoundTab t = tabs[sd.outer];
                o = F::mul(eq.scale[e], F::load(t.in, t.dtype_in, p << eq.stride_log2[e]));
                od = F::zero();
            } else {
                seg_load<F>(tabs[sd.outer], p, rk, o, od);
            }
            if (cg) {
                acc[D] = F::add(acc[D], F::mul(sl.get(inner_slot), o));
            } else {
#pragma unroll
                for (int x = 0; x < NP; x++) {
                    if (!(SKIP_ONE && x == 1)) acc[x] = F::add(acc[x], F::mul(sl.get(inner_slot + x), o));
                    if (x < NP - 1 && e < 0) o = F::add(o, od);
                }
            }
        }
    }
    grid_sum_publish<F, D + 1>(acc, rs, out);
}

// ---- resident kernel for the last rounds ---------------------------------------
//
// Once a round has only a few hundred pairs, launching a kernel per round costs
// more than the round.  sc_tail_generic stays resident instead: one block runs
// every remaining round, hands each round's sums to the host through mapped
// memory and waits there for the challenge (about 4 us per exchange, measured).
// With so little work per round the latency of one thread's chain of
// multiplications is what counts, so the block spreads a round as widely as it
// can: binding over (pair, table), evaluation over (pair, point).  Every wait
// is bounded: when the host does not answer within wait_ns the kernel records
// that in the mailbox and returns.

constexpr uint32_t kTailAbort = 0xFFFFFFFFu;
constexpr unsigned long long kTailHelloNs = 50ull * 1000 * 1000;  // 50 ms for the host's first sign of life
constexpr uint32_t kTailMaxTables = 96;

// Mailbox in mapped pinned host memory.  Everything travels as 16-byte chunks
// {8 bytes of data, sequence number, pad}: a chunk is written and read as one
// transaction, so a reader that sees the sequence number it waits for has the
// data that belongs to it, and neither side needs a system-wide fence (those
// cost more than a microsecond each on the device).
struct TailBox {
    // host -> device: the challenge that ends round i carries sequence number i + 1; kTailAbort: leave now
    TailChunk chal[4];
    // host -> device, written right after the launch call returns: sequence number 1 = "the host runs beside you"
    TailChunk hello;
    uint32_t pad0[12];
    // device -> host
    volatile uint32_t status;  // 0 running, 2 gave up waiting for a challenge, 3 no hello: launches block the host
    uint32_t pad[15];
    TailChunk evals[kMaxAccTail * 4];      // sums of round i: sequence number i + 1
    TailChunk finals[kTailMaxTables * 4];  // final evaluations: sequence number n_rounds + 1
};

static_assert(sizeof(TailBox) <= 8192, "the context reserves 8 KiB for the mailbox");

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void chunk_load(const TailChunk* c, uint64_t& data, uint32_t& seq) {
    uint32_t lo, hi, unused = 0;
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(lo), "=r"(hi), "=r"(seq), "+r"(unused) : "l"(c) : "memory");
    data = (uint64_t)lo | ((uint64_t)hi << 32);
}
// The kernel can only trade messages with a host that runs while it does.  Under a profiler that serialises
// launches, or with blocking launches, the launch call returns only when the kernel has ended: the hello never
// comes, the kernel says so and leaves at once, and the host goes back to one launch per round.
__device__ __forceinline__ bool tail_hello(TailBox* box, unsigned long long limit_ns) {
    const unsigned long long t0 = global_ns();
    for (;;) {
        uint64_t d;
        uint32_t s;
        chunk_load(&box->hello, d, s);
        if (s == 1) return true;
        if (s == kTailAbort) return false;
        if (global_ns() - t0 > limit_ns) {
            box->status = 3;
            return false;
        }
    }
}

// Waits for the challenge with sequence number `want`: lane i of the calling warp polls chunk i, because every look at
// host memory is a trip over the bus (about a microsecond) and the chunks of one challenge must not queue up behind
// each other.  All 32 lanes call; returns 0 when the challenge has arrived (lane i then holds its 64-bit word i in
// `word`), 1 on abort or time-out.
template <class E>
__device__ __forceinline__ int tail_wait(TailBox* box, uint32_t want, unsigned long long wait_ns, uint64_t& word) {
    constexpr int W8 = (int)(sizeof(E) / 8);
    const int lane = threadIdx.x & 31;
    const unsigned long long t0 = global_ns();
    for (;;) {
        uint32_t s = want;
        if (lane < W8) chunk_load(&box->chal[lane], word, s);
        if (__all_sync(0xffffffffu, s == want)) return 0;
        if (__any_sync(0xffffffffu, s == kTailAbort)) return 1;
        const bool late = global_ns() - t0 > wait_ns;
        if (__any_sync(0xffffffffu, late)) {
            if (lane == 0) box->status = 2;
            return 1;
        }
    }
}

constexpr int kTailThreads = 512;
constexpr uint32_t kTailBlocks = 8;   // blocks of the cluster that runs larger rounds (the portable size)
// Pairs from which one block goes on alone (at most): the cluster divides a round's products by eight and adds two
// cluster barriers, which pays for BN254 rounds of more than 32 pairs (n = 8: 105 -> 100 us a proof) and makes no
// difference to Goldilocks rounds of up to 256 (n = 10: 102.4 us handed over at 32 pairs, 103.6 at 256).
constexpr uint32_t kTailAloneFr = 32, kTailAloneGl = 256;
// Pairs the slots of even and of odd rounds are laid out for, nb pairs of a block in the first round: a cluster's first
// block needs room for all that is left when it goes on alone, in whichever set that falls.
__host__ __device__ __forceinline__ size_t tail_slot_pairs(size_t nb, uint32_t blocks, uint32_t alone, int set) {
    const size_t own = set ? (nb + 1) / 2 : nb, gathered = blocks > 1 ? (size_t)alone : 0;
    return own > gathered ? own : gathered;
}
constexpr int kTailProgBytes = 8 * 1024;  // the term program is staged in shared memory when it fits

// Shared-memory slots addressed by pair instead of by thread: slot s of pair p, n pairs in the round.
template <class F>
struct PairSlots {
    typedef typename F::E E;
    static constexpr int W = sizeof(E) / 16;
    uint4* base;
    uint32_t n;
    __device__ __forceinline__ E get(uint32_t s, uint32_t p) const {
        E v;
        uint4* q = (uint4*)&v;
#pragma unroll
        for (int w = 0; w < W; w++) q[w] = base[((size_t)s * W + w) * n + p];
        return v;
    }
    __device__ __forceinline__ void put(uint32_t s, uint32_t p, const E& v) const {
        const uint4* q = (const uint4*)&v;
#pragma unroll
        for (int w = 0; w < W; w++) base[((size_t)s * W + w) * n + p] = q[w];
    }
    // value of table j at the integer point x: f(0) + x * (f(1) - f(0)) by repeated addition
    __device__ __forceinline__ E at(uint32_t j, uint32_t p, uint32_t x) const {
        E v = get(2 * j, p);
        if (x) {
            const E d = get(2 * j + 1, p);
            for (uint32_t q = 0; q < x; q++) v = F::add(v, d);
        }
        return v;
    }
};

template <class F>
__device__ __noinline__ typename F::E eval_program_at(const PairSlots<F>& sl, uint32_t p, uint32_t x,
                                                      const ProgGroup* groups, uint32_t n_groups,
                                                      const ProgTerm<F>* terms) {
    typedef typename F::E E;
    E total = F::zero();
    for (uint32_t g = 0; g < n_groups; g++) {
        const ProgGroup pg = groups[g];
        E inner = F::zero(), run = F::zero();
        for (uint32_t t = pg.term_begin; t < pg.term_end; t++) {
            const ProgTerm<F>& tm = terms[t];
            const uint32_t nf = tm.n_factors;
            if (tm.op == kOpFold) {
                for (uint32_t j = 0; j < nf; j++) inner = F::mul(inner, sl.at(tm.idx[j], p, x));
                continue;
            }
            if (tm.op == kOpConst) {
                inner = F::add(inner, tm.coeff);
                continue;
            }
            E prod;
            if (nf == 0) {
                prod = F::one();
            } else {
                prod = sl.at(tm.idx[0], p, x);
                for (uint32_t j = 1; j < nf; j++) prod = F::mul(prod, sl.at(tm.idx[j], p, x));
            }
            run = F::add(run, prod);
            if (tm.run_last) {
                if (tm.neg) inner = F::sub(inner, run);
                else inner = F::add(inner, tm.coeff_is_one ? run : F::mul(run, tm.coeff));
                run = F::zero();
            }
        }
        if (pg.outer != kNoOuter) inner = F::mul(inner, sl.at(pg.outer, p, x));
        total = F::add(total, inner);
    }
    return total;
}

// Sums v over the n (a power of two) neighbouring threads of its segment; threads of whole segments call together.
// The first thread of a segment, or for n > 32 of the segment's part in a warp, ends up with the sum.
template <class F>
__device__ __forceinline__ typename F::E segment_sum(typename F::E v, uint32_t n) {
    for (uint32_t off = (n < 32 ? n : 32) >> 1; off > 0; off >>= 1) v = F::add(v, F::shfl_down(v, (int)off));
    return v;
}

// One block, or a cluster of kTailBlocks blocks while a round has more than `alone` pairs: every block then holds a
// contiguous part of the pairs, partial sums and the challenge travel through distributed shared memory, and the first
// block goes on alone.  (Blocks of a cluster are resident together, so their barriers end; the one wait for the host
// is bounded, and its outcome is handed to all.)  Per round of 2^(n_rounds - round - 1) pairs:
//   A. items (pair, table): bind the previous challenge and fill the pair's slots.  The values to bind are the slots of
//      the round before (two sets of slots, used in turn); only the first round reads tables from memory.  The bound
//      tables are stored all the same, so that the kernel can be started again at any round;
//   B. items (pair, point): evaluate the program at that point;
//   C. sums over the pairs of each point, by shuffles and one exchange between warps; the first warp posts them and
//      waits for the challenge.
// Latency is all that counts here: one thread's chain of products, barriers, and trips to memory and to the host.
// Dynamic shared memory: [program copy | round descriptors | slots of even rounds | slots of odd rounds].
// Product of three tables over BN254, n = 8: 14.1 us a round with the tables read back from memory, a tree of
// barriers for the sums and a challenge read chunk by chunk, 11.2 us since (Goldilocks 9.5, 7.1); with the cluster
// three more rounds are resident: n = 12 201 -> 153 us a proof (Goldilocks 148 -> 129), n = 20 631 -> 555 us.
template <class F, int D>
__global__ void __launch_bounds__(kTailThreads)
    sc_tail_generic(const RoundTab* __restrict__ tabs_all, uint32_t k, const ProgGroup* __restrict__ groups_g,
                    uint32_t n_groups, const ProgTerm<F>* __restrict__ terms_g, uint32_t n_prog_terms,
                    typename F::E r, uint32_t first_round, uint32_t n_rounds, TailBox* box,
                    unsigned long long wait_ns, uint32_t prog_in_smem, uint32_t slots_offset, uint32_t alone) {
    typedef typename F::E E;
    namespace cg = cooperative_groups;
    constexpr int W8 = sizeof(E) / 8;
    cg::cluster_group cluster = cg::this_cluster();
    uint32_t blocks = cluster.num_blocks();
    const uint32_t rank = cluster.block_rank();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(16) E sh_r;
    __shared__ int sh_stop;
    __shared__ typename F::FoldKey sh_key;  // the current challenge in the form the folds multiply by
    __shared__ E sh_sum[2 * kTailThreads / 32];
    __shared__ __align__(16) E sh_part[D + 1][kTailBlocks];
    const ProgGroup* groups = groups_g;
    const ProgTerm<F>* terms = terms_g;
    unsigned char* cursor = smem_raw;
    if (prog_in_smem) {
        ProgTerm<F>* st = (ProgTerm<F>*)cursor;
        cursor += (size_t)n_prog_terms * sizeof(ProgTerm<F>);
        ProgGroup* sg = (ProgGroup*)cursor;
        for (uint32_t i = threadIdx.x; i < n_prog_terms; i += blockDim.x) st[i] = terms_g[i];
        for (uint32_t i = threadIdx.x; i < n_groups; i += blockDim.x) sg[i] = groups_g[i];
        groups = sg;
        terms = st;
    }
    // round descriptors, double-buffered: the next round's are fetched while this round computes
    RoundTab* tabs_buf[2] = {(RoundTab*)(smem_raw + slots_offset - 2 * (size_t)k * sizeof(RoundTab)),
                             (RoundTab*)(smem_raw + slots_offset - (size_t)k * sizeof(RoundTab))};
    for (uint32_t j = threadIdx.x; j < k; j += blockDim.x) tabs_buf[0][j] = tabs_all[(size_t)first_round * k + j];
    const RoundTab* tabs = tabs_buf[0];
    uint32_t nb = (1u << (n_rounds - first_round - 1)) / blocks;  // pairs of this block
    const size_t set_words = (size_t)2 * k * PairSlots<F>::W * tail_slot_pairs(nb, blocks, alone, 0);
    PairSlots<F> sl, old;
    sl.base = old.base = (uint4*)(smem_raw + slots_offset);
    sl.n = old.n = nb;
    if (blocks > 1) cluster.sync();  // every block has started: its shared memory may be written
    if (threadIdx.x == 0) {
        if (rank == 0) {
            const int stop = tail_hello(box, kTailHelloNs) ? 0 : 1;
            for (uint32_t b = 0; b < blocks; b++) *cluster.map_shared_rank(&sh_stop, b) = stop;
        }
        sh_r = r;
    }
    F::fold_key_block(r, &sh_key);
    if (blocks > 1) cluster.sync();
    else __syncthreads();
    if (sh_stop) return;
    for (uint32_t round = first_round; round < n_rounds; round++) {
        const bool gather = round > first_round && blocks > 1 && nb * blocks <= 2 * alone;
        if (round > first_round) {
            old = sl;
            nb = gather ? nb * blocks / 2 : nb / 2;
            sl.n = nb;
            sl.base = (uint4*)(smem_raw + slots_offset) + (((round - first_round) & 1) ? set_words : 0);
        }
        tabs = tabs_buf[(round - first_round) & 1];
        if (round + 1 < n_rounds) {
            RoundTab* nxt = tabs_buf[(round + 1 - first_round) & 1];
            for (uint32_t j = threadIdx.x; j < k; j += blockDim.x) nxt[j] = tabs_all[(size_t)(round + 1) * k + j];
        }
        // A
        const uint64_t p0 = gather ? 0 : (uint64_t)rank * nb;  // first pair of this block
        if (!gather || rank == 0) {
            for (uint32_t w = threadIdx.x; w < nb * k; w += blockDim.x) {
                const uint32_t j = w / nb, p = w % nb;
                const RoundTab t = tabs[j];
                E f0, f1;
                if (t.out) {
                    E a0, b0, da, db;
                    if (round > first_round) {
                        PairSlots<F> src = old;
                        uint32_t q = 2 * p;
                        if (gather) {  // a block held 2 * alone / kTailBlocks pairs, an even number
                            src.base = cluster.map_shared_rank(old.base, q / old.n);
                            q %= old.n;
                        }
                        a0 = src.get(2 * j, q);
                        da = src.get(2 * j + 1, q);
                        b0 = src.get(2 * j, q + 1);
                        db = src.get(2 * j + 1, q + 1);
                    } else {
                        E a1, b1;
                        F::load_pair(t.in, t.dtype_in, 2 * (p0 + p), a0, a1);
                        F::load_pair(t.in, t.dtype_in, 2 * (p0 + p) + 1, b0, b1);
                        da = F::sub(a1, a0);
                        db = F::sub(b1, b0);
                    }
                    f0 = F::add(a0, F::mul_key(sh_key, da));
                    f1 = F::add(b0, F::mul_key(sh_key, db));
                    F::store(t.out, 2 * (p0 + p), f0);
                    F::store(t.out, 2 * (p0 + p) + 1, f1);
                } else if (t.shift < 0) {
                    F::load_pair(t.in, t.dtype_in, p0 + p, f0, f1);
                } else {
                    f0 = F::load(t.in, t.dtype_in, (p0 + p) >> t.shift);
                    f1 = f0;
                }
                sl.put(2 * j, p, f0);
                sl.put(2 * j + 1, p, F::sub(f1, f0));
            }
        }
        if (gather) {
            cluster.sync();  // the other blocks' slots have been read
            if (rank != 0) return;
            blocks = 1;
        }
        __syncthreads();
        // B: the points are 0, 1, .., D in round 0 and 0, 2, .., D later (index 1 is left out); at most two items per
        // thread (nb * n_points <= 2 * blockDim)
        const uint32_t n_points = round > 0 ? D : D + 1;
        const uint32_t n_items = nb * n_points;
        const uint32_t parts = nb > 32 ? nb / 32 : 1;  // partial sums per point
        for (uint32_t w0 = 0; w0 < n_items; w0 += blockDim.x) {
            const uint32_t w = w0 + threadIdx.x;
            if ((w & ~31u) >= n_items) continue;  // whole warps: the sums below shuffle
            E v = F::zero();
            const uint32_t xi = w / nb, p = w % nb;
            if (w < n_items) {
                const uint32_t x = (round > 0 && xi >= 1) ? xi + 1 : xi;
                v = eval_program_at<F>(sl, p, x, groups, n_groups, terms);
            }
            v = segment_sum<F>(v, nb);
            if (w < n_items && (p & 31) == 0) sh_sum[xi * parts + p / 32] = v;
        }
        __syncthreads();
        // C
        if (threadIdx.x < 32) {
            const uint32_t lane = threadIdx.x;
            // n_points segments of `parts` partial sums (at most 32 sums in all: n_items <= 2 * kTailThreads)
            E v = lane < n_points * parts ? sh_sum[lane] : F::zero();
            v = segment_sum<F>(v, parts);
            if (lane < n_points * parts && lane % parts == 0) {
                const uint32_t xi = lane / parts;
                if (blocks > 1) {
                    cluster.map_shared_rank(&sh_part[0][0], 0)[xi * kTailBlocks + rank] = v;
                } else {
                    const uint32_t x = (round > 0 && xi >= 1) ? xi + 1 : xi;
                    chunks_store<E>(&box->evals[x * W8], v, round + 1);
                }
            }
            __syncwarp();
        }
        if (blocks > 1) cluster.sync();
        if (rank == 0 && threadIdx.x < 32) {
            const uint32_t lane = threadIdx.x;
            if (blocks > 1) {
                for (uint32_t x0 = 0; x0 < n_points; x0 += 32 / kTailBlocks) {  // four points at a time
                    const uint32_t xi = x0 + lane / kTailBlocks;
                    E v = xi < n_points ? sh_part[xi][lane % kTailBlocks] : F::zero();
                    v = segment_sum<F>(v, kTailBlocks);
                    if (xi < n_points && lane % kTailBlocks == 0) {
                        const uint32_t x = (round > 0 && xi >= 1) ? xi + 1 : xi;
                        chunks_store<E>(&box->evals[x * W8], v, round + 1);
                    }
                }
            }
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
        r = sh_r;
        F::fold_key_block(r, &sh_key);
        __syncthreads();
    }
    // r ends the last round: one value per table (the last round had one pair, its slots are in sl)
    for (uint32_t j = threadIdx.x; j < k; j += blockDim.x)
        chunks_store<E>(&box->finals[j * (sizeof(E) / 8)], F::add(sl.get(2 * j, 0), F::mul(r, sl.get(2 * j + 1, 0))), n_rounds + 1);
}

// ---- host side ---------------------------------------------------------------

// A monomial of a group's inner sum on the host: coeff * product of f.
template <class F>
struct ProgMono {
    typename F::E coeff;
    std::vector<uint16_t> f;
};

// Steps and field multiplications of a monomial list evaluated as it stands: constants summed into one
// kOpConst, the rest sorted into runs of equal coefficients.
template <class F>
inline uint32_t emit_flat(std::vector<ProgMono<F>> monos, std::vector<ProgTerm<F>>& out) {
    typedef typename F::E E;
    uint32_t cost = 0;
    E c = F::zero();
    bool have_c = false;
    std::vector<ProgMono<F>> rest;
    for (auto& m : monos) {
        if (m.f.empty()) {
            c = F::add(c, m.coeff);
            have_c = true;
        } else {
            rest.push_back(std::move(m));
        }
    }
    if (have_c && !F::is_zero(c)) {
        ProgTerm<F> pt;
        memset(&pt, 0, sizeof pt);
        pt.coeff = c;
        pt.op = kOpConst;
        out.push_back(pt);
    }
    // equal coefficients next to each other (stable: otherwise the caller's order), the last of each run marked
    std::stable_sort(rest.begin(), rest.end(),
                     [](const ProgMono<F>& x, const ProgMono<F>& y) { return memcmp(&x.coeff, &y.coeff, sizeof(E)) < 0; });
    for (size_t t = 0; t < rest.size(); t++) {
        ProgTerm<F> pt;
        memset(&pt, 0, sizeof pt);
        pt.coeff = rest[t].coeff;
        pt.op = kOpTerm;
        pt.coeff_is_one = F::is_one(pt.coeff) ? 1 : 0;
        pt.neg = F::is_one(F::neg(pt.coeff)) ? 1 : 0;
        pt.n_factors = (uint16_t)rest[t].f.size();
        for (size_t j = 0; j < rest[t].f.size(); j++) pt.idx[j] = rest[t].f[j];
        pt.run_last = (t + 1 == rest.size() || memcmp(&rest[t].coeff, &rest[t + 1].coeff, sizeof(E)) != 0) ? 1 : 0;
        cost += pt.n_factors - 1;
        if (pt.run_last && !pt.coeff_is_one && !pt.neg) cost++;
        out.push_back(pt);
    }
    return cost;
}

// The cheaper of the list as it stands and  f * (monomials with f, f taken out once) + (monomials without f),
// f the table in most monomials, the first part planned the same way.  Returns the multiplications per
// evaluation; appends the steps to `out`.
template <class F>
inline uint32_t emit_chain(const std::vector<ProgMono<F>>& monos, uint32_t k, std::vector<ProgTerm<F>>& out) {
    std::vector<ProgTerm<F>> flat;
    const uint32_t flat_cost = emit_flat<F>(monos, flat);
    std::vector<uint32_t> count(k, 0);
    for (const auto& m : monos)
        for (size_t j = 0; j < m.f.size(); j++) {
            bool first = true;
            for (size_t q = 0; q < j; q++)
                if (m.f[q] == m.f[j]) first = false;
            if (first) count[m.f[j]]++;
        }
    uint32_t best = 0, best_n = 0;
    for (uint32_t j = 0; j < k; j++)
        if (count[j] > best_n) {
            best_n = count[j];
            best = j;
        }
    if (best_n >= 2 && monos.size() <= 4096) {
        std::vector<ProgMono<F>> with, without;
        for (const auto& m : monos) {
            size_t pos = m.f.size();
            for (size_t j = 0; j < m.f.size(); j++)
                if (m.f[j] == best) {
                    pos = j;
                    break;
                }
            if (pos == m.f.size()) {
                without.push_back(m);
            } else {
                ProgMono<F> r = m;
                r.f.erase(r.f.begin() + pos);
                with.push_back(std::move(r));
            }
        }
        std::vector<ProgTerm<F>> chain;
        uint32_t cost = emit_chain<F>(with, k, chain);
        ProgTerm<F> fold;
        memset(&fold, 0, sizeof fold);
        fold.op = kOpFold;
        fold.n_factors = 1;
        fold.idx[0] = (uint16_t)best;
        chain.push_back(fold);
        cost += 1 + emit_flat<F>(without, chain);
        if (cost < flat_cost) {
            out.insert(out.end(), chain.begin(), chain.end());
            return cost;
        }
    }
    out.insert(out.end(), flat.begin(), flat.end());
    return flat_cost;
}

// Groups terms by a shared table, greedily: the table that occurs in most of the
// still ungrouped terms (at least two) becomes the outer factor of those terms.
// Tables listed in `prefer` (eq tables) become outer factors first, whatever their counts.
// Inside a group the remaining monomials become a Horner chain where that saves multiplications (emit_chain).
template <class F>
inline void compile_program(const dpb_term* terms, uint32_t n_terms, uint32_t k, std::vector<ProgGroup>& groups,
                            std::vector<ProgTerm<F>>& prog, const std::vector<bool>& prefer = std::vector<bool>(),
                            uint32_t* mults_per_point = nullptr,
                            std::vector<std::vector<ProgMono<F>>>* group_monos = nullptr) {
    typedef typename F::E E;
    std::vector<bool> used(n_terms, false);
    uint32_t left = n_terms;
    std::vector<ProgMono<F>> monos;
    auto take = [&](uint32_t t, int drop) {  // drop: position of the factor that became the outer table, or -1
        ProgMono<F> m;
        memcpy(&m.coeff, terms[t].coeff, sizeof(E));
        for (uint32_t j = 0; j < terms[t].n_factors; j++)
            if ((int)j != drop) m.f.push_back(terms[t].idx[j]);
        monos.push_back(std::move(m));
    };
    while (left > 0) {
        std::vector<uint32_t> count(k, 0);
        for (uint32_t t = 0; t < n_terms; t++) {
            if (used[t]) continue;
            for (uint32_t j = 0; j < terms[t].n_factors; j++) {
                bool first = true;
                for (uint32_t q = 0; q < j; q++)
                    if (terms[t].idx[q] == terms[t].idx[j]) first = false;
                if (first) count[terms[t].idx[j]]++;
            }
        }
        uint32_t best = 0, best_n = 0;
        bool best_pref = false;
        for (uint32_t j = 0; j < k; j++) {
            const bool pref = j < prefer.size() && prefer[j] && count[j] > 0;
            if ((pref && !best_pref) || (pref == best_pref && count[j] > best_n)) {
                best_n = count[j];
                best = j;
                best_pref = pref;
            }
        }
        if (best_pref && best_n < 2) best_n = 2;  // an eq table leads its group even when a single term uses it
        ProgGroup g;
        g.pad = 0;
        g.term_begin = (uint16_t)prog.size();
        monos.clear();
        if (best_n >= 2) {
            g.outer = (uint16_t)best;
            for (uint32_t t = 0; t < n_terms; t++) {
                if (used[t]) continue;
                int pos = -1;
                for (uint32_t j = 0; j < terms[t].n_factors; j++)
                    if (terms[t].idx[j] == best) {
                        pos = (int)j;
                        break;
                    }
                if (pos < 0) continue;
                take(t, pos);
                used[t] = true;
                left--;
            }
        } else {
            g.outer = kNoOuter;
            for (uint32_t t = 0; t < n_terms; t++) {
                if (used[t]) continue;
                take(t, -1);
                used[t] = true;
                left--;
            }
        }
        if (group_monos) group_monos->push_back(monos);
        const uint32_t cost = emit_chain<F>(monos, k, prog) + (g.outer != kNoOuter ? 1 : 0);
        if (mults_per_point) *mults_per_point += cost;
        g.term_end = (uint16_t)prog.size();
        groups.push_back(g);
    }
}

// Cuts the groups compile_program made into segments for sc_round_seg: inside a group, the connected components of
// "monomials that share a table", in the order of their first monomial; a group's constants form a component
// without tables.  Every table no term touches gets a place in a segment without steps, so that it is still bound
// and stored.  Returns false when a component has more than kSegTables tables (the caller keeps the unsegmented
// kernels) or when nothing would be gained (a single segment holds every table).
template <class F>
inline bool compile_segments(const std::vector<ProgGroup>& groups, const std::vector<std::vector<ProgMono<F>>>& group_monos,
                             uint32_t k, std::vector<SegDesc>& segs, std::vector<ProgTerm<F>>& prog, uint32_t* max_tabs) {
    if (groups.size() != group_monos.size() || groups.size() > 32) return false;
    std::vector<bool> covered(k, false);
    uint32_t widest = 1;
    for (size_t g = 0; g < groups.size(); g++) {
        const auto& monos = group_monos[g];
        if (groups[g].outer != kNoOuter) covered[groups[g].outer] = true;
        // union-find over the tables of this group's monomials
        std::vector<int> parent(k);
        for (uint32_t j = 0; j < k; j++) parent[j] = (int)j;
        auto find = [&](int x) {
            while (parent[x] != x) x = parent[x] = parent[parent[x]];
            return x;
        };
        for (const auto& m : monos)
            for (size_t j = 1; j < m.f.size(); j++) parent[find(m.f[j])] = find(m.f[0]);
        std::vector<int> comp_of_root(k, -1);
        std::vector<std::vector<ProgMono<F>>> comp_monos;
        int const_comp = -1;
        for (const auto& m : monos) {
            int c;
            if (m.f.empty()) {
                if (const_comp < 0) {
                    const_comp = (int)comp_monos.size();
                    comp_monos.emplace_back();
                }
                c = const_comp;
            } else {
                const int root = find(m.f[0]);
                if (comp_of_root[root] < 0) {
                    comp_of_root[root] = (int)comp_monos.size();
                    comp_monos.emplace_back();
                }
                c = comp_of_root[root];
            }
            comp_monos[c].push_back(m);
        }
        if (comp_monos.empty()) comp_monos.emplace_back();  // a group of nothing but its outer table cannot occur; keep a segment
        for (size_t c = 0; c < comp_monos.size(); c++) {
            std::vector<uint16_t> tabs;
            for (const auto& m : comp_monos[c])
                for (uint16_t t : m.f)
                    if (std::find(tabs.begin(), tabs.end(), t) == tabs.end()) tabs.push_back(t);
            if (tabs.size() > (size_t)kSegTables) return false;
            std::sort(tabs.begin(), tabs.end());
            std::vector<ProgMono<F>> local = comp_monos[c];
            for (auto& m : local)
                for (auto& t : m.f) t = (uint16_t)(std::find(tabs.begin(), tabs.end(), t) - tabs.begin());
            if (prog.size() + 4 * local.size() + 8 > 65535) return false;
            SegDesc sd;
            memset(&sd, 0, sizeof sd);
            sd.group = (uint16_t)g;
            sd.outer = groups[g].outer;
            sd.n_tabs = (uint16_t)tabs.size();
            for (size_t j = 0; j < tabs.size(); j++) {
                sd.tab[j] = tabs[j];
                covered[tabs[j]] = true;
            }
            sd.term_begin = (uint16_t)prog.size();
            emit_chain<F>(local, (uint32_t)tabs.size(), prog);
            sd.term_end = (uint16_t)prog.size();
            sd.first = c == 0;
            sd.last = c + 1 == comp_monos.size();
            widest = std::max<uint32_t>(widest, (uint32_t)tabs.size());
            segs.push_back(sd);
        }
    }
    // tables outside every term: bound and stored by segments without steps
    SegDesc rest;
    memset(&rest, 0, sizeof rest);
    rest.outer = kNoOuter;
    for (uint32_t j = 0; j < k; j++) {
        if (covered[j]) continue;
        rest.tab[rest.n_tabs++] = (uint16_t)j;
        if (rest.n_tabs == kSegTables) {
            segs.push_back(rest);
            widest = std::max<uint32_t>(widest, rest.n_tabs);
            rest.n_tabs = 0;
        }
    }
    if (rest.n_tabs) {
        segs.push_back(rest);
        widest = std::max<uint32_t>(widest, rest.n_tabs);
    }
    *max_tabs = widest;
    return segs.size() > 1 && (uint32_t)(2 * widest) <= k;
}

// Value at x of the polynomial of degree <= D with the given values at 0..D.
// w[j] = 1 / prod_{m != j} (j - m), computed once by lagrange_weights.
template <class F>
inline void lagrange_weights(int D, typename F::E* w) {
    typedef typename F::E E;
    for (int j = 0; j <= D; j++) {
        E den = F::one();
        for (int m = 0; m <= D; m++) {
            if (m == j) continue;
            const E diff = j > m ? F::from_u64((uint64_t)(j - m)) : F::neg(F::from_u64((uint64_t)(m - j)));
            den = F::mul(den, diff);
        }
        w[j] = F::inv(den);
    }
}
template <class F>
inline typename F::E lagrange_eval(int D, const typename F::E* evals, const typename F::E* w, const typename F::E& x) {
    typedef typename F::E E;
    E total = F::zero();
    for (int j = 0; j <= D; j++) {
        E term = F::mul(evals[j], w[j]);
        for (int m = 0; m <= D; m++)
            if (m != j) term = F::mul(term, F::sub(x, F::from_u64((uint64_t)m)));
        total = F::add(total, term);
    }
    return total;
}

}  // namespace dpb

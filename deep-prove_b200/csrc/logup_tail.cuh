// The last rounds of a logup-GKR layer in one resident kernel, from the layer's own formula.
//
// sc_tail_generic walks a layer's term list: per instance five dependent products and their running sums, one thread
// after the other's tables through memory, on one SM.  Most of a batched logup proof is rounds of a few hundred pairs
// or fewer, and there the latency of that chain is what the proof waits for.  Here
//  * an instance is the tables C, D, U, A of  g = C U + A D  (U = B + lambda D; a lookup's input layer has A = -1 and
//    U = lambda D - 1, which need no tables), all linear in the original tables, so that they are bound like them and
//    the originals are read off at the end.  They live in shared memory for all rounds; nothing is written back: when
//    the host was held up beyond the kernel's limit, the rounds so far are played again from the tables the first of
//    them read;
//  * a round is sampled at 0 and infinity (and 1 in round 0), items (instance, pair) over the threads, a pair weighted
//    by the eq table of the open variables (the entries at the stride of the round: nothing to bind), an instance by
//    its alpha once per round;
//  * a cluster of eight blocks runs the rounds that are too large for one: every block holds a contiguous eighth of the
//    pairs, partial sums and the challenge travel through distributed shared memory, and one block goes on alone once
//    32 pairs (BN254; 256 Goldilocks, fewer with many tables) are left.  Blocks of a cluster are resident together, so their barriers end; the one wait for the host
//    is bounded and its outcome is handed to all.
// Measured, BN254, three instances of 2^21 rows: 144 rounds of up to 256 pairs took 3460 us in sc_tail_generic and 32
// rounds of up to 2048 pairs 1100 us as fold + evaluation launches and the gaps between them; 176 rounds take 2730 us
// here (15.5 us each, of which the host's transcript and the bus take 6).  A lookup of 2^10 rows: 1100 us and 680 us.
#pragma once
#include <cooperative_groups.h>

#include "logup_tail.hpp"
#include "generic_round.cuh"
#include "lazy_sum.cuh"

namespace dpb {

namespace cg = cooperative_groups;

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

// entry e of an original table in the kernel's first round
template <class F>
__device__ __forceinline__ typename F::E logup_tail_load(const RoundTab& t, uint64_t e, const typename F::E& r) {
    typedef typename F::E E;
    if (!t.out) return F::load(t.in, t.dtype_in, e);
    E a, b;
    F::load_pair(t.in, t.dtype_in, e, a, b);
    return F::add(a, F::mul(r, F::sub(b, a)));
}

template <class F>
__global__ void __launch_bounds__(kTailThreads)
    sc_tail_logup(const RoundTab* __restrict__ tabs, const LogupTailInst* __restrict__ inst_g,
                  const typename F::E* __restrict__ consts_g, uint32_t n_inst, uint32_t n_tabs, typename F::E lambda,
                  const typename F::E* __restrict__ eq, uint32_t eq_stride_log2, typename F::E r, uint32_t first_round,
                  uint32_t n_rounds, uint32_t alone, TailBox* box, unsigned long long wait_ns) {
    typedef typename F::E E;
    constexpr int W8 = sizeof(E) / 8;
    cg::cluster_group cluster = cg::this_cluster();
    uint32_t blocks = cluster.num_blocks();
    const uint32_t rank = cluster.block_rank();
    // [alpha, sep, constant per instance | W of the first round | tables of even rounds | of odd rounds | instances]
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ __align__(16) E sh_r;
    __shared__ int sh_stop;
    __shared__ typename F::FoldKey sh_key;
    __shared__ __align__(16) E sh_part[3][kLogupTailBlocks];
    __shared__ __align__(16) E sh_sum[3][kLogupTailMaxInst];
    const uint32_t first_pairs = (1u << (n_rounds - first_round - 1)) / blocks;  // of this block
    E* consts = (E*)smem_raw;
    E* weights = consts + 3 * n_inst;
    uint4* const tab_mem = (uint4*)(weights + logup_tail_weights(first_pairs, blocks, alone));
    const size_t set_words = (size_t)n_tabs * TailTabs<F>::W * logup_tail_set_entries(first_pairs, blocks, alone, 0);
    LogupTailInst* inst = (LogupTailInst*)(tab_mem + set_words +
                                           (size_t)n_tabs * TailTabs<F>::W * logup_tail_set_entries(first_pairs, blocks, alone, 1));
    for (uint32_t i = threadIdx.x; i < 3 * n_inst; i += blockDim.x) consts[i] = consts_g[i];
    for (uint32_t i = threadIdx.x; i < n_inst * (uint32_t)(sizeof(LogupTailInst) / 4); i += blockDim.x)
        ((uint32_t*)inst)[i] = ((const uint32_t*)inst_g)[i];
    for (uint32_t p = threadIdx.x; p < first_pairs; p += blockDim.x)
        weights[p] = F::load(eq, F::kChalDtype, ((uint64_t)rank * first_pairs + p) << eq_stride_log2);
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
            const LogupTailInst in = inst[i];
            const uint32_t slot = t - in.tab0;
            E v;
            auto column_sum = [&](uint32_t half) {  // c + column_0 + s column_1 of the low or the high halves
                const uint32_t col = in.first + (in.kind == kLogupTable ? 2u : 0u) + half * in.ncol;
                E x = F::add(consts[3 * i + 2], logup_tail_load<F>(tabs[col], e0 + e, r));
                if (in.ncol == 2) x = F::add(x, F::mul(consts[3 * i + 1], logup_tail_load<F>(tabs[col + 1], e0 + e, r)));
                return x;
            };
            const bool inner = in.kind == kLogupInner;
            if (slot == 0) {
                v = inner ? logup_tail_load<F>(tabs[in.first + 2], e0 + e, r) : column_sum(0);
            } else if (slot == 1) {
                v = inner ? logup_tail_load<F>(tabs[in.first + 3], e0 + e, r) : column_sum(1);
            } else if (in.kind != kLogupLookup && slot < 4) {
                v = logup_tail_load<F>(tabs[in.first + (slot == 2 ? 1u : 0u)], e0 + e, r);
                if (slot == 2) {
                    const E d = inner ? logup_tail_load<F>(tabs[in.first + 3], e0 + e, r) : column_sum(1);
                    v = F::add(v, F::mul(lambda, d));
                }
            } else {  // the second column's halves, for the end
                const uint32_t half = (slot & 1u);
                v = logup_tail_load<F>(tabs[in.first + (in.kind == kLogupTable ? 2u : 0u) + half * 2 + 1], e0 + e, r);
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
                static_assert(kTailAloneGl <= 3 * kLogupTailMaxInst, "the weights pass through sh_sum");
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
                const LogupTailInst in = inst[i];
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
                const E al = consts[3 * (s / parts)];
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
        const LogupTailInst in = inst[i];
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
        const uint32_t extra = in.kind == kLogupTable ? 4 : 2;
        for (uint32_t half = 0; half < 2; half++) {
            E x = F::sub(half ? d : c, consts[3 * i + 2]);
            if (in.ncol == 2) {
                const E y = final_of(extra + half);
                post(col + half * 2 + 1, y);
                x = F::sub(x, F::mul(consts[3 * i + 1], y));
            }
            post(col + half * in.ncol, x);
        }
    }
}

}  // namespace dpb

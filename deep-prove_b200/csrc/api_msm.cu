// C ABI: multi-scalar multiplication over BN254 G1, the arithmetic of the commitment scheme's commit
// (HyperKZG commits to a multilinear polynomial as sum_i evals[i] * G_i over the SRS's G1 points;
// CommittedPolynomial::batch_commit, zkml/src/poly_commit/context.rs:56-90, one MSM per chunk of at most 2^20
// evaluations).
//
// Bucket method (Pippenger) with windows of c bits:
//   1. msm_count      per scalar and window: which bucket it goes to (its c-bit digit; zero digits are skipped);
//                     a histogram of the (window, bucket) keys
//   2. msm_scan_*     exclusive prefix sums of the histogram: where every bucket's list starts
//   3. msm_scatter    the point indices, grouped by bucket
//   4. msm_segments   the index list is cut into equal runs, one per thread, whatever buckets they belong to; a bucket
//                     that ends where it began in the same run is written at once, the pieces of one that spans runs
//                     are added up inside the block; msm_join adds what spans blocks
//   5. msm_reduce     per window sum_b b * B_b, as plain sums over the buckets whose number has a given bit set: four
//                     buckets per thread, then a tree in shared memory (msm_reduce over 512 buckets, msm_reduce_blocks
//                     over a window's blocks)
//   6. host           the sixteen sums per window and the windows put together in one chain of doublings, one
//                     inversion for the affine result.
// Integer tables (DPB_FR_I32 / DPB_FR_I64) enter as magnitudes: a negative scalar adds the negated point, and only
// the one to four windows their bits reach are ever touched: committing to quantised tensors and 16-bit lookup
// columns costs a fraction of a commit to full-width scalars.
#include <vector>

#include "../../include/dpb_pcs.h"
#include "common.cuh"
#include "g1_bn254.cuh"

struct dpb_g1_bases {
    dpb_ctx* ctx = nullptr;
    uint64_t n = 0;
    dpb::G1Affine* dev = nullptr;
};

namespace dpb {

struct MsmScalars {
    const void* ptr;
    int dtype;  // DPB_FR (Montgomery), DPB_FR_I32, DPB_FR_I64
};

// the scalar as a 256-bit magnitude (canonical integer below r) and a sign
__device__ __forceinline__ void msm_scalar(const MsmScalars& s, uint64_t i, uint64_t (&mag)[4], bool& neg) {
    neg = false;
    if (s.dtype == DPB_FR) {
        const Fr v = fr_from_mont(FrFam::load(s.ptr, DPB_FR, i));
        mag[0] = v.l[0];
        mag[1] = v.l[1];
        mag[2] = v.l[2];
        mag[3] = v.l[3];
        return;
    }
    const int64_t x = s.dtype == DPB_FR_I32 ? (int64_t)((const int32_t*)s.ptr)[i] : ((const int64_t*)s.ptr)[i];
    neg = x < 0;
    mag[0] = neg ? (uint64_t)0 - (uint64_t)x : (uint64_t)x;
    mag[1] = mag[2] = mag[3] = 0;
}
__device__ __forceinline__ uint32_t msm_digit(const uint64_t (&mag)[4], uint32_t w, uint32_t c) {
    const uint32_t bit = w * c, limb = bit >> 6, off = bit & 63;
    if (limb >= 4) return 0;
    uint64_t v = mag[limb] >> off;
    if (off + c > 64 && limb + 1 < 4) v |= mag[limb + 1] << (64 - off);
    return (uint32_t)(v & ((1ull << c) - 1));
}

// Lanes of a warp that hold the same key add their count with one atomic (a column of a few distinct values would
// otherwise send a million atomics to the same few counters).  Returns the lane's rank among them and, in every
// lane of the group, the value the leader's atomicAdd returned.
__device__ __forceinline__ uint32_t msm_group_add(uint32_t* counter, uint64_t key, bool take, unsigned active,
                                                  uint32_t& rank) {
    const unsigned peers = __match_any_sync(active, take ? key : ~0ull);
    const int leader = __ffs(peers) - 1;
    const unsigned lane = threadIdx.x & 31;
    rank = __popc(peers & ((1u << lane) - 1));
    uint32_t base = 0;
    if (take && (int)lane == leader) base = atomicAdd(counter, (uint32_t)__popc(peers));
    return __shfl_sync(peers, base, leader);
}

__global__ void __launch_bounds__(kThreads)
    msm_count(MsmScalars s, uint64_t n, uint32_t c, uint32_t windows, uint32_t* __restrict__ counts) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const unsigned active = __activemask();
        uint64_t mag[4];
        bool neg;
        msm_scalar(s, i, mag, neg);
        for (uint32_t w = 0; w < windows; w++) {
            const uint32_t d = msm_digit(mag, w, c);
            const size_t key = ((size_t)w << c) + d;
            uint32_t rank;
            msm_group_add(&counts[key], key, d != 0, active, rank);
        }
    }
}

// Exclusive scan of the histogram in three small launches: sums of tiles of 4096 counters, a scan of the tile sums
// by one block, and the scan inside every tile (all global accesses coalesced, the serial part in shared memory).
constexpr uint32_t kScanTile = 4096, kScanThreads = 256, kScanPer = kScanTile / kScanThreads;

__global__ void __launch_bounds__(kScanThreads)
    msm_scan_tile_sums(const uint32_t* __restrict__ counts, uint64_t n, uint32_t* __restrict__ tile_sums) {
    __shared__ uint32_t sh[kScanThreads];
    const uint64_t base = (uint64_t)blockIdx.x * kScanTile;
    uint32_t sum = 0;
    for (uint32_t j = 0; j < kScanPer; j++) {
        const uint64_t i = base + (uint64_t)j * kScanThreads + threadIdx.x;
        if (i < n) sum += counts[i];
    }
    sh[threadIdx.x] = sum;
    __syncthreads();
    for (uint32_t s = kScanThreads / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = sh[0];
}

// in place: tile_sums[t] becomes the sum of the tiles before t (n_tiles is at most a few thousand)
__global__ void __launch_bounds__(1024) msm_scan_tiles(uint32_t* __restrict__ tile_sums, uint32_t n_tiles) {
    __shared__ uint32_t part[1024];
    const uint32_t per = (n_tiles + blockDim.x - 1) / blockDim.x;
    const uint32_t lo = threadIdx.x * per, hi = lo + per < n_tiles ? lo + per : n_tiles;
    uint32_t sum = 0;
    for (uint32_t i = lo; i < hi; i++) sum += tile_sums[i];
    part[threadIdx.x] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t run = 0;
        for (uint32_t t = 0; t < blockDim.x; t++) {
            const uint32_t v = part[t];
            part[t] = run;
            run += v;
        }
    }
    __syncthreads();
    uint32_t run = part[threadIdx.x];
    for (uint32_t i = lo; i < hi; i++) {
        const uint32_t v = tile_sums[i];
        tile_sums[i] = run;
        run += v;
    }
}

__global__ void __launch_bounds__(kScanThreads)
    msm_scan_in_tiles(const uint32_t* __restrict__ counts, const uint32_t* __restrict__ tile_offsets, uint64_t n,
                      uint32_t* __restrict__ offsets) {
    __shared__ uint32_t vals[kScanTile];
    __shared__ uint32_t part[kScanThreads];
    const uint64_t base = (uint64_t)blockIdx.x * kScanTile;
    for (uint32_t j = 0; j < kScanPer; j++) {
        const uint32_t k = j * kScanThreads + threadIdx.x;
        vals[k] = base + k < n ? counts[base + k] : 0u;
    }
    __syncthreads();
    uint32_t sum = 0;
    for (uint32_t j = 0; j < kScanPer; j++) sum += vals[threadIdx.x * kScanPer + j];
    part[threadIdx.x] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t run = tile_offsets[blockIdx.x];
        for (uint32_t t = 0; t < kScanThreads; t++) {
            const uint32_t v = part[t];
            part[t] = run;
            run += v;
        }
    }
    __syncthreads();
    uint32_t run = part[threadIdx.x];
    for (uint32_t j = 0; j < kScanPer; j++) {
        const uint32_t k = threadIdx.x * kScanPer + j;
        const uint32_t v = vals[k];
        vals[k] = run;
        run += v;
    }
    __syncthreads();
    for (uint32_t j = 0; j < kScanPer; j++) {
        const uint32_t k = j * kScanThreads + threadIdx.x;
        if (base + k < n) offsets[base + k] = vals[k];
    }
}

__global__ void __launch_bounds__(kThreads)
    msm_scatter(MsmScalars s, uint64_t n, uint32_t c, uint32_t windows, const uint32_t* __restrict__ offsets,
                uint32_t* __restrict__ cursor, uint32_t* __restrict__ items) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const unsigned active = __activemask();
        uint64_t mag[4];
        bool neg;
        msm_scalar(s, i, mag, neg);
        for (uint32_t w = 0; w < windows; w++) {
            const uint32_t d = msm_digit(mag, w, c);
            const size_t key = ((size_t)w << c) + d;
            uint32_t rank;
            const uint32_t at = msm_group_add(&cursor[key], key, d != 0, active, rank);
            if (d) items[offsets[key] + at + rank] = (uint32_t)i | (neg ? 0x80000000u : 0u);
        }
    }
}

// Bucket sums.  The scatter leaves the point indices grouped by bucket, in the order of the buckets, so the list is cut
// into equal runs, one per thread of a grid that fills the GPU once: every lane of a warp makes the same number of
// additions whether the digits are uniform (16 points a bucket at 2^20 points), crowd a few buckets or are almost all
// one value.  (With a thread per bucket a warp waits for its fullest bucket, 27 points where the mean is 16, and
// buckets of more than 96 points need kernels of their own: six integer columns of 2^20 committed together took 3944 us
// that way; equal runs and the bit sums below took 2099 us, four lanes per addition in the trees and the host's share
// next to the kernels 1784 us.)  A run begins inside a bucket as a rule and ends inside another: those two pieces meet
// their neighbours' in shared memory.
//
// Pieces of a span of runs (a thread's, later a part of the block's, at last the block's):
//   L  the sum of the span's first points, of a bucket that began before the span and ends inside it
//   R  the sum of its last points, of a bucket that begins inside the span and goes on after it
//   W  (kept in L's place) the whole span belongs to one bucket that began before and goes on after
// Two neighbouring spans meet in at most one addition: R or W of the left one with L or W of the right one.  R + L
// completes a bucket; all those pairs are added at once, so that only buckets that span three runs or more go through
// the levels of the tree.
constexpr int kSegThreads = 128;
constexpr int kSegBlocks = 4;            // resident blocks per SM at 128 registers
constexpr uint32_t kSegMinRun = 2;       // an addition of the run and a level of the tree take about as long
constexpr uint32_t kHasL = 1, kHasR = 2, kWhole = 4;

struct MsmEdge {
    G1Sum L, R;
    uint32_t flags, key_r, pad[2];
};

// last key whose list starts at or before item j, at or after `from` (offsets[from] <= j)
__device__ __forceinline__ uint32_t msm_key_of(const uint32_t* __restrict__ offsets, uint32_t n_keys, uint32_t from, uint32_t j) {
    uint32_t lo = from, hi = n_keys;
    for (uint32_t step = 1; lo + step < hi; step <<= 1) {  // the next key as a rule: look near first
        if (offsets[lo + step] > j) {
            hi = lo + step;
            break;
        }
        lo += step;
    }
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (offsets[mid] <= j) lo = mid;
        else hi = mid;
    }
    return lo;
}

// *to = *x + *y: one copy of the addition for every step of a tree, its operands in memory
__device__ __noinline__ void msm_add(G1Sum* to, const G1Sum* x, const G1Sum* y) { *to = g1_add(*x, *y); }

// The same by four neighbouring lanes, for the levels of a tree that leave lanes idle: the fourteen products of the
// addition in four steps of one product per lane (a warp alone on its scheduler issues a product in about 0.3 us
// whatever the number of its lanes that take part).  All four lanes are called with the same pointers.
__device__ __noinline__ void msm_add4(G1Sum* to, const G1Sum* x, const G1Sum* y) {
    const uint32_t lane = threadIdx.x & 31, q = lane & 3;
    const uint32_t quad = 0xfu << (lane & ~3u);
    auto from = [&](const Fq& v, int src) {
        Fq r;
#pragma unroll
        for (int i = 0; i < 4; i++) r.l[i] = __shfl_sync(quad, v.l[i], src, 4);
        return r;
    };
    const bool x_inf = g1_is_infinity(*x), y_inf = g1_is_infinity(*y);
    __syncwarp(quad);
    if (x_inf || y_inf) {
        const Fq* src = (const Fq*)(x_inf ? y : x);
        ((Fq*)to)[q] = src[q];
        return;
    }
    // 1: U1, U2, S1, S2 of lanes 0..3
    const Fq* mine = (const Fq*)(q & 1 ? y : x);    // its X or Y
    const Fq* other = (const Fq*)(q & 1 ? x : y);   // with this one's ZZ or ZZZ
    const uint32_t h = q >> 1;
    const Fq v1 = fq_mul(mine[h], other[2 + h]);
    Fq d = from(v1, (int)(q ^ 1));
    d = q & 1 ? fq_sub(v1, d) : fq_sub(d, v1);  // P in lanes 0 and 1, R in lanes 2 and 3
    const unsigned zero = __ballot_sync(quad, fq_is_zero(d)) >> (lane & ~3u);
    if (zero & 1) {  // the same point or opposite points
        if (q == 0) *to = zero & 4 ? g1_double(*x) : g1_infinity();
        __syncwarp(quad);
        return;
    }
    // 2: PP, ZZ1 ZZ2, RR, ZZZ1 ZZZ2
    const Fq v2 = fq_mul(q & 1 ? mine[2 + h] : d, q & 1 ? other[2 + h] : d);
    // 3: P PP, ZZ1 ZZ2 PP, U1 PP
    const Fq pp = from(v2, 0), u1 = from(v1, 0);
    const Fq v3 = fq_mul(q == 0 ? d : q == 1 ? v2 : u1, pp);
    // 4: S1 PPP, -, R (Q - X), ZZZ1 ZZZ2 PPP
    const Fq ppp = from(v3, 0), s1 = from(v1, 2);
    const Fq X = fq_sub(fq_sub(v2, ppp), fq_dbl(v3));  // lane 2: RR - PPP - 2 Q
    const Fq v4 = fq_mul(q == 0 ? s1 : q == 2 ? d : v2, q == 2 ? fq_sub(v3, X) : ppp);
    const Fq s1ppp = from(v4, 0);
    if (q == 1) to->ZZ = v3;
    if (q == 2) {
        to->X = X;
        to->Y = fq_sub(v4, s1ppp);
    }
    if (q == 3) to->ZZZ = v4;
}

// Joins span `a` with the span `b` to its right, by four lanes; the result is span a.  The whole of a span lies in its L; r[a] is
// where its R lies, key_r[a] the bucket R belongs to.
struct MsmSpans {
    uint32_t* flags;
    uint32_t* key_r;
    uint32_t* r;
};
template <class Left, class Right>
__device__ __forceinline__ void msm_meet(const MsmSpans& sp, uint32_t a, uint32_t b, const Left& left, const Right& right,
                                         G1Sum* __restrict__ buckets) {
    const uint32_t fa = sp.flags[a], fb = sp.flags[b];
    uint32_t f = (fa & kHasL) | (fb & kHasR);
    if ((fa & (kHasR | kWhole)) && (fb & (kHasL | kWhole))) {
        G1Sum* x = fa & kWhole ? left(a) : right(sp.r[a]);
        G1Sum* to = (fa | fb) & kWhole ? x : &buckets[sp.key_r[a]];
        msm_add4(to, x, left(b));
        if (fa & fb & kWhole) f = kWhole;
        else if (fa & kWhole) f |= kHasL;
        else if (fb & kWhole) f |= kHasR;
    }
    __syncwarp(0xfu << (threadIdx.x & 28));  // all four have read
    if (threadIdx.x & 3) return;
    if (!(fb & kWhole)) {
        sp.key_r[a] = sp.key_r[b];
        sp.r[a] = sp.r[b];
    }
    sp.flags[a] = f;
}

// Bound by the multiplier: ten products per point (1216 multiply-adds), the points gathered from L2.  2^20 points: 284 us
// for 16-bit values and 266 us for 12-bit ones, where the multiply-adds alone take 147.
__global__ void __launch_bounds__(kSegThreads, kSegBlocks)
    msm_segments(const G1Affine* __restrict__ bases, const uint32_t* __restrict__ offsets,
                 const uint32_t* __restrict__ counts, const uint32_t* __restrict__ items, uint32_t n_keys,
                 G1Sum* __restrict__ buckets, MsmEdge* __restrict__ edges) {
    __shared__ G1Sum L[kSegThreads], R[kSegThreads];
    __shared__ uint32_t flags[kSegThreads], key_r[kSegThreads], r_at[kSegThreads];
    const uint32_t total = offsets[n_keys - 1] + counts[n_keys - 1], t = threadIdx.x;
    const uint32_t threads = gridDim.x * kSegThreads;
    uint32_t run = (uint32_t)(((uint64_t)total + threads - 1) / threads);
    if (run < kSegMinRun) run = kSegMinRun;
    const uint64_t start64 = (uint64_t)(blockIdx.x * kSegThreads + t) * run;
    const uint32_t start = start64 < total ? (uint32_t)start64 : total;
    const uint32_t end = total - start < run ? total : start + run;
    uint32_t f = 0, key = 0;
    if (start < end) {
        key = msm_key_of(offsets, n_keys, 0, start);
        uint32_t key_end = offsets[key] + counts[key];
        bool before = offsets[key] < start;  // the bucket at hand began before this run
        G1Sum acc = g1_infinity();
        for (uint32_t j = start; j < end; j++) {
            if (j == key_end) {
                if (before) {
                    L[t] = acc;
                    f |= kHasL;
                } else {
                    buckets[key] = acc;
                }
                key = msm_key_of(offsets, n_keys, key, j);
                key_end = offsets[key] + counts[key];
                before = false;
                acc = g1_infinity();
            }
            const uint32_t it = items[j];
            G1Affine p = bases[it & 0x7fffffffu];
            if (it & 0x80000000u) p = g1_affine_neg(p);
            acc = g1_add_mixed(acc, p);
        }
        if (before) {
            L[t] = acc;
            f |= key_end > end ? kWhole : kHasL;
        } else if (key_end > end) {
            R[t] = acc;
            f |= kHasR;
        } else {
            buckets[key] = acc;
        }
    }
    flags[t] = f;
    key_r[t] = key;
    r_at[t] = t;
    __syncthreads();
    // buckets of two runs, all at once
    const bool pair = t + 1 < kSegThreads && (f & kHasR) && (flags[t + 1] & kHasL);
    if (pair) msm_add(&buckets[key_r[t]], &R[t], &L[t + 1]);
    __syncthreads();
    if (pair) {
        atomicAnd(&flags[t], ~kHasR);
        atomicAnd(&flags[t + 1], ~kHasL);
    }
    __syncthreads();
    const MsmSpans sp = {flags, key_r, r_at};
    for (uint32_t s = 1; s < kSegThreads; s <<= 1) {
        for (uint32_t a = 2 * s * (t / 4); a < kSegThreads; a += 2 * s * (kSegThreads / 4))
            msm_meet(sp, a, a + s, [&](uint32_t i) { return &L[i]; }, [&](uint32_t i) { return &R[i]; }, buckets);
        __syncthreads();
    }
    MsmEdge& e = edges[blockIdx.x];
    if (t == 0) {
        e.flags = flags[0];
        e.key_r = key_r[0];
        if (flags[0] & (kHasL | kWhole)) e.L = L[0];
    }
    if (t == 32 && (flags[0] & kHasR)) e.R = R[r_at[0]];
}

// The pieces that span blocks of msm_segments (at most a few hundred blocks).  Block 0 takes the buckets that span
// three blocks or more through the levels of the tree, the others the pairs, 128 each: the two sets are disjoint.
constexpr int kJoinThreads = 512, kJoinStep = 128, kJoinMax = 2048;
__global__ void __launch_bounds__(kJoinThreads)
    msm_join(MsmEdge* __restrict__ edges, uint32_t n, G1Sum* __restrict__ buckets) {
    __shared__ uint32_t flags[kJoinMax], key_r[kJoinMax], r_at[kJoinMax];
    const uint32_t t = threadIdx.x;
    if (blockIdx.x > 0) {
        const uint32_t i = (blockIdx.x - 1) * kJoinStep + t;
        if (t < kJoinStep && i + 1 < n && (edges[i].flags & kHasR) && (edges[i + 1].flags & kHasL))
            msm_add(&buckets[edges[i].key_r], &edges[i].R, &edges[i + 1].L);
        return;
    }
    bool left = false;
    for (uint32_t i = t; i < n; i += kJoinThreads) {
        uint32_t f = edges[i].flags;
        if ((f & kHasR) && i + 1 < n && (edges[i + 1].flags & kHasL)) f &= ~kHasR;
        if ((f & kHasL) && i > 0 && (edges[i - 1].flags & kHasR)) f &= ~kHasL;
        flags[i] = f;
        key_r[i] = edges[i].key_r;
        r_at[i] = i;
        left = left || f != 0;
    }
    if (!__syncthreads_or(left)) return;
    const MsmSpans sp = {flags, key_r, r_at};
    for (uint32_t s = 1; s < n; s <<= 1) {
        for (uint32_t a = 2 * s * (t / 4); a + s < n; a += 2 * s * (kJoinThreads / 4))
            msm_meet(sp, a, a + s, [&](uint32_t i) { return &edges[i].L; }, [&](uint32_t i) { return &edges[i].R; }, buckets);
        __syncthreads();
    }
}

// Bound by the latency of its dependent additions (a block of 512 buckets: five, then seven levels): 106 + 38 us for two
// windows of 2^16 buckets where runs of 16 buckets with running sums took 440.
// sum_b b B_b of a window as plain sums: over the buckets whose number has bit k set, for every k.  Pairs of spans of
// 2^l elements join by adding their sums bit by bit; the right one's total is the new bit l.  In place: element 0 of
// a span holds its total, element 2^k the sum over the elements with bit k set.  l + 1 additions per pair, two per
// element over all levels (as many as a running sum takes), none waiting for another of its level.
// sums of a block: 0: sum of (b mod 4) B_b; 1..7: of the B_b with bit 2..8 of b set; 8: of all
constexpr int kReduceThreads = 128, kReduceLevels = 7, kReducePer = 4;
constexpr uint32_t kReduceSpan = kReduceThreads * kReducePer, kBlockSums = kReduceLevels + 2;
// sums of a window: 0..7 the blocks' added up; 8..14: of all B_b with bit 9..15 of b set
constexpr uint32_t kWindowSums = 16;
// which of them enters with weight 2^bit, or -1
static int msm_sum_of_bit(uint32_t bit) { return bit == 0 ? 0 : bit == 1 ? -1 : (int)bit - 1; }

__global__ void __launch_bounds__(kReduceThreads, 4)
    msm_reduce(const G1Sum* __restrict__ buckets, const uint32_t* __restrict__ counts, uint32_t c, uint32_t blocks_per_window,
               G1Sum* __restrict__ part) {
    __shared__ G1Sum S[kReduceThreads], T[kReduceThreads];
    const uint32_t w = blockIdx.x / blocks_per_window, blk = blockIdx.x % blocks_per_window, t = threadIdx.x;
    const uint32_t first = blk * kReduceSpan + t * kReducePer;
    S[t] = T[t] = g1_infinity();
    bool any = false;
#pragma unroll 1
    for (int b = kReducePer - 1; b >= 0; b--) {  // S = sum of b B_b, T = sum of B_b
        const size_t key = ((size_t)w << c) + first + b;
        if (first + b < (1u << c) && counts[key]) {  // the bucket of digit 0 has no points
            msm_add(&T[t], &T[t], &buckets[key]);
            any = true;
        }
        if (b) msm_add(&S[t], &S[t], &T[t]);
    }
    if (__syncthreads_or(any)) {
#pragma unroll 1
        for (uint32_t l = 0; l < kReduceLevels; l++) {
            const uint32_t s = 1u << l, pairs = kReduceThreads >> (l + 1);
            for (uint32_t a = t / 4; a < pairs * (l + 2); a += kReduceThreads / 4) {
                // the last `pairs` additions are the plain sums S
                const bool bits = a < pairs * (l + 1);
                const uint32_t pair = bits ? a / (l + 1) : a - pairs * (l + 1), k = bits ? a % (l + 1) : 0;
                G1Sum* x = (bits ? T : S) + (pair << (l + 1)) + (k ? 1u << (k - 1) : 0u);
                msm_add4(x, x, x + s);
            }
            __syncthreads();
        }
    }
    if (t < kBlockSums) part[(size_t)blockIdx.x * kBlockSums + t] = t == 0 ? S[0] : t == kBlockSums - 1 ? T[0] : T[1u << (t - 1)];
}

// one block per window and sum: the sums 0..7 over the window's blocks, the blocks' totals by the bits of the block
__global__ void __launch_bounds__(kReduceThreads, 4)
    msm_reduce_blocks(const G1Sum* __restrict__ part, uint32_t blocks_per_window, G1Sum* __restrict__ sums) {
    __shared__ G1Sum T[kReduceThreads];
    const uint32_t w = blockIdx.x / kBlockSums, v = blockIdx.x % kBlockSums, t = threadIdx.x;
    T[t] = t < blocks_per_window ? part[((size_t)w * blocks_per_window + t) * kBlockSums + v] : g1_infinity();
    const bool bits = v == kBlockSums - 1;
    __syncthreads();
#pragma unroll 1
    for (uint32_t l = 0; l < kReduceLevels && (1u << l) < blocks_per_window; l++) {
        const uint32_t sums_per = bits ? l + 1 : 1;
        for (uint32_t a = t / 4; a < (kReduceThreads >> (l + 1)) * sums_per; a += kReduceThreads / 4) {
            const uint32_t k = a % sums_per;
            G1Sum* x = T + ((a / sums_per) << (l + 1)) + (k ? 1u << (k - 1) : 0u);
            msm_add4(x, x, x + (1u << l));
        }
        __syncthreads();
    }
    G1Sum* out = sums + (size_t)w * kWindowSums;
    if (!bits) {
        if (t == 0) out[v] = T[0];
    } else if (t < kReduceLevels) {
        out[kBlockSums - 1 + t] = (1u << t) < blocks_per_window ? T[1u << t] : g1_infinity();
    } else if (t == kReduceLevels) {
        out[kWindowSums - 1] = g1_infinity();
    }
}

__global__ void __launch_bounds__(kThreads) msm_bases_to_mont(G1Affine* p, uint64_t n, unsigned int* bad) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    G1Affine a = p[i];
    if (!g1_affine_is_infinity(a)) {
        if (fq_geq_q(a.x) || fq_geq_q(a.y)) {
            atomicAdd(bad, 1u);
            return;
        }
        a.x = fq_to_mont(a.x);
        a.y = fq_to_mont(a.y);
        if (!g1_affine_on_curve(a)) atomicAdd(bad, 1u);
    }
    p[i] = a;
}

// point i = (first + i) * G for the generator G = (1, 2): valid, distinct points for benchmarks and tests
__global__ void __launch_bounds__(kThreads) msm_synthetic_bases(G1Affine* out, uint64_t n, uint32_t first) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    G1Affine g;
    Fq one, two;
    one.l[0] = 1;
    two.l[0] = 2;
    one.l[1] = one.l[2] = one.l[3] = two.l[1] = two.l[2] = two.l[3] = 0;
    g.x = fq_to_mont(one);
    g.y = fq_to_mont(two);
    out[i] = g1_to_affine(g1_mul_small(g1_from_affine(g), first + (uint32_t)i));
}

static uint32_t msm_window_bits(uint64_t n) {
    uint32_t lg = 0;
    while ((1ull << lg) < n) lg++;
    if (lg >= 18) return 16;
    if (lg >= 14) return 13;
    if (lg >= 10) return 10;
    return 8;
}

constexpr uint32_t kMsmGroup = dpb_ctx::kMsmGroup;
constexpr size_t kMsmHostBytes = 1 << 20;         // pinned staging for their window sums

// One commitment: its layout in one block of device memory [counts | offsets | cursor | items | scan tiles | buckets |
// block edges | block sums | window sums].
struct MsmJob {
    uint64_t n = 0;
    uint32_t c = 0, windows = 0, blocks_per_window = 0, n_tiles = 0, segment_blocks = 0;
    size_t n_keys = 0, n_sums = 0, host_off = 0;
    size_t o_counts = 0, o_offsets = 0, o_cursor = 0, o_items = 0, o_tiles = 0, o_buckets = 0, o_edges = 0, o_part = 0,
           o_sums = 0;
    void* slab = nullptr;
};

static int msm_plan(dpb_ctx* ctx, const dpb_g1_bases* bases, const dpb_mle* scalars, MsmJob& job) {
    if (scalars->dtype != DPB_FR && scalars->dtype != DPB_FR_I32 && scalars->dtype != DPB_FR_I64)
        return fail(DPB_EINVAL, "scalars must be a BN254 table (DPB_FR, DPB_FR_I32 or DPB_FR_I64), not dtype %d", scalars->dtype);
    const uint64_t n = scalars->len;
    if (n > bases->n)
        return fail(DPB_EINVAL, "%llu scalars but only %llu points", (unsigned long long)n, (unsigned long long)bases->n);
    job.n = n;
    job.c = msm_window_bits(n);
    const uint32_t scalar_bits = scalars->dtype == DPB_FR ? 254 : scalars->dtype == DPB_FR_I32 ? 32 : 64;
    job.windows = (scalar_bits + job.c - 1) / job.c;
    job.n_keys = (size_t)job.windows << job.c;
    job.blocks_per_window = (uint32_t)(((1ull << job.c) + kReduceSpan - 1) / kReduceSpan);
    job.n_sums = (size_t)job.windows * kWindowSums;
    job.segment_blocks = std::min<uint32_t>((uint32_t)ctx->sm_count * kSegBlocks, kJoinMax);
    const uint64_t most = ((uint64_t)n * job.windows + kSegThreads * kSegMinRun - 1) / (kSegThreads * kSegMinRun);
    if (most < job.segment_blocks) job.segment_blocks = (uint32_t)most;
    job.n_tiles = (uint32_t)((job.n_keys + kScanTile - 1) / kScanTile);
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off = (off + bytes + 255) & ~(size_t)255;
        return o;
    };
    job.o_counts = take(job.n_keys * 4);
    job.o_offsets = take(job.n_keys * 4);
    job.o_cursor = take(job.n_keys * 4);
    job.o_items = take((size_t)n * job.windows * 4);
    job.o_tiles = take((size_t)job.n_tiles * 4);
    job.o_buckets = take(job.n_keys * sizeof(G1Sum));
    job.o_edges = take((size_t)job.segment_blocks * sizeof(MsmEdge));
    job.o_part = take((size_t)job.windows * job.blocks_per_window * kBlockSums * sizeof(G1Sum));
    job.o_sums = take(job.n_sums * sizeof(G1Sum));
    return device_alloc(ctx, off, &job.slab);
}

// every kernel of one commitment and the copy of its window sums to `h_part` (pinned), on stream `st`
static cudaError_t msm_launch(dpb_ctx* ctx, const dpb_g1_bases* bases, const dpb_mle* scalars, const MsmJob& job,
                              cudaStream_t st, G1Sum* h_sums) {
    char* base = (char*)job.slab;
    uint32_t* counts = (uint32_t*)(base + job.o_counts);
    uint32_t* offsets = (uint32_t*)(base + job.o_offsets);
    uint32_t* cursor = (uint32_t*)(base + job.o_cursor);
    uint32_t* items = (uint32_t*)(base + job.o_items);
    uint32_t* tile_sums = (uint32_t*)(base + job.o_tiles);
    G1Sum* buckets = (G1Sum*)(base + job.o_buckets);
    MsmEdge* edges = (MsmEdge*)(base + job.o_edges);
    G1Sum* part = (G1Sum*)(base + job.o_part);
    G1Sum* sums = (G1Sum*)(base + job.o_sums);
    MsmScalars s;
    s.ptr = scalars->ptr;
    s.dtype = scalars->dtype;
    const uint64_t n = job.n;
    const uint32_t c = job.c, windows = job.windows;
    const size_t n_keys = job.n_keys;
    cudaError_t e = cudaMemsetAsync(counts, 0, job.o_items - job.o_counts, st);  // counts, offsets, cursor
    if (e != cudaSuccess) return e;
    msm_count<<<grid_for(ctx, n), kThreads, 0, st>>>(s, n, c, windows, counts);
    msm_scan_tile_sums<<<job.n_tiles, kScanThreads, 0, st>>>(counts, n_keys, tile_sums);
    msm_scan_tiles<<<1, 1024, 0, st>>>(tile_sums, job.n_tiles);
    msm_scan_in_tiles<<<job.n_tiles, kScanThreads, 0, st>>>(counts, tile_sums, n_keys, offsets);
    msm_scatter<<<grid_for(ctx, n), kThreads, 0, st>>>(s, n, c, windows, offsets, cursor, items);
    msm_segments<<<job.segment_blocks, kSegThreads, 0, st>>>(bases->dev, offsets, counts, items, (uint32_t)n_keys, buckets,
                                                             edges);
    msm_join<<<1 + (job.segment_blocks + kJoinStep - 1) / kJoinStep, kJoinThreads, 0, st>>>(edges, job.segment_blocks, buckets);
    msm_reduce<<<windows * job.blocks_per_window, kReduceThreads, 0, st>>>(buckets, counts, c, job.blocks_per_window, part);
    msm_reduce_blocks<<<windows * kBlockSums, kReduceThreads, 0, st>>>(part, job.blocks_per_window, sums);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return cudaMemcpyAsync(h_sums, sums, job.n_sums * sizeof(G1Sum), cudaMemcpyDeviceToHost, st);
}

// host: bit by bit from the top, total = 2 total + the sums that enter at this bit of this window; one inversion for
// the affine result
static void msm_finish(const MsmJob& job, const G1Sum* h_sums, Fq* xy) {
    G1Sum total = g1_infinity();
    for (uint32_t w = job.windows; w-- > 0;) {
        for (uint32_t bit = job.c; bit-- > 0;) {
            total = g1_double(total);
            const int at = msm_sum_of_bit(bit);
            if (at >= 0) total = g1_add(total, h_sums[(size_t)w * kWindowSums + at]);
        }
    }
    const G1Affine a = g1_to_affine(total);
    if (g1_affine_is_infinity(a)) {
        xy[0] = xy[1] = fq_zero();
    } else {
        xy[0] = fq_from_mont(a.x);
        xy[1] = fq_from_mont(a.y);
    }
}

static int msm_done_events(dpb_ctx* ctx, uint32_t n) {
    for (uint32_t j = 0; j < n; j++)
        if (!ctx->msm_done[j]) DPB_CUDA(cudaEventCreateWithFlags(&ctx->msm_done[j], cudaEventDisableTiming));
    return DPB_OK;
}

static int msm_side_streams(dpb_ctx* ctx) {
    if (ctx->msm_stream[0]) return DPB_OK;
    for (int q = 0; q < dpb_ctx::kMsmStreams; q++) DPB_CUDA(cudaStreamCreateWithFlags(&ctx->msm_stream[q], cudaStreamNonBlocking));
    for (int q = 0; q <= dpb_ctx::kMsmStreams; q++) DPB_CUDA(cudaEventCreateWithFlags(&ctx->msm_ev[q], cudaEventDisableTiming));
    return DPB_OK;
}

}  // namespace dpb

using namespace dpb;

extern "C" {

int dpb_g1_bases_from_host(dpb_ctx* ctx, const void* affine_xy, uint64_t n, dpb_g1_bases** out) {
    if (!ctx || !affine_xy || !out) return fail(DPB_EINVAL, "null argument");
    if (n == 0 || n > (1ull << 31)) return fail(DPB_EINVAL, "number of points %llu outside 1..2^31", (unsigned long long)n);
    dpb_g1_bases* b = new (std::nothrow) dpb_g1_bases();
    if (!b) return fail(DPB_ENOMEM, "host allocation failed");
    b->ctx = ctx;
    b->n = n;
    void* p = nullptr;
    int rc = device_alloc(ctx, n * sizeof(G1Affine), &p);
    if (rc != DPB_OK) {
        delete b;
        return rc;
    }
    b->dev = (G1Affine*)p;
    unsigned int* bad = nullptr;
    rc = device_alloc(ctx, sizeof(unsigned int), (void**)&bad);
    unsigned int h_bad = 0;
    cudaError_t e = cudaSuccess;
    if (rc == DPB_OK) {
        e = cudaMemcpyAsync(p, affine_xy, n * sizeof(G1Affine), cudaMemcpyHostToDevice, ctx->stream);
        if (e == cudaSuccess) e = cudaMemsetAsync(bad, 0, sizeof(unsigned int), ctx->stream);
        if (e == cudaSuccess) {
            msm_bases_to_mont<<<(uint32_t)((n + kThreads - 1) / kThreads), kThreads, 0, ctx->stream>>>(b->dev, n, bad);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaMemcpyAsync(&h_bad, bad, sizeof(unsigned int), cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    }
    device_free(ctx, bad);
    if (rc == DPB_OK && e != cudaSuccess) rc = fail(DPB_ECUDA, "uploading G1 points: %s", cudaGetErrorString(e));
    if (rc == DPB_OK && h_bad) rc = fail(DPB_EINVAL, "%u points are not on the curve or have coordinates >= q", h_bad);
    if (rc != DPB_OK) {
        device_free(ctx, p);
        delete b;
        return rc;
    }
    *out = b;
    return DPB_OK;
}

int dpb_g1_bases_synthetic(dpb_ctx* ctx, uint64_t n, uint32_t first_multiple, dpb_g1_bases** out) {
    if (!ctx || !out) return fail(DPB_EINVAL, "null argument");
    if (n == 0 || first_multiple == 0 || n + first_multiple > (1ull << 31))
        return fail(DPB_EINVAL, "multiples %u .. %llu of the generator are outside 1..2^31", first_multiple,
                    (unsigned long long)(n + first_multiple - 1));
    dpb_g1_bases* b = new (std::nothrow) dpb_g1_bases();
    if (!b) return fail(DPB_ENOMEM, "host allocation failed");
    b->ctx = ctx;
    b->n = n;
    void* p = nullptr;
    int rc = device_alloc(ctx, n * sizeof(G1Affine), &p);
    if (rc != DPB_OK) {
        delete b;
        return rc;
    }
    b->dev = (G1Affine*)p;
    msm_synthetic_bases<<<(uint32_t)((n + kThreads - 1) / kThreads), kThreads, 0, ctx->stream>>>(b->dev, n, first_multiple);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        device_free(ctx, p);
        delete b;
        return fail(DPB_ECUDA, "synthetic bases: %s", cudaGetErrorString(e));
    }
    *out = b;
    return DPB_OK;
}

uint64_t dpb_g1_bases_len(const dpb_g1_bases* b) { return b ? b->n : 0; }

void dpb_g1_bases_free(dpb_g1_bases* b) {
    if (!b) return;
    device_free(b->ctx, b->dev);
    delete b;
}

int dpb_msm_g1(dpb_ctx* ctx, const dpb_g1_bases* bases, const dpb_mle* scalars, void* out_affine_xy) {
    dpb_mle* one[1] = {const_cast<dpb_mle*>(scalars)};
    if (!scalars) return fail(DPB_EINVAL, "null argument");
    return dpb_pcs_batch_commit(ctx, bases, one, 1, out_affine_xy);
}

int dpb_pcs_batch_commit(dpb_ctx* ctx, const dpb_g1_bases* bases, dpb_mle* const* polys, uint32_t n_polys,
                         void* out_affine_xy) {
    if (!ctx || !bases || !polys || !out_affine_xy) return fail(DPB_EINVAL, "null argument");
    if (bases->ctx != ctx) return fail(DPB_EINVAL, "the bases belong to another context");
    for (uint32_t i = 0; i < n_polys; i++) {
        if (!polys[i]) return fail(DPB_EINVAL, "polynomial %u is null", i);
        if (polys[i]->ctx != ctx) return fail(DPB_EINVAL, "polynomial %u belongs to another context", i);
    }
    if (n_polys > 1) DPB_TRY(msm_side_streams(ctx));
    DPB_TRY(msm_done_events(ctx, std::min<uint32_t>(kMsmGroup, n_polys)));
    // groups of commitments in flight together: their kernels are short chains of curve additions that leave most
    // of the GPU idle one at a time
    for (uint32_t first = 0; first < n_polys; first += kMsmGroup) {
        const uint32_t cnt = std::min<uint32_t>(kMsmGroup, n_polys - first);
        std::vector<MsmJob> jobs(cnt);
        std::vector<Fq> xy(2 * (size_t)cnt);  // handed out when the whole group is done
        int rc = DPB_OK;
        size_t host_off = 0;
        for (uint32_t j = 0; j < cnt && rc == DPB_OK; j++) {
            rc = msm_plan(ctx, bases, polys[first + j], jobs[j]);
            jobs[j].host_off = host_off;
            host_off += jobs[j].n_sums * sizeof(G1Sum);
        }
        if (rc == DPB_OK && host_off > kMsmHostBytes) rc = fail(DPB_EINVAL, "commitment staging of %zu bytes", host_off);
        cudaError_t e = cudaSuccess;
        if (rc == DPB_OK) {
            if (!ctx->msm_host) e = cudaHostAlloc(&ctx->msm_host, kMsmHostBytes, cudaHostAllocDefault);
            const bool side = cnt > 1;
            if (e == cudaSuccess && side) {
                // the side streams start after everything this context has queued (the scalars' producers included)
                e = cudaEventRecord(ctx->msm_ev[dpb_ctx::kMsmStreams], ctx->stream);
                for (int q = 0; q < dpb_ctx::kMsmStreams && e == cudaSuccess; q++)
                    e = cudaStreamWaitEvent(ctx->msm_stream[q], ctx->msm_ev[dpb_ctx::kMsmStreams], 0);
            }
            for (uint32_t j = 0; j < cnt && e == cudaSuccess; j++) {
                cudaStream_t st = side ? ctx->msm_stream[j % dpb_ctx::kMsmStreams] : ctx->stream;
                e = msm_launch(ctx, bases, polys[first + j], jobs[j], st, (G1Sum*)((char*)ctx->msm_host + jobs[j].host_off));
                if (e == cudaSuccess) e = cudaEventRecord(ctx->msm_done[j], st);
            }
            if (side) {
                // ... and this context's stream goes on after them (even when a launch failed: the slabs are freed below)
                for (int q = 0; q < dpb_ctx::kMsmStreams; q++) {
                    cudaEventRecord(ctx->msm_ev[q], ctx->msm_stream[q]);
                    cudaStreamWaitEvent(ctx->stream, ctx->msm_ev[q], 0);
                }
            }
            // the host's share of a commitment while the kernels of the next ones run
            for (uint32_t j = 0; j < cnt && e == cudaSuccess; j++) {
                e = cudaEventSynchronize(ctx->msm_done[j]);
                if (e == cudaSuccess)
                    msm_finish(jobs[j], (const G1Sum*)((const char*)ctx->msm_host + jobs[j].host_off), &xy[2 * j]);
            }
            const cudaError_t es = cudaStreamSynchronize(ctx->stream);
            if (e == cudaSuccess) e = es;
        }
        for (auto& job : jobs) device_free(ctx, job.slab);
        if (rc != DPB_OK) return rc;
        if (e != cudaSuccess) return fail(DPB_ECUDA, "msm: %s", cudaGetErrorString(e));
        memcpy((char*)out_affine_xy + (size_t)first * 64, xy.data(), (size_t)cnt * 64);
    }
    return DPB_OK;
}

}  // extern "C"

// Launches of the claim-batching rounds (eq_pairs.cuh).
#include "eq_pairs.hpp"

#include "eq_pairs.cuh"

namespace dpb {

template <class F>
void eq_pairs_launch_round(dpb_ctx* ctx, const EqPairPlan& p, uint32_t round, const typename F::E& r) {
    typedef typename F::E E;
    const uint32_t n = (uint32_t)p.terms.size();
    // two resident blocks per SM; every block walks tiles
    uint32_t blocks = std::min<uint32_t>(p.tiles[round], (uint32_t)ctx->sm_count * 2);
    if (blocks > ctx->max_blocks) blocks = ctx->max_blocks;
    E* s = (E*)p.d_s;
    eq_pairs_round<F><<<blocks, kThreads, 0, ctx->stream>>>(
        (const EqPairTerm*)p.d_terms, n, (const E*)p.d_points, p.d_prefix + (size_t)round * (n + 1), p.per_thread[round], round,
        r, EqPairKey<F>::make(r), s + (size_t)((round + 1) & 1) * n, s + (size_t)(round & 1) * n, reduce_scratch<F>(ctx),
        (E*)ctx->round_out);
}

template <class F>
void eq_pairs_launch_finals(dpb_ctx* ctx, const EqPairPlan& p, uint32_t round, const typename F::E& r, typename F::E* out) {
    typedef typename F::E E;
    const uint32_t n = (uint32_t)p.terms.size();
    eq_pairs_finals<F><<<(n + kThreads - 1) / kThreads, kThreads, 0, ctx->stream>>>(
        (const EqPairTerm*)p.d_terms, n, (const E*)p.d_points, round, r, (const E*)p.d_s + (size_t)(round & 1) * n, out);
}

template void eq_pairs_launch_round<FrFam>(dpb_ctx*, const EqPairPlan&, uint32_t, const Fr&);
template void eq_pairs_launch_round<GlFam>(dpb_ctx*, const EqPairPlan&, uint32_t, const Gl2&);
template void eq_pairs_launch_finals<FrFam>(dpb_ctx*, const EqPairPlan&, uint32_t, const Fr&, Fr*);
template void eq_pairs_launch_finals<GlFam>(dpb_ctx*, const EqPairPlan&, uint32_t, const Gl2&, Gl2*);

}  // namespace dpb

// Host side of the claim-batching rounds (eq_pairs.cuh): the plan a sumcheck keeps, and the launches.
#pragma once
#include "common.cuh"

namespace dpb {

struct EqPairPlan {
    struct Term {
        uint32_t f, eq;  // table ids
    };
    std::vector<Term> terms;  // empty: the sumcheck is not of this form
    // per round: pairs a thread takes of a tile, tiles in all
    std::vector<uint32_t> per_thread, tiles;
    const void* d_terms = nullptr;         // EqPairTerm[n_terms]
    const void* d_points = nullptr;        // the eq tables' points, end to end
    const uint32_t* d_prefix = nullptr;    // [rounds][n_terms + 1]
    void* d_s = nullptr;                   // [2][n_terms]
};

// Publishes the three samples of a degree-2 product round (the slots of fused_v2.cuh) as every round kernel does.
template <class F>
void eq_pairs_launch_round(dpb_ctx* ctx, const EqPairPlan& p, uint32_t round, const typename F::E& r);
// Every table's value at the point into out[table id]; r is the challenge that ended `round`, the last one.
template <class F>
void eq_pairs_launch_finals(dpb_ctx* ctx, const EqPairPlan& p, uint32_t round, const typename F::E& r, typename F::E* out);

}  // namespace dpb

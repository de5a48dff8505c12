// The sumcheck of one logup-GKR layer, from the layer's own formula (logup_layer.cuh has the kernels, logup_layer.cu the
// state machine).  Used by the batched logup prover in place of a general sumcheck over the layer's term list.
#pragma once
#include "common.cuh"

namespace dpb {

struct LogupLayerSc;

// Starts the sumcheck of  sum_j alpha_j eq (n_lo d_hi + n_hi d_lo + lambda d_lo d_hi)  over `num_vars` variables: the
// instances' tables in order (LogupHintInst), then the eq table.  partial: the instances are spread over the ranks of the
// context's communicator and every round's sums are added over the ranks.  *out = nullptr when the layer is not of the
// form the kernels take (the caller then runs the general sumcheck).
int logup_layer_begin(dpb_ctx* ctx, uint32_t num_vars, dpb_mle* const* mles, uint32_t k, const LogupHintInst* inst, uint32_t n_inst,
                      const void* lambda, bool partial, LogupLayerSc** out);
// The round message: 4 challenge elements, the polynomial at 0..3.
int logup_layer_round(LogupLayerSc* sc, const void* prev_challenge, void* out_evals);
// Every table's value at the point, k challenge elements.
int logup_layer_finish(LogupLayerSc* sc, const void* last_challenge, void* out);
void logup_layer_free(LogupLayerSc* sc);

}  // namespace dpb

// Host side of the resident last-rounds kernel of a logup layer (logup_tail.cuh).
#pragma once
#include "common.cuh"

namespace dpb {

constexpr uint32_t kLogupTailBlocks = 8;     // the cluster (the portable size)
constexpr uint32_t kLogupTailMaxInst = 128;

struct LogupTailInst {
    uint16_t kind;   // kLogup*
    uint16_t first;  // index of the first original table
    uint16_t ncol;
    uint16_t tab0;   // first of the instance's tables in shared memory
};

// Shape of the kernel for one sumcheck.
struct LogupTailPlan {
    bool ok = false;
    uint32_t n_inst = 0, n_tabs = 0, eq_table = 0;
    uint32_t start = 0;      // first round it can run
    uint32_t alone = 0;      // pairs from which a cluster goes on with one block
    const void* d_inst = nullptr;    // LogupTailInst[n_inst]
    const void* d_consts = nullptr;  // alpha, sep, constant per instance
};

// Blocks and dynamic shared memory of a launch whose first round has `pairs` pairs; 0 blocks: does not fit.
uint32_t logup_tail_blocks(const LogupTailPlan& p, uint64_t pairs, size_t elem, size_t* smem);

// tabs: this round's descriptors (RoundTab) of the original tables; eq: the eq table's original entries.
template <class F>
int logup_tail_launch(dpb_ctx* ctx, const LogupTailPlan& p, const void* tabs, const void* eq, uint32_t eq_stride_log2,
                      const typename F::E& lambda, const typename F::E& r, uint32_t first_round, uint32_t n_rounds);

}  // namespace dpb

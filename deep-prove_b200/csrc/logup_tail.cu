// Launch of the resident last-rounds kernel of a logup layer (logup_tail.cuh).
#include "logup_tail.cuh"

namespace dpb {

constexpr size_t kLogupTailSmem = 200 * 1024;

uint32_t logup_tail_blocks(const LogupTailPlan& p, uint64_t pairs, size_t elem, size_t* smem) {
    const uint32_t blocks = pairs > p.alone ? kLogupTailBlocks : 1;
    if (pairs % blocks) return 0;
    const uint64_t nb = pairs / blocks;
    if (nb < 1 || nb > 256 || nb * p.n_inst > 2 * (uint64_t)kTailThreads) return 0;
    const size_t bytes = (3 * (size_t)p.n_inst + logup_tail_weights(nb, blocks, p.alone)) * elem + logup_tail_set_entries(nb, blocks, p.alone, 0) * p.n_tabs * elem +
                         logup_tail_set_entries(nb, blocks, p.alone, 1) * p.n_tabs * elem + p.n_inst * sizeof(LogupTailInst);
    if (bytes > kLogupTailSmem) return 0;
    *smem = bytes;
    return blocks;
}

template <class F>
int logup_tail_launch(dpb_ctx* ctx, const LogupTailPlan& p, const void* tabs, const void* eq, uint32_t eq_stride_log2,
                      const typename F::E& lambda, const typename F::E& r, uint32_t first_round, uint32_t n_rounds) {
    typedef typename F::E E;
    size_t smem = 0;
    const uint32_t blocks = logup_tail_blocks(p, 1ull << (n_rounds - first_round - 1), sizeof(E), &smem);
    if (!blocks) return fail(DPB_EINVAL, "the last rounds of this logup layer do not fit");
    DPB_CUDA(cudaFuncSetAttribute(sc_tail_logup<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLogupTailSmem));
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof cfg);
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kTailThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->tail_stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = blocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    DPB_CUDA(cudaLaunchKernelEx(&cfg, sc_tail_logup<F>, (const RoundTab*)tabs, (const LogupTailInst*)p.d_inst, (const E*)p.d_consts,
                                p.n_inst, p.n_tabs, lambda, (const E*)eq, eq_stride_log2, r, first_round, n_rounds, p.alone,
                                (TailBox*)ctx->tail_box_dev, ctx->tail_wait_ns));
    return DPB_OK;
}

template int logup_tail_launch<FrFam>(dpb_ctx*, const LogupTailPlan&, const void*, const void*, uint32_t, const Fr&, const Fr&,
                                      uint32_t, uint32_t);
template int logup_tail_launch<GlFam>(dpb_ctx*, const LogupTailPlan&, const void*, const void*, uint32_t, const Gl2&, const Gl2&,
                                      uint32_t, uint32_t);

}  // namespace dpb

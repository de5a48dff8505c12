// The sumcheck of one logup-GKR layer: its state machine (begin / round / finish) over the kernels of logup_layer.cuh.
#include "logup_layer.hpp"

#include <algorithm>

#include "comm.cuh"
#include "fused_v2.cuh"
#include "logup_layer.cuh"
#include "tail_host.hpp"

namespace dpb {

constexpr size_t kLogupTailSmem = 200 * 1024;
constexpr size_t kLogupRoundSmem = 64 * 1024;

struct LogupLayerSc {
    dpb_ctx* ctx = nullptr;
    bool gl = false, partial = false, finished = false;
    uint32_t n = 0, k = 0, n_inst = 0, round = 0;
    uint32_t eq_table = 0;
    std::vector<dpb_mle*> mles;          // borrowed
    std::vector<LogupHintInst> inst;
    void* slab = nullptr;                // slots' buffers, instances, constants, keys, rows, final values
    const void *d_inst = nullptr, *d_consts = nullptr, *d_alphas = nullptr;
    void *d_rows = nullptr, *d_final = nullptr;
    bool int_rows = false;               // BN254, every input column holds integers
    std::vector<LgRows> h_rows;
    std::vector<uint8_t> q, inv_q, inv_zp;  // the eq table's point; 1 / q_i; 1 / prod_{k < j} (1 - q_k), j = 0..n
    alignas(16) uint8_t S[32] = {0};     // prod eq(q_k, r_k) over the bound variables
    alignas(16) uint8_t lambda[32] = {0};
    alignas(16) uint8_t h[4 * 32] = {0};  // the previous round's H(0), h1, h2 and its q
    std::vector<uint8_t> point;          // the challenges so far
    // the resident kernel
    uint32_t tail_start = ~0u, tail_first = 0, tail_tabs = 0, alone = 0;
    bool extra = false, tail_active = false;
};

template <class F>
static typename F::E get(const void* p, size_t i) {
    typename F::E e;
    memcpy(&e, (const char*)p + i * sizeof(e), sizeof(e));
    return e;
}

// blocks of a launch whose first round has `pairs` pairs and its dynamic shared memory; 0: does not fit
template <class F>
static uint32_t tail_blocks(const LogupLayerSc* sc, uint64_t pairs, uint32_t alone, size_t* smem) {
    typedef typename F::E E;
    const uint32_t blocks = pairs > alone ? kLogupTailBlocks : 1;
    const uint64_t nb = pairs / blocks;
    if (pairs % blocks || nb < 1 || nb > 256 || nb * sc->n_inst > 2 * (uint64_t)kTailThreads) return 0;
    const size_t bytes = sc->n_inst * (sizeof(LgConst<F>) + sizeof(LgInst)) + logup_tail_weights(nb, blocks, alone) * sizeof(E) +
                         (logup_tail_set_entries(nb, blocks, alone, 0) + logup_tail_set_entries(nb, blocks, alone, 1)) * sc->tail_tabs * sizeof(E);
    if (bytes > kLogupTailSmem) return 0;
    *smem = bytes;
    return blocks;
}

// The most pairs the resident kernel takes, with as few of them as need be left to one block.
template <class F>
static uint64_t plan_tail(LogupLayerSc* sc) {
    uint64_t best = 0;
    for (uint32_t alone = sc->gl ? kTailAloneGl : kTailAloneFr; alone >= 4; alone /= 2) {
        size_t smem;
        if (!tail_blocks<F>(sc, alone, alone, &smem)) continue;  // what is left for one block has to fit as well
        for (uint64_t pairs = 256 * kLogupTailBlocks; pairs > best; pairs /= 2)
            if (tail_blocks<F>(sc, pairs, alone, &smem)) {
                best = pairs;
                sc->alone = alone;
            }
    }
    return best;
}

template <class F>
static int begin_impl(LogupLayerSc* sc, bool* usable) {
    typedef typename F::E E;
    dpb_ctx* ctx = sc->ctx;
    const E one = F::one();
    const dpb_mle* eq = sc->mles[sc->eq_table];
    if (eq->eq_point.size() != (size_t)sc->n * sizeof(E) || eq->len != (1ull << sc->n) || eq->dtype != F::kChalDtype) return DPB_OK;
    sc->q = eq->eq_point;
    for (uint32_t i = 0; i < sc->n; i++) {  // their inverses are needed
        const E q = get<F>(sc->q.data(), i);
        if (F::is_zero(q) || F::is_zero(F::sub(one, q))) return DPB_OK;
    }
    memcpy(sc->S, &one, sizeof(E));
    const E lam = get<F>(sc->lambda, 0);
    if (F::is_zero(lam)) return DPB_OK;  // the layer's degree would be lower
    // instances
    std::vector<LgInst> di(sc->n_inst);
    std::vector<LgConst<F>> dc(sc->n_inst);
    std::vector<typename AlphaSum<F>::Key> da(sc->n_inst);
    size_t slots = 0;
    bool input_layer = false;
    sc->int_rows = sizeof(E) == 32;
    for (uint32_t i = 0; i < sc->n_inst; i++) {
        const LogupHintInst& h = sc->inst[i];
        LgInst& d = di[i];
        memset(&d, 0, sizeof d);
        memset((void*)&dc[i], 0, sizeof(LgConst<F>));
        dc[i].alpha = get<F>(h.alpha, 0);
        if (F::is_zero(dc[i].alpha)) return DPB_OK;
        dc[i].sep = get<F>(h.sep, 0);
        dc[i].c = get<F>(h.constant, 0);
        da[i] = F::fold_key(dc[i].alpha);
        d.kind = (uint16_t)h.kind;
        d.ncol = (uint16_t)h.ncol;
        d.first = (uint16_t)h.first;
        const uint32_t n_orig = h.kind == kLogupInner ? 4 : 2 * h.ncol + (h.kind == kLogupTable ? 2 : 0);
        for (uint32_t j = 0; j < n_orig; j++) {
            const dpb_mle* m = sc->mles[h.first + j];
            if (m->len != (1ull << sc->n) || m->ctx != ctx || is_gl(m->dtype) != sc->gl) return DPB_OK;
            d.orig[j] = m->ptr;
            d.dtype[j] = (int8_t)m->dtype;
            const bool column = h.kind != kLogupInner && j >= (h.kind == kLogupTable ? 2u : 0u);
            if (column && !is_int_dtype(m->dtype)) sc->int_rows = false;
        }
        if (h.kind != kLogupInner) input_layer = true;
        slots += lg_slots(d);
    }
    sc->int_rows = sc->int_rows && input_layer;
    // the resident kernel: from the originals it binds the second columns as well; started later it leaves the columns'
    // values to one evaluation at the end
    for (int attempt = 0; attempt < 2; attempt++) {
        sc->extra = attempt == 0 && input_layer;
        uint32_t tabs = 0;
        for (uint32_t i = 0; i < sc->n_inst; i++) {
            di[i].tab0 = (uint16_t)tabs;
            tabs += lg_slots(di[i]) + (sc->extra && di[i].kind != kLogupInner && di[i].ncol == 2 ? 2 : 0);
        }
        sc->tail_tabs = tabs;
        sc->tail_start = ~0u;
        if ((size_t)sc->k * (sizeof(E) / 8) > (size_t)kTailMaxTables * 4) break;  // the mailbox
        const uint64_t most = plan_tail<F>(sc);
        if (most) {
            uint32_t i = 0;
            while ((1ull << (sc->n - i - 1)) > most) i++;
            sc->tail_start = i;
        }
        if (!sc->extra || sc->tail_start <= 1) break;
    }
    // one block of device memory: [slots' buffers | final values | rows | instances, constants, keys]
    const size_t per_slot = sc->n >= 2 ? (1ull << (sc->n - 1)) + (1ull << (sc->n - 2)) : 1;
    size_t off = slots * per_slot * sizeof(E);
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off = (off + bytes + 31) & ~(size_t)31;
        return o;
    };
    const size_t o_final = take(4 * (size_t)sc->n_inst * sizeof(E)), o_rows = take(sc->int_rows ? sc->n_inst * sizeof(LgRows) : 0),
                 o_inst = take(di.size() * sizeof(LgInst)), o_consts = take(dc.size() * sizeof(LgConst<F>)),
                 o_alphas = take(da.size() * sizeof(da[0])), end = off;
    if (ctx->slab_cache && !ctx->slab_cache_busy && end <= ctx->slab_cache_bytes) {
        sc->slab = ctx->slab_cache;  // as dpb_sumcheck_begin does
        ctx->slab_cache_busy = true;
    } else {
        DPB_TRY(device_alloc(ctx, end, &sc->slab));
        if (!ctx->slab_cache_busy && end <= kSlabCacheMax) {
            device_free(ctx, ctx->slab_cache);
            ctx->slab_cache = sc->slab;
            ctx->slab_cache_bytes = end;
            ctx->slab_cache_busy = true;
        }
    }
    char* base = (char*)sc->slab;
    E* buf = (E*)base;
    for (auto& d : di)
        for (uint32_t s = 0; s < lg_slots(d); s++) {
            d.buf[s][0] = buf;
            d.buf[s][1] = sc->n >= 2 ? buf + (1ull << (sc->n - 1)) : buf;
            buf += per_slot;
        }
    sc->d_final = base + o_final;
    sc->d_rows = base + o_rows;
    sc->d_inst = base + o_inst;
    sc->d_consts = base + o_consts;
    sc->d_alphas = base + o_alphas;
    std::vector<uint8_t> blob(end - o_inst, 0);
    memcpy(blob.data(), di.data(), di.size() * sizeof(LgInst));
    memcpy(blob.data() + (o_consts - o_inst), (const void*)dc.data(), dc.size() * sizeof(LgConst<F>));
    memcpy(blob.data() + (o_alphas - o_inst), (const void*)da.data(), da.size() * sizeof(da[0]));
    DPB_TRY(upload_small(ctx, base + o_inst, blob.data(), blob.size()));
    *usable = true;
    return DPB_OK;
}

// 1 / q_i and 1 / prod_{k < j} (1 - q_k), made while the first kernel works: one inversion for all (Montgomery's trick)
template <class F>
static void make_inverses(LogupLayerSc* sc) {
    typedef typename F::E E;
    if (!sc->inv_q.empty()) return;
    const E one = F::one();
    std::vector<E> vals;
    for (uint32_t i = 0; i < sc->n; i++) vals.push_back(get<F>(sc->q.data(), i));
    E zp = one;
    vals.push_back(zp);
    for (uint32_t i = 0; i < sc->n; i++) {
        zp = F::mul(zp, F::sub(one, get<F>(sc->q.data(), i)));
        vals.push_back(zp);
    }
    std::vector<E> pre(vals.size() + 1, one), inv(vals.size());
    for (size_t a = 0; a < vals.size(); a++) pre[a + 1] = F::mul(pre[a], vals[a]);
    E all = F::inv(pre[vals.size()]);
    for (size_t a = vals.size(); a-- > 0;) {
        inv[a] = F::mul(all, pre[a]);
        all = F::mul(all, vals[a]);
    }
    sc->inv_q.assign((const uint8_t*)inv.data(), (const uint8_t*)(inv.data() + sc->n));
    sc->inv_zp.assign((const uint8_t*)(inv.data() + sc->n), (const uint8_t*)(inv.data() + inv.size()));
}

// Rows for the integer columns of round 0 or 1 (LgRows).
static int upload_rows(LogupLayerSc* sc, int mode, const Fr& r) {
    std::vector<LgRows> rows(sc->n_inst);
    const Fr two31 = fr_from_u64(0x80000000ull);
    for (uint32_t i = 0; i < sc->n_inst; i++) {
        const LogupHintInst& h = sc->inst[i];
        LgRows& w = rows[i];
        memset(&w, 0, sizeof w);
        if (h.kind == kLogupInner) continue;
        Fr s = fr_zero(), c;
        if (h.ncol == 2) memcpy(&s, h.sep, sizeof s);
        memcpy(&c, h.constant, sizeof c);
        const Fr a = mode == kLgBind ? fr_sub(fr_one(), r) : fr_one(), b = mode == kLgBind ? r : fr_zero();
        fr_fixed_row(a, 8, w.row[0]);
        fr_fixed_row(b, 8, w.row[1]);
        fr_fixed_row(fr_mul(s, a), 8, w.row[2]);
        fr_fixed_row(fr_mul(s, b), 8, w.row[3]);
        c = fr_sub(c, fr_mul(two31, fr_add(fr_one(), s)));
        for (int j = 0; j < 4; j++) {
            w.c[2 * j] = (uint32_t)c.l[j];
            w.c[2 * j + 1] = (uint32_t)(c.l[j] >> 32);
        }
    }
    return upload_small(sc->ctx, sc->d_rows, rows.data(), rows.size() * sizeof(LgRows));
}
static int upload_rows(LogupLayerSc*, int, const Gl2&) { return DPB_OK; }

template <class F, int MODE, int KIND>
static int launch_round(LogupLayerSc* sc, uint32_t round, const typename F::E& r) {
    typedef typename F::E E;
    typedef typename AlphaSum<F>::Key Key;
    dpb_ctx* ctx = sc->ctx;
    const uint64_t n_pairs = 1ull << (sc->n - round - 1);
    // blocks of 128 threads, of 64 when the pairs do not fill the GPU even then; and when they still do not, the
    // instances are cut into slices that run as blocks of their own
    const uint64_t per_sm = sizeof(E) == 16 ? 4 : MODE == kLgSlots ? 3 : 2;
    const uint32_t threads = n_pairs < (uint64_t)ctx->sm_count * 128 ? 64 : 128;
    const uint64_t room = (uint64_t)ctx->sm_count * per_sm * (128 / threads);
    uint64_t blocks_x = std::min<uint64_t>((n_pairs + threads - 1) / threads, std::min<uint64_t>(room, ctx->max_blocks));
    uint32_t per_slice = sc->n_inst, slices = 1;
    const size_t per_inst = sizeof(Key) + sizeof(LgInst);
    const uint32_t most = (uint32_t)(kLogupRoundSmem / per_inst);  // instances a block keeps on chip
    if (blocks_x < room) per_slice = (sc->n_inst + (uint32_t)(room / blocks_x) - 1) / (uint32_t)(room / blocks_x);
    per_slice = std::max(1u, std::min(per_slice, most));
    slices = (sc->n_inst + per_slice - 1) / per_slice;
    if (blocks_x * slices > ctx->max_blocks) blocks_x = std::max<uint64_t>(1, ctx->max_blocks / slices);
    if (MODE != kLgSlots && sc->int_rows) DPB_TRY(upload_rows(sc, MODE, r));
    DPB_CUDA(cudaFuncSetAttribute(logup_layer_round<F, MODE, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLogupRoundSmem));
    logup_layer_round<F, MODE, KIND><<<(uint32_t)(blocks_x * slices), threads, per_slice * per_inst, ctx->stream>>>(
        (const LgInst*)sc->d_inst, (const LgConst<F>*)sc->d_consts, (const Key*)sc->d_alphas,
        MODE != kLgSlots && sc->int_rows ? (const LgRows*)sc->d_rows : nullptr, sc->n_inst, F::fold_key(r),
        F::fold_key(get<F>(sc->lambda, 0)), (const E*)sc->mles[sc->eq_table]->ptr, round + 1, n_pairs, round & 1, (uint32_t)blocks_x,
        per_slice, reduce_scratch<F>(ctx), (E*)ctx->round_out);
    DPB_CUDA(cudaGetLastError());
    ctx->sumcheck_launches++;
    return DPB_OK;
}

template <class F, int KIND>
static int launch_round(LogupLayerSc* sc, uint32_t round, const typename F::E& r) {
    return round == 0   ? launch_round<F, kLgOriginal, KIND>(sc, round, r)
           : round == 1 ? launch_round<F, kLgBind, KIND>(sc, round, r)
                        : launch_round<F, kLgSlots, KIND == kLogupTable ? kLogupInner : KIND>(sc, round, r);
}

// (Re)starts the resident kernel at its first round; r is the challenge that ended the round before.
template <class F, int MODE>
static int launch_tail(LogupLayerSc* sc, const typename F::E& r) {
    typedef typename F::E E;
    dpb_ctx* ctx = sc->ctx;
    size_t smem = 0;
    const uint32_t blocks = tail_blocks<F>(sc, 1ull << (sc->n - sc->tail_first - 1), sc->alone, &smem);
    if (!blocks) return fail(DPB_EINVAL, "the last rounds of this logup layer do not fit");
    DPB_CUDA(cudaFuncSetAttribute(sc_tail_logup<F, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLogupTailSmem));
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
    DPB_CUDA(cudaLaunchKernelEx(&cfg, sc_tail_logup<F, MODE>, (const LgInst*)sc->d_inst, (const LgConst<F>*)sc->d_consts, sc->n_inst,
                                sc->tail_tabs, sc->extra ? 1u : 0u, get<F>(sc->lambda, 0), (const E*)sc->mles[sc->eq_table]->ptr,
                                sc->tail_first + 1, r, sc->tail_first & 1, sc->tail_first, sc->n, sc->alone,
                                (TailBox*)ctx->tail_box_dev, ctx->tail_wait_ns));
    return DPB_OK;
}
template <class F>
static int start_tail(LogupLayerSc* sc, const typename F::E& r) {
    dpb_ctx* ctx = sc->ctx;
    TailBox* box = (TailBox*)ctx->tail_box_host;
    memset(box, 0, sizeof(TailBox));  // sequence numbers of an earlier run must not be mistaken for this one's
    std::atomic_thread_fence(std::memory_order_seq_cst);
    // the kernel runs on its own stream, after everything this context has queued so far
    DPB_CUDA(cudaEventRecord(ctx->tail_ev[0], ctx->stream));
    DPB_CUDA(cudaStreamWaitEvent(ctx->tail_stream, ctx->tail_ev[0], 0));
    DPB_TRY((sc->tail_first == 0   ? launch_tail<F, kLgOriginal>(sc, r)
             : sc->tail_first == 1 ? launch_tail<F, kLgBind>(sc, r)
                                   : launch_tail<F, kLgSlots>(sc, r)));
    // first sign of life, as soon as the launch call is back (the kernel waits 50 ms for it)
    ((volatile TailChunk*)&box->hello)->seq = 1;
    DPB_CUDA(cudaEventRecord(ctx->tail_ev[1], ctx->tail_stream));
    ctx->sumcheck_launches++;
    return DPB_OK;
}

// the resident kernel's samples of round j: at 0, 1 (round 0 only) and infinity
template <class F>
static int take_samples(LogupLayerSc* sc, uint32_t j, typename F::E* raw) {
    TailBox* box = (TailBox*)sc->ctx->tail_box_host;
    uint32_t x = 0;
    return tail_wait_host(sc->ctx, box, [&] {
        while (x <= 2) {
            if (j > 0 && x == 1) {
                x++;
                continue;
            }
            if (!tail_take<typename F::E>(box->evals, x, j + 1, &raw[x])) return false;
            x++;
        }
        return true;
    });
}

// The kernel gave up waiting (the host was held up): start it again and play the rounds before `upto` with the
// challenges they had, and the challenge after them.
template <class F>
static int replay(LogupLayerSc* sc, uint32_t upto) {
    typedef typename F::E E;
    dpb_ctx* ctx = sc->ctx;
    DPB_CUDA(cudaStreamSynchronize(ctx->tail_stream));  // it has returned; make that certain
    const E r0 = sc->tail_first ? get<F>(sc->point.data(), sc->tail_first - 1) : F::zero();
    DPB_TRY(start_tail<F>(sc, r0));
    for (uint32_t j = sc->tail_first; j < upto; j++) {
        E raw[3];
        const int rc = take_samples<F>(sc, j, raw);
        if (rc != DPB_OK) return rc < 0 ? rc : fail(DPB_ETIMEOUT, "the resident round kernel gave up waiting for a challenge");
        const E ch = get<F>(sc->point.data(), j);
        tail_post<E>(ctx, &ch, j + 1);
    }
    return DPB_OK;
}

static void leave_tail(LogupLayerSc* sc) {
    sc->tail_active = false;
    sc->ctx->tail_owner = nullptr;
}

static void log_profile(LogupLayerSc* sc, uint32_t round, size_t elem) {
    dpb_ctx* ctx = sc->ctx;
    float ms = 0.f;
    cudaEventSynchronize(ctx->prof_ev[1]);
    cudaEventElapsedTime(&ms, ctx->prof_ev[0], ctx->prof_ev[1]);
    // minimum traffic of this round: every table read once, bound slots written once, the eq entries of the pairs
    const uint64_t v = sc->n - round;
    uint64_t bytes = elem << (v - 1);
    for (const auto& h : sc->inst) {
        const uint32_t n_orig = h.kind == kLogupInner ? 4 : 2 * h.ncol + (h.kind == kLogupTable ? 2 : 0);
        const uint64_t n_slots = h.kind == kLogupLookup ? 2 : 4;
        if (round < 2)
            for (uint32_t j = 0; j < n_orig; j++) bytes += dtype_size(sc->mles[h.first + j]->dtype) << sc->n;
        else
            bytes += n_slots * (elem << (v + 1));
        if (round > 0) bytes += n_slots * (elem << v);
    }
    for (auto& e : ctx->prof_log)
        if (e.round == round && e.alg_bytes_per_launch == bytes && strcmp(e.kernel, "logup_layer_round") == 0) {
            e.launches++;
            e.total_ms += ms;
            return;
        }
    dpb_profile_entry e;
    memset(&e, 0, sizeof e);
    strncpy(e.kernel, "logup_layer_round", sizeof(e.kernel) - 1);
    e.round = round;
    e.launches = 1;
    e.total_ms = ms;
    e.alg_bytes_per_launch = bytes;
    ctx->prof_log.push_back(e);
}

template <class F>
static int round_impl(LogupLayerSc* sc, const void* prev_challenge, void* out_evals) {
    typedef typename F::E E;
    dpb_ctx* ctx = sc->ctx;
    const uint32_t i = sc->round;
    const E one = F::one();
    E r = F::zero(), S = get<F>(sc->S, 0);
    E* h = (E*)sc->h;
    if (i > 0) {
        r = get<F>(prev_challenge, 0);
        sc->point.insert(sc->point.end(), (const uint8_t*)&r, (const uint8_t*)&r + sizeof(E));
        const E q = get<F>(sc->q.data(), i - 1);
        S = F::mul(S, F::add(F::mul(q, r), F::mul(F::sub(one, q), F::sub(one, r))));
        memcpy(sc->S, &S, sizeof(E));
    }
    // with `extra` the kernel binds the second columns too, from the originals: rounds 0 and 1 only
    const bool can_start = i >= sc->tail_start && !(sc->extra && i > 1);
    bool tail = sc->tail_active || (ctx->tail_enabled && !sc->partial && !ctx->profile && can_start && ctx->tail_owner == nullptr);
    const bool first = tail && !sc->tail_active;
    // the samples go to the host's chunk area, this rank's slot of the shared segment, or a collective
    const size_t msg_bytes = 3 * sizeof(E);
    const bool shared_xch = sc->partial && ctx->xch_host != nullptr;
    auto launch = [&]() -> int {
        if (shared_xch) {
            ctx->xseq++;
            ctx->chunk_out_dev = (char*)ctx->xch_dev + xch_slot_offset(ctx->rank, ctx->xseq);
            ctx->round_out = nullptr;
            ctx->done_value = ctx->xseq;
        } else {
            ctx->round_out = sc->partial ? (void*)((char*)ctx->gather_dev + (size_t)ctx->rank * msg_bytes) : ctx->result_dev;
            ctx->done_seq++;
            ctx->done_value = ctx->done_seq;
            ctx->chunk_out_dev = sc->partial ? nullptr : ctx->result_dev;
        }
        if (ctx->profile) DPB_CUDA(cudaEventRecord(ctx->prof_ev[0], ctx->stream));
        const int kind = sc->inst[0].kind;
        DPB_TRY((kind == kLogupInner    ? launch_round<F, kLogupInner>(sc, i, r)
                 : kind == kLogupLookup ? launch_round<F, kLogupLookup>(sc, i, r)
                                        : launch_round<F, kLogupTable>(sc, i, r)));
        if (ctx->profile) DPB_CUDA(cudaEventRecord(ctx->prof_ev[1], ctx->stream));
        return DPB_OK;
    };
    if (first) {
        sc->tail_first = i;
        DPB_TRY(start_tail<F>(sc, r));
        sc->tail_active = true;
        ctx->tail_owner = sc;
    } else if (tail) {
        tail_post<E>(ctx, &r, i);
    } else {
        DPB_TRY(launch());
    }
    // while the kernel works: the claim s(0) + s(1) (the previous round's polynomial at r) and the scalars
    make_inverses<F>(sc);
    E claim = F::zero();
    if (i > 0) {
        const E l = F::add(F::sub(one, h[3]), F::mul(F::sub(F::add(h[3], h[3]), one), r));
        claim = F::mul(l, F::add(h[0], F::mul(r, F::add(h[1], F::mul(r, h[2])))));
    }
    const E q = get<F>(sc->q.data(), i), q0 = F::sub(one, q), inv_q = get<F>(sc->inv_q.data(), i);
    const E kappa = F::mul(S, get<F>(sc->inv_zp.data(), i + 1));
    E raw[3];
    if (tail) {
        int rc = take_samples<F>(sc, i, raw);
        if (rc == kTailNoHost) {
            // launches block this host thread: nothing has run; this context runs one launch per round from now on
            cudaStreamSynchronize(ctx->tail_stream);
            ctx->tail_enabled = false;
            leave_tail(sc);
            tail = false;
            DPB_TRY(launch());
        } else {
            if (rc == kTailGaveUp && !first) {
                DPB_TRY(replay<F>(sc, i));
                rc = take_samples<F>(sc, i, raw);
            }
            if (rc == kTailGaveUp) return fail(DPB_ETIMEOUT, "the resident round kernel gave up waiting for a challenge");
            if (rc != DPB_OK) return rc;
        }
    }
    if (!tail) {
        if (sc->partial) {
            if (shared_xch) DPB_TRY(xch_collect(ctx, ctx->xseq, msg_bytes, ctx->gather_host, 60.0));
            else DPB_TRY(allgather_to_host(ctx, ctx->round_out, msg_bytes));
            for (uint32_t x = 0; x < 3; x++) {
                raw[x] = get<F>(ctx->gather_host, x);
                for (int g = 1; g < ctx->nranks; g++) raw[x] = F::add(raw[x], get<F>(ctx->gather_host, (size_t)g * 3 + x));
            }
        } else {
            DPB_TRY(wait_round_chunks(ctx, msg_bytes, raw));
        }
        if (ctx->profile) log_profile(sc, i, sizeof(E));
    }
    const E H0 = F::mul(kappa, raw[0]), Hi = F::mul(kappa, raw[2]);
    // s(0) + s(1) = (1 - q) H(0) + q H(1)
    const E H1 = i == 0 ? F::mul(kappa, raw[1]) : F::mul(F::sub(claim, F::mul(q0, H0)), inv_q);
    const E h1 = F::sub(F::sub(H1, H0), Hi);
    // H(x) = H0 + h1 x + Hi x^2 by differences; s(x) = ((1 - q) + (2 q - 1) x) H(x)
    const E slope = F::sub(q, q0), step2 = F::add(Hi, Hi);
    E H = H0, step = F::add(h1, Hi), l = q0;
    for (uint32_t x = 0; x <= 3; x++) {
        const E v = F::mul(l, H);
        memcpy((char*)out_evals + x * sizeof(E), &v, sizeof(E));
        H = F::add(H, step);
        step = F::add(step, step2);
        l = F::add(l, slope);
    }
    h[0] = H0;
    h[1] = h1;
    h[2] = Hi;
    h[3] = q;
    sc->round++;
    return DPB_OK;
}

template <class F>
static int finish_impl(LogupLayerSc* sc, const void* last_challenge, void* out_raw) {
    typedef typename F::E E;
    dpb_ctx* ctx = sc->ctx;
    const E r = get<F>(last_challenge, 0), one = F::one(), lam = get<F>(sc->lambda, 0);
    sc->point.insert(sc->point.end(), (const uint8_t*)&r, (const uint8_t*)&r + sizeof(E));
    std::vector<E> out(sc->k);
    bool columns = false;  // the input columns' values are still missing
    if (sc->tail_active) {
        TailBox* box = (TailBox*)ctx->tail_box_host;
        tail_post<E>(ctx, &r, sc->n);
        std::vector<uint32_t> want;  // the tables the kernel reports
        for (const auto& h : sc->inst) {
            const uint32_t n = h.kind == kLogupInner ? 4 : (h.kind == kLogupTable ? 2 : 0) + (sc->extra ? 2 * h.ncol : 0);
            for (uint32_t j = 0; j < n; j++) want.push_back(h.first + j);
            if (h.kind != kLogupInner && !sc->extra) columns = true;
        }
        // the kernel ends with these values; when it has none to report its end is what is waited for
        size_t j = 0;
        auto take = [&] {
            while (j < want.size()) {
                if (!tail_take<E>(box->finals, want[j], sc->n + 1, &out[want[j]])) return false;
                j++;
            }
            return true;
        };
        int rc = tail_wait_host(ctx, box, take);
        if (rc == kTailGaveUp) {
            rc = replay<F>(sc, sc->n);
            if (rc == DPB_OK) rc = tail_wait_host(ctx, box, take);
            if (rc == kTailGaveUp) rc = fail(DPB_ETIMEOUT, "the resident round kernel gave up waiting for a challenge");
        }
        // later work of this context (frees, the next sumcheck) is ordered after the kernel's end
        cudaStreamWaitEvent(ctx->stream, ctx->tail_ev[1], 0);
        leave_tail(sc);
        if (rc != DPB_OK) return rc;
    } else {
        std::vector<E> slots(4 * (size_t)sc->n_inst);
        logup_layer_finals<F><<<(sc->n_inst + 127) / 128, 128, 0, ctx->stream>>>(
            (const LgInst*)sc->d_inst, (const LgConst<F>*)sc->d_consts, sc->n_inst, F::fold_key(r), F::fold_key(lam), sc->n - 1, (E*)sc->d_final);
        DPB_CUDA(cudaGetLastError());
        ctx->sumcheck_launches++;
        DPB_CUDA(cudaMemcpyAsync(slots.data(), sc->d_final, slots.size() * sizeof(E), cudaMemcpyDeviceToHost, ctx->stream));
        DPB_CUDA(cudaStreamSynchronize(ctx->stream));
        for (uint32_t i = 0; i < sc->n_inst; i++) {
            const auto& h = sc->inst[i];
            const E *v = &slots[4 * (size_t)i], c = v[0], d = v[1];
            if (h.kind != kLogupLookup) {
                out[h.first] = v[3];
                out[h.first + 1] = F::sub(v[2], F::mul(lam, d));
            }
            if (h.kind == kLogupInner) {
                out[h.first + 2] = c;
                out[h.first + 3] = d;
            } else {
                columns = true;
            }
        }
    }
    if (columns) {
        std::vector<dpb_mle*> tabs;
        std::vector<uint32_t> place;
        for (const auto& h : sc->inst) {
            if (h.kind == kLogupInner) continue;
            const uint32_t col = h.first + (h.kind == kLogupTable ? 2 : 0);
            for (uint32_t j = 0; j < 2 * h.ncol; j++) {
                tabs.push_back(sc->mles[col + j]);
                place.push_back(col + j);
            }
        }
        std::vector<E> vals(tabs.size());
        DPB_TRY(dpb_mle_evaluate_many(ctx, tabs.data(), (uint32_t)tabs.size(), sc->point.data(), sc->n, vals.data()));
        for (size_t j = 0; j < vals.size(); j++) out[place[j]] = vals[j];
    }
    // the eq table at the point: the product of eq(q_k, r_k)
    const E q = get<F>(sc->q.data(), sc->n - 1);
    out[sc->eq_table] = F::mul(get<F>(sc->S, 0), F::add(F::mul(q, r), F::mul(F::sub(one, q), F::sub(one, r))));
    memcpy(out_raw, out.data(), out.size() * sizeof(E));
    sc->finished = true;
    return DPB_OK;
}

int logup_layer_begin(dpb_ctx* ctx, uint32_t num_vars, dpb_mle* const* mles, uint32_t k, const LogupHintInst* inst, uint32_t n_inst,
                      const void* lambda, bool partial, LogupLayerSc** out) {
    *out = nullptr;
    if (!ctx || !mles || !inst || !lambda) return fail(DPB_EINVAL, "null argument");
    if (num_vars < 1 || num_vars > 40 || n_inst == 0 || n_inst > kLogupMaxInst || k < 2 || getenv("DPB_NO_LOGUP_KERNEL")) return DPB_OK;
    for (uint32_t j = 0; j < k; j++)
        if (!mles[j]) return DPB_OK;
    // the tables are exactly the instances', in order, and the eq table
    uint32_t next = 0;
    for (uint32_t i = 0; i < n_inst; i++) {
        const LogupHintInst& h = inst[i];
        if (h.first != next || h.kind != inst[0].kind) return DPB_OK;
        if (h.kind == kLogupInner) next += 4;
        else if ((h.kind == kLogupLookup || h.kind == kLogupTable) && (h.ncol == 1 || h.ncol == 2))
            next += 2 * h.ncol + (h.kind == kLogupTable ? 2 : 0);
        else return DPB_OK;
    }
    if (next + 1 != k) return DPB_OK;
    if (partial && ctx->nranks > 1 && !ctx->nccl_comm) return fail(DPB_ESTATE, "the context has no communicator (dpb_comm_init)");
    LogupLayerSc* sc = new (std::nothrow) LogupLayerSc();
    if (!sc) return fail(DPB_ENOMEM, "host allocation failed");
    sc->ctx = ctx;
    sc->gl = is_gl(mles[next]->dtype);
    sc->partial = partial && ctx->nranks > 1;
    sc->n = num_vars;
    sc->k = k;
    sc->n_inst = n_inst;
    sc->eq_table = next;
    sc->mles.assign(mles, mles + k);
    sc->inst.assign(inst, inst + n_inst);
    memcpy(sc->lambda, lambda, sc->gl ? 16 : 32);
    bool usable = false;
    const int rc = sc->gl ? begin_impl<GlFam>(sc, &usable) : begin_impl<FrFam>(sc, &usable);
    if (rc != DPB_OK || !usable) {
        logup_layer_free(sc);
        return rc;
    }
    *out = sc;
    return DPB_OK;
}

int logup_layer_round(LogupLayerSc* sc, const void* prev_challenge, void* out_evals) {
    if (sc->round >= sc->n || (sc->round > 0) != (prev_challenge != nullptr)) return fail(DPB_ESTATE, "logup layer round out of order");
    return sc->gl ? round_impl<GlFam>(sc, prev_challenge, out_evals) : round_impl<FrFam>(sc, prev_challenge, out_evals);
}

int logup_layer_finish(LogupLayerSc* sc, const void* last_challenge, void* out) {
    if (sc->finished || sc->round != sc->n || !last_challenge) return fail(DPB_ESTATE, "logup layer finished out of order");
    return sc->gl ? finish_impl<GlFam>(sc, last_challenge, out) : finish_impl<FrFam>(sc, last_challenge, out);
}

void logup_layer_free(LogupLayerSc* sc) {
    if (!sc) return;
    dpb_ctx* ctx = sc->ctx;
    if (sc->tail_active) {
        // dropped before its end: tell the kernel to leave and wait for it (bounded by the kernel's own limit)
        TailBox* box = (TailBox*)ctx->tail_box_host;
        for (int i = 0; i < 4; i++) ((volatile TailChunk*)box->chal)[i].seq = kTailAbort;
        std::atomic_thread_fence(std::memory_order_seq_cst);
        cudaStreamSynchronize(ctx->tail_stream);
        leave_tail(sc);
    }
    if (sc->slab && sc->slab == ctx->slab_cache) ctx->slab_cache_busy = false;
    else device_free(ctx, sc->slab);
    delete sc;
}

}  // namespace dpb

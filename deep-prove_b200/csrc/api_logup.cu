// C ABI: logup-GKR fraction tree of one instance, every level resident on the
// device (the batched prover walks the levels top-down and needs all of them,
// zkml/src/lookup/logup_gkr/prover.rs:144-147).
#include <algorithm>

#include "common.cuh"
#include "logup_kernels.cuh"

using namespace dpb;

struct dpb_logup {
    dpb_ctx* ctx = nullptr;
    bool gl = false;
    uint32_t m = 0;        // columns have 2^m entries
    void* slab = nullptr;  // all levels, numerators then denominators per level
    std::vector<void*> num, den;  // level l (1-based) at index l-1, 2^(m-l) entries each
};

namespace dpb {

static int check_spec(dpb_ctx* ctx, const LogupSpec& p) {
    if (!p.columns || !p.constant || !p.sep) return fail(DPB_EINVAL, "null argument");
    if (p.kind != DPB_LOGUP_LOOKUP && p.kind != DPB_LOGUP_TABLE) return fail(DPB_EINVAL, "unknown kind %d", p.kind);
    if (p.n_cols < 1 || p.n_cols > (uint32_t)kMaxLogupCols)
        return fail(DPB_EINVAL, "No column evals were provided or too many (%u, max %d)", p.n_cols, kMaxLogupCols);
    if ((p.kind == DPB_LOGUP_TABLE) != (p.mult != nullptr))
        return fail(DPB_EINVAL, "multiplicities are required for tables and only for tables");
    for (uint32_t j = 0; j < p.n_cols; j++)
        if (!p.columns[j] || p.columns[j]->ctx != ctx) return fail(DPB_EINVAL, "column %u is null or foreign", j);
    const uint64_t len = p.columns[0]->len;
    const bool gl = is_gl(p.columns[0]->dtype);
    for (uint32_t j = 1; j < p.n_cols; j++) {
        if (p.columns[j]->len != len) return fail(DPB_EINVAL, "All sets of evaluations should be the same length");
        if (is_gl(p.columns[j]->dtype) != gl) return fail(DPB_EINVAL, "columns mix fields");
    }
    if (p.mult && (p.mult->len != len || is_gl(p.mult->dtype) != gl))
        return fail(DPB_EINVAL, "Multiplicities length was not equal to column evaluations length, multiplicities: %llu, columns: %llu",
                    (unsigned long long)p.mult->len, (unsigned long long)len);
    if (len < 4) return fail(DPB_EINVAL, "columns need at least 4 entries, got %llu", (unsigned long long)len);
    return DPB_OK;
}

static void int_rows(LogupTree<FrFam>& t, uint32_t j) {
    for (int half = 0; half < 2; half++) fr_fixed_row(t.sep_pow[j], 8 + half, t.rows[j][half]);
}
static void int_rows(LogupTree<GlFam>&, uint32_t) {}

// From this many rows, or fractions of a level, of all trees together a BN254 level is a launch of its own (level 1: of
// trees over field columns).  Two levels at a time and so, four columns: 2^19 rows 134 and 133 us, 2^20 196 and 181.
constexpr uint64_t kLogupSingle = 1ull << 20;

// The levels of `cnt` of the call's n trees.
template <class F, bool ONE>
static void launch_trees(dpb_ctx* ctx, const LogupTree<F>* dt, const LogupTree<F>* trees, uint32_t cnt, uint32_t n, typename F::E* outputs) {
    uint32_t max_m = 0;
    bool any_rows = false, all_rows = true;
    for (uint32_t i = 0; i < cnt; i++) {
        max_m = std::max(max_m, trees[i].m);
        any_rows |= trees[i].int_rows != 0;
        all_rows &= trees[i].int_rows != 0;
    }
    auto grid = [&](uint32_t items_log2) {  // per tree; all trees together fill the GPU
        const uint64_t want = ((1ull << items_log2) + kThreads - 1) / kThreads, cap = ((uint64_t)ctx->sm_count * 8 + n - 1) / n;
        return dim3((uint32_t)std::max<uint64_t>(1, std::min(want, cap)), cnt);
    };
    const LogupTree<F>& one = trees[0];
    constexpr bool kFr = sizeof(typename F::E) == 32;
    auto single = [&](uint32_t l) { return ((uint64_t)n << (max_m - l)) >= kLogupSingle; };
    const bool split = kFr && !all_rows && single(0);
    if (!split || any_rows) logup_leaf_levels<F, ONE><<<grid(max_m - 2), kThreads, 0, ctx->stream>>>(dt, one, split);
    if constexpr (kFr) {
        if (split) {
            logup_leaf_level<F, ONE><<<grid(max_m - 1), kThreads, 0, ctx->stream>>>(dt, one);
            logup_one_level<F, ONE><<<grid(max_m - 2), kThreads, 0, ctx->stream>>>(dt, one, 1);
        }
    }
    for (uint32_t l = 2; l + 2 <= max_m && (1ull << (max_m - l)) > kLogupSmall; l += 2) {
        if constexpr (kFr) {
            if (single(l)) {
                logup_one_level<F, ONE><<<grid(max_m - l - 1), kThreads, 0, ctx->stream>>>(dt, one, l);
                logup_one_level<F, ONE><<<grid(max_m - l - 2), kThreads, 0, ctx->stream>>>(dt, one, l + 1);
                continue;
            }
        }
        logup_two_levels<F, ONE><<<grid(max_m - l - 2), kThreads, 0, ctx->stream>>>(dt, one, l);
    }
    logup_small_levels<F, ONE><<<cnt, kThreads, 0, ctx->stream>>>(dt, one, outputs);
}

// The trees' levels, and their outputs (4 elements each) to the host when asked for.
template <class F>
static int build_trees(dpb_ctx* ctx, const LogupSpec* specs, uint32_t n, dpb_logup** out, void* host_outputs) {
    typedef typename F::E E;
    std::vector<LogupTree<F>> trees(n);
    for (uint32_t i = 0; i < n; i++) {
        const LogupSpec& p = specs[i];
        dpb_logup* lu = out[i];
        LogupTree<F>& t = trees[i];
        memset((void*)&t, 0, sizeof t);
        const uint32_t m = lu->m;
        DPB_TRY(device_alloc(ctx, logup_level_offset(m, m) * sizeof(E), &lu->slab));
        for (uint32_t l = 1; l < m; l++) {
            lu->num.push_back((E*)lu->slab + logup_level_offset(m, l));
            lu->den.push_back((E*)lu->slab + logup_level_offset(m, l) + (1ull << (m - l)));
        }
        t.slab = (E*)lu->slab;
        t.m = m;
        t.n_cols = p.n_cols;
        t.is_table = p.kind == DPB_LOGUP_TABLE;
        if (p.mult) {
            t.mult = p.mult->ptr;
            t.mult_dtype = p.mult->dtype;
        }
        memcpy(&t.constant, p.constant, sizeof(E));
        E sep, pw = F::one();
        memcpy(&sep, p.sep, sizeof(E));
        t.int_rows = sizeof(E) == 32;
        E sum = F::zero();
        for (uint32_t j = 0; j < p.n_cols; j++) {
            t.col[j] = p.columns[j]->ptr;
            t.dtype[j] = p.columns[j]->dtype;
            if (!is_int_dtype(t.dtype[j])) t.int_rows = 0;
            t.sep_pow[j] = pw;
            sum = F::add(sum, pw);
            pw = F::mul(pw, sep);
        }
        t.int_constant = F::sub(t.constant, F::mul(F::from_u64(0x80000000ull), sum));
        for (uint32_t j = 0; t.int_rows && j < p.n_cols; j++) int_rows(t, j);
    }
    // one tree goes to the kernels as a parameter, several through memory: [trees | outputs]
    char* d = nullptr;
    const size_t o_out = n > 1 ? (n * sizeof(LogupTree<F>) + 31) & ~(size_t)31 : 0;
    if (n > 1 || host_outputs) DPB_TRY(device_alloc(ctx, o_out + (size_t)n * 4 * sizeof(E), (void**)&d));
    E* outputs = d ? (E*)(d + o_out) : nullptr;
    int rc = n > 1 ? upload_small(ctx, d, trees.data(), n * sizeof(LogupTree<F>)) : DPB_OK;
    if (rc == DPB_OK) {
        for (uint32_t first = 0; first < n; first += 65535) {  // the grid's second dimension
            const uint32_t cnt = std::min<uint32_t>(65535, n - first);
            if (n > 1) launch_trees<F, false>(ctx, (const LogupTree<F>*)d + first, trees.data() + first, cnt, n, outputs ? outputs + 4 * (size_t)first : nullptr);
            else launch_trees<F, true>(ctx, nullptr, trees.data(), 1, 1, outputs);
        }
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess && host_outputs) {
            TracePhase t_out("logup.outputs");
            e = cudaMemcpyAsync(host_outputs, outputs, (size_t)n * 4 * sizeof(E), cudaMemcpyDeviceToHost, ctx->stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
        }
        if (e != cudaSuccess) rc = fail(DPB_ECUDA, "logup trees: %s", cudaGetErrorString(e));
    }
    device_free(ctx, d);
    return rc;
}

int logup_build_batch(dpb_ctx* ctx, const LogupSpec* specs, uint32_t n, dpb_logup** out, void* host_outputs) {
    if (!ctx || !specs || !out || n == 0) return fail(DPB_EINVAL, "null argument");
    for (uint32_t i = 0; i < n; i++) {
        out[i] = nullptr;
        DPB_TRY(check_spec(ctx, specs[i]));
        if (is_gl(specs[i].columns[0]->dtype) != is_gl(specs[0].columns[0]->dtype))
            return fail(DPB_EINVAL, "instance %u is of another field", i);
    }
    const bool gl = is_gl(specs[0].columns[0]->dtype);
    int rc = DPB_OK;
    for (uint32_t i = 0; i < n && rc == DPB_OK; i++) {
        out[i] = new (std::nothrow) dpb_logup();
        if (!out[i]) {
            rc = fail(DPB_ENOMEM, "host allocation failed");
            break;
        }
        out[i]->ctx = ctx;
        out[i]->gl = gl;
        out[i]->m = log2u(specs[i].columns[0]->len);
    }
    if (rc == DPB_OK) rc = gl ? build_trees<GlFam>(ctx, specs, n, out, host_outputs) : build_trees<FrFam>(ctx, specs, n, out, host_outputs);
    if (rc != DPB_OK)
        for (uint32_t i = 0; i < n; i++) {
            dpb_logup_free(out[i]);
            out[i] = nullptr;
        }
    return rc;
}

}  // namespace dpb

extern "C" {

int dpb_logup_build(dpb_ctx* ctx, int kind, dpb_mle* const* columns, uint32_t n_cols,
                    const dpb_mle* mult, const void* constant_chal, const void* sep_chal,
                    dpb_logup** out) {
    if (!ctx || !columns || !constant_chal || !sep_chal || !out) return fail(DPB_EINVAL, "null argument");
    LogupSpec p;
    p.kind = kind;
    p.columns = columns;
    p.n_cols = n_cols;
    p.mult = mult;
    p.constant = constant_chal;
    p.sep = sep_chal;
    dpb_logup* lu = nullptr;
    DPB_TRY(logup_build_batch(ctx, &p, 1, &lu, nullptr));
    *out = lu;
    return DPB_OK;
}

uint32_t dpb_logup_num_levels(const dpb_logup* lu) { return lu ? lu->m - 1 : 0; }

int dpb_logup_level(const dpb_logup* lu, uint32_t level, dpb_mle* out_views[4]) {
    if (!lu || !out_views) return fail(DPB_EINVAL, "null argument");
    if (level < 1 || level > lu->m - 1) return fail(DPB_EINVAL, "level %u outside 1..%u", level, lu->m - 1);
    const uint64_t half = 1ull << (lu->m - level - 1);
    const size_t es = lu->gl ? 16 : 32;
    const int dt = lu->gl ? DPB_GL_EXT : DPB_FR;
    char* base[2] = {(char*)lu->num[level - 1], (char*)lu->den[level - 1]};
    for (int a = 0; a < 2; a++) {
        for (int h = 0; h < 2; h++) {
            dpb_mle* v = new (std::nothrow) dpb_mle();
            if (!v) return fail(DPB_ENOMEM, "host allocation failed");
            v->ctx = lu->ctx;
            v->dtype = dt;
            v->len = half;
            v->ptr = base[a] + (size_t)h * half * es;
            v->owns = false;
            out_views[a * 2 + h] = v;
        }
    }
    return DPB_OK;
}

int dpb_logup_outputs(const dpb_logup* lu, void* out4) {
    if (!lu || !out4) return fail(DPB_EINVAL, "null argument");
    const size_t es = lu->gl ? 16 : 32;
    const uint32_t top = lu->m - 1;
    dpb_ctx* ctx = lu->ctx;
    DPB_CUDA(cudaMemcpyAsync(out4, lu->num[top - 1], 2 * es, cudaMemcpyDeviceToHost, ctx->stream));
    DPB_CUDA(cudaMemcpyAsync((char*)out4 + 2 * es, lu->den[top - 1], 2 * es, cudaMemcpyDeviceToHost, ctx->stream));
    DPB_CUDA(cudaStreamSynchronize(ctx->stream));
    return DPB_OK;
}

int dpb_logup_outputs_batch(const dpb_logup* const* lus, uint32_t n, void* out) {
    if (!lus || !out || n == 0) return fail(DPB_EINVAL, "null argument");
    for (uint32_t i = 0; i < n; i++)
        if (!lus[i] || lus[i]->ctx != lus[0]->ctx || lus[i]->gl != lus[0]->gl)
            return fail(DPB_EINVAL, "tree %u is null, of another context or of another field", i);
    dpb_ctx* ctx = lus[0]->ctx;
    const size_t es = lus[0]->gl ? 16 : 32;
    // gathered on the device, then one copy to the host and one wait, instead of one of each per tree
    void* gathered = nullptr;
    DPB_TRY(device_alloc(ctx, (size_t)n * 4 * es, &gathered));
    cudaError_t e = cudaSuccess;
    for (uint32_t i = 0; i < n && e == cudaSuccess; i++) {
        const uint32_t top = lus[i]->m - 1;
        char* dst = (char*)gathered + (size_t)i * 4 * es;
        e = cudaMemcpyAsync(dst, lus[i]->num[top - 1], 2 * es, cudaMemcpyDeviceToDevice, ctx->stream);
        if (e == cudaSuccess) e = cudaMemcpyAsync(dst + 2 * es, lus[i]->den[top - 1], 2 * es, cudaMemcpyDeviceToDevice, ctx->stream);
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(out, gathered, (size_t)n * 4 * es, cudaMemcpyDeviceToHost, ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
    device_free(ctx, gathered);
    if (e != cudaSuccess) return fail(DPB_ECUDA, "logup outputs: %s", cudaGetErrorString(e));
    return DPB_OK;
}

void dpb_logup_free(dpb_logup* lu) {
    if (!lu) return;
    device_free(lu->ctx, lu->slab);
    delete lu;
}

}  // extern "C"

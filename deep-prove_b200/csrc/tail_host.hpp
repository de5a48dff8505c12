// Host side of the mailbox between a resident kernel and the prover's thread (TailBox, generic_round.cuh).
#pragma once
#include <atomic>
#include <chrono>
#include <thread>

#include "common.cuh"
#include "generic_round.cuh"

namespace dpb {

// Polls the mailbox until `ready` holds; bounded, and the stream is queried now and then so that a
// kernel that died or returned early surfaces as an error.
constexpr int kTailNoHost = 1;  // internal: the kernel found that launches block the host; fall back to launches
constexpr int kTailGaveUp = 2;  // internal: the kernel's wait for a challenge ran out and it returned

template <class Ready>
static int tail_wait_host(dpb_ctx* ctx, TailBox* box, Ready ready) {
    uint64_t spins = 0;
    std::chrono::steady_clock::time_point t0;
    while (!ready()) {
        if (box->status == 3) return kTailNoHost;
        if (box->status == 2) {
            // the host may have been held up between the two looks: what it waits for can have come first
            std::atomic_thread_fence(std::memory_order_acquire);
            if (ready()) break;
            return kTailGaveUp;
        }
        if ((++spins & 0xFFF) == 0) {
            cudaError_t e = cudaStreamQuery(ctx->tail_stream);
            if (e != cudaSuccess && e != cudaErrorNotReady)
                return fail(DPB_ECUDA, "resident round kernel: %s", cudaGetErrorString(e));
            if (e == cudaSuccess && box->status != 2 && box->status != 3 && !ready())
                return fail(DPB_ECUDA, "the resident round kernel returned without a result (%s)",
                            cudaGetErrorString(cudaGetLastError()));
            if (spins == 0x1000) t0 = std::chrono::steady_clock::now();
            else if (std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count() > 120.0)
                return fail(DPB_ETIMEOUT, "the resident round kernel did not answer within 120 s");
        }
    }
    std::atomic_thread_fence(std::memory_order_acquire);
    return DPB_OK;
}

// the challenge as chunks: data first, then the sequence numbers
template <class E>
static void tail_post(dpb_ctx* ctx, const void* chal, uint32_t seq) {
    TailBox* box = (TailBox*)ctx->tail_box_host;
    if (ctx->tail_posts++ == ctx->tail_hold_post)
        std::this_thread::sleep_for(std::chrono::milliseconds(ctx->tail_hold_ms));  // dpb_resident_hold
    const uint64_t* w = (const uint64_t*)chal;
    constexpr int W8 = sizeof(E) / 8;
    for (int i = 0; i < W8; i++) ((volatile TailChunk*)box->chal)[i].data = w[i];
    std::atomic_thread_fence(std::memory_order_release);
    for (int i = 0; i < W8; i++) ((volatile TailChunk*)box->chal)[i].seq = seq;
}
// element `idx` of a chunk array, once every chunk of it carries `seq`
template <class E>
static bool tail_take(const TailChunk* base, uint32_t idx, uint32_t seq, E* out) {
    constexpr int W8 = sizeof(E) / 8;
    const volatile TailChunk* c = (const volatile TailChunk*)base + (size_t)idx * W8;
    uint64_t* w = (uint64_t*)out;
    for (int i = 0; i < W8; i++) {
        if (c[i].seq != seq) return false;
        std::atomic_thread_fence(std::memory_order_acquire);
        w[i] = c[i].data;
    }
    return true;
}

// Collects the sums of the round just launched from the chunk area in mapped host memory: every chunk carries
// the launch's sequence number once it has arrived.  The stream is queried now and then so that a failed launch
// surfaces, and the wait is bounded.
static int wait_round_chunks(dpb_ctx* ctx, size_t msg_bytes, void* out) {
    const unsigned int want = ctx->done_value;
    const volatile TailChunk* c = (const volatile TailChunk*)ctx->result_host;
    uint64_t* dst = (uint64_t*)out;
    uint64_t spins = 0;
    std::chrono::steady_clock::time_point t0;
    for (size_t w = 0; w < msg_bytes / 8; w++) {
        while (c[w].seq != want) {
            if ((++spins & 0xFFF) == 0) {
                cudaError_t e = cudaStreamQuery(ctx->stream);
                if (e != cudaSuccess && e != cudaErrorNotReady) return fail(DPB_ECUDA, "round kernel: %s", cudaGetErrorString(e));
                if (e == cudaSuccess && c[w].seq != want) {
                    // the stream drained without the result: the launch itself failed
                    e = cudaGetLastError();
                    if (c[w].seq == want) break;
                    return fail(DPB_ECUDA, "round kernel did not deliver its result (%s)", cudaGetErrorString(e));
                }
                if (spins == 0x1000) t0 = std::chrono::steady_clock::now();
                else if (std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count() > 120.0)
                    return fail(DPB_ETIMEOUT, "round kernel did not finish within 120 s");
            }
        }
        std::atomic_thread_fence(std::memory_order_acquire);
        dst[w] = c[w].data;
    }
    return DPB_OK;
}

}  // namespace dpb

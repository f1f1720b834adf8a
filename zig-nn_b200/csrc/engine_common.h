// Pieces shared by the device-resident engines (engine.cu: GPT-2 and Gemma-3, engine_decoder.cu): the owner of an
// engine's device memory and the recorded decode steps.
#pragma once
#include <string.h>

#include <vector>

#include "zq_internal.h"

namespace zq {
namespace {

struct DeviceArena {
    std::vector<void*> ptrs;
    size_t total = 0;
    ~DeviceArena() {
        for (void* p : ptrs) cudaFree(p);
    }
    int alloc(void** out, size_t bytes) {
        cudaError_t e = cudaMalloc(out, bytes ? bytes : 4);
        if (e != cudaSuccess) return alloc_fail(e);
        ptrs.push_back(*out);
        total += bytes;
        return ZQ_OK;
    }
    template <typename T>
    int alloc_n(T** out, size_t n) {
        return alloc(reinterpret_cast<void**>(out), n * sizeof(T));
    }
    int upload_f32(float** out, const float* host, size_t n, cudaStream_t st) {
        if (!host) return ZQ_ERR_BAD_ARG;
        int rc = alloc_n(out, n);
        if (rc != ZQ_OK) return rc;
        ZQ_CUDA(cudaMemcpyAsync(*out, host, n * sizeof(float), cudaMemcpyHostToDevice, st));
        return ZQ_OK;
    }
};

// Rows of a step of several sequences, as kernel arguments: copies from the caller's arrays would have to be waited for, and the
// device would idle while the host launches the step (10 us of a 380 us step of six sequences, 8 of 1600 for eight of Gemma-3-1B).
constexpr uint32_t kStepRows = 256;
struct StepRows {
    uint32_t token[kStepRows], pos[kStepRows], slot[kStepRows];
};
__global__ void set_step_rows_kernel(const __grid_constant__ StepRows rows, uint32_t n, uint32_t* tokens, uint32_t* pos, uint32_t* slots) {
    const uint32_t i = threadIdx.x;
    if (i >= n) return;
    tokens[i] = rows.token[i];
    pos[i] = rows.pos[i];
    if (slots) slots[i] = rows.slot[i];
}
// Row r: token h_tokens[r] of sequence h_seqs[r] (null: r) at position lens[that sequence]. Such a step advances the host's
// lengths, so a recording of it could not be replayed: it is refused.
inline int set_step_rows(const uint32_t* h_seqs, const uint32_t* h_tokens, const uint32_t* lens, uint32_t n, void* d_tokens,
                         void* d_pos, void* d_slots, cudaStream_t st) {
    uint32_t *tokens = static_cast<uint32_t*>(d_tokens), *pos = static_cast<uint32_t*>(d_pos), *slots = static_cast<uint32_t*>(d_slots);
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    ZQ_CUDA(cudaStreamIsCapturing(st, &capture));
    if (capture != cudaStreamCaptureStatusNone) return cuda_fail(cudaErrorStreamCaptureUnsupported);
    for (uint32_t r0 = 0; r0 < n; r0 += kStepRows) {
        const uint32_t m = n - r0 < kStepRows ? n - r0 : kStepRows;
        StepRows rows;
        for (uint32_t i = 0; i < m; ++i) {
            rows.slot[i] = h_seqs ? h_seqs[r0 + i] : r0 + i;
            rows.token[i] = h_tokens[r0 + i];
            rows.pos[i] = lens[rows.slot[i]];
        }
        set_step_rows_kernel<<<1, kStepRows, 0, st>>>(rows, m, tokens + r0, pos + r0, slots ? slots + r0 : nullptr);
        ZQ_LAUNCH_CHECK();
    }
    return ZQ_OK;
}

// A decode step is a fixed launch sequence whose only varying inputs live in device memory, so it is
// captured once per variant and replayed. The first use of a variant runs eagerly (function
// attributes get set and launch errors surface outside capture); the second captures on the
// engine's own stream (the caller's may be the legacy default stream, which cannot capture); every
// use from then on is one graph launch on the caller's stream.
enum StepVariant { STEP_CACHE_ONLY = 0, STEP_LOGITS = 1, STEP_GREEDY = 2, STEP_BATCH = 3, STEP_VARIANTS = 4 };

struct StepGraphs {
    cudaGraphExec_t exec[STEP_VARIANTS] = {nullptr, nullptr, nullptr, nullptr};
    bool warmed[STEP_VARIANTS] = {false, false, false, false};
    cudaStream_t capture_stream = nullptr;
    bool disabled = false;
    ~StepGraphs() {
        for (cudaGraphExec_t e : exec)
            if (e) cudaGraphExecDestroy(e);
        if (capture_stream) cudaStreamDestroy(capture_stream);
    }
    template <typename Body>
    int run(int variant, cudaStream_t st, Body&& body) {
        if (disabled) return body(st);
        if (!warmed[variant]) {
            warmed[variant] = true;
            return body(st);
        }
        if (!exec[variant]) {
            if (!capture_stream) ZQ_CUDA(cudaStreamCreateWithFlags(&capture_stream, cudaStreamNonBlocking));
            ZQ_CUDA(cudaStreamBeginCapture(capture_stream, cudaStreamCaptureModeThreadLocal));
            const int rc = body(capture_stream);
            cudaGraph_t graph = nullptr;
            const cudaError_t e = cudaStreamEndCapture(capture_stream, &graph);
            if (rc != ZQ_OK || e != cudaSuccess) {
                if (graph) cudaGraphDestroy(graph);
                return rc != ZQ_OK ? rc : cuda_fail(e);
            }
            const cudaError_t ei = cudaGraphInstantiate(&exec[variant], graph, 0);
            cudaGraphDestroy(graph);
            if (ei != cudaSuccess) {
                exec[variant] = nullptr;
                return cuda_fail(ei);
            }
        }
        ZQ_CUDA(cudaGraphLaunch(exec[variant], st));
        return ZQ_OK;
    }
};

}  // namespace
}  // namespace zq

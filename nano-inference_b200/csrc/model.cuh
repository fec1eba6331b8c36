// The loaded model as the decode and the M-token step see it.
#pragma once
#include "decode_kernel.cuh"
#include "gemm_dig.cuh"
#include "buffer_set.cuh"
#include "pass_graphs.cuh"

#include <tuple>
#include <vector>

namespace mi {
// what a captured pass depends on besides the buffers: tokens, attention grid, kind of meta block, the cache
struct PassKey {
    int M, regime, ragged; const void* kc; const void* vc; int max_seq;
    bool operator<(const PassKey& o) const { return std::tie(M, regime, ragged, kc, vc, max_seq) < std::tie(o.M, o.regime, o.ragged, o.kc, o.vc, o.max_seq); }
};
// device buffers of the M-token step (all [tokens][...], token-major)
struct VerifyBufs {
    int cap = 0, cap_logits = 0;       // tokens the buffers hold
    BufferSet mem;                     // the allocations behind the pointers below; clears them when it frees
    float* X = nullptr;                // residual stream [M][E]
    double* part = nullptr; int ldp = 0;    // sums of a projection per K range [range][M][ldp]
    float* Y = nullptr;                // fp32 rows of the QKV and gate/up products (more than kMaxFusedTok tokens)
    float* q = nullptr;                // [M][NQ] after bias and RoPE, natural order
    TokX xf{}, attf{}, actf{};         // q8_0 of the normed input, the attention output and SwiGLU, in operand order
    uint8_t* dig = nullptr; int* dig_info = nullptr; long long* dig_bias = nullptr;     // digits of one product's activations (more than kMaxFusedTok tokens)
    float* att = nullptr;              // [M][NQ]
    float* logits = nullptr;           // [M][V]
    int* meta = nullptr; int* h_meta = nullptr;         // tokens | positions | slots, or tokens | first position; its pinned image
    int* out = nullptr;                // [M]
    PassGraphs<PassKey> graphs;        // cudaGraphExec_t
    double* attn_part = nullptr;       // chunk sums of the attention (attn_tok.cu)
    float* pick = nullptr; unsigned* pick_cnt = nullptr;         // greedy pick: candidates per slice, arrival counters (self-clearing)
    float* margins = nullptr;          // [M] greedy logit minus the runner-up
};
}

struct mi_model {
    int device = 0;
    int L = 0, E = 0, FF = 0, NH = 0, NKV = 0, HD = 0, KVD = 0, V = 0, G = 0;
    float eps = 1e-6f, rope_base = 1e6f;
    int max_seq = 0, grid = 0, max_chunks = 0, attn_ctas = 0;
    bool one_batch = true;                 // every CTA has at most one batch of units per job (what the range builds of the decode kernel take)
    int tp_rank = 0, tp_world = 1;
    bool tied = false;
    int requantized = 0;                  // matrices that were stored in another block format and re-quantized at load
    int64_t weight_bytes_q4 = 0;          // algorithmic q4_0 bytes streamed per token (18 bytes / 32 weights)
    std::vector<void*> allocs;            // everything cudaMalloc'ed for this model
    std::vector<mi::Job> jobs;
    mi::DecodeParams P{};                     // device pointers filled in; per-call fields set at launch
    int* d_in_tokens = nullptr; int in_capacity = 0;
    int* d_out_tokens = nullptr; int out_capacity = 0;
    // kernel-sequence engine as a replayed CUDA graph (decode.cu, step_graph): one graph per context range, the control
    // block the graph's first and last node read (device memory, refilled per call), the step's token and margin
    void* step_graph[4] = {}; unsigned long long step_graph_wait[4] = {};
    void* d_seq_ctl = nullptr; int* d_step_out = nullptr; float* d_step_margin = nullptr;
    int stop_token = -1;                  // see mi_model_set_stop_token
    int last_count = 0;                   // steps (tokens) the last decode / generate call produced: fewer than asked after a stop
    float* d_margins = nullptr; int last_steps = 0;   // top-1 minus top-2 logit of every step of the last decode call
    size_t smem = 0;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    unsigned long long* prof_buf = nullptr;
    float* best_buf = nullptr;           // {best logit value, greedy token (int bits)}
    int qkv_rows = 0;
    int* tp_flags = nullptr;              // host-driven peer exchange: flags, epoch, gathered argmax candidates (see tp_peer.cu)
    void* tp_peer[8][3] = {};             // per rank: exchange block, (unused), flag block (own entries = local pointers)
    unsigned long long errors_seen = 0;   // value of the context's error count when this model last cleared its counters
    bool tp_peer_on = false;
    std::vector<void*> ipc_opened;        // peer mappings to close
    int* d_pos = nullptr;                 // [2]: device-resident position for position-free launch sequences; the tag epoch
    std::vector<mi_weight> views;         // [4L+1] whole matrices in job order (QKV, O, gate/up, down per layer; lm_head), for the M-token step
    std::vector<mi::LayerPtrs> layer_ptrs;    // host copy of the per-layer norm / bias pointers
    int products = 0;                     // mi_model_debug_products
    mi::VerifyBufs vb;                    // buffers of the M-token step, allocated on first use
};


namespace mi {

void free_verify_bufs(mi_model* m);
int reset_after_error(mi_ctx* ctx, mi_model* m);

template <typename T>
int dev_alloc(mi_ctx* ctx, mi_model* m, T** p, size_t n, bool zero = true) {
    *p = nullptr;
    if (n == 0) n = 1;
    cudaError_t e = cudaMalloc((void**)p, n * sizeof(T));
    if (e != cudaSuccess) return set_error(ctx, MI_ERR_NOMEM, "model: cudaMalloc(%zu) failed: %s", n * sizeof(T), cudaGetErrorString(e));
    m->allocs.push_back(*p);
    if (zero) {
        // the fill runs on the legacy stream, which the context's own (non-blocking) stream does not wait for:
        // finish it here, before anything enqueued later can write the buffer
        e = cudaMemset(*p, 0, n * sizeof(T));
        if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);
        if (e != cudaSuccess) return set_error(ctx, MI_ERR_CUDA, "model: cudaMemset failed");
    }
    return MI_OK;
}

}  // namespace mi

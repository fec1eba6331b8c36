// The M-token step: several tokens in one pass over the weights - up to 16 drafted tokens with logits (mi_verify), up to 512
// prompt tokens (mi_prefill), up to 64 sequences of their own (mi_batch_step) - and the stand-alone split-KV attention
// entry point.
//
// Replaces forward_batch (reference src/cuda_infer.cu:990-1029: quant_x_q8_batch,
// gemv_dp4a_batch<T>, rope / kv_store / attention per token) and the M-token path of the
// persistent kernel (reference src/mega.cu:246-299 gemv_seq, :414-521 attention).
//
// One pass is a sequence of launches per layer
//     norm+q8 (M tokens) -> QKV product + RoPE + fp16 KV store -> attention (M queries)
//     -> O product -> residual + norm+q8 -> gate/up product + SwiGLU + q8 -> down product
// and finally norm+q8 -> lm_head product -> greedy pick per token.  Every token goes through the
// expressions of the single-token decode kernel (same quantizer, same sums carried in double), so its
// logits do not depend on how many tokens share the pass.
// Above 16 tokens RoPE and SwiGLU are kernels of their own, and each product goes over digits (gemm_dig.cu) where that is faster (choose_gemm_dig;
// 333 tokens of the 1.5B shape 8040 -> 5718 us, 64 sequences of the 3B shape 4657 -> 3674); the kernel before it then writes the digits.
#include "model.cuh"
#include "attn_tok.cuh"

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <type_traits>

using namespace mi;

namespace {

constexpr int VMAX = 16;                    // tokens of one mi_verify call
constexpr int BMAX = 64;                    // sequences of one batched pass
constexpr int PMAX = 512;                   // prompt tokens of one pass
constexpr int kMaxRanges = 8;               // K ranges of a split product (plan_gemm_tok)

// x = (embedding row | X) (+ the projection's sum over its K ranges, rounded to fp32 once), committed to X;
// q8_0(rmsnorm(x) * w) (src/cpu_infer.cpp:40-46) in operand order.  One CTA per token, four consecutive elements per
// thread: every load of a thread is requested before the first is used, a block of 32 is eight threads.  Token m0 + blockIdx.x
// of X is token blockIdx.x of the output.  DIG: the digits of a product that takes all of K at once as well; a form of its own, because passes of few
// tokens pay for that code without running it (5 tokens of the 1.5B shape at 2000 positions 1161 us per pass with it, 1132 before it; 16 sequences of the 3B shape 2094 / 2074).
template <int R, bool DIG>
__global__ void __launch_bounds__(R == 1 ? 512 : 1024) vf_norm_quant(const DecodeParams P, const int* __restrict__ tokens, bool embed, int m0, float* X, const double* part,
                                                       int ranges, long long range_stride, int ldp, const float* __restrict__ w, TokX out, DigX dig) {
    __shared__ double red[32];
    const int E = P.E, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5, mo = blockIdx.x, m = m0 + mo;
    float4 wv[R];
    #pragma unroll
    for (int r = 0; r < R; r++) {
        const int e = (tid + r * blockDim.x) * 4;
        wv[r] = e < E ? __ldg(reinterpret_cast<const float4*>(w + e)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    pdl_launch_dependents(); pdl_wait_prior();
    float v[R][4];
    double ss = 0.0;
    #pragma unroll
    for (int r = 0; r < R; r++) {
        const int e = (tid + r * blockDim.x) * 4;
        if (e >= E) { v[r][0] = v[r][1] = v[r][2] = v[r][3] = 0.f; continue; }
        float4 x;
        if (embed) {
            const int token = __ldg(tokens + m), b = e >> 5, k = e & 31;
            if (P.emb_q8) {                                           // a Q8_0 row as stored: int8 * d (src/gguf.h:112-118)
                const uint8_t* bp = P.emb_q8 + ((size_t)token * (E / 32) + b) * 34;
                const float d = __half2float(__ldg(reinterpret_cast<const __half*>(bp)));
                const unsigned short q01 = __ldg(reinterpret_cast<const unsigned short*>(bp + 2 + k)), q23 = __ldg(reinterpret_cast<const unsigned short*>(bp + 4 + k));
                x = make_float4(__fmul_rn(__int2float_rn((int)(int8_t)(q01 & 0xff)), d), __fmul_rn(__int2float_rn((int)(int8_t)(q01 >> 8)), d),
                                __fmul_rn(__int2float_rn((int)(int8_t)(q23 & 0xff)), d), __fmul_rn(__int2float_rn((int)(int8_t)(q23 >> 8)), d));
            } else {                                                  // value (nibble - 8) * d (src/gguf.h:94-102)
                const int g = token >> 5, rr = token & 31, kb = P.emb_kb, t = b / kb, kk = b - t * kb;
                const uint8_t* tile = P.emb_base + ((size_t)g * P.emb_nt + t) * (kb * kTileRowBytes);
                const unsigned q = __ldg(reinterpret_cast<const unsigned*>(tile + ((size_t)kk * 32 + rr) * 16 + (k & 15))) >> (k < 16 ? 0 : 4);
                const float d = __half2float(__ldg(reinterpret_cast<const __half*>(tile + (size_t)kb * 512 + ((size_t)rr * kb + kk) * 2)));
                x = make_float4(__fmul_rn(__int2float_rn((int)(q & 15) - 8), d), __fmul_rn(__int2float_rn((int)(q >> 8 & 15) - 8), d),
                                __fmul_rn(__int2float_rn((int)(q >> 16 & 15) - 8), d), __fmul_rn(__int2float_rn((int)(q >> 24 & 15) - 8), d));
            }
        } else {
            x = *reinterpret_cast<const float4*>(X + (size_t)m * E + e);
        }
        v[r][0] = x.x; v[r][1] = x.y; v[r][2] = x.z; v[r][3] = x.w;
        if (part) {
            const double* pp = part + (size_t)m * ldp + e;
            double s[4] = {0.0, 0.0, 0.0, 0.0};
            // (a row of ranges is requested four at a time, and what remains together: a loop over single ones waits for each)
            auto add = [&](auto count, int q0) {
                constexpr int U = decltype(count)::value;
                double2 a[U], b[U];
                #pragma unroll
                for (int u = 0; u < U; u++) {
                    const double2* p2 = reinterpret_cast<const double2*>(pp + (q0 + u) * range_stride);
                    a[u] = __ldcg(p2); b[u] = __ldcg(p2 + 1);
                }
                #pragma unroll
                for (int u = 0; u < U; u++) { s[0] = __dadd_rn(s[0], a[u].x); s[1] = __dadd_rn(s[1], a[u].y); s[2] = __dadd_rn(s[2], b[u].x); s[3] = __dadd_rn(s[3], b[u].y); }
            };
            int q0 = 0;
            #pragma unroll 1
            for (; q0 + 4 <= ranges; q0 += 4) add(std::integral_constant<int, 4>{}, q0);
            if (ranges - q0 == 3) add(std::integral_constant<int, 3>{}, q0);
            else if (ranges - q0 == 2) add(std::integral_constant<int, 2>{}, q0);
            else if (ranges - q0 == 1) add(std::integral_constant<int, 1>{}, q0);
            #pragma unroll
            for (int i = 0; i < 4; i++) v[r][i] = __fadd_rn(v[r][i], __double2float_rn(s[i]));
        }
        if (embed || part) *reinterpret_cast<float4*>(X + (size_t)m * E + e) = make_float4(v[r][0], v[r][1], v[r][2], v[r][3]);
        #pragma unroll
        for (int i = 0; i < 4; i++) { const double d = v[r][i]; ss = __fma_rn(d, d, ss); }
    }
    #pragma unroll
    for (int o = 16; o; o >>= 1) ss = __dadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, o));
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    double tot = lane < nw ? red[lane] : 0.0;
    #pragma unroll
    for (int o = 16; o; o >>= 1) tot = __dadd_rn(tot, __shfl_xor_sync(0xffffffffu, tot, o));
    const float mean = __double2float_rn(div_known(tot, (double)E, P.inv_e));
    const float scale = __fdiv_rn(1.f, __fsqrt_rn(__fadd_rn(mean, P.eps)));
    [[maybe_unused]] unsigned q[R], h[R];
    [[maybe_unused]] DigRange mine;
    #pragma unroll
    for (int r = 0; r < R; r++) {
        const int e = (tid + r * blockDim.x) * 4;
        if constexpr (DIG) q[r] = h[r] = 0;
        if (((tid & ~31) + r * (int)blockDim.x) * 4 >= E) break;      // warp-uniform: the folds below are warp-wide
        const float ww[4] = {wv[r].x, wv[r].y, wv[r].z, wv[r].w};
        float a = 0.f;
        #pragma unroll
        for (int i = 0; i < 4; i++) { v[r][i] = __fmul_rn(__fmul_rn(v[r][i], scale), ww[i]); a = fmaxf(a, fabsf(v[r][i])); }
        a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, 1));
        a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, 2));
        a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, 4));
        const float inv = a > 0.f ? __fdiv_rn(127.f, a) : 0.f;
        unsigned qw = 0;
        #pragma unroll
        for (int i = 0; i < 4; i++) qw |= ((unsigned)__float2int_rn(__fmul_rn(v[r][i], inv)) & 0xffu) << (8 * i);
        if (e < E) {
            out.q[tok_word(out.J, e >> 5, mo, e & 31)] = qw;
            if constexpr (DIG) {
                const __half d = __float2half_rn(__fdiv_rn(a, 127.f));
                if ((tid & 7) == 0) out.d[tok_scale(out.J, e >> 5, mo)] = tok_scale_value(d);
                q[r] = qw; h[r] = __half_as_ushort(d);
                mine.add(h[r], __dp4a((int)qw, 0x01010101, 0));
            } else if ((tid & 7) == 0) out.d[tok_scale(out.J, e >> 5, mo)] = tok_scale_value(__float2half_rn(__fdiv_rn(a, 127.f)));
        }
    }
    if constexpr (!DIG) return;
    else {
    __shared__ DigReduce dred;
    const DigRange all = mine.over_cta(dred);
    if (tid == 0) { dig.info[mo] = all.unit() | all.planes() << 8; dig.bias[mo] = all.total(); }
    const int tt = mo / dig.T, t = mo - tt * dig.T;
    #pragma unroll
    for (int r = 0; r < R; r++) {
        const int e = (tid + r * blockDim.x) * 4;
        if (e >= E) break;
        unsigned d[4];
        dig_word(q[r], all.factor(h[r]), d);
        #pragma unroll
        for (int j = 0; j < 4; j++) *reinterpret_cast<unsigned*>(dig.q + dig_offset(dig, E / 32, tt, e >> 5, e >> 4 & 1, j, t) + (e & 15)) = d[j];
        if (3 * dig.T + t < dig_rows(dig.T)) *reinterpret_cast<unsigned*>(dig.q + dig_offset(dig, E / 32, tt, e >> 5, e >> 4 & 1, 0, 3 * dig.T + t) + (e & 15)) = 0;      // rows of padding
    }
    }
}

// The QKV product's epilogue as a kernel of its own (more than kMaxFusedTok tokens): one warp per 32 rows and token of y (bias added)
__global__ void __launch_bounds__(256) vf_rope(const RopeParams r, const float* y, int rows) {
    const int n = blockIdx.y, row0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * 32, lane = threadIdx.x & 31;
    pdl_launch_dependents(); pdl_wait_prior();
    if (row0 >= rows) return;
    rope_store(r, row0 + lane, n, __ldcg(y + (size_t)n * rows + row0 + lane));
}

// The gate/up product's epilogue likewise: one warp per q8_0 block and token (few tokens: four elements per lane, as in swiglu_digits_kernel,
// make a longer chain, 32 tokens of the 1.5B shape 1769 us instead of 1738); the rows of y come as (gate, up) groups of 32
__global__ void __launch_bounds__(256) vf_swiglu(const float* y, int FF, TokX act) {
    const int n = blockIdx.y, b = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    pdl_launch_dependents(); pdl_wait_prior();
    if (b >= FF / 32) return;
    const float* v = y + (size_t)n * 2 * FF + (size_t)b * 64 + lane;
    store_tok_block(act, b, n, lane, swiglu(__ldcg(v), __ldcg(v + 32)));
}

// greedy pick of every token, lowest index on ties (src/cpu_infer.cpp:153-154), and its logit margin (greedy logit minus the
// largest other one) in one reading of the logits.  grid = (slices, tokens): every CTA reduces its slice to {best, row, second};
// the last CTA of a token to arrive merges the slices and clears the counter for the next pass.  A NaN in row 0 wins like +inf
// and any other NaN never does, as in the single-token step.
constexpr int kPickSlices = 37;                                      // four tokens fill the machine
__global__ void __launch_bounds__(512) vf_pick(const float* logits, long long stride, int V, int* out, float* margins, float* slices, unsigned* cnt, int* cur_token) {
    __shared__ float sb[16], s2[16]; __shared__ int si[16]; __shared__ unsigned s_prev;
    pdl_launch_dependents(); pdl_wait_prior();
    const int m = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const float* lg = logits + (size_t)m * stride;
    const int per = (V + gridDim.x - 1) / gridDim.x, r0 = blockIdx.x * per, r1 = min(V, r0 + per);
    Cand c; c.best = -INFINITY; c.idx = 0x7fffffff; c.second = -INFINITY;
    constexpr int U = 8;                                              // loads in flight
    for (int r = r0 + tid; r < r1; r += U * blockDim.x) {
        float v[U];
        #pragma unroll
        for (int u = 0; u < U; u++) v[u] = r + u * (int)blockDim.x < r1 ? __ldcg(lg + r + u * blockDim.x) : -INFINITY;
        #pragma unroll
        for (int u = 0; u < U; u++) {
            const int q = r + u * (int)blockDim.x;
            if (q < r1) c.add(q == 0 && v[u] != v[u] ? INFINITY : v[u], q);
        }
    }
    c.warp_reduce();
    if (lane == 0) { sb[warp] = c.best; si[warp] = c.idx; s2[warp] = c.second; }
    __syncthreads();
    float* sl = slices + (size_t)m * kPickSlices * 3;
    if (tid == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); w++) { Cand o; o.best = sb[w]; o.idx = si[w]; o.second = s2[w]; c.merge(o); }
        __stcg(sl + blockIdx.x * 3, c.best); __stcg(sl + blockIdx.x * 3 + 1, __int_as_float(c.idx)); __stcg(sl + blockIdx.x * 3 + 2, c.second);
        __threadfence();
        s_prev = atomicAdd(cnt + m, 1u);
    }
    __syncthreads();
    if (s_prev != gridDim.x - 1 || warp != 0) return;
    __threadfence();
    c.best = -INFINITY; c.idx = 0x7fffffff; c.second = -INFINITY;
    for (int q = lane; q < (int)gridDim.x; q += 32) {
        Cand o; o.best = __ldcg(sl + q * 3); o.idx = __float_as_int(__ldcg(sl + q * 3 + 1)); o.second = __ldcg(sl + q * 3 + 2);
        c.merge(o);
    }
    c.warp_reduce();
    if (lane == 0) {
        const int tok = c.idx == 0x7fffffff ? 0 : c.idx;
        out[m] = tok; margins[m] = __fsub_rn(c.best, c.second); cnt[m] = 0;
        if (m == (int)gridDim.y - 1) *cur_token = tok;               // the single-token loop continues from the last token's pick
    }
}

void destroy_graph(void* g) { cudaGraphExecDestroy((cudaGraphExec_t)g); }

void release_bufs(VerifyBufs& b) {
    b.mem.release([](void* p) { cudaFree(p); });
    b.cap = b.cap_logits = 0;
}

// Buffers of a pass over up to M tokens (logits for up to ML of them).  They grow in steps and are kept; graphs that point into
// replaced ones go with them.  After an allocation that failed there are none, and the next call starts over.
int ensure_bufs(mi_ctx* ctx, mi_model* m, int M, int ML) {
    VerifyBufs& b = m->vb;
    if (b.cap >= M && b.cap_logits >= ML) return MI_OK;
    MI_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (!b.h_meta && cudaMallocHost((void**)&b.h_meta, (3 * PMAX + 4) * sizeof(int)) != cudaSuccess) {
        b.h_meta = nullptr;
        return set_error(ctx, MI_ERR_NOMEM, "M-token step: pinned allocation failed");
    }
    b.graphs.drop_graphs(destroy_graph);
    const int cap = std::max(b.cap, M <= VMAX ? VMAX : M <= BMAX ? BMAX : PMAX), capl = std::max(b.cap_logits, ML <= VMAX ? VMAX : BMAX);
    release_bufs(b);
    auto take = [&](auto** p, size_t n) -> int {
        const size_t bytes = std::max<size_t>(n, 4) * sizeof(**p);
        if (!b.mem.take(p, bytes, [](void** q, size_t k) { return cudaMalloc(q, k) == cudaSuccess; }))
            return set_error(ctx, MI_ERR_NOMEM, "M-token step: cudaMalloc(%zu) failed: %s", bytes, cudaGetErrorString(cudaGetLastError()));
        MI_CUDA(ctx, cudaMemsetAsync(*p, 0, bytes, ctx->stream));
        return MI_OK;
    };
    auto take_tok = [&](TokX* x, int n, int tokens) -> int {
        const size_t J = (size_t)(tokens + 7) / 8 + kMaxTokNT;         // a pass may pad its token groups to whole tiles
        int st = take(&x->q, (size_t)(n / 32) * J * 64);
        return st ? st : take(&x->d, (size_t)(n / 32) * J * 8);
    };
    const int E = m->E, FF = m->FF, NQ = m->NH * m->HD;
    b.ldp = (E + 31) / 32 * 32;
    int st;
    if ((st = take(&b.X, (size_t)cap * E)) || (st = take(&b.part, (size_t)kMaxRanges * cap * b.ldp)) || (st = take(&b.q, (size_t)cap * NQ)) ||
        (st = take_tok(&b.xf, E, cap)) || (st = take_tok(&b.attf, NQ, cap)) || (st = take_tok(&b.actf, FF, cap)) ||
        (st = take(&b.att, (size_t)cap * NQ)) || (st = take(&b.Y, cap > kMaxFusedTok ? (size_t)cap * std::max(2 * FF, m->qkv_rows) : 0)) || (st = take(&b.logits, (size_t)capl * m->V)) ||
        (st = take(&b.dig, cap > kMaxFusedTok ? dig_bytes(std::max(std::max(E, NQ), FF) / 32, cap) : 0)) || (st = take(&b.dig_info, (size_t)kMaxRanges * cap)) ||
        (st = take(&b.dig_bias, (size_t)kMaxRanges * cap)) || (st = take(&b.meta, (size_t)3 * cap + 4)) || (st = take(&b.out, (size_t)cap)) || (st = take(&b.margins, (size_t)cap)) ||
        (st = take(&b.attn_part, attn_part_max(ctx, m->NH, m->NKV, m->HD))) ||
        (st = take(&b.pick, (size_t)capl * kPickSlices * 3)) || (st = take(&b.pick_cnt, (size_t)capl))) {
        cudaStreamSynchronize(ctx->stream);                            // (the fills of those that were made)
        release_bufs(b);
        return st;
    }
    b.cap = cap; b.cap_logits = capl;
    return MI_OK;
}

}  // namespace

void mi::free_verify_bufs(mi_model* m) {
    m->vb.graphs.drop_graphs(destroy_graph);
    release_bufs(m->vb);
    if (m->vb.h_meta) cudaFreeHost(m->vb.h_meta);
}

namespace {

// What a pass works on: M tokens, their ids and positions in device memory (meta: ids | positions | slots, or ids | first
// position for consecutive positions of one sequence), and the cache they live in.
struct Pass {
    int M;
    bool ragged;                                   // every token has a position and a cache slab of its own
    __half* kc; __half* vc; int max_seq; long long slab_stride;
    int lp_max;                                    // longest causal range among the tokens
    int head;                                      // whose logits are wanted
};
enum { HEAD_ALL, HEAD_LAST, HEAD_NONE };

// Positions that a launch sequence is planned for: captured passes of up to 160 cached positions share one plan, for 128 (one chunk: see
// plan_attn_tok; 48 sequences of the 1.5B shape at 40 positions 2.32 ms with the plan for 160, which cuts them, 2.23 so), beyond that those up to
// 512, 768, 1024, 1536, .. (the plan only cuts the ranges, it is right for any position).
int attn_bucket(int lp_max) {
    if (lp_max <= 160) return 128;
    int b = 512;
    while (b < lp_max) b *= 2;
    return b > 512 && lp_max <= b / 4 * 3 ? b / 4 * 3 : b;
}

// Every launch may overlap its predecessor's tail (each kernel waits before it touches what the predecessor wrote);
// MINFER_VERIFY_PDL=0 restores plain stream order.
int enqueue_pass(mi_ctx* ctx, mi_model* m, const Pass& a) {
    VerifyBufs& b = m->vb;
    const int E = m->E, L = m->L, V = m->V, M = a.M, NQ = m->NH * m->HD;
    DecodeParams P = m->P;
    P.kc = a.kc; P.vc = a.vc; P.max_seq = a.max_seq;
    const int* tokens = b.meta; const int* pos0 = b.meta + M; const int* pos_arr = a.ragged ? b.meta + M : nullptr; const int* slot_arr = a.ragged ? b.meta + 2 * M : nullptr;
    P.prof = nullptr;
    TokX xf = b.xf, attf = b.attf, actf = b.actf;
    const std::vector<LayerPtrs>& lp = m->layer_ptrs;
    const AttnPlan pa = plan_attn_tok(ctx, m->NH, m->NKV, m->HD, M, a.head == HEAD_ALL ? attn_bucket(a.lp_max) : a.lp_max, a.ragged);      // (the others are not captured)
    static const bool pdl = [] { const char* e = getenv("MINFER_VERIFY_PDL"); return !(e && atoi(e) == 0); }();
    const bool fused = M <= kMaxFusedTok;
    const int ML = a.head == HEAD_LAST ? 1 : M;
    const mi_weight* const mats[5] = {&m->views[0], &m->views[1], &m->views[2], &m->views[3], &m->views[4 * L]};
    GemmPlan plans[5];
    TokTiling tiles;
    int st;
    if ((st = plan_pass_products(ctx, mats, L, M, a.head == HEAD_NONE ? 0 : ML, &tiles, plans))) return st;
    const GemmPlan &po = plans[1], &pd = plans[3];
    xf.J = attf.J = actf.J = tiles.J();
    // the plans of the layer under way: which product goes over digits depends on the layer's rows too
    DigPlan dp[5];
    bool dig[5];
    int planned[5] = {-1, -1, -1, -1, -1};                             // rows out of the digits' range that dp and dig are for
    auto plan = [&](int i, const mi_weight* w) {
        if (planned[i] == w->bad_rows) return;
        const int Mi = i == 4 ? ML : M;
        dig[i] = m->products == 0 ? choose_gemm_dig(ctx, w, i, Mi, plans[i], &dp[i]) : m->products > 0 && Mi > kMaxFusedTok && plan_gemm_dig(ctx, w, i == 1 || i == 3, Mi, &dp[i]);
        planned[i] = w->bad_rows;
    };
    auto digits_for = [&](int i) { return dig[i] ? DigX{b.dig, b.dig_info, b.dig_bias, dp[i].T, dp[i].TT} : DigX{nullptr, nullptr, nullptr, 1, 1}; };
    // The product over digits has them from the kernel that makes its activations, but for the attention's output.
    auto product = [&](int i, const mi_weight* w, int mode, const GemmParams& gp) -> int {
        if (!dig[i]) return launch_gemm_tok(ctx, w, plans[i], mode, false, gp, pdl);
        if (i == 1) { const int s = launch_tok_digits(ctx, w, dp[i], gp.x, digits_for(i), gp.M, pdl); if (s) return s; }
        return launch_gemm_dig(ctx, w, dp[i], mode, digits_for(i), gp, pdl);
    };
    int d_ranges = 0;                                                  // K ranges of the down projection before
    const int nt_norm = std::min(1024, (E / 4 + 31) / 32 * 32);
    GemmParams g{};
    g.M = M;
    auto norm = [&](bool embed, int m0, int count, int ranges, const float* w, const TokX& out, const DigX& x) -> int {
        const auto kern = E <= 2048 ? (x.q ? vf_norm_quant<1, true> : vf_norm_quant<1, false>) : (x.q ? vf_norm_quant<2, true> : vf_norm_quant<2, false>);
        MI_CUDA(ctx, launch_k(pdl, kern, dim3(count), dim3(nt_norm), 0, ctx->stream, P, tokens, embed, m0, b.X, (const double*)(ranges ? b.part : nullptr), ranges,
                              (long long)M * b.ldp, b.ldp, w, out, x));
        return MI_OK;
    };
    for (int l = 0; l < L; l++) {
        const mi_weight *wqkv = &m->views[4 * l], *wo = &m->views[4 * l + 1], *wgu = &m->views[4 * l + 2], *wdn = &m->views[4 * l + 3];
        plan(0, wqkv); plan(1, wo); plan(2, wgu); plan(3, wdn);
        if ((st = norm(l == 0, 0, M, d_ranges, lp[l].attn_norm, xf, digits_for(0)))) return st;
        GemmParams gq = g;
        gq.x = xf; gq.bias = lp[l].bqkv; gq.y = b.Y;
        gq.rope = RopeParams{b.q, NQ, m->HD, P.kc, P.vc, m->KVD, a.slab_stride, l, a.max_seq, P.rope_cs, P.rope_freq, P.rope_rows, pos0, pos_arr, slot_arr};
        if ((st = product(0, wqkv, fused ? GEMM_QKV : GEMM_PLAIN, gq))) return st;
        if (!fused) MI_CUDA(ctx, launch_k(pdl, vf_rope, dim3(((int)wqkv->rows / 32 + 7) / 8, M), dim3(256), 0, ctx->stream, gq.rope, (const float*)b.Y, (int)wqkv->rows));
        const AttnParams at{b.q, P.kc, P.vc, M, m->NH, m->NKV, m->HD, m->KVD, l, a.max_seq, pos0, 0, pos_arr, slot_arr, a.slab_stride, b.att, attf, b.attn_part, 1, 1, 1};
        if ((st = launch_attn_tok(ctx, at, pa, pdl))) return st;
        GemmParams go = g; go.x = attf; go.part = b.part; go.ldp = b.ldp;
        if ((st = product(1, wo, GEMM_PART, go))) return st;
        if ((st = norm(false, 0, M, dig[1] ? dp[1].ksg : po.ksg, lp[l].ffn_norm, xf, digits_for(2)))) return st;
        GemmParams gg = g; gg.x = xf; gg.act = actf; gg.y = b.Y;
        if ((st = product(2, wgu, fused ? GEMM_GU : GEMM_PLAIN, gg))) return st;
        if (dig[3]) { if ((st = launch_swiglu_digits(ctx, wdn, dp[3], b.Y, actf, digits_for(3), M, pdl))) return st; }
        else if (!fused) MI_CUDA(ctx, launch_k(pdl, vf_swiglu, dim3((m->FF / 32 + 7) / 8, M), dim3(256), 0, ctx->stream, (const float*)b.Y, m->FF, actf));
        GemmParams gd = g; gd.x = actf; gd.part = b.part; gd.ldp = b.ldp;
        if ((st = product(3, wdn, GEMM_PART, gd))) return st;
        d_ranges = dig[3] ? dp[3].ksg : pd.ksg;
    }
    if (a.head == HEAD_NONE) return MI_OK;
    plan(4, &m->views[4 * L]);
    TokX lf = b.xf; lf.J = ML == M ? tiles.J() : tok_tiling(ML).J();
    if ((st = norm(false, M - ML, ML, d_ranges, m->P.out_norm, lf, digits_for(4)))) return st;
    GemmParams gl = g; gl.M = ML; gl.x = lf; gl.y = b.logits;
    if ((st = product(4, &m->views[4 * L], GEMM_PLAIN, gl))) return st;
    MI_CUDA(ctx, launch_k(pdl, vf_pick, dim3(kPickSlices, ML), dim3(512), 0, ctx->stream, (const float*)b.logits, (long long)V, V, b.out, b.margins, b.pick, b.pick_cnt,
                          m->P.cur_token));
    return MI_OK;
}

// The pass as a CUDA graph: the launch sequence is fixed by the number of tokens, the range of positions that its attention
// grid covers and the cache; tokens and positions live in device memory.  The first pass of a kind runs plainly, the second
// is captured - on a stream of its own, the caller's may be the legacy default stream - and replayed from then on.
// MINFER_VERIFY_GRAPH=0 runs everything plainly.  `start`: recorded when the pass is about to run, behind any capturing (which the host does for
// milliseconds while the stream waits; the time of a pass is what it costs from then on), or null.
int run_pass(mi_ctx* ctx, mi_model* m, const Pass& a, cudaEvent_t start) {
    VerifyBufs& b = m->vb;
    auto plainly = [&]() -> int {
        if (start) MI_CUDA(ctx, cudaEventRecord(start, ctx->stream));
        return enqueue_pass(ctx, m, a);
    };
    static const bool use_graph = [] { const char* e = getenv("MINFER_VERIFY_GRAPH"); return !(e && atoi(e) == 0); }();
    const int regime = attn_bucket(a.lp_max);
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (!use_graph || a.head != HEAD_ALL || cudaStreamIsCapturing(ctx->stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) return plainly();
    const PassKey key{a.M, regime, a.ragged ? 1 : 0, (const void*)a.kc, (const void*)a.vc, a.max_seq};
    bool again;
    void* graph = b.graphs.use(key, &again, destroy_graph);
    if (!graph) {
        if (!again) return plainly();
        cudaStream_t cs = nullptr, user = ctx->stream;
        MI_CUDA(ctx, cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
        cudaError_t e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
        int st = MI_OK;
        cudaGraph_t g = nullptr;
        if (e == cudaSuccess) {
            ctx->stream = cs;
            st = enqueue_pass(ctx, m, a);
            ctx->stream = user;
            e = cudaStreamEndCapture(cs, &g);
        }
        cudaStreamDestroy(cs);
        if (st != MI_OK) { if (g) cudaGraphDestroy(g); return st; }
        if (e != cudaSuccess) { if (g) cudaGraphDestroy(g); return set_error(ctx, MI_ERR_CUDA, "verify: stream capture failed: %s", cudaGetErrorString(e)); }
        cudaGraphExec_t ge = nullptr;
        e = cudaGraphInstantiate(&ge, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) return set_error(ctx, MI_ERR_CUDA, "verify: graph instantiation failed: %s", cudaGetErrorString(e));
        graph = ge;
        b.graphs.put(key, graph, destroy_graph);                       // (no pass is in flight here: every call ends with a wait)
    }
    if (start) MI_CUDA(ctx, cudaEventRecord(start, ctx->stream));
    MI_CUDA(ctx, cudaGraphLaunch((cudaGraphExec_t)graph, ctx->stream));
    return MI_OK;
}

}  // namespace

extern "C" int mi_verify(mi_ctx* ctx, mi_model* m, const int32_t* tokens_host, int M, int pos0, int32_t* out_tokens_host,
                         float* logits_dev, float* elapsed_ms) {
    if (!ctx) return MI_ERR_INVALID;
    if (!m || !tokens_host) return set_error(ctx, MI_ERR_INVALID, "verify: null argument");
    if (M < 1 || M > VMAX) return set_error(ctx, MI_ERR_LIMIT, "verify: M=%d tokens per pass; this entry point takes 1..%d", M, VMAX);
    if (pos0 < 0 || pos0 + M > m->max_seq)
        return set_error(ctx, MI_ERR_LIMIT, "verify: positions %d..%d exceed the KV cache of %d", pos0, pos0 + M - 1, m->max_seq);
    if (m->tp_world != 1) return set_error(ctx, MI_ERR_UNSUPPORTED, "verify: the M-token step runs on an unsharded model");
    for (int i = 0; i < M; i++)
        if (tokens_host[i] < 0 || tokens_host[i] >= m->V) return set_error(ctx, MI_ERR_INVALID, "verify: token id %d out of range", tokens_host[i]);
    MI_CUDA(ctx, cudaSetDevice(ctx->device));
    int st;
    if ((st = ensure_bufs(ctx, m, M, M))) return st;
    VerifyBufs& b = m->vb;
    if ((st = mi::reset_after_error(ctx, m))) return st;
    memcpy(b.h_meta, tokens_host, (size_t)M * 4);                     // pinned: free again once the call has synchronized below
    b.h_meta[M] = pos0;
    MI_CUDA(ctx, cudaMemcpyAsync(b.meta, b.h_meta, (size_t)(M + 1) * 4, cudaMemcpyHostToDevice, ctx->stream));
    if ((st = run_pass(ctx, m, Pass{M, false, m->P.kc, m->P.vc, m->max_seq, 0, pos0 + M, HEAD_ALL}, m->ev0))) return st;
    MI_CUDA(ctx, cudaEventRecord(m->ev1, ctx->stream));
    if (logits_dev) MI_CUDA(ctx, cudaMemcpyAsync(logits_dev, b.logits, (size_t)M * m->V * 4, cudaMemcpyDeviceToDevice, ctx->stream));
    if (out_tokens_host) MI_CUDA(ctx, cudaMemcpyAsync(b.h_meta, b.out, (size_t)M * 4, cudaMemcpyDeviceToHost, ctx->stream));
    st = mi_ctx_sync(ctx);
    if (st != MI_OK) return st;
    if (out_tokens_host) memcpy(out_tokens_host, b.h_meta, (size_t)M * 4);
    if (elapsed_ms) MI_CUDA(ctx, cudaEventElapsedTime(elapsed_ms, m->ev0, m->ev1));
    return MI_OK;
}

extern "C" int mi_prefill(mi_ctx* ctx, mi_model* m, const int32_t* tokens_host, int n, int pos0, int32_t* next_token_host, float* elapsed_ms) {
    if (!ctx) return MI_ERR_INVALID;
    if (!m || !tokens_host || n < 1) return set_error(ctx, MI_ERR_INVALID, "prefill: null argument, or no tokens");
    if (pos0 < 0 || (long long)pos0 + n > m->max_seq)
        return set_error(ctx, MI_ERR_LIMIT, "prefill: positions %d..%lld exceed the KV cache of %d", pos0, (long long)pos0 + n - 1, m->max_seq);
    if (m->tp_world != 1) return set_error(ctx, MI_ERR_UNSUPPORTED, "prefill: the M-token step runs on an unsharded model");
    for (int i = 0; i < n; i++)
        if (tokens_host[i] < 0 || tokens_host[i] >= m->V) return set_error(ctx, MI_ERR_INVALID, "prefill: token id %d out of range", tokens_host[i]);
    MI_CUDA(ctx, cudaSetDevice(ctx->device));
    int st;
    if ((st = ensure_bufs(ctx, m, std::min(n, PMAX), 1))) return st;
    VerifyBufs& b = m->vb;
    if ((st = mi::reset_after_error(ctx, m))) return st;
    MI_CUDA(ctx, cudaEventRecord(m->ev0, ctx->stream));
    // passes of equal size (to one token), so that the last one is not a small one at a large one's latency
    const int passes = (n + PMAX - 1) / PMAX;
    for (int k = 0; k < passes; k++) {
        const int i0 = (int)((long long)n * k / passes), M = (int)((long long)n * (k + 1) / passes) - i0;
        if (k > 0) MI_CUDA(ctx, cudaEventSynchronize(m->ev1));         // the pinned block has been copied
        memcpy(b.h_meta, tokens_host + i0, (size_t)M * 4);
        b.h_meta[M] = pos0 + i0;
        MI_CUDA(ctx, cudaMemcpyAsync(b.meta, b.h_meta, (size_t)(M + 1) * 4, cudaMemcpyHostToDevice, ctx->stream));
        MI_CUDA(ctx, cudaEventRecord(m->ev1, ctx->stream));
        if ((st = run_pass(ctx, m, Pass{M, false, m->P.kc, m->P.vc, m->max_seq, 0, pos0 + i0 + M, k == passes - 1 ? HEAD_LAST : HEAD_NONE}, nullptr))) return st;
    }
    MI_CUDA(ctx, cudaEventRecord(m->ev1, ctx->stream));
    if (next_token_host) MI_CUDA(ctx, cudaMemcpyAsync(b.h_meta, b.out, 4, cudaMemcpyDeviceToHost, ctx->stream));
    if ((st = mi_ctx_sync(ctx))) return st;
    if (next_token_host) *next_token_host = b.h_meta[0];
    if (elapsed_ms) MI_CUDA(ctx, cudaEventElapsedTime(elapsed_ms, m->ev0, m->ev1));
    return MI_OK;
}

extern "C" int mi_model_debug_products(mi_ctx* ctx, mi_model* m, int which) {
    if (!ctx) return MI_ERR_INVALID;
    if (!m || which < -1 || which > 1) return set_error(ctx, MI_ERR_INVALID, "debug_products: %d", which);
    MI_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    m->products = which;
    m->vb.graphs.drop_graphs(destroy_graph);
    return MI_OK;
}

extern "C" int mi_verify_margins(mi_ctx* ctx, mi_model* m, int n, float* margins_host) {
    if (!ctx) return MI_ERR_INVALID;
    if (!m || !margins_host || n < 0 || n > VMAX || !m->vb.margins) return set_error(ctx, MI_ERR_INVALID, "verify_margins: bad argument, or no M-token pass has run");
    if (n == 0) return MI_OK;
    MI_CUDA(ctx, cudaMemcpyAsync(margins_host, m->vb.margins, (size_t)n * 4, cudaMemcpyDeviceToHost, ctx->stream));
    MI_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return MI_OK;
}

extern "C" int mi_attn_splitkv(mi_ctx* ctx, const float* q_dev, const uint16_t* kcache_dev, const uint16_t* vcache_dev, int n_head,
                               int n_head_kv, int head_dim, int pos0, int M, float* out_dev) {
    if (!ctx) return MI_ERR_INVALID;
    if (!q_dev || !kcache_dev || !vcache_dev || !out_dev) return set_error(ctx, MI_ERR_INVALID, "attention: null argument");
    if (M < 1 || M > VMAX) return set_error(ctx, MI_ERR_LIMIT, "attention: M=%d queries per call; this entry point takes 1..%d", M, VMAX);
    if (n_head <= 0 || n_head_kv <= 0 || n_head % n_head_kv || pos0 < 0) return set_error(ctx, MI_ERR_INVALID, "attention: bad head counts or position");
    MI_CUDA(ctx, cudaSetDevice(ctx->device));
    AttnPlan plan = plan_attn_tok(ctx, n_head, n_head_kv, head_dim, M, pos0 + M, false);
    // inside a stream capture nothing may be allocated: without the scratch the range stays in one piece
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (plan.part_doubles > ctx->part_count && cudaStreamIsCapturing(ctx->stream, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusActive) { plan.nch = 1; plan.part_doubles = 0; }
    int st = ensure_scratch(ctx, plan.part_doubles, 0);
    if (st != MI_OK) return st;
    const AttnParams p{q_dev, reinterpret_cast<const __half*>(kcache_dev), reinterpret_cast<const __half*>(vcache_dev), M, n_head, n_head_kv, head_dim, n_head_kv * head_dim,
                       0, 0, nullptr, pos0, nullptr, nullptr, 0, out_dev, TokX{nullptr, nullptr, 0}, ctx->part, 1, 1, 0};
    return launch_attn_tok(ctx, p, plan, true);
}

// ---- batched decode of independent sequences -------------------------------------------------------------
// One step of up to B sequences per call: the current token of each goes through ONE pass over the weights as a column
// of the M-token step (up to 64 columns per pass; larger batches run several passes), with its own position and its
// own slab of a KV cache that belongs to the batch object.  Every column is processed exactly as if it were alone, so
// a sequence's ids and logits are the bits of its batch-1 run, whatever else shares the pass.  The reference serves one
// sequence at a time (README.md:54); the closest code is gemv_dp4a_batch<T> (src/cuda_infer.cu:183-222).
struct mi_batch {
    mi_model* model = nullptr;
    int n_slots = 0, max_seq = 0;
    __half* kc = nullptr; __half* vc = nullptr;       // [slot][layer][max_seq][KVD]
    long long slab_stride = 0;
};

extern "C" int mi_batch_create(mi_ctx* ctx, mi_model* m, int n_slots, int max_seq, mi_batch** out) {
    if (!ctx) return MI_ERR_INVALID;
    if (!m || !out || n_slots < 1 || max_seq < 1) return set_error(ctx, MI_ERR_INVALID, "batch_create: bad argument");
    if (m->tp_world != 1) return set_error(ctx, MI_ERR_UNSUPPORTED, "batch_create: the M-token step runs on an unsharded model");
    *out = nullptr;
    MI_CUDA(ctx, cudaSetDevice(ctx->device));
    mi_batch* b = new (std::nothrow) mi_batch();
    if (!b) return set_error(ctx, MI_ERR_NOMEM, "batch_create: host allocation failed");
    b->model = m; b->n_slots = n_slots; b->max_seq = max_seq;
    b->slab_stride = (long long)m->L * max_seq * m->KVD;
    const size_t bytes = (size_t)n_slots * (size_t)b->slab_stride * sizeof(__half);
    if (cudaMalloc(&b->kc, bytes) != cudaSuccess || cudaMalloc(&b->vc, bytes) != cudaSuccess) {
        cudaFree(b->kc); cudaFree(b->vc); delete b;
        return set_error(ctx, MI_ERR_NOMEM, "batch_create: %d KV slabs of %zu bytes do not fit", n_slots, bytes / n_slots);
    }
    *out = b;
    return MI_OK;
}

extern "C" int mi_batch_free(mi_ctx* ctx, mi_batch* b) {
    if (!b) return MI_OK;
    if (ctx) { cudaSetDevice(ctx->device); cudaStreamSynchronize(ctx->stream); }
    cudaFree(b->kc); cudaFree(b->vc);
    delete b;
    return MI_OK;
}

extern "C" int mi_batch_step(mi_ctx* ctx, mi_batch* b, int n, const int32_t* tokens_host, const int32_t* slots_host, const int32_t* positions_host,
                             int32_t* out_tokens_host, float* logits_dev, float* elapsed_ms) {
    if (!ctx) return MI_ERR_INVALID;
    if (!b || !tokens_host || !slots_host || !positions_host || n < 1) return set_error(ctx, MI_ERR_INVALID, "batch_step: bad argument");
    mi_model* m = b->model;
    for (int i = 0; i < n; i++) {
        if (tokens_host[i] < 0 || tokens_host[i] >= m->V) return set_error(ctx, MI_ERR_INVALID, "batch_step: token id %d out of range", tokens_host[i]);
        if (slots_host[i] < 0 || slots_host[i] >= b->n_slots) return set_error(ctx, MI_ERR_INVALID, "batch_step: slot %d of %d", slots_host[i], b->n_slots);
        if (positions_host[i] < 0 || positions_host[i] >= b->max_seq)
            return set_error(ctx, MI_ERR_LIMIT, "batch_step: position %d outside the KV slab of %d", positions_host[i], b->max_seq);
        for (int j = 0; j < i; j++)
            if (slots_host[j] == slots_host[i]) return set_error(ctx, MI_ERR_INVALID, "batch_step: slot %d appears twice in one step", slots_host[i]);
    }
    MI_CUDA(ctx, cudaSetDevice(ctx->device));
    int st;
    if ((st = ensure_bufs(ctx, m, std::min(n, BMAX), std::min(n, BMAX)))) return st;
    VerifyBufs& vb = m->vb;
    if ((st = mi::reset_after_error(ctx, m))) return st;
    for (int i0 = 0; i0 < n; i0 += BMAX) {
        const int M = std::min(BMAX, n - i0);
        memcpy(vb.h_meta, tokens_host + i0, (size_t)M * 4);
        memcpy(vb.h_meta + M, positions_host + i0, (size_t)M * 4);
        memcpy(vb.h_meta + 2 * M, slots_host + i0, (size_t)M * 4);
        const int lp_max = *std::max_element(positions_host + i0, positions_host + i0 + M) + 1;
        MI_CUDA(ctx, cudaMemcpyAsync(vb.meta, vb.h_meta, (size_t)3 * M * 4, cudaMemcpyHostToDevice, ctx->stream));
        if ((st = run_pass(ctx, m, Pass{M, true, b->kc, b->vc, b->max_seq, b->slab_stride, lp_max, HEAD_ALL}, i0 == 0 ? m->ev0 : nullptr))) return st;
        if (logits_dev) MI_CUDA(ctx, cudaMemcpyAsync(logits_dev + (size_t)i0 * m->V, vb.logits, (size_t)M * m->V * 4, cudaMemcpyDeviceToDevice, ctx->stream));
        if (i0 + BMAX >= n) MI_CUDA(ctx, cudaEventRecord(m->ev1, ctx->stream));
        if (out_tokens_host) MI_CUDA(ctx, cudaMemcpyAsync(vb.h_meta, vb.out, (size_t)M * 4, cudaMemcpyDeviceToHost, ctx->stream));
        if ((st = mi_ctx_sync(ctx))) return st;                                    // (the pinned block is filled again by the next pass)
        if (out_tokens_host) memcpy(out_tokens_host + i0, vb.h_meta, (size_t)M * 4);
    }
    if (elapsed_ms) MI_CUDA(ctx, cudaEventElapsedTime(elapsed_ms, m->ev0, m->ev1));
    return MI_OK;
}

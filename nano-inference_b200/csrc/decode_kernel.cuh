// The fused decode step for sm_100a: one persistent kernel that runs any range of
// the per-token phases
//     per layer:  QKV  (residual add -> rmsnorm -> q8 -> GEMV -> +bias, RoPE, q / k / v)
//                 ATTN (split-KV attention over the fp16 cache, merge, -> q8)
//                 O    (GEMV)
//                 GU   (residual add -> rmsnorm -> q8 -> gate & up GEMV -> SwiGLU -> q8)
//                 DOWN (GEMV, K-split over CTAs, folded by the split-0 CTA)
//     finally:    LM   (residual add -> rmsnorm -> q8 -> lm_head GEMV -> argmax)
// for any range of steps.  Launched with one phase per launch it is a plain
// kernel sequence; launched cooperatively (all CTAs resident) over all phases and
// steps it is the persistent decode loop.
//
// No grid barrier.  The reference's persistent kernel separates its phases by a
// grid-wide barrier (src/mega.cu:123-134, five per layer).  Here every value that
// one CTA hands to another travels as a TAGGED WORD: 8 bytes = {32-bit payload,
// 32-bit tag}, written and read as one naturally aligned 64-bit access (single-copy
// atomic).  The tag numbers the (step, phase) that produced the value.  A consumer
// simply loads the words it needs and looks at their tags; words that are not there
// yet are polled (bounded by a time budget).  There is no separate flag, hence no
// release fence before it and no second round trip after it (what travels beside the words, rows of the KV cache and partial sums of
// the long-range attention, has fences of its own): a phase boundary costs
// one store-to-load hop through the L2 instead of arrive + poll + reload, and a CTA
// waits only for the values it actually consumes.  Buffers are reused every layer;
// a word is overwritten only after every reader has passed on, because the
// writer's own inputs descend from outputs of those readers.  The readers of q / k / v, of
// the attention output, of the activations, of chunk maxima and of partial sums publish something of the same phase
// that the next writer needs.  The words of the O and of the down projection are read by every GEMV CTA: one with
// a unit of QKV or of gate/up has read both before it publishes that unit's rows, which all later writers of either need (a unit of O alone or of down alone
// protects one of the two).  A CTA with neither publishes in its place a word of the attention phase, which says
// that it has read them and which the CTAs of the O projection await with the attention output (bystanders).
// (A GPU of a tensor-parallel group that has no unit of gate/up, fewer groups of 32 than GPUs, is not held by this.)  A reader that
// nevertheless fell behind would see a wrong tag and time out - never wrong data.
// The same words, stored additionally into the other GPUs' copies of the buffers
// over NVLink (plain 8-byte peer stores), are the whole tensor-parallel exchange.
//
// The residual stream lives in shared memory: every CTA adds the same projection
// outputs to its own copy (the arithmetic is deterministic, all copies hold the
// same bits), so it never travels.  The first GEMV CTA also writes it to global memory
// for launches that start in the middle of a step, and for inspection.
//
// Work split.  Every GEMV phase is a "job" over a tiled q4_0 matrix.  For the
// per-layer matrices a unit is a 32-row group (gate/up: a pair of groups), half of one where that leaves no CTA
// with two, or (group, K-split), and belongs to a CTA: its eight warps take the tiles of all its units round-robin and
// fold their double partial sums through shared memory.  Where a down projection has
// fewer row groups than the grid has CTAs and halves would be too many, its K dimension is split
// across CTAs; splits 1.. hand their double partial sums (two tagged words each) to
// the CTA of split 0, which adds them in split order and publishes the fp32 row.
// The lm_head has thousands of row groups: there a unit is a row group and belongs
// to one warp.
//
// Weight streaming.  The whole tile sequence of a warp - across phases, layers
// and steps - follows from shapes and indices alone, so a ninth warp keeps the eight
// private shared-memory rings full with bulk copies that run ahead of
// the phase boundaries: weights are immutable, the HBM stream never waits for a
// phase, only for ring space.
//
// Numerics follow the reference (paths relative to its root): quantizer
// src/cuda_infer.cu:80-89; block dot src/mega.cu:151-165; RMSNorm / RoPE / SwiGLU /
// argmax src/cpu_infer.cpp:40-61,147,153-154; split-KV merge
// src/cuda_infer.cu:650-702.  Every sum that feeds a stored tensor (GEMV rows,
// RMSNorm sum of squares, attention scores, softmax denominator and weighted
// values) is carried in double and rounded to fp32 once; exp, cos and sin come
// from the double math library.  A q8_0 quantizer is discontinuous, so this is
// what lets two engines (or two split / step / shard configurations of this one)
// agree bit for bit: every term of a GEMV sum is a multiple of 2^-48 (fp16 x fp16 x
// integer), so while a sum stays below 2^5 in magnitude the double additions are
// exact and the fp32 value cannot depend on their order; beyond that it has been
// observed, not proved.  Each token is processed exactly as if it were alone.
#pragma once
#include "gemv_core.cuh"
#include "decode_deal.cuh"
// functions that sit out of line to keep the loop body small; the short-context build inlines them instead, because every
// call site inside the step loop, executed or not, makes the compiler keep the loop's values where a call preserves them
#if defined(MI_LEAN) && MI_LEAN
#define MI_COLD_FN static __device__ __forceinline__
#else
#define MI_COLD_FN static __device__ __noinline__
#endif

// The kernel exists in several builds.  The default one carries no profiling code and no peer stores.  A translation unit
// that defines MI_PROF 1 before including this file gets the instrumented build (timer marks between the hot instructions
// cost a few percent when merely compiled in); MI_TP 1 gives the tensor-parallel build, whose publishing stores also go to
// the other GPUs; MI_LEAN 1 gives the short-context build, which holds no attention code but that of the dedicated attention
// CTAs (launched only for step ranges that end within kShortAttnMax positions on a model with such CTAs: without the other
// attention variants in the same function the GEMV CTAs' loop keeps its values in registers); MI_LEAN 2 is the same idea for
// more than kShortAttnMax positions (attention_split); MI_SMALL 1 makes either one for narrow models (lean_shape).  They live in
// different inline namespaces, so all can be linked into one library and picked at launch time.
#ifndef MI_PROF
#define MI_PROF 0
#endif
#ifndef MI_TP
#define MI_TP 0
#endif
#ifndef MI_LEAN
#define MI_LEAN 0
#endif
#ifndef MI_SMALL
#define MI_SMALL 0
#endif
#if MI_PROF && MI_SMALL && MI_LEAN == 2
#define MI_KVARIANT profsmalllong
#elif MI_PROF && MI_SMALL && MI_LEAN
#define MI_KVARIANT profsmall
#elif MI_PROF && !MI_TP && MI_LEAN == 2
#define MI_KVARIANT proflong
#elif MI_SMALL && MI_LEAN == 2
#define MI_KVARIANT leansmalllong
#elif MI_SMALL && MI_LEAN
#define MI_KVARIANT leansmall
#elif MI_PROF && MI_TP && MI_LEAN
#define MI_KVARIANT tpxproflean
#elif MI_PROF && MI_LEAN
#define MI_KVARIANT proflean
#elif MI_PROF
#define MI_KVARIANT prof
#elif MI_TP && MI_LEAN
#define MI_KVARIANT tpxlean
#elif MI_TP
#define MI_KVARIANT tpx
#elif MI_LEAN == 2
#define MI_KVARIANT leanlong
#elif MI_LEAN
#define MI_KVARIANT lean
#else
#define MI_KVARIANT fast
#endif

namespace mi {

constexpr int DNT_ALL = DNT + 32; // and one warp that requests the weights
constexpr int DS = 3;             // ring slots per warp
constexpr int DSLOT = 4608;       // bytes per slot: the largest tile (8 blocks)
constexpr int kAttnChunk = 32;    // smallest KV range worth its own CTA
constexpr int kShortAttnMax = 256;      // up to this many cached positions one CTA handles the whole range of a query head (attention_short)
constexpr int kMaxWorldTP = 8;
constexpr int kXCopies = 8;       // copies of the exchange block (see Pub)

// profile slots: 2*k = staging of phase kind k, 2*k+1 = its main work; 12 = time spent waiting for tagged words, 13 = step prologue
enum { kProfWait = 12, kProfStep = 13, kProfSlots = 32 };

// What a CTA does in the per-layer jobs, listed by the host (all layers are dealt alike): 32-bit words, [kind] = offset of the job's first batch, or 0.
// A batch is up to kBatchUnits units; its tiles, numbered unit by unit, accumulator by accumulator (gate, up), along K, go round-robin over the eight warps:
//   [0] number of units | offset of the next batch << 8, or 0      [1 + b] unit b: its q8_0 block (gate/up), else its first row
//   [5 + b] K-split of unit b | number of warps with tiles of a sum << 8 | first of them << 16 (gate), << 20 (up)
//   [9 + w] offset of warp w's list | number of its tiles << 16;  list entry: first block | sum (2 b + accumulator) << 16 | last of the sum << 20 | second half of the rows << 21
// Where twice the row groups of a job are no more than the CTAs, its units are half row groups (DecodeParams::half_rows): both CTAs of a group read its tiles, the second one from
// the L2, and a lane has a row of sixteen and half of a tile's blocks.  The down projection of the 1.5B shape is 35 tiles on 96 CTAs instead of 48 so.
enum { kBatchGroup = 1, kBatchUnit = kBatchGroup + kBatchUnits, kBatchList = kBatchUnit + kBatchUnits, kBatchWords = kBatchList + 8 };

struct LayerPtrs { const float* attn_norm; const float* ffn_norm; const float* bqkv; };

// Tensor parallelism inside the kernel: the other GPUs' exchange blocks (CUDA IPC mappings).  on == 0: single GPU, or
// exchanges done by the host program between launches.
struct TpPeerParams {
    int on, rank, world, pad_;
    unsigned long long* xw_peer[kMaxWorldTP];     // exchange block on every GPU (own entry = local block)
};

// Offsets (in 8-byte words) of the tagged vectors inside the exchange block.  q8_0 vectors are stored as
// [n/4] words of four int8 values followed by [n/32 (+1 if odd)] words of {fp16 scale bits | int16 sum of the block's values << 16}.
struct XwLayout {
    int qkv;        // [qkv rows, padded to 32]   fp32 bits: q | k | v after bias and RoPE, packed (pair-adjacent) order
    int att;        // q8_0 of the merged attention output [NH*HD]; behind its scales a word of every CTA without a unit of QKV and gate/up (see bystanders)
    int o;          // [E] fp32 bits: O projection
    int act;        // q8_0 of SwiGLU(gate, up) [FF]                                     (pushed to the other GPUs)
    int down;       // [E] fp32 bits: down projection                                    (pushed)
    int dpart;      // [E/32][kMaxKSplit-1][32][2]: double partial sums (lo, hi) of the down K-splits 1..
    int cand;       // [kMaxWorldTP][grid][4]: argmax candidates {best value}, {its row}, {second-best value}, -   (pushed)
    int attm;       // [NH][max_chunks] fp32 bits: maximum of every chunk of the long-range attention
    int tokw;       // [2]: the token picked by the step that just ended, for the attention CTAs (written only under a stop rule)
    int attdone;    // [2][attn_ctas]: by step parity, "this attention CTA has left the step" (see rows_ordered)
    int total;
};

// Host-mapped (pinned, device-visible) memory through which a running generation hands its tokens to the host
// (src/mega.cu:1130-1137): the kernel fills tokens / margins / ns from entry `base` on and raises *count.
struct TokenRing { int* count; int* tokens; float* margins; unsigned long long* ns; int capacity, base; };

struct DecodeParams {
    int L, E, FF, NH, NKV, HD, KVD, V;
    float eps;
    double inv_e;                    // 1 / E
    const unsigned* work; int work_stride, work_smem;      // per GEMV CTA: its list (see above); whether it goes to shared memory
    int fold_at;                                           // byte of the shared memory where the sums of a batch meet (decode_fold_at)
    int seen_first, seen_n, att_scales;                    // GEMV CTAs without a unit of QKV and gate/up (bystanders); scales of the attention output and those CTAs' words
    int kb[5], ks_down, half_rows;                         // tile depths by JobKind, K-splits of the down projection, which jobs' units are half row groups (bit per JobKind)
    int lm_units, lm_nt, lm_off;                           // lm_head: row groups and tiles of one, first row group
    const unsigned long long* tile_tab;   // per warp: source address | kb code of every tile of one step, in consumption order
    const unsigned* tile_start;      // [grid*DNW][4L+2]: index of each job's first tile in the warp's list (last = count)
    int tile_stride;                 // entries reserved per warp in tile_tab
    const LayerPtrs* layers;         // [L]
    const float* out_norm;
    const float* rope_freq;          // [HD/2]: base^(-2i/HD), computed on the host with powf
    const float* rope_cs;            // [rope_rows][HD]: cos then sin of every position's HD/2 angles, made once at load (rope_cs_kernel)
    int rope_rows;                   // = the model's max_seq at load
    const uint8_t* emb_base;         // tiled token embedding (may alias the lm_head)
    int emb_nt, emb_kb;
    const uint8_t* emb_q8;           // or, when set: the embedding as stored Q8_0 rows (34-byte blocks), read instead of emb_base
    // residual stream as committed by CTA 0: read by a launch that starts in the middle of a step, and by tests
    float* h_in;                     // at the input of the current layer
    float* h_mid;                    // after the attention block
    // the exchange block: every vector one CTA hands to another, as tagged words
    unsigned long long* xw; XwLayout xo;
    int copies;                      // how many copies of the block consumers read (1: tensor parallelism, whose exchanges write the first one only)
    // Tag of (step s of the launch, phase p) = epoch + s * (5L+1) + p + 1.  The epoch lives in device memory and the kernel
    // advances it itself: a launch whose phase range ends a step leaves it past every tag the launch used (a launch that
    // gave up on a wait: further still).  Replayed launch sequences and calls after a failure therefore never meet a stale
    // word with a matching tag; launches that continue a step (phase range not starting at 0) share its epoch.
    unsigned* epoch_dev;
    unsigned long long wait_ns;      // time budget of every device-side wait
    int drop_phase;                  // test hook: the producers of this phase publish nothing (-1: none), so that its consumers' waits run out
    int hold_us;                     // test hook of the instrumented builds: CTA prof_cta comes this much late to every norm prologue
    float* att;                      // merged attention output, fp32, for inspection
    __half* kc; __half* vc; int max_seq;       // [L][max_seq][KVD]
    double* attn_part; int max_chunks, split_sub;       // [NH][max_chunks][HD+2]: weighted sums and denominator of every chunk (attention_split)
    float* out_margins;              // optional [n_steps]: top-1 minus top-2 logit of every step
    TokenRing ring;                  // optional: host-mapped ring the first GEMV CTA publishes every step's token into
    float* best_val;                 // value of the best logit (tensor parallelism with host-side exchange: this GPU's rows only)
    const int* in_tokens; int n_forced; int* out_tokens; int* cur_token;
    int stop_token;                  // >= 0: a run over whole steps ends after the step that picks this token as the next input
                                     // (text generation's end-of-sequence rule, src/mega.cu:868-874); -1: off
    float* logits; long long logits_stride;    // optional [n_steps][stride]
    int pos0;
    const int* pos_dev;              // optional: first position read from device memory instead (a captured launch sequence stays position-free)
    int* err;
    unsigned long long* prof;        // optional [32]: nanoseconds per phase part on CTA prof_cta (see kProf*)
    int prof_cta;
    // CTAs [0, attn_ctas) do nothing but attention; the GEMV phases (and the greedy pick) are dealt over the other
    // CTAs [attn_ctas, grid).  At short context one CTA per query head runs attention, and a CTA that also carried GEMV
    // units would walk both phases' code every layer; kept apart, each CTA's instructions stay in its instruction cache.
    // 0: every CTA does everything.  Beyond kShortAttnMax positions the GEMV CTAs take attention chunks as well.
    int attn_ctas;
    TpPeerParams tp;
};

// number of KV chunks for a causal range of Lp positions (host and device agree)
__host__ __device__ inline int attn_chunks(int Lp, int max_chunks) {
    int n = (Lp + kAttnChunk - 1) / kAttnChunk;
    return n < 1 ? 1 : (n > max_chunks ? max_chunks : n);
}
__host__ __device__ inline int q8_words(int n) { return n / 4 + (n / 32 + 1) / 2 * 2; }     // tagged words of a q8_0 vector of n values

#ifdef __CUDACC__
inline namespace MI_KVARIANT {

struct DecodeSmem {
    uint8_t* ring; uint64_t* bars; const unsigned* work; LayerPtrs* lp; float* cs; double* red; double* fold; float* h; uint8_t* stage;
};

constexpr int kWorkSmem = 512;                        // words of a CTA's list that fit the shared memory

// attention_split: positions per step (as many as the shared memory allows: a chunk that fits one step has all its rows requested
// before q is waited for; 8192 positions in two steps of 64 instead of one of 112: 3.9 instead of 2 us for the scores), words of
// chunk maxima a lane polls (up to 160 chunks per kv head), layout of its staging area
constexpr int kSplitSubMin = 64, kSplitSubMax = 128, kMaxChunkWords = 5;
struct SplitSmem {
    int HD, sub;
    __host__ __device__ int kld() const { return 2 * HD + 64; }                          // row strides: fragment loads without bank conflicts
    __host__ __device__ int vld() const { return 2 * HD + 32; }
    __host__ __device__ int scl() const { return sub + 4; }
    __host__ __device__ int wt() const { return 8 * HD * 8; }                            // q comes first
    __host__ __device__ int k() const { return wt() + 8 * sub * 8; }
    __host__ __device__ int v() const { return k() + sub * kld(); }
    __host__ __device__ int sc() const { return v() + sub * vld(); }
    __host__ __device__ int st() const { return sc() + 8 * scl() * 4; }
    __host__ __device__ int red() const { return st() + 8 * 3 * 8; }
    __host__ __device__ int bytes() const { return red() + DNW * 33 * 8; }
};

__host__ __device__ inline size_t decode_stage_bytes(int E, int FF, int HD, int sub) {
    const int maxin = E > FF ? E : FF;
    size_t a = (size_t)maxin + (size_t)(maxin / 32) * 8;               // xq, xs (bystanders' words behind the latter: where there are any, maxin is below 32 times the grid and b is more than enough)
    const size_t split = SplitSmem{HD, sub}.bytes();
    const size_t shrt = (size_t)(8 * (HD / 8 + 2) + 256 + DNW * HD + DNW) * 8 + 1024;                // attention_short
    const size_t b = split > shrt ? split : shrt;
    return ((a > b ? a : b) + 127) / 128 * 128;
}
// where the sums of a batch of `units` meet ([unit][acc][warp][lane] doubles), behind everything else
__host__ __device__ inline size_t decode_fold_at(int E, int FF, int HD, int sub) {
    return (size_t)DNW * DS * DSLOT + 512 + kWorkSmem * 4 + 64 * sizeof(LayerPtrs) + 1024 + 256 +
           ((size_t)E * 4 + 127) / 128 * 128 + decode_stage_bytes(E, FF, HD, sub);
}
__host__ __device__ inline size_t decode_smem_bytes(int E, int FF, int HD, int sub, int units) {
    return decode_fold_at(E, FF, HD, sub) + (size_t)units * 2 * DNW * 32 * 8;
}

// close the current profile interval: charge the time since t to slot k (CTA 0, thread 0 only).
// The sums live in shared memory and are flushed once at kernel exit, so a mark costs a
// timer read and a shared-memory add, not a global round trip on the critical path.
#if MI_PROF
__shared__ unsigned long long s_prof[kProfSlots];
__shared__ unsigned long long s_prof_t;          // start of the open interval (thread 0 of the profiled CTA)
#endif
__device__ __forceinline__ void prof_mark(const DecodeParams& P, int k) {
#if MI_PROF
    if (P.prof && (int)blockIdx.x == P.prof_cta && threadIdx.x == 0) { const unsigned long long n = gtime_ns(); s_prof[k] += n - s_prof_t; s_prof_t = n; }
#endif
}

// A greedy-pick candidate: best value, its row (lowest row wins ties), and the runner-up value.
struct Cand {
    float best; int idx; float second;
    __device__ __forceinline__ void add(float v, int r) {
        if (v > best || (v == best && r < idx)) { second = best; best = v; idx = r; }
        else if (v > second) second = v;
    }
    __device__ __forceinline__ void merge(const Cand& o) {
        if (o.best > best || (o.best == best && o.idx < idx)) { second = fmaxf(best, o.second); best = o.best; idx = o.idx; }
        else second = fmaxf(second, o.best);
    }
    __device__ __forceinline__ void warp_reduce() {
        #pragma unroll
        for (int s = 16; s; s >>= 1) {
            Cand o;
            o.best = __shfl_xor_sync(0xffffffffu, best, s); o.idx = __shfl_xor_sync(0xffffffffu, idx, s); o.second = __shfl_xor_sync(0xffffffffu, second, s);
            merge(o);
        }
    }
};

// Barriers of the warps that compute (the one that requests weights has no part in them)
__device__ __forceinline__ void cta__syncthreads() { asm volatile("bar.sync 1, %0;" ::"n"(DNT) : "memory"); }
__device__ __forceinline__ int cta__syncthreads_and(int p) {
    int r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.and.pred q, 1, %2, p;\n\tselp.s32 %0, 1, 0, q;\n\t}" : "=r"(r) : "r"(p), "n"(DNT) : "memory");
    return r;
}

// ---- tagged words ---------------------------------------------------------------------
// One 64-bit access carries value and tag together, so there is nothing to order between them.
// The accesses are volatile: they are performed at the L2 (the point where all SMs of this GPU,
// and peers storing over NVLink, meet), once each, in program order.
__device__ __forceinline__ unsigned long long tw_ld(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.volatile.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void tw_ld2(const unsigned long long* p, unsigned long long& a, unsigned long long& b) {   // 16-byte aligned pair; each word is checked on its own
    asm volatile("ld.volatile.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ void tw_st(unsigned long long* p, unsigned tag, unsigned payload) {
    asm volatile("st.volatile.global.u64 [%0], %1;" ::"l"(p), "l"(((unsigned long long)tag << 32) | payload) : "memory");
}
__device__ __forceinline__ bool tw_is(unsigned long long w, unsigned tag) { return (unsigned)(w >> 32) == tag; }

// Where a phase publishes.  What (nearly) every CTA reads goes into kXCopies copies of the exchange block, and CTA i reads copy i % P.copies: a vector is a hundred lines of the
// L2 or less, each read by 142 CTAs, and the slices that hold several of them were what the words waited for.  Where a copy's lines lie decides much: a model loaded
// eight times in one process, us per token, mean (least - most), with 1, 2, 4 and 8 copies:
//   1.5B shape 582 (570 - 608), 547 (541 - 556), 521 (515 - 535), 521 (516 - 526)        behind 8192 positions 868 (809 - 920), 832 (773 - 870), 780 (753 - 856), 819 (790 - 842)
//   0.5B shape 371 (347 - 383), 382 (378 - 384), 372 (366 - 376), 369 (366 - 373)        3B shape 827 (797 - 855), 817 (803 - 844), 797 (787 - 802), 801 (793 - 830)
// Words with few readers are in the first copy only.  The tensor-parallel build, whose shared vectors also go into every other GPU's block, writes and reads the first copy alone
// (that build without a peer, mean of eight loads: 1.5B shape 536, with the vectors that stay on this GPU in eight copies 577).  A sharded model that the host drives writes
// all copies and reads the first: one store there would be a test in every publish here (0.6 % of that form's time against 0.9 % of every token).
struct Pub {
    unsigned long long* xw; unsigned tag; bool mute; int stride;
#if MI_TP
    const TpPeerParams* tp;
#endif
    __device__ __forceinline__ void local(int off, unsigned payload) const { if (!mute) tw_st(xw + off, tag, payload); }
    __device__ __forceinline__ void all(int off, unsigned payload) const {
        if (mute) return;
        #pragma unroll
        for (int r = 0; r < (MI_TP ? 1 : kXCopies); r++) tw_st(xw + off + r * stride, tag, payload);
    }
    __device__ __forceinline__ void shared(int off, unsigned payload) const {
        all(off, payload);
#if MI_TP
        if (mute) return;
        if (tp->on) {
            for (int p = 0; p < tp->world; p++) if (p != tp->rank) tw_st(tp->xw_peer[p] + off, tag, payload);
        }
#endif
    }
};
__device__ __forceinline__ const unsigned long long* xw_read(const DecodeParams& P) { return P.xw + (blockIdx.x & (unsigned)(P.copies - 1)) * (size_t)P.xo.total; }

// Poll one word until it carries `tag`.  Gives up (false) when the time budget has run out or another CTA has reported
// an error; the caller then leaves the kernel through its error path.
MI_COLD_FN bool tw_spin(const unsigned long long* p, unsigned tag, unsigned long long budget_ns, const int* err) {
    unsigned long long t0 = 0;
    #pragma unroll 1
    for (unsigned it = 1; !tw_is(tw_ld(p), tag); it++) {
        if ((it & 31u) == 0) {
            const unsigned long long now = gtime_ns();
            if (t0 == 0) t0 = now;
            if (now - t0 > budget_ns || *reinterpret_cast<const volatile int*>(err) != 0) return false;
        }
    }
    return true;
}

// What a warp does that misses words: every lane fetches its missing words again at once.  Each 64th round the lowest lane that misses one polls that word alone, looks at the time and
// at the error word, and the other lanes sit at the vote.  (One lane polling from the start, which keeps one load of a warp in flight instead of
// thirty-two, costs a round trip behind the last word: tensor-parallel build without a peer, mean of eight loads, 1.5B shape 561 us per token so and 536, 0.5B 464 and 441, 3B 826 and 800; with a pause
// of 40 or 150 ns between polls, one load each, 594 and 604 where 585 was without.)
// Called by all lanes of a warp with the first missing address of each (null: none).  Returns 0 when
// no lane misses anything, 1 when the lanes are to fetch their missing words again, -1 when the wait gave up.
__device__ __forceinline__ int tw_wait_warp(const unsigned long long* miss, unsigned tag, unsigned long long budget_ns, const int* err, unsigned round) {
    const unsigned mm = __ballot_sync(0xffffffffu, miss != nullptr);
    if (!mm) return 0;
    if ((round & 63u) != 63u) return 1;
    const int leader = __ffs(mm) - 1;
    int r = 1;
    if ((int)(threadIdx.x & 31) == leader) r = tw_spin(miss, tag, budget_ns, err) ? 1 : -1;
    return __shfl_sync(0xffffffffu, r, leader);
}

// Load the N words addr(k) (k with bit k of `valid` set) and return their payloads once all carry `tag`.  All loads are
// issued before any is looked at; while some word is not there yet, every lane fetches
// its missing words again (tw_wait_warp).  All 32 lanes of a warp must call.
template <int N, class AddrFn>
__device__ __forceinline__ bool tw_poll(const DecodeParams& P, unsigned tag, unsigned valid, AddrFn addr, unsigned (&out)[N]) {
    unsigned long long w[N];
    #pragma unroll
    for (int k = 0; k < N; k++) w[k] = (valid >> k & 1u) ? tw_ld(addr(k)) : ((unsigned long long)tag << 32);
    for (unsigned round = 0;; round++) {
        const unsigned long long* miss = nullptr;
        #pragma unroll
        for (int k = N - 1; k >= 0; k--) if (!tw_is(w[k], tag)) miss = addr(k);
        const int st = tw_wait_warp(miss, tag, P.wait_ns, P.err, round);
        if (st == 0) break;
        if (st < 0) return false;
        #pragma unroll
        for (int k = 0; k < N; k++) if (!tw_is(w[k], tag)) w[k] = tw_ld(addr(k));
    }
    #pragma unroll
    for (int k = 0; k < N; k++) out[k] = (unsigned)w[k];
    return true;
}

// N 16-byte pairs of words, pair k at `base + off[k]` (where bit k of `valid` is set), their payloads in a and b.  As tw_poll, in few instructions: a lane that misses
// anything fetches all of its pairs again.
// Among the last NPAD pairs, word `pad` is one that nobody writes.
template <int N, int NPAD = 0>
__device__ __forceinline__ bool tw_poll_pairs(const DecodeParams& P, unsigned tag, unsigned valid, const unsigned long long* base, const int (&off)[N], unsigned (&a)[N], unsigned (&b)[N],
                                              int pad = -1) {
    const unsigned long long none = (unsigned long long)tag << 32;
    unsigned round = 0;
    #pragma unroll 1
    for (;;) {
        unsigned long long wa[N], wb[N];
        #pragma unroll
        for (int k = 0; k < N; k++) {
            wa[k] = wb[k] = none;
            if (valid >> k & 1u) tw_ld2(base + off[k], wa[k], wb[k]);
        }
        int miss = -1;
        #pragma unroll
        for (int k = 0; k < N; k++) {
            if (!tw_is(wa[k], tag)) miss = off[k];
            if (!tw_is(wb[k], tag) && !(k >= N - NPAD && off[k] + 1 == pad)) miss = off[k] + 1;
            a[k] = (unsigned)wa[k]; b[k] = (unsigned)wb[k];
        }
        const int st = tw_wait_warp(miss >= 0 ? base + miss : nullptr, tag, P.wait_ns, P.err, round++);
        if (st <= 0) return st == 0;
    }
}

// ---- the per-warp weight stream -----------------------------------------------
// The order in which a warp consumes tiles is a pure function of shapes and indices, so the host lists it once per model: entry k of a warp's
// list is the global address of its k-th tile of a step (16-byte aligned; the low two bits carry log2 of the tile depth).  A ninth warp walks
// the lists, a lane per ring, wrapping at the end of the launch's job range, and requests a tile whenever a slot is free.  (A copy takes the warp that issues it
// some 400 clocks; issued by the computing warps, between tiles or behind a phase, that was a tenth of a token and left copies to be made in bursts, so that
// the tiles of the next phase were missing.)
struct WarpStream {
    const uint8_t* ring; uint64_t* full; uint64_t* empty;
    unsigned out, phase;             // slot of the next tile, parity of its barrier
    int warp;                        // warp in CTA
    int gcta, ggrid;                 // this CTA's index among the CTAs that carry GEMV units, their number

    __device__ __forceinline__ void init(const DecodeSmem& sm, const DecodeParams& P, int warp_) {
        warp = warp_;
        ring = sm.ring + (size_t)warp * DS * DSLOT; full = sm.bars + warp * DS; empty = full + DNW * DS;
        gcta = (int)blockIdx.x - P.attn_ctas; ggrid = (int)gridDim.x - P.attn_ctas;
        out = phase = 0;
    }
    // waits for the next tile; release() when every lane is through with it
    __device__ __forceinline__ bool acquire() const {
        unsigned long long t0 = 0;
        #pragma unroll 1
        for (unsigned i = 1; !mbar_try_wait(&full[out], phase); i++) {
            if ((i & 255u) == 0) {
                const unsigned long long now = gtime_ns();
                if (t0 == 0) t0 = now;
                if (now - t0 > kWaitBudgetNs) return false;
            }
        }
        return true;
    }
    __device__ __forceinline__ const uint8_t* tile() const { return ring + (size_t)out * DSLOT; }
    __device__ __forceinline__ void release(int lane) {
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&empty[out])) : "memory");
        if (++out == DS) { out = 0; phase ^= 1u; }
    }
};
// The ninth warp: lane r < 8 keeps ring r full until the launch's tiles have been requested, or the computing warps have left (quit).  Then it sees its copies land: they
// target this CTA's shared memory.
__device__ __forceinline__ void stream_weights(const DecodeSmem& sm, const DecodeParams& P, int lane, int steps, int j0, int j1, const volatile int* quit) {
    const int r = lane & (DNW - 1), slot = ((int)blockIdx.x - P.attn_ctas) * DNW + r, nj = 4 * P.L + 2;
    uint8_t* ring = sm.ring + (size_t)r * DS * DSLOT;
    uint64_t* full = sm.bars + r * DS; uint64_t* empty = full + DNW * DS;
    const unsigned long long* tab = P.tile_tab + (size_t)slot * P.tile_stride;
    const unsigned e0 = __ldg(P.tile_start + (size_t)slot * nj + j0), e1 = __ldg(P.tile_start + (size_t)slot * nj + j1);
    long long left = lane < DNW && j0 < j1 ? (long long)steps * (e1 - e0) : 0;
    unsigned c = e0, in = 0, lap = 0;
    int issued = 0;
    const uint64_t policy = l2_policy_evict_first();          // a weight byte leaves the HBM once per token: also where two CTAs read a tile (halves) the second finds it in the L2 (1.5B shape: 868.4 MB read, 868.3 of weights)
    unsigned long long next = left > 0 ? __ldg(tab + c) : 0ull;
    while (__any_sync(0xffffffffu, left > 0) && !__any_sync(0xffffffffu, *quit != 0)) {
        const bool go = left > 0 && (lap == 0 || mbar_try_wait(&empty[in], (lap - 1) & 1));        // (the first lap finds the slots empty)
        if (go) {
            const int tb = kTileRowBytes << (int)(next & 3ull);
            mbar_expect_tx(&full[in], tb);
            bulk_g2s_hint(ring + (size_t)in * DSLOT, reinterpret_cast<const void*>(next & ~15ull), tb, &full[in], policy);
            issued++; left--;
            if (++in == DS) { in = 0; lap++; }
            if (++c == e1) c = e0;
            if (left > 0) next = __ldg(tab + c);
        }
        if (!__any_sync(0xffffffffu, go)) __nanosleep(64);
    }
    if (lane < DNW)
        for (int k = max(0, issued - DS); k < issued; k++) (void)mbar_wait_bounded(&full[k % DS], (k / DS) & 1);
}

// The per-token loop body must stay small: it is executed phase after phase by every SM, and measured, the kernel ran
// 15 % faster once the four GEMV phases shared one copy of their code.  So the double-precision exponential has one
// out-of-line copy, and the variants a given model never takes (other tile depths, other norm widths) sit out of line
// instead of between the hot instructions.
MI_COLD_FN double exp_shared(double x) { return exp(x); }
// A tile's contribution to the lane's row: the GEMV's terms (blk_acc) from fewer operations.  What bounds it is the integer pipe (an SM makes 64 dp4a a clock, two
// clocks for a warp on its sub-partition, and logic operations with an immediate twice that: 27 clocks of it per block), and, for the few tiles of a small phase, latency.  So the high
// nibbles stay where they are, as bytes 16 n, and the dot product is 16 (low - 8 sum x) + high; its 16 is in xs_s, a sixteenth of each block's scale (a power of two: all
// products stay exact) beside -8 times the sum of the block's activations.  The dot product starts at 2^31, so that below the exponent bits of 2^52 it is a double without a
// conversion (of which an SM makes 16 a clock).  Tried: the blocks on int8 MMAs, one column of the
// activations per block (the same throughput, twice the latency); nibbles made signed bytes with an exclusive or (three-operand logic: 38 clocks); sixteen warps with half a
// tile each (680 us per token of the 1.5B shape: the pipe is as full with eight, and barriers and polls cost more).
__device__ __forceinline__ int dp4a_us(unsigned w, int x, int c) { int r; asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(w), "r"(x), "r"(c)); return r; }
struct BlockScale { float d16; int m8s; };                    // a sixteenth of the scale, -8 times the sum of the values
__device__ __forceinline__ BlockScale block_scale(float d, int sum) { BlockScale b; b.d16 = __fmul_rn(d, 0.0625f); b.m8s = -8 * sum; return b; }
template <int KB> struct TileRegs { uint4 w[KB]; unsigned d[(KB + 1) / 2]; };          // a lane's row of KB blocks
template <int KB>
__device__ __forceinline__ void tile_load(const uint8_t* tile, int lane, TileRegs<KB>& r) {
    const uint8_t* sp = tile + KB * 512 + lane * (KB * 2);
    if constexpr (KB == 8) { const uint4 v = *reinterpret_cast<const uint4*>(sp); r.d[0] = v.x; r.d[1] = v.y; r.d[2] = v.z; r.d[3] = v.w; }
    else if constexpr (KB == 4) { const uint2 v = *reinterpret_cast<const uint2*>(sp); r.d[0] = v.x; r.d[1] = v.y; }
    else if constexpr (KB == 2) r.d[0] = *reinterpret_cast<const unsigned*>(sp);
    else r.d[0] = *reinterpret_cast<const unsigned short*>(sp);
    #pragma unroll
    for (int k = 0; k < KB; k++) r.w[k] = reinterpret_cast<const uint4*>(tile)[k * 32 + lane];
}
template <int KB>
__device__ __forceinline__ double tile_dot(const TileRegs<KB>& r, int b0, const int8_t* xq_s, const BlockScale* xs_s, double acc) {
    #pragma unroll
    for (int k = 0; k < KB; k++) {
        const uint4 w = r.w[k];
        const int4 xa = *reinterpret_cast<const int4*>(xq_s + (b0 + k) * 32), xc = *reinterpret_cast<const int4*>(xq_s + (b0 + k) * 32 + 16);
        const BlockScale x = xs_s[b0 + k];
        constexpr unsigned L = 0x0F0F0F0Fu, H = 0xF0F0F0F0u;
        int c = dp4a_us(w.x & L, xa.x, x.m8s), d = dp4a_us(w.x & H, xc.x, (int)0x80000000);
        c = dp4a_us(w.y & L, xa.y, c); d = dp4a_us(w.y & H, xc.y, d);
        c = dp4a_us(w.z & L, xa.z, c); d = dp4a_us(w.z & H, xc.z, d);
        c = dp4a_us(w.w & L, xa.w, c); d = dp4a_us(w.w & H, xc.w, d);
        acc = __fma_rn((double)__fmul_rn(__half2float(__ushort_as_half((unsigned short)(r.d[k / 2] >> 16 * (k & 1)))), x.d16),
                       __dsub_rn(__hiloint2double(0x43300000, c * 16 + d), 4503601774854144.0), acc);      // 2^52 + 2^31
    }
    return acc;
}
// The same for sixteen rows of a tile (second: the latter ones): lane 16 j + r has row r and the j-th half of the blocks
template <int KB>
__device__ __forceinline__ void tile_load_half(const uint8_t* tile, int lane, bool second, TileRegs<KB / 2>& r) {
    const int row = (lane & 15) + (second ? 16 : 0), j = lane >> 4;
    const uint8_t* sp = tile + KB * 512 + row * (KB * 2) + j * KB;
    if constexpr (KB == 8) { const uint2 v = *reinterpret_cast<const uint2*>(sp); r.d[0] = v.x; r.d[1] = v.y; }
    else r.d[0] = *reinterpret_cast<const unsigned*>(sp);
    #pragma unroll
    for (int k = 0; k < KB / 2; k++) r.w[k] = reinterpret_cast<const uint4*>(tile)[(j * (KB / 2) + k) * 32 + row];
}
template <int KB>
static __device__ __noinline__ double tile_dot_rare(const uint8_t* tile, int lane, int b0, const int8_t* xq_s, const BlockScale* xs_s, double acc) {
    TileRegs<KB> r;
    tile_load<KB>(tile, lane, r);
    return tile_dot<KB>(r, b0, xq_s, xs_s, acc);
}
// A tile in registers, and its product: the two are apart because the first tile of a phase is read before its input is there.  lean_shape(): tiles
// are 8 blocks deep, or (small build) 8 or 4; the general build reads its tiles where it needs them.
struct WarpTile {
#if MI_LEAN
    TileRegs<8> t;
    template <int N> __device__ __forceinline__ void keep(const TileRegs<N>& r) {
        #pragma unroll
        for (int k = 0; k < N; k++) { t.w[k] = r.w[k]; t.d[k / 2] = r.d[k / 2]; }
    }
    template <int N> __device__ __forceinline__ TileRegs<N> first() const {
        TileRegs<N> r;
        #pragma unroll
        for (int k = 0; k < N; k++) { r.w[k] = t.w[k]; r.d[k / 2] = t.d[k / 2]; }
        return r;
    }
    // half: the tile belongs to a unit of sixteen rows; second: the latter ones
    __device__ __forceinline__ void load(WarpStream& ws, int lane, int kb, bool half, bool second) {
        if (MI_SMALL && kb == 4) {
            if (half) { TileRegs<2> r; tile_load_half<4>(ws.tile(), lane, second, r); keep<2>(r); }
            else { TileRegs<4> r; tile_load<4>(ws.tile(), lane, r); keep<4>(r); }
        } else if (half) { TileRegs<4> r; tile_load_half<8>(ws.tile(), lane, second, r); keep<4>(r); }
        else tile_load<8>(ws.tile(), lane, t);
        ws.release(lane);
    }
    __device__ __forceinline__ double dot(WarpStream&, int lane, int kb, bool half, bool, int b0, const int8_t* xq_s, const BlockScale* xs_s, double acc) const {
        if (half) {
            b0 += (lane >> 4) * (kb >> 1);
            if (MI_SMALL && kb == 4) return tile_dot<2>(first<2>(), b0, xq_s, xs_s, acc);
            return tile_dot<4>(first<4>(), b0, xq_s, xs_s, acc);
        }
        if (MI_SMALL && kb == 4) return tile_dot<4>(first<4>(), b0, xq_s, xs_s, acc);
        return tile_dot<8>(t, b0, xq_s, xs_s, acc);
    }
#else
    const uint8_t* at;
    __device__ __forceinline__ void load(const WarpStream& ws, int, int, bool, bool) { at = ws.tile(); }
    __device__ __forceinline__ double dot(WarpStream& ws, int lane, int kb, bool half, bool second, int b0, const int8_t* xq_s, const BlockScale* xs_s, double acc) const {
        if (half) {                                        // (tiles of 8 or 4 blocks)
            b0 += (lane >> 4) * (kb >> 1);
            if (kb == 8) { TileRegs<4> r; tile_load_half<8>(at, lane, second, r); acc = tile_dot<4>(r, b0, xq_s, xs_s, acc); }
            else { TileRegs<2> r; tile_load_half<4>(at, lane, second, r); acc = tile_dot<2>(r, b0, xq_s, xs_s, acc); }
        } else if (kb == 8) {
            TileRegs<8> r;
            tile_load<8>(at, lane, r);
            acc = tile_dot<8>(r, b0, xq_s, xs_s, acc);
        } else acc = kb == 4 ? tile_dot_rare<4>(at, lane, b0, xq_s, xs_s, acc) : kb == 2 ? tile_dot_rare<2>(at, lane, b0, xq_s, xs_s, acc) : tile_dot_rare<1>(at, lane, b0, xq_s, xs_s, acc);
        ws.release(lane);
        return acc;
    }
#endif
};

// q8_0 of one 32-element block held one element per lane; returns the int8 value, and through
// d_out / s_out (all lanes) the fp16 scale and the integer sum of the block's values.
__device__ __forceinline__ int quant_block_warp2(float v, __half& d_out, int& s_out) {
    const float a = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(v))));
    const bool odd = threadIdx.x & 1;                       // (one division for 127 / a and a / 127)
    const float r = __fdiv_rn(odd ? a : 127.f, odd ? 127.f : a), iv = __shfl_sync(0xffffffffu, r, 0);
    const int q = __float2int_rn(__fmul_rn(v, a > 0.f ? iv : 0.f));
    s_out = __reduce_add_sync(0xffffffffu, q);
    d_out = __float2half_rn(__shfl_sync(0xffffffffu, r, 1));
    return q;
}
// Publish one q8_0 block (lane = element) as tagged words: lanes 0, 4, 8, .. store four int8 values each, lane 1
// the scale word.  qoff / soff: word offsets of the vector's value and scale parts; b: block index.
template <bool SHARED>
__device__ __forceinline__ void publish_q8_block(const Pub& pub, int qoff, int soff, int b, int lane, int q, __half d, int s) {
    unsigned v = (unsigned)q & 0xffu;
    v |= __shfl_down_sync(0xffffffffu, v, 1) << 8;
    v |= __shfl_down_sync(0xffffffffu, v, 2) << 16;
    const unsigned sw = (unsigned)__half_as_ushort(d) | ((unsigned)s << 16);
    if ((lane & 3) == 0) { if (SHARED) pub.shared(qoff + b * 8 + (lane >> 2), v); else pub.all(qoff + b * 8 + (lane >> 2), v); }
    if (lane == 0) { if (SHARED) pub.shared(soff + b, sw); else pub.all(soff + b, sw); }
}

// A per-layer job, before its input is there: the CTA's first batch, and this warp's first tile (range builds: in registers), so that behind the last word
// that arrives there are only the activations to be read.
struct JobStart { unsigned at; bool ok; float bias; WarpTile t; };
// bias: added to complete sums by the epilogue, which needs those of its unit's rows
__device__ __forceinline__ float batch_bias(const unsigned* work, unsigned at, int warp, int lane, bool half, const float* __restrict__ bias) {
    return bias && warp < (int)(work[at] & 255u) ? __ldg(bias + work[at + kBatchGroup + warp] + (half ? lane & 15 : lane)) : 0.f;
}
__device__ __forceinline__ JobStart begin_cta_job(WarpStream& ws, const unsigned* work, int kind, int kb, bool half, int lane, const float* __restrict__ bias) {
    JobStart st;
    st.at = work[kind]; st.ok = true; st.bias = 0.f;
    if (st.at) {
        st.bias = batch_bias(work, st.at, ws.warp, lane, half, bias);
        const unsigned list = work[st.at + kBatchList + ws.warp];
        if (list >> 16) { st.ok = ws.acquire(); st.t.load(ws, lane, kb, half, work[list & 0xffffu] >> 21 & 1u); }
    }
    return st;
}

__device__ __forceinline__ double tree_sum8(double a, double b, double c, double d, double e, double f, double g, double h) {
    return __dadd_rn(__dadd_rn(__dadd_rn(a, b), __dadd_rn(c, d)), __dadd_rn(__dadd_rn(e, f), __dadd_rn(g, h)));
}
// The job's batches: the warps' shares of every sum meet in shared memory, and warp b adds those of unit b and calls epi(g, lane, v0, v1, bias) with
// the complete sums rounded to fp32.  A job that is K-split across CTAs (ks > 1; down projection)
// adds one hop: the CTAs of splits 1.. publish their double partial sums as tagged word pairs,
// the CTA of split 0 waits for them, adds them to its own in split order and calls epi.
// Every warp passes the same number of barriers, also after a wait gave up.
template <class Epi>
__device__ __forceinline__ bool run_cta_job(WarpStream& ws, const DecodeParams& P, const DecodeSmem& sm, const JobStart& st, int kb, int ks, bool two, bool half, int lane,
                                            const int8_t* xq_s, const BlockScale* xs_s, const float* __restrict__ bias, const Pub& pub, Epi epi) {
    bool ok = st.ok;
    unsigned at = st.at;
    if (!at) return ok;
    const unsigned* work = sm.work;
    WarpTile t = st.t;
    float bv = st.bias;
    for (;;) {
        const unsigned list = work[at + kBatchList + ws.warp], head = work[at];
        const unsigned* item = work + (list & 0xffffu);
        int n = (int)(list >> 16);
        if (n) {
            double acc = 0.0;
            for (;;) {
                const unsigned it = *item++;
                acc = t.dot(ws, lane, kb, half, it >> 21 & 1u, (int)(it & 0xffffu), xq_s, xs_s, acc);
                if (it >> 20 & 1u) { sm.fold[((it >> 16 & 7u) * DNW + ws.warp) * 32 + lane] = acc; acc = 0.0; }
                if (--n == 0) break;
                if (ok) ok = ws.acquire();
                t.load(ws, lane, kb, half, *item >> 21 & 1u);
            }
        }
        prof_mark(P, 18);
        cta__syncthreads();
        if (ws.warp < (int)(head & 255u)) {
            const unsigned gg = work[at + kBatchGroup + ws.warp], u = work[at + kBatchUnit + ws.warp];
            const double* f0 = sm.fold + ws.warp * (2 * DNW * 32) + lane;
            double v0 = 0.0, v1 = 0.0;
            #pragma unroll 1
            for (int a = two ? 1 : 0; a >= 0; a--) {                    // up, then gate
                const double* f = f0 + a * (DNW * 32);
                const unsigned p0 = a ? u >> 20 : u >> 16;
                const int n8 = (int)(u >> 8 & 15u);
                double v[DNW];
                #pragma unroll
                for (int q = 0; q < DNW; q++) { const double x = f[((p0 + q) & (DNW - 1)) * 32]; v[q] = q < n8 ? x : 0.0; }
                v1 = v0;
                v0 = tree_sum8(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]);
            }
            if (half) v0 = __dadd_rn(v0, __shfl_xor_sync(0xffffffffu, v0, 16));          // (the two halves of the blocks)
            bool whole = true;
            if (ks > 1) {
                const int sp = (int)(u & 255u), to = P.xo.dpart + ((int)gg * (kMaxKSplit - 1) + lane) * 2;
                whole = sp == 0;
                if (!whole) {
                    const unsigned long long bits = (unsigned long long)__double_as_longlong(v0);
                    pub.local(to + (sp - 1) * 64, (unsigned)bits);
                    pub.local(to + (sp - 1) * 64 + 1, (unsigned)(bits >> 32));
                } else {
                    #pragma unroll 1
                    for (int q = 0; q < ks - 1; q++) {
                        const int off[1] = {to + q * 64};
                        unsigned lo[1], hi[1];
                        const bool got = tw_poll_pairs<1>(P, pub.tag, 1u, P.xw, off, lo, hi);      // all lanes, always
                        ok = __all_sync(0xffffffffu, (ok && got) ? 1 : 0) != 0;
                        v0 = __dadd_rn(v0, __hiloint2double((int)hi[0], (int)lo[0]));
                    }
                    whole = ok;
                }
            }
            if (whole) epi((int)gg, lane, __double2float_rn(v0), __double2float_rn(v1), bv);
        }
        prof_mark(P, 19);
#if MI_LEAN
        return ok;                                                      // (a range build runs only where one batch is all there is)
#endif
        at = head >> 8;
        if (!at) return ok;
        bv = batch_bias(work, at, ws.warp, lane, half, bias);
        const unsigned next = work[at + kBatchList + ws.warp];
        if (next >> 16) {
            if (ok) ok = ws.acquire();
            t.load(ws, lane, kb, half, work[next & 0xffffu] >> 21 & 1u);
        }
        cta__syncthreads();                                                // the sums have been read
    }
}

// lm_head: a unit (row group) belongs to one warp; epi(g, lane, v).
template <class Epi>
__device__ __forceinline__ bool run_warp_job(WarpStream& ws, int /* in phase order */, const DecodeParams& P, int lane, const int8_t* xq_s, const BlockScale* xs_s, Epi epi) {
    const int nt = P.lm_nt, kb = P.kb[JOB_LM], n_units = P.lm_units, off = P.lm_off;
    bool ok = true;
    WarpTile h;
    for (int u = ws.warp * ws.ggrid + ws.gcta; u < n_units && ok; u += ws.ggrid * DNW) {       // (consecutive units land on different SMs)
        double acc = 0.0;
        for (int t = 0; t < nt && ok; t++) {
            if (!(ok = ws.acquire())) break;
            h.load(ws, lane, kb, false, false);
            acc = h.dot(ws, lane, kb, false, false, t * kb, xq_s, xs_s, acc);
        }
        if (ok) epi(u + off, lane, __double2float_rn(acc));
    }
    return ok;
}

// ---- activation staging (whole CTA; returns a CTA-uniform ok) -----------------------

// warp-wide maximum of arbitrary finite floats (or -inf): order-preserving key
__device__ __forceinline__ float warp_max_float(float a) {
    const unsigned b = __float_as_uint(a), key = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
    const unsigned m = __reduce_max_sync(0xffffffffu, key);
    return __uint_as_float((m & 0x80000000u) ? (m & 0x7fffffffu) : ~m);
}

// Residual add + RMSNorm + q8_0 staging:
//   x = h (this CTA's copy of the residual stream in shared memory; or gsrc, the copy the first GEMV CTA committed to
//       global memory, when the launch starts here; or the embedding row of `token`)
//       + the projection output published as tagged fp32 words at addw   [if addw]
//   h = x;  the first GEMV CTA also commits x to global memory;
//   xq_s / xs_s = q8_0( x * (1/sqrt(float(ss/n) + eps)) * w )   (src/cpu_infer.cpp:40-46).
// What bounds it is a chain of latencies behind the last word that arrives, so a thread keeps its elements in registers from the words to the int8
// values and nothing on the way branches (a branch, taken or not, is some 16 clocks, an integer operation 2 per warp).  Warp w owns the runs of 64
// elements w, w+8, ...; a lane has two consecutive ones of each, so a warp's load of tagged words is one contiguous 512-byte run of
// 16-byte pairs, and a q8_0 block is half a warp.  Sum of squares in double (every x*x is exact there); the lanes' sums are added by two FP64 MMAs
// against ones (the first adds four lanes each and leaves two of eight sums per lane, the second adds the four pairs), where five rounds of 64-bit shuffles took three
// times as long.
// h_s must hold the residual stream already (residual_init below puts the embedding row, or the copy committed to global
// memory, there with this same thread mapping, so no barrier is needed in between).
__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}
__device__ __forceinline__ double warp_sum(double v) {
    double c[2] = {0.0, 0.0}, d[2] = {0.0, 0.0};
    dmma884(c, 1.0, v);
    dmma884(d, 1.0, __dadd_rn(c[0], c[1]));
    return d[0];
}
// ok: whether this warp's part of the phase before was complete.
template <int NC>
__device__ __forceinline__ bool stage_norm_q8_t(bool ok, const DecodeParams& P, float* h_s,
                                                const unsigned long long* addw, unsigned tag, float* commit, const float* __restrict__ w,
                                                int E, float eps, double* red, int8_t* xq_s, BlockScale* xs_s) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float2 x[NC], wv[NC];
    int e[NC];
    unsigned valid = 0;
    #pragma unroll
    for (int k = 0; k < NC; k++) {
        const int at = (warp + k * DNW) * 64 + 2 * lane;
        valid |= at < E ? 1u << k : 0u;
        e[k] = at < E ? at : 0;                              // every address is valid; a lane past the vector stores nothing
        wv[k] = __ldg(reinterpret_cast<const float2*>(w + e[k]));
        x[k] = *reinterpret_cast<const float2*>(h_s + e[k]);
    }
    if (addw) {
        unsigned a[NC], b[NC];
        prof_mark(P, 27);
        ok = tw_poll_pairs<NC>(P, tag, (1u << NC) - 1u, addw, e, a, b) && ok;
        prof_mark(P, kProfWait);
        #pragma unroll
        for (int k = 0; k < NC; k++) { x[k].x = __fadd_rn(x[k].x, __uint_as_float(a[k])); x[k].y = __fadd_rn(x[k].y, __uint_as_float(b[k])); }
        prof_mark(P, 28);
    }
    double s2[2] = {0.0, 0.0};                           // two chains
    #pragma unroll
    for (int k = 0; k < NC; k++) {
        const bool live = valid >> k & 1u;
        const double x0 = live ? x[k].x : 0.f, x1 = live ? x[k].y : 0.f;
        s2[0] = __fma_rn(x0, x0, s2[0]); s2[1] = __fma_rn(x1, x1, s2[1]);
    }
    const double ss = warp_sum(__dadd_rn(s2[0], s2[1]));
    if (lane == 0) red[warp] = ss;
    #pragma unroll
    for (int k = 0; k < NC; k++) if (valid >> k & 1u) *reinterpret_cast<float2*>(h_s + e[k]) = x[k];
    if (commit && (int)blockIdx.x == P.attn_ctas) {
        #pragma unroll
        for (int k = 0; k < NC; k++) if (valid >> k & 1u) __stcg(reinterpret_cast<float2*>(commit + e[k]), x[k]);
    }
    prof_mark(P, 23);
    if (!cta__syncthreads_and(ok ? 1 : 0)) return false;
    prof_mark(P, 24);
    const double2* r2 = reinterpret_cast<const double2*>(red);
    const double2 ra = r2[0], rb = r2[1], rc = r2[2], rd = r2[3];
    const float mean = __double2float_rn(div_known(tree_sum8(ra.x, ra.y, rb.x, rb.y, rc.x, rc.y, rd.x, rd.y), (double)E, P.inv_e));
    const float scale = __fdiv_rn(1.f, __fsqrt_rn(__fadd_rn(mean, eps)));
    float m[NC];
    #pragma unroll
    for (int k = 0; k < NC; k++) {
        x[k].x = __fmul_rn(__fmul_rn(x[k].x, scale), wv[k].x); x[k].y = __fmul_rn(__fmul_rn(x[k].y, scale), wv[k].y);
        m[k] = fmaxf(fmaxf(0.f, fabsf(x[k].x)), fabsf(x[k].y));        // (a NaN does not count)
    }
    #pragma unroll
    for (int o = 1; o < 16; o <<= 1)
        #pragma unroll
        for (int k = 0; k < NC; k++) m[k] = fmaxf(m[k], __shfl_xor_sync(0xffffffffu, m[k], o));
    // one division for up to eight runs: lane 2 k of a half warp has 127 / (its half's maximum of run k), lane 2 k + 1 that maximum / 127
    // (a division has a branch: two for each run were half of this pass)
    #pragma unroll
    for (int k0 = 0; k0 < NC; k0 += 8) {
        const int mk = k0 + ((lane & 15) >> 1);
        float a = m[k0];
        #pragma unroll
        for (int k = k0 + 1; k < k0 + 8 && k < NC; k++) if (mk == k) a = m[k];
        const bool odd = lane & 1;
        const float d = __fdiv_rn(odd ? a : 127.f, odd ? 127.f : a);
        const int mine = (warp + mk * DNW) * 64 + 2 * (lane & 16);          // first element of the lane's block
        int sum[8];
        #pragma unroll
        for (int k = k0; k < k0 + 8 && k < NC; k++) {
            const float iv = __shfl_sync(0xffffffffu, d, (lane & 16) + 2 * (k - k0)), inv = m[k] > 0.f ? iv : 0.f;
            const int q0 = __float2int_rn(__fmul_rn(x[k].x, inv)), q1 = __float2int_rn(__fmul_rn(x[k].y, inv));
            if (valid >> k & 1u) *reinterpret_cast<unsigned short*>(xq_s + e[k]) = (unsigned short)__byte_perm((unsigned)q0, (unsigned)q1, 0x0040);
            sum[k - k0] = q0 + q1;
        }
        #pragma unroll
        for (int o = 1; o < 16; o <<= 1)
            #pragma unroll
            for (int k = k0; k < k0 + 8 && k < NC; k++) sum[k - k0] += __shfl_xor_sync(0xffffffffu, sum[k - k0], o);
        int sm = sum[0];
        #pragma unroll
        for (int k = k0 + 1; k < k0 + 8 && k < NC; k++) if (mk == k) sm = sum[k - k0];
        if (odd && mk < NC && mine < E) xs_s[mine >> 5] = block_scale(__half2float(__float2half_rn(d)), sm);
    }
    prof_mark(P, 25);
    cta__syncthreads();
    prof_mark(P, 26);
    return true;
}

// The compiler knows nothing of k from here on: it would otherwise make a copy of what follows for each value that k has had.
__device__ __forceinline__ void same_code(int& k) { asm volatile("" : "+r"(k)); }

// The residual stream into this CTA's shared memory, where a step or a launch begins: the embedding row of `token`
// (value (nibble - 8) * d, src/gguf.h:94-102; or a Q8_0 row as stored, int8 * d, src/gguf.h:112-118 and src/mega.cu:639-642),
// or the copy the first GEMV CTA committed to global memory (a launch that starts in mid-step).  Thread mapping of the norm
// prologue's gathering pass: each thread later reads only what it wrote here.
__device__ __forceinline__ void residual_init(const DecodeParams& P, float* h_s, const float* gsrc, int token, int E) {
    const int tid = threadIdx.x, nb = E / 32;
    #pragma unroll 1
    for (int e = 2 * tid; e < E; e += 2 * DNT) {
        const int b = e >> 5, i = e & 31;                  // elements i and i + 1 of block b
        float2 x;
        if (gsrc) x = __ldcg(reinterpret_cast<const float2*>(gsrc + e));
        else if (P.emb_q8) {
            const uint8_t* bp = P.emb_q8 + ((size_t)token * nb + b) * 34;
            const float d = __half2float(__ldg(reinterpret_cast<const __half*>(bp)));
            const unsigned q = __ldg(reinterpret_cast<const unsigned short*>(bp + 2 + i));
            x = make_float2(__fmul_rn(__int2float_rn((int)(int8_t)(q & 0xff)), d), __fmul_rn(__int2float_rn((int)(int8_t)(q >> 8)), d));
        } else {
            const int g = token >> 5, r = token & 31, kb = P.emb_kb, t = b / kb, kk = b % kb;
            const uint8_t* tile = P.emb_base + ((size_t)g * P.emb_nt + t) * (kb * kTileRowBytes);
            const unsigned q = (unsigned)__ldg(reinterpret_cast<const unsigned short*>(tile + ((size_t)kk * 32 + r) * 16 + (i & 15))) >> (i < 16 ? 0 : 4);
            const float d = __half2float(__ldg(reinterpret_cast<const __half*>(tile + (size_t)kb * 512 + ((size_t)r * kb + kk) * 2)));
            x = make_float2(__fmul_rn(__int2float_rn((int)(q & 15) - 8), d), __fmul_rn(__int2float_rn((int)(q >> 8 & 15) - 8), d));
        }
        *reinterpret_cast<float2*>(h_s + e) = x;
    }
}

#define MI_NORM_ARGS bool ok, const DecodeParams& P, float* h_s, const unsigned long long* addw, unsigned tag, \
                     float* commit, const float* __restrict__ w, int E, float eps, double* red, int8_t* xq_s, BlockScale* xs_s
#define MI_NORM_PASS ok, P, h_s, addw, tag, commit, w, E, eps, red, xq_s, xs_s
// runs of 64 elements per warp (NC): as many as the widest vector of a call needs
static __device__ __noinline__ bool stage_norm_q8_rare(MI_NORM_ARGS) {
    if (E <= 512) return stage_norm_q8_t<1>(MI_NORM_PASS);
    if (E <= 1024) return stage_norm_q8_t<2>(MI_NORM_PASS);
    if (E <= 4096) return stage_norm_q8_t<8>(MI_NORM_PASS);
    return stage_norm_q8_t<16>(MI_NORM_PASS);
}
// NC_MAX: the most that a model of this head shape has in a range build
template <int NC_MAX>
__device__ __forceinline__ bool stage_norm_q8u(MI_NORM_ARGS) {
#if MI_LEAN
    return stage_norm_q8_t<NC_MAX>(MI_NORM_PASS);           // lean_shape(): 1024 < E <= 2048, or (small build) 512 < E <= 1024
#else
    if (E > 1024 && E <= 2048) return stage_norm_q8_t<4>(MI_NORM_PASS);
    return stage_norm_q8_rare(MI_NORM_PASS);
#endif
}
// E is a multiple of HD * G: the largest one within the range build's widths, in runs of 64 over the warps
__host__ __device__ constexpr int norm_chunks(int HD, int G) { return ((MI_SMALL ? 1024 : 2048) / (HD * G) * (HD * G) + 64 * DNW - 1) / (64 * DNW); }

// A q8_0 vector published as tagged words by other CTAs -> shared memory: int8 values, and per block what
// tile_dot wants of its scale and sum.  Thread t takes the 16-byte word pairs t, t + 256, ... of the values (NV at most) and of the scales (NS); all of a
// thread's loads are in flight together.  nw: scales, and words behind them that have to be there too (what is stored of those nobody reads).
template <int NV, int NS>
__device__ __forceinline__ bool stage_poll_q8_t(bool ok, const DecodeParams& P, const unsigned long long* vw, int n, int nw, unsigned tag, int8_t* xq_s, BlockScale* xs_s) {
    const int tid = threadIdx.x, nq2 = n / 8;
    int off[NV + NS];
    unsigned valid = 0, a[NV + NS], b[NV + NS];
    #pragma unroll
    for (int k = 0; k < NV + NS; k++) {
        const int pr = tid + (k < NV ? k : k - NV) * DNT;
        off[k] = k < NV ? 2 * pr : 2 * nq2 + 2 * pr;
        valid |= (k < NV ? pr < nq2 : 2 * pr < nw) ? 1u << k : 0u;
    }
    ok = tw_poll_pairs<NV + NS, NS>(P, tag, valid, vw, off, a, b, nw & 1 ? 2 * nq2 + nw : -1) && ok;
    #pragma unroll
    for (int k = 0; k < NV; k++) if (valid >> k & 1u) reinterpret_cast<uint2*>(xq_s)[tid + k * DNT] = make_uint2(a[k], b[k]);
    #pragma unroll
    for (int k = NV; k < NV + NS; k++) {
        auto scale = [](unsigned sw) { return block_scale(__half2float(__ushort_as_half((unsigned short)(sw & 0xffffu))), (int)(short)(sw >> 16)); };
        const int blk = off[k] - 2 * nq2;
        if (valid >> k & 1u) { xs_s[blk] = scale(a[k]); if (blk + 1 < nw) xs_s[blk + 1] = scale(b[k]); }
    }
    return cta__syncthreads_and(ok ? 1 : 0) != 0;
}
// as many pairs as the longest vector wants; one form per build, so that all phases run the same instructions (lean_shape(): at most 8 pairs of values per thread)
__device__ __forceinline__ bool stage_poll_q8(bool ok, const DecodeParams& P, const unsigned long long* vw, int n, int nw, unsigned tag, int8_t* xq_s, BlockScale* xs_s) {
    return stage_poll_q8_t<MI_LEAN ? 8 : 16, MI_LEAN ? 1 : 2>(ok, P, vw, n, nw, tag, xq_s, xs_s);
}

// ---- attention over a long causal range --------------------------------------------------
// CTA = (kv head, chunk of the causal range), all query heads of the group at once, then one CTA per 32-dim block of the
// output merges the chunks.  What bounds it is the FP64 pipe (2 HD FMAs per head and position) and a chain of latencies, so
//   * both products are FP64 MMAs (m8n8k4: a group's heads are the rows): one issue slot per 256 FMAs, and a K or V element is
//     converted to double once for the whole group.  (The scalar form of this phase took 26 us per layer at 8192 positions,
//     most of it conversions and broadcast loads beside the FMAs.)
//   * the chunk's K and V rows are requested (asynchronous copies into shared memory) before the CTA waits for q: they do not
//     depend on this layer's projection, so their latency passes while the projection finishes;
//   * a chunk leaves its weighted sums and denominator in global memory and, behind a fence, its maximum as a tagged word.  Whoever
//     merges polls those words: no counter to reset, and 48 CTAs (1.5B shape) read 38 KB each where the last CTA of a kv head to
//     arrive read 460 KB alone.
// Scores: double dot products rounded to fp32 once, scaled in fp32; weights, denominator and sums in double, running maximum across
// steps, common maximum across chunks.  Returns false if a wait gave up (CTA-uniform).
__device__ __forceinline__ void cp_async16(void* dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void fence_acq_rel_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ double half_to_double(unsigned w) { return (double)__half2float(__ushort_as_half((unsigned short)w)); }

template <int HD, int G>
__device__ __forceinline__ bool attention_split(const DecodeParams& P, int l, int pos, uint8_t* stage, unsigned tag_in, const Pub pub) {
    const SplitSmem lay{HD, P.split_sub};
    constexpr int KLD = 2 * HD + 64, VLD = 2 * HD + 32;
    const int SUB = P.split_sub, SCL = lay.scl();
    constexpr int NTW = HD >= 64 ? HD / 64 : 1, VW = HD / 8 / NTW, SW = HD + 2;      // 8-dim tiles per warp of the value product, warps that have some; doubles per partial
    double* qs = reinterpret_cast<double*>(stage); double* wt = reinterpret_cast<double*>(stage + lay.wt());      // q [dim of a lane][lane], weights [step of 4][lane]
    uint8_t* ks = stage + lay.k(); uint8_t* vs = stage + lay.v();
    float* sc = reinterpret_cast<float*>(stage + lay.sc());
    double* rm = reinterpret_cast<double*>(stage + lay.st()); double* rl = rm + 8; double* rf = rl + 8;                    // per head: running maximum, denominator, rescale factor
    double* red = reinterpret_cast<double*>(stage + lay.red());
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int Lp = pos + 1, nch = attn_chunks(Lp, min(P.max_chunks, (int)gridDim.x / P.NKV)), nq = P.NH * HD;
    bool ok = true;
    if ((int)blockIdx.x < P.NKV * nch) {
        const int kvh = blockIdx.x / nch, ch = blockIdx.x - kvh * nch, h0 = kvh * G;
        const int p0 = (int)((long long)ch * Lp / nch), p1 = (int)((long long)(ch + 1) * Lp / nch), n = p1 - p0, nsub = (n + SUB - 1) / SUB;
        const bool has_new = ch == nch - 1;
        const size_t lbase = (size_t)l * P.max_seq * P.KVD + (size_t)kvh * HD;
        auto sub_begin = [&](int s) { return p0 + n * s / nsub; };
        auto copy_rows = [&](uint8_t* dst, int ld, const __half* src, int s) {
            const int b0 = sub_begin(s), np = min(sub_begin(s + 1), pos) - b0;             // the new position is not in the cache yet
            for (int i = tid; i < np * (HD / 8); i += DNT) {
                const int r = i / (HD / 8), c = i - r * (HD / 8);
                cp_async16(dst + r * ld + c * 16, src + lbase + (size_t)(b0 + r) * P.KVD + c * 8);
            }
            cp_async_commit();
        };
        // rows of earlier positions: written before this launch, or by steps that the greedy pick orders before this one (rows_ordered)
        copy_rows(ks, KLD, P.kc, 0); copy_rows(vs, VLD, P.vc, 0);
        // q of the group, and k / v of the new position (packed order: dim d of a head sits at 2d (d < HD/2) or 2(d-HD/2)+1)
        constexpr int QN = (G * HD + DNT - 1) / DNT;
        unsigned qw[QN + 2], valid = 0;
        #pragma unroll
        for (int k = 0; k < QN; k++) if (tid + k * DNT < G * HD) valid |= 1u << k;
        if (has_new && tid < HD) valid |= 3u << QN;
        const unsigned long long* qv = xw_read(P) + P.xo.qkv;
        const int dk = tid < HD / 2 ? 2 * tid : 2 * (tid - HD / 2) + 1;
        const bool okq = tw_poll(P, tag_in, valid, [&](int k) -> const unsigned long long* {
            if (k < QN) {
                const int i = tid + k * DNT, j = i / HD, d = i % HD, pk = d < HD / 2 ? 2 * d : 2 * (d - HD / 2) + 1;
                return qv + (size_t)(h0 + j) * HD + pk;
            }
            return k == QN ? qv + nq + (size_t)kvh * HD + dk : qv + nq + P.KVD + (size_t)kvh * HD + tid;
        }, qw);
        // the order the MMA reads q in: lane (row, t) takes the 16-byte pieces t, t + 4, .. of a row
        auto qslot = [](int row, int d) { return ((d >> 5) * 8 + (d & 7)) * 32 + row * 4 + ((d >> 3) & 3); };
        #pragma unroll
        for (int k = 0; k < QN; k++) {
            const int i = tid + k * DNT;
            if (i < G * HD) { const int j = i / HD, d = i % HD; qs[qslot(j, d)] = (double)__uint_as_float(qw[k]); }
        }
        for (int i = tid + G * HD; i < 8 * HD; i += DNT) qs[qslot(i / HD, i % HD)] = 0.0;
        const __half knew = __float2half_rn(__uint_as_float(qw[QN])), vnew = __float2half_rn(__uint_as_float(qw[QN + 1]));
        if (has_new && tid < HD) { P.kc[lbase + (size_t)pos * P.KVD + tid] = knew; P.vc[lbase + (size_t)pos * P.KVD + tid] = vnew; }
        if (tid < 8) { rm[tid] = -INFINITY; rl[tid] = 0.0; }
        prof_mark(P, 14);
        const float inv = __fdiv_rn(1.f, __fsqrt_rn((float)HD));
        double o[2][NTW][2];                        // two chains
        #pragma unroll
        for (int c = 0; c < 2; c++)
            #pragma unroll
            for (int i = 0; i < NTW; i++) o[c][i][0] = o[c][i][1] = 0.0;
        #pragma unroll 1
        for (int s = 0; s < nsub; s++) {
            const int b0 = sub_begin(s), np = sub_begin(s + 1) - b0;
            cp_async_wait<1>();                     // the K rows (the V rows were requested after them)
            if (has_new && s == nsub - 1 && tid < HD) {
                reinterpret_cast<__half*>(ks + (pos - b0) * KLD)[tid] = knew;
                reinterpret_cast<__half*>(vs + (pos - b0) * VLD)[tid] = vnew;
            }
            if (s == 0) { if (!cta__syncthreads_and(okq ? 1 : 0)) { ok = false; break; } } else cta__syncthreads();
            // scores: warp = every 8th group of 8 positions
            #pragma unroll 1
            for (int t = warp; t * 8 < np; t += DNW) {
                const uint8_t* kr = ks + min(t * 8 + g, np - 1) * KLD + t4 * 16;
                double c[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
                #pragma unroll
                for (int i = 0; i < HD / 32; i++) {
                    const uint4 kw = *reinterpret_cast<const uint4*>(kr + i * 64);
                    const unsigned w[4] = {kw.x, kw.y, kw.z, kw.w};
                    #pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const double* a = qs + (i * 8 + e * 2) * 32 + lane;
                        dmma884(c[0], a[0], half_to_double(w[e] & 0xffffu)); dmma884(c[1], a[32], half_to_double(w[e] >> 16));
                    }
                }
                #pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int pp = t * 8 + 2 * t4 + e;
                    if (pp < SUB) sc[g * SCL + pp] = pp < np ? __fmul_rn(__double2float_rn(__dadd_rn(c[0][e], c[1][e])), inv) : -INFINITY;
                }
            }
            cta__syncthreads();
            prof_mark(P, 27);
            if (s + 1 < nsub) copy_rows(ks, KLD, P.kc, s + 1); else cp_async_commit();
            // weights: one warp per head
            if (warp < G) {
                float x[kSplitSubMax / 32], m = -INFINITY;
                #pragma unroll
                for (int i = 0; i < kSplitSubMax / 32; i++) { x[i] = lane + 32 * i < np ? sc[warp * SCL + lane + 32 * i] : -INFINITY; m = fmaxf(m, x[i]); }
                m = warp_max_float(m);
                const double mo = rm[warp], mn = fmax(mo, (double)m);
                double ls = 0.0;
                #pragma unroll
                for (int i = 0; i < kSplitSubMax / 32; i++) {
                    if (32 * i >= np) break;                                               // warp-uniform
                    const double w = lane + 32 * i < np ? exp_shared((double)x[i] - mn) : 0.0;
                    const int pp = lane + 32 * i;
                    if (pp < SUB) wt[(pp >> 2) * 32 + warp * 4 + (pp & 3)] = w;
                    ls = __dadd_rn(ls, w);
                }
                #pragma unroll
                for (int q = 16; q; q >>= 1) ls = __dadd_rn(ls, __shfl_xor_sync(0xffffffffu, ls, q));
                if (lane == 0) {
                    const double f = mo == mn ? 1.0 : mo == -INFINITY ? 0.0 : exp_shared(mo - mn);
                    rf[warp] = f; rm[warp] = mn; rl[warp] = __fma_rn(rl[warp], f, ls);
                }
            }
            cp_async_wait<1>();                     // the V rows
            cta__syncthreads();
            prof_mark(P, 29);
            // values: warp = HD/8 dims, all positions
            if (warp < VW) {
                if (s > 0) {
                    const double f = g < G ? rf[g] : 1.0;
                    #pragma unroll
                    for (int c = 0; c < 2; c++)
                        #pragma unroll
                        for (int i = 0; i < NTW; i++) { o[c][i][0] = __dmul_rn(o[c][i][0], f); o[c][i][1] = __dmul_rn(o[c][i][1], f); }
                }
                const uint8_t* vr = vs + (warp * (8 * NTW) + g * NTW) * 2;
                #pragma unroll 2
                for (int u = 0; u * 4 < np; u += 2) {
                    #pragma unroll
                    for (int c = 0; c < 2; c++) {
                        if ((u + c) * 4 >= np) break;                                      // warp-uniform
                        const uint8_t* v = vr + min((u + c) * 4 + t4, np - 1) * VLD;
                        const double w = wt[(u + c) * 32 + lane];
                        if constexpr (NTW == 2) {
                            const unsigned vw = *reinterpret_cast<const unsigned*>(v);
                            dmma884(o[c][0], w, half_to_double(vw & 0xffffu)); dmma884(o[c][NTW - 1], w, half_to_double(vw >> 16));
                        } else {
                            dmma884(o[c][0], w, half_to_double(*reinterpret_cast<const unsigned short*>(v)));
                        }
                    }
                }
            }
            cta__syncthreads();                        // scores, weights and V rows may be written again
            if (s + 1 < nsub) copy_rows(vs, VLD, P.vc, s + 1);
        }
        if (!ok) cp_async_wait<0>();                // copies in flight target the staging area
        prof_mark(P, 15);
        if (ok) {
            if (warp < VW && g < G) {
                double* gp = P.attn_part + ((size_t)(h0 + g) * P.max_chunks + ch) * SW;
                #pragma unroll
                for (int i = 0; i < NTW; i++)
                    #pragma unroll
                    for (int e = 0; e < 2; e++) __stcg(gp + warp * (8 * NTW) + (2 * t4 + e) * NTW + i, __dadd_rn(o[0][i][e], o[1][i][e]));
            }
            if (tid < G) __stcg(P.attn_part + ((size_t)(h0 + tid) * P.max_chunks + ch) * SW + HD, rl[tid]);
            cta__syncthreads();
            if (tid < G) {
                fence_acq_rel_gpu();                // the partial, and the new position's rows, before the word that announces them
                pub.local(P.xo.attm + (h0 + tid) * P.max_chunks + ch, __float_as_uint((float)rm[tid]));
            }
        }
        prof_mark(P, 16);
    }
    // merge: one CTA per 32-dim block of a head, its warps share the chunks; lane = dim
    const int nblk = P.NH * (HD / 32);
    for (int b = blockIdx.x; b < nblk && ok; b += gridDim.x) {
        const int head = b / (HD / 32), d0 = (b - head * (HD / 32)) * 32;
        unsigned mw[kMaxChunkWords], valid = 0;
        #pragma unroll
        for (int k = 0; k < kMaxChunkWords; k++) if (lane + 32 * k < nch) valid |= 1u << k;
        const unsigned long long* mv = P.xw + P.xo.attm + (size_t)head * P.max_chunks;
        const bool okm = tw_poll(P, pub.tag, valid, [&](int k) { return mv + lane + 32 * k; }, mw);
        fence_acq_rel_gpu();
        __syncwarp();                               // a lane reads sums whose words other lanes polled
        float m = -INFINITY;
        #pragma unroll
        for (int k = 0; k < kMaxChunkWords; k++) if (valid >> k & 1u) m = fmaxf(m, __uint_as_float(mw[k]));
        m = warp_max_float(m);
        // this warp's chunks: warp, warp + 8, ..; lane i prepares the factor of the i-th
        const int mine = (nch - warp + DNW - 1) / DNW;
        const double* gp = P.attn_part + ((size_t)head * P.max_chunks + warp) * SW;
        double f_l = 0.0;
        {
            const int c = warp + DNW * lane;                                               // its maximum is word c / 32 of lane c % 32
            unsigned w = 0;
            #pragma unroll
            for (int k = 0; k < kMaxChunkWords; k++) { const unsigned x = __shfl_sync(0xffffffffu, mw[k], c & 31); if ((c >> 5) == k) w = x; }
            const float mc = __uint_as_float(w);
            if (lane < mine) f_l = mc == -INFINITY ? 0.0 : exp_shared((double)mc - (double)m);
        }
        double ob = 0.0, lb = lane < mine ? __dmul_rn(__ldcg(gp + (size_t)lane * DNW * SW + HD), f_l) : 0.0;
        for (int i0 = 0; i0 < mine; i0 += 8) {
            double v[8];
            #pragma unroll
            for (int u = 0; u < 8; u++) v[u] = __ldcg(gp + (size_t)min(i0 + u, mine - 1) * DNW * SW + d0 + lane);
            #pragma unroll
            for (int u = 0; u < 8; u++) {
                const double f = __shfl_sync(0xffffffffu, f_l, (i0 + u) & 31);
                if (i0 + u < mine) ob = __fma_rn(v[u], f, ob);
            }
        }
        #pragma unroll
        for (int q = 16; q; q >>= 1) lb = __dadd_rn(lb, __shfl_xor_sync(0xffffffffu, lb, q));
        cta__syncthreads();                            // the buffer below is free (a second block of this CTA)
        red[warp * 33 + lane] = ob;
        if (lane == 0) red[warp * 33 + 32] = lb;
        ok = cta__syncthreads_and(okm ? 1 : 0) != 0;
        if (warp == 0 && ok) {
            double den = red[32];
            ob = red[lane];
            #pragma unroll
            for (int w = 1; w < DNW; w++) { ob = __dadd_rn(ob, red[w * 33 + lane]); den = __dadd_rn(den, red[w * 33 + 32]); }
            const float v = __double2float_rn(__ddiv_rn(ob, den));
            const int e = head * HD + d0 + lane;
            __stcg(P.att + e, v);
            __half dq; int sq;
            const int qv8 = quant_block_warp2(v, dq, sq);
            publish_q8_block<false>(pub, P.xo.att, P.xo.att + P.NH * HD / 4, e >> 5, lane, qv8, dq, sq);
        }
    }
    prof_mark(P, 17);
    return ok;
}

// ---- attention over a short causal range (at most 256 positions): one CTA per query head ---------------
// The whole range of a head fits one CTA, so the softmax is computed the way the reference's CPU program writes it
// (src/cpu_infer.cpp:121-140): all scores, their maximum, exp(score - max) once per position, then the weighted sum of the
// V rows and the division - no running maximum, no rescaling, no merge of partial states.
//   pass 1  warp w takes a contiguous eighth of the positions; eight lanes share a position (HD/8 dims each), the dot
//           product is carried in double and folded over the eight lanes; score = fp32(dot) * 1/sqrt(HD) in fp32;
//   max     every warp scans the scores in shared memory; thread t computes the weight of position t (one double exp);
//   pass 2  warp w, same positions: lane = dims {lane + 32 i}; o += w[p] * V[p], l += w[p] in position order;
//   finish  warp i (i < HD/32) adds the eight warps' partial sums in warp order, divides, rounds to fp32, quantizes its
//           32-dim block to q8_0 and publishes it.
// Same interface as attention_split.
template <int HD, int GQ>
static __device__ __noinline__ bool attention_short(const DecodeParams& P, int l, int pos, uint8_t* stage, unsigned tag_in, const Pub pub) {
    constexpr int DPW = HD / 32;
    constexpr int LPP = 8, DPL = HD / LPP, QSTR = DPL + 2;                 // lanes per position in pass 1, dims per lane, padded stride
    constexpr int KV4 = DPL * 2 / 16 > 0 ? DPL * 2 / 16 : 1;              // 16-byte loads per lane and position
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if ((int)blockIdx.x >= P.NH) return true;
    const int head = blockIdx.x, kvh = head / GQ, Lp = pos + 1;
    double* qs = reinterpret_cast<double*>(stage);                         // [LPP][QSTR]
    double* wt = qs + LPP * QSTR;                                          // [256] weights
    double* ow = wt + 256;                                                 // [DNW][HD] partial outputs
    double* lw = ow + DNW * HD;                                            // [DNW] partial denominators
    float* sc = reinterpret_cast<float*>(lw + DNW);                        // [256] scores
    const int nq = P.NH * HD;
    unsigned qw[3], valid = 0;
    if (tid < HD) valid = 7u;
    const unsigned long long* qv = xw_read(P) + P.xo.qkv;
    const int dk = tid < HD / 2 ? 2 * tid : 2 * (tid - HD / 2) + 1;    // packed slot of dim `tid`
    const bool okq = tw_poll(P, tag_in, valid, [&](int k) -> const unsigned long long* {
        return k == 0 ? qv + (size_t)head * HD + dk : k == 1 ? qv + nq + (size_t)kvh * HD + dk : qv + nq + P.KVD + (size_t)kvh * HD + tid;
    }, qw);
    if (tid < HD) {
        qs[(tid / DPL) * QSTR + tid % DPL] = (double)__uint_as_float(qw[0]);
        // CTAs that share a kv head store the same bits
        P.kc[((size_t)l * P.max_seq + pos) * P.KVD + (size_t)kvh * HD + tid] = __float2half_rn(__uint_as_float(qw[1]));
        P.vc[((size_t)l * P.max_seq + pos) * P.KVD + (size_t)kvh * HD + tid] = __float2half_rn(__uint_as_float(qw[2]));
    }
    if (!cta__syncthreads_and(okq ? 1 : 0)) return false;
    prof_mark(P, 14);
    const float inv = __fdiv_rn(1.f, __fsqrt_rn((float)HD));
    const int a0 = (int)((long long)Lp * warp / DNW), a1 = (int)((long long)Lp * (warp + 1) / DNW);      // at most 32 positions
    const __half* kbase = P.kc + ((size_t)l * P.max_seq) * P.KVD + (size_t)kvh * HD;
    const __half* vbase = P.vc + ((size_t)l * P.max_seq) * P.KVD + (size_t)kvh * HD;
    const int np = a1 - a0;
    // pass 1: four positions per sweep, rounds of four sweeps whose K rows are all requested before the first is used
    {
        const int sub = lane >> 3, li = lane & 7;
        const double* qj = qs + li * QSTR;
        #pragma unroll 1
        for (int s0 = 0; s0 * 4 < np; s0 += 4) {
            uint4 kraw[4][KV4];
            #pragma unroll
            for (int u = 0; u < 4; u++) {
                if ((s0 + u) * 4 >= np) continue;                          // warp-uniform
                const int pi = min((s0 + u) * 4 + sub, np - 1);
                const __half* kr = kbase + (size_t)(a0 + pi) * P.KVD + li * DPL;
                if constexpr (DPL >= 8) {
                    #pragma unroll
                    for (int c = 0; c < KV4; c++) kraw[u][c] = __ldcg(reinterpret_cast<const uint4*>(kr) + c);
                } else {
                    const uint2 k2 = __ldcg(reinterpret_cast<const uint2*>(kr));
                    kraw[u][0] = make_uint4(k2.x, k2.y, 0u, 0u);
                }
            }
            #pragma unroll
            for (int u = 0; u < 4; u++) {
                if ((s0 + u) * 4 < np) {                                   // warp-uniform
                    const int pi = (s0 + u) * 4 + sub;
                    double acc = 0.0;
                    #pragma unroll
                    for (int c = 0; c < KV4; c++) {
                        const __half2* hh = reinterpret_cast<const __half2*>(&kraw[u][c]);
                        #pragma unroll
                        for (int e = 0; e < 4; e++) {
                            if (c * 8 + 2 * e < DPL) {
                                const float2 f = __half22float2(hh[e]);
                                const double2 qq = *reinterpret_cast<const double2*>(qj + c * 8 + 2 * e);
                                acc = __fma_rn(qq.x, (double)f.x, acc);
                                acc = __fma_rn(qq.y, (double)f.y, acc);
                            }
                        }
                    }
                    #pragma unroll
                    for (int sft = 1; sft <= 4; sft <<= 1) acc = __dadd_rn(acc, __shfl_xor_sync(0xffffffffu, acc, sft));
                    if (li == 0 && pi < np) sc[a0 + pi] = __fmul_rn(__double2float_rn(acc), inv);
                }
            }
        }
    }
    prof_mark(P, 27);
    // the V rows of this warp's positions: requested now, used after the weights are known
    // (lane = the dim pairs {2 lane, 2 lane + 1} + 64 j: one 4-byte load per pair; head_dim 32: lane = dim)
    // (the first sixteen; a warp has more only beyond 128 positions, and fetches those when it gets there)
    constexpr int VB = 16, VP = DPW >= 2 ? DPW / 2 : 1;
    unsigned vh[VB][VP];
    auto load_v = [&](int r) {
        #pragma unroll
        for (int u = 0; u < VB; u++) {
            const __half* vrow = vbase + (size_t)(a0 + min(r * VB + u, max(np - 1, 0))) * P.KVD;
            if constexpr (DPW >= 2) {
                #pragma unroll
                for (int j = 0; j < VP; j++) vh[u][j] = __ldcg(reinterpret_cast<const unsigned*>(vrow) + lane + 32 * j);
            } else {
                vh[u][0] = __ldcg(reinterpret_cast<const unsigned short*>(vrow) + lane);
            }
        }
    };
    if (np > 0) load_v(0);
    prof_mark(P, 28);
    cta__syncthreads();
    prof_mark(P, 15);
    // maximum over the whole range (every warp scans all scores), then one weight per thread
    float mx = -INFINITY;
    #pragma unroll
    for (int i = 0; i < 8; i++) if (lane + 32 * i < Lp) mx = fmaxf(mx, sc[lane + 32 * i]);
    mx = warp_max_float(mx);
    if (tid < Lp) wt[tid] = exp_shared((double)sc[tid] - (double)mx);
    prof_mark(P, 29);
    cta__syncthreads();
    prof_mark(P, 30);
    // pass 2
    double o[DPW], ls = 0.0;
    #pragma unroll
    for (int i = 0; i < DPW; i++) o[i] = 0.0;
    #pragma unroll 1
    for (int r = 0; r * VB < np; r++) {
        if (r > 0) load_v(r);
        #pragma unroll
        for (int u = 0; u < VB; u++) {
            if (r * VB + u < np) {
                const double w = wt[a0 + r * VB + u];
                ls = __dadd_rn(ls, w);
                if constexpr (DPW >= 2) {
                    #pragma unroll
                    for (int j = 0; j < VP; j++) {
                        const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&vh[u][j]));
                        o[2 * j] = __fma_rn(w, (double)f.x, o[2 * j]);
                        o[2 * j + 1] = __fma_rn(w, (double)f.y, o[2 * j + 1]);
                    }
                } else {
                    o[0] = __fma_rn(w, (double)__half2float(__ushort_as_half((unsigned short)vh[u][0])), o[0]);
                }
            }
        }
    }
    if constexpr (DPW >= 2) {
        #pragma unroll
        for (int j = 0; j < VP; j++) *reinterpret_cast<double2*>(ow + warp * HD + 2 * (lane + 32 * j)) = make_double2(o[2 * j], o[2 * j + 1]);
    } else {
        ow[warp * HD + lane] = o[0];
    }
    if (lane == 0) lw[warp] = ls;
    prof_mark(P, 31);
    // the new position's K / V rows (plain stores above) are performed before anything this CTA publishes
    if (tid < HD) __threadfence();
    cta__syncthreads();
    prof_mark(P, 16);
    if (warp < DPW) {
        const int d = warp * 32 + lane;
        double ob = ow[d], ll = lw[0];
        #pragma unroll
        for (int w = 1; w < DNW; w++) { ob = __dadd_rn(ob, ow[w * HD + d]); ll = __dadd_rn(ll, lw[w]); }
        const float v = __double2float_rn(__ddiv_rn(ob, ll));
        const int e = head * HD + d;
        __stcg(P.att + e, v);
        __half dq; int sq;
        const int qv8 = quant_block_warp2(v, dq, sq);
        publish_q8_block<false>(pub, P.xo.att, P.xo.att + P.NH * HD / 4, e >> 5, lane, qv8, dq, sq);
    }
    prof_mark(P, 17);
    return true;
}

// ---- short-range attention on the CTAs set aside for it ------------------------------------------------
// A CTA of [0, attn_ctas) handles HPC query heads of one kv head and nothing else, which buys two things.  (1) The K and V
// rows of the cached positions are known long before the layer's q arrives, so the CTA copies them into shared memory
// ahead of time (asynchronous 16-byte copies, rows padded by 16 bytes against bank conflicts; requested as soon as the layer before has left
// the buffer): between q's arrival and the published output there is
// no global load at all.  (2) One fp16 -> double conversion of a K or V element serves all HPC heads.
// The new position's K and V come with q as tagged words; they go into the shared-memory rows directly and to the global
// cache after the output has been published (fenced before this CTA's next output, which is what later readers wait for).
// The two passes and the softmax are attention_short's; a dot product is added in another order (eight partial sums over an eighth of the dimensions
// each, in a tree), in double and rounded to fp32 once: the same bits in every test, observed and not proved.
constexpr int kAttnRows = kShortAttnMax;
template <int HD> __host__ __device__ constexpr int attn_row_bytes() { return 2 * HD + 16; }
__host__ __device__ inline size_t attn_dedicated_smem(int HD, int HPC) {
    return (size_t)2 * kAttnRows * (2 * HD + 16) + (size_t)HPC * (HD + 16) * 8 + (size_t)HPC * kAttnRows * 8 + (size_t)DNW * HPC * HD * 8 +
           (size_t)DNW * HPC * 8 + (size_t)HPC * kAttnRows * 4 + (size_t)DNW * HPC * kAttnRows * 8 + 64;
}
// query heads per attention CTA: two where the group size is even (1.5B: six CTAs of two heads; three heads per CTA
// measured 4.5 us per layer on the critical path), one where it is odd or at most two
__host__ __device__ constexpr int attn_heads_per_cta(int G) { return G % 2 == 0 && G > 2 ? 2 : 1; }

// Returns a CTA-uniform ok.
template <int HD, int GQ, int HPC>
__device__ __forceinline__ bool attention_dedicated(const DecodeParams& P, int l, int pos, uint8_t* smem, unsigned tag_in, const Pub pub) {
    constexpr int DPW = HD / 32, RSB = attn_row_bytes<HD>();
    constexpr int LPP = 8, DPL = HD / LPP, QSTR = DPL + 2;
    constexpr int QN = (HPC * HD + DNT - 1) / DNT;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int h0 = (int)blockIdx.x * HPC, kvh = h0 / GQ, Lp = pos + 1, nq = P.NH * HD;
    uint8_t* Kb = smem; uint8_t* Vb = smem + (size_t)kAttnRows * RSB;
    double* qs = reinterpret_cast<double*>(smem + (size_t)2 * kAttnRows * RSB);   // [HPC][LPP][QSTR]
    double* wt = qs + HPC * LPP * QSTR;                                         // [HPC][rows]
    double* ow = wt + HPC * kAttnRows;                                          // [DNW][HPC][HD]
    double* lw = ow + DNW * HPC * HD;                                           // [DNW][HPC]
    double* pd = lw + DNW * HPC;                                                // [DNW][HPC][rows] partial scores
    float* sc = reinterpret_cast<float*>(pd + DNW * HPC * kAttnRows);           // [HPC][rows]
    // the rows of the earlier positions: requested before q is waited for (this CTA has nothing else to do)
    #pragma unroll 2
    for (int i = tid; i < pos * (HD / 8); i += DNT) {
        const int r = i / (HD / 8), c = (i % (HD / 8)) * 16;
        const size_t row = ((size_t)l * P.max_seq + r) * P.KVD + (size_t)kvh * HD + c / 2;
        cp_async16(Kb + r * RSB + c, P.kc + row);
        cp_async16(Vb + r * RSB + c, P.vc + row);
    }
    cp_async_commit();
    // q of this CTA's heads and k / v of the new position (tagged words, packed order: dim d sits at 2d (d < HD/2) or 2(d-HD/2)+1)
    unsigned qw[QN + 2], valid = 0;
    #pragma unroll
    for (int k = 0; k < QN; k++) if (tid + k * DNT < HPC * HD) valid |= 1u << k;
    if (tid < HD) valid |= 3u << QN;
    const unsigned long long* qv = xw_read(P) + P.xo.qkv;
    const int dk = tid < HD / 2 ? 2 * tid : 2 * (tid - HD / 2) + 1;
    bool ok = tw_poll(P, tag_in, valid, [&](int k) -> const unsigned long long* {
        if (k < QN) {
            const int i = tid + k * DNT, j = i / HD, d = i % HD, pk = d < HD / 2 ? 2 * d : 2 * (d - HD / 2) + 1;
            return qv + (size_t)(h0 + j) * HD + pk;
        }
        return k == QN ? qv + nq + (size_t)kvh * HD + dk : qv + nq + P.KVD + (size_t)kvh * HD + tid;
    }, qw);
    #pragma unroll
    for (int k = 0; k < QN; k++) {
        const int i = tid + k * DNT;
        if (i < HPC * HD) { const int j = i / HD, d = i % HD; qs[(j * LPP + d / DPL) * QSTR + d % DPL] = (double)__uint_as_float(qw[k]); }
    }
    const __half knew = __float2half_rn(__uint_as_float(qw[QN])), vnew = __float2half_rn(__uint_as_float(qw[QN + 1]));
    if (tid < HD) {
        reinterpret_cast<__half*>(Kb + (size_t)pos * RSB)[tid] = knew;
        reinterpret_cast<__half*>(Vb + (size_t)pos * RSB)[tid] = vnew;
    }
    prof_mark(P, 14);
    cp_async_wait<0>();
    if (!cta__syncthreads_and(ok ? 1 : 0)) return false;
    prof_mark(P, 27);
    const float inv = __fdiv_rn(1.f, __fsqrt_rn((float)HD));
    const int a0 = (int)((long long)Lp * warp / DNW), a1 = (int)((long long)Lp * (warp + 1) / DNW), np = a1 - a0;
    // pass 1: a warp takes an eighth of the dimensions, q of which stays in its registers, lane = position: one fp16 -> double
    // conversion of a K element serves all heads, and the eight partial dot products meet in shared memory.  (A thread per position
    // over all dimensions reads q as broadcasts, 128 of them per warp at four cycles each: 1.25 us per layer at a hundred positions.)
    // Rows are 16 bytes longer than their data, so the eight lanes of a quarter warp cover all banks.
    {
        constexpr int DW = HD / DNW;                                            // dims of a warp
        double qr[HPC][DW];
        #pragma unroll
        for (int j = 0; j < HPC; j++)
            #pragma unroll
            for (int e = 0; e < DW; e++) qr[j][e] = qs[(j * LPP + (warp * DW + e) / DPL) * QSTR + (warp * DW + e) % DPL];
        #pragma unroll 1
        for (int p0 = 0; p0 < Lp; p0 += 32) {
            const uint8_t* kr = Kb + (size_t)min(p0 + lane, Lp - 1) * RSB + warp * (DW * 2);
            unsigned kw[DW / 2];
            if constexpr (DW >= 8) {
                #pragma unroll
                for (int c = 0; c < DW / 8; c++) { const uint4 v = reinterpret_cast<const uint4*>(kr)[c]; kw[4 * c] = v.x; kw[4 * c + 1] = v.y; kw[4 * c + 2] = v.z; kw[4 * c + 3] = v.w; }
            } else {
                const uint2 v = *reinterpret_cast<const uint2*>(kr); kw[0] = v.x; kw[1] = v.y;
            }
            double acc[HPC][2];                                                 // two chains per head
            #pragma unroll
            for (int j = 0; j < HPC; j++) acc[j][0] = acc[j][1] = 0.0;
            #pragma unroll
            for (int e = 0; e < DW / 2; e++) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&kw[e]));
                const double k0 = f.x, k1 = f.y;
                #pragma unroll
                for (int j = 0; j < HPC; j++) { acc[j][0] = __fma_rn(qr[j][2 * e], k0, acc[j][0]); acc[j][1] = __fma_rn(qr[j][2 * e + 1], k1, acc[j][1]); }
            }
            #pragma unroll
            for (int j = 0; j < HPC; j++) pd[(warp * HPC + j) * kAttnRows + p0 + lane] = __dadd_rn(acc[j][0], acc[j][1]);
        }
    }
    cta__syncthreads();
    if (tid < Lp) {
        #pragma unroll
        for (int j = 0; j < HPC; j++) {
            const double* p = pd + j * kAttnRows + tid;
            constexpr int S = HPC * kAttnRows;
            sc[j * kAttnRows + tid] = __fmul_rn(__double2float_rn(tree_sum8(p[0], p[S], p[2 * S], p[3 * S], p[4 * S], p[5 * S], p[6 * S], p[7 * S])), inv);
        }
    }
    cta__syncthreads();
    prof_mark(P, 15);
    // per head: maximum over the whole range, then one weight per (head, position)
    float mx[HPC];
    #pragma unroll
    for (int j = 0; j < HPC; j++) {
        float m = -INFINITY;
        #pragma unroll
        for (int i = 0; i < kAttnRows / 32; i++) if (lane + 32 * i < Lp) m = fmaxf(m, sc[j * kAttnRows + lane + 32 * i]);
        mx[j] = warp_max_float(m);
    }
    for (int idx = tid; idx < HPC * Lp; idx += DNT) {
        const int j = idx / Lp, p = idx - j * Lp;
        float mj = mx[0];
        #pragma unroll
        for (int jj = 1; jj < HPC; jj++) if (j == jj) mj = mx[jj];
        wt[j * kAttnRows + p] = exp_shared((double)sc[j * kAttnRows + p] - (double)mj);
    }
    prof_mark(P, 29);
    cta__syncthreads();
    prof_mark(P, 30);
    // pass 2: lane = the dim pairs {2 lane, 2 lane + 1} + 64 jj (head_dim 32: lane = dim)
    constexpr int VP = DPW >= 2 ? DPW / 2 : 1;
    double o[HPC][DPW], ls[HPC];
    #pragma unroll
    for (int j = 0; j < HPC; j++) {
        ls[j] = 0.0;
        #pragma unroll
        for (int i = 0; i < DPW; i++) o[j][i] = 0.0;
    }
    #pragma unroll 2
    for (int u = 0; u < np; u++) {
        const uint8_t* vrow = Vb + (size_t)(a0 + u) * RSB;
        double vd[DPW];
        if constexpr (DPW >= 2) {
            #pragma unroll
            for (int jj = 0; jj < VP; jj++) {
                const float2 f = __half22float2(reinterpret_cast<const __half2*>(vrow)[lane + 32 * jj]);
                vd[2 * jj] = (double)f.x; vd[2 * jj + 1] = (double)f.y;
            }
        } else {
            vd[0] = (double)__half2float(reinterpret_cast<const __half*>(vrow)[lane]);
        }
        #pragma unroll
        for (int j = 0; j < HPC; j++) {
            const double w = wt[j * kAttnRows + a0 + u];
            ls[j] = __dadd_rn(ls[j], w);
            #pragma unroll
            for (int i = 0; i < DPW; i++) o[j][i] = __fma_rn(w, vd[i], o[j][i]);
        }
    }
    #pragma unroll
    for (int j = 0; j < HPC; j++) {
        double* od = ow + (size_t)(warp * HPC + j) * HD;
        if constexpr (DPW >= 2) {
            #pragma unroll
            for (int jj = 0; jj < VP; jj++) *reinterpret_cast<double2*>(od + 2 * (lane + 32 * jj)) = make_double2(o[j][2 * jj], o[j][2 * jj + 1]);
        } else {
            od[lane] = o[j][0];
        }
        if (lane == 0) lw[warp * HPC + j] = ls[j];
    }
    prof_mark(P, 31);
    cta__syncthreads();
    prof_mark(P, 16);
    // finish: one 32-dim block of one head per warp and round
    for (int b = warp; b < HPC * DPW; b += DNW) {
        const int j = b / DPW, d = (b % DPW) * 32 + lane;
        double ob = ow[(size_t)j * HD + d], ll = lw[j];
        #pragma unroll
        for (int w = 1; w < DNW; w++) { ob = __dadd_rn(ob, ow[(size_t)(w * HPC + j) * HD + d]); ll = __dadd_rn(ll, lw[w * HPC + j]); }
        const float v = __double2float_rn(__ddiv_rn(ob, ll));
        const int e = (h0 + j) * HD + d;
        __stcg(P.att + e, v);
        __half dq; int sq;
        const int qv8 = quant_block_warp2(v, dq, sq);
        publish_q8_block<false>(pub, P.xo.att, P.xo.att + P.NH * HD / 4, e >> 5, lane, qv8, dq, sq);
    }
    prof_mark(P, 17);
    // the new position into the global cache (CTAs that share a kv head store the same bits); performed before this CTA publishes anything else
    if (tid < HD) {
        P.kc[((size_t)l * P.max_seq + pos) * P.KVD + (size_t)kvh * HD + tid] = knew;
        P.vc[((size_t)l * P.max_seq + pos) * P.KVD + (size_t)kvh * HD + tid] = vnew;
        __threadfence();
    }
    cta__syncthreads();                                  // the buffer is free, the stores are fenced
    return true;
}

// The whole life of a CTA that does nothing but attention: every step, every layer, wait for q, attend, publish.  One call
// at the top of the kernel, out of line: its registers and instructions are its own, and the CTAs that carry the GEMV phases
// never see any of it (measured: an out-of-line call inside their per-layer loop, or this code inlined into it, costs the
// GEMV phases 10 - 25 %).
// whether this build holds the attention variant a position needs (the host picks the build by the launch's positions)
__device__ __forceinline__ bool lean_regime_ok(int pos, int attn_ctas) {
#if MI_LEAN == 1
    return pos + 1 <= kShortAttnMax && attn_ctas > 0;
#elif MI_LEAN == 2
    return pos + 1 > kShortAttnMax;
#else
    return true;
#endif
}

// Where rows of the cache that one CTA writes in a step become readable by every CTA in the next one.  attention_split requests the rows
// of earlier positions before it has polled anything of its layer, and the tagged words that its CTA has polled since the last
// step carry no order for them: they came from CTAs that had passed on other words without a fence.  So the greedy pick, which every GEMV CTA
// publishes to and polls once per step, is an ordering point in the builds that have attention_split: a CTA's candidate is
// stored behind a fence (and behind a barrier, so the fence speaks for all its threads), and a CTA's threads fence once they
// have polled all candidates.  The attention CTAs, which take chunks as well but have no part in the pick, say behind a fence that they have left the step
// (attdone; two sets by step parity, because an attention CTA may leave the next step before a GEMV CTA has looked), and poll the
// candidates before their next step.  No candidate is overwritten before they have: every CTA below attn_ctas has a chunk in every layer
// (attn_ctas <= 7 NKV, and there are at least 9 NKV chunks or as many as the grid holds), so the next pick descends from it.
// Two fences per step where the chain of a step is a hundred and forty hops.
constexpr bool kRowsCross = MI_LEAN != 1;
__device__ __forceinline__ int attdone_off(const DecodeParams& P, int step) { return P.xo.attdone + (step & 1) * P.attn_ctas; }

// attention CTAs, before a step that reads rows of the step before it; tag: that step's pick.  Whole CTA, returns a CTA-uniform ok.
static __device__ __noinline__ bool rows_ordered(const DecodeParams& P, unsigned tag, int step) {
    const int n_cand = (P.tp.on ? P.tp.world : 1) * ((int)gridDim.x - P.attn_ctas), n = n_cand + P.attn_ctas, done = attdone_off(P, step);
    bool ok = true;
    for (int i0 = 0; i0 < n && ok; i0 += DNT) {
        const int i = i0 + (int)threadIdx.x;
        unsigned w[1];
        ok = tw_poll(P, tag, i < n ? 1u : 0u, [&](int) { return i < n_cand ? xw_read(P) + P.xo.cand + i * 4 : P.xw + done + i - n_cand; }, w);
    }
    fence_acq_rel_gpu();
    return cta__syncthreads_and(ok ? 1 : 0) != 0;
}

template <int HD, int G>
static __device__ __noinline__ void attn_cta_main(const DecodeParams& P, int step0, int step1, int ph0, int ph1, uint8_t* smem, uint8_t* stage) {
    const int nph = 5 * P.L + 1;
    pdl_launch_dependents();
    pdl_wait_prior();
    const unsigned epoch = __ldcg(P.epoch_dev);
    const int pos_base = P.pos_dev ? __ldcg(P.pos_dev) : P.pos0;
    bool ok = true;
    int err_code = MI_ERR_TIMEOUT;
#if MI_PROF
    const long long prof_c0 = clock64(); const unsigned long long prof_t0 = gtime_ns();
    if (threadIdx.x == 0) s_prof_t = prof_t0;
#endif
    for (int step = step0; step < step1 && ok; step++) {
        const int pos = pos_base + step;
        if (pos < 0 || pos >= P.max_seq || !lean_regime_ok(pos, P.attn_ctas)) { ok = false; err_code = MI_ERR_LIMIT; break; }
        const unsigned tag0 = epoch + (unsigned)(step - step0) * (unsigned)nph + 1u;
        if (P.stop_token >= 0 && step > step0 && step >= P.n_forced && ph0 == 0 && ph1 == nph) {
            // the stop rule: learn the token the previous step picked (its lm_head phase carries tag tag0 - 1)
            unsigned tw[1];
            const bool got = tw_poll(P, tag0 - 1u, 1u, [&](int) { return P.xw + P.xo.tokw; }, tw);
            ok = cta__syncthreads_and(got ? 1 : 0) != 0;
            if (!ok || (int)tw[0] == P.stop_token) break;
        }
        // (only a launch over whole steps has more than one)
        if (kRowsCross && step > step0 && ph0 == 0 && ph1 == nph && pos + 1 > kShortAttnMax && !(ok = rows_ordered(P, tag0 - 1u, step - 1))) break;
        for (int l = max(0, (ph0 + 3) / 5); 5 * l + 1 < ph1 && l < P.L && ok; l++) {
            const int ph = 5 * l + 1;
            Pub pub;
            pub.xw = P.xw; pub.tag = tag0 + (unsigned)ph; pub.mute = ph == P.drop_phase; pub.stride = P.xo.total;
#if MI_TP
            pub.tp = &P.tp;
#endif
#if MI_LEAN <= 1
            if (pos + 1 <= kShortAttnMax) ok = attention_dedicated<HD, G, attn_heads_per_cta(G)>(P, l, pos, smem, pub.tag - 1u, pub);
#endif
#if MI_LEAN == 0
            else ok = attention_split<HD, G>(P, l, pos, stage, pub.tag - 1u, pub);
#elif MI_LEAN == 2
            ok = attention_split<HD, G>(P, l, pos, stage, pub.tag - 1u, pub);
#endif
            ok = cta__syncthreads_and(ok ? 1 : 0) != 0;
            prof_mark(P, 3);
        }
        if (kRowsCross && ok && ph1 == nph && threadIdx.x == 0) {
            fence_acq_rel_gpu();
            tw_st(P.xw + attdone_off(P, step) + blockIdx.x, tag0 + (unsigned)nph - 1u, 1u);
        }
    }
#if MI_PROF
    if (P.prof && (int)blockIdx.x == P.prof_cta) {
        if (threadIdx.x == 0) { s_prof[8] = (unsigned long long)(clock64() - prof_c0); s_prof[9] = gtime_ns() - prof_t0; }
        cta__syncthreads();
        if (threadIdx.x < kProfSlots) P.prof[threadIdx.x] += s_prof[threadIdx.x];
    }
#endif
    if (!ok && (threadIdx.x & 31) == 0) atomicMax(P.err, err_code);
}

// ---- the kernel ---------------------------------------------------------------------
template <int HD, int G>
__global__ void __launch_bounds__(DNT_ALL, 1)
decode_kernel(const __grid_constant__ DecodeParams P, int step0, int step1, int ph0, int ph1) {
    extern __shared__ __align__(128) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int njobs = 4 * P.L + 1, nph = 5 * P.L + 1;
    DecodeSmem sm;
    sm.ring = smem;
    sm.bars = reinterpret_cast<uint64_t*>(smem + (size_t)DNW * DS * DSLOT);
    unsigned* work_s = reinterpret_cast<unsigned*>(smem + (size_t)DNW * DS * DSLOT + 512);
    uint8_t* after_jobs = reinterpret_cast<uint8_t*>(work_s + kWorkSmem);
    sm.lp = reinterpret_cast<LayerPtrs*>(after_jobs);              // [<= 64]
    after_jobs += 64 * sizeof(LayerPtrs);
    sm.cs = reinterpret_cast<float*>(after_jobs);                 // [HD]: cos then sin
    sm.red = reinterpret_cast<double*>(after_jobs + 1024);         // 32 doubles
    sm.h = reinterpret_cast<float*>(after_jobs + 1024 + 256);
    sm.stage = after_jobs + 1024 + 256 + ((size_t)P.E * 4 + 127) / 128 * 128;
    sm.fold = reinterpret_cast<double*>(smem + P.fold_at);
    __shared__ int s_tok;
    __shared__ int s_quit;                             // the computing warps have left
#if MI_PROF
    if (tid < kProfSlots) s_prof[tid] = 0;
#endif

    for (int i = tid; i < P.L * (int)(sizeof(LayerPtrs) / 4); i += DNT_ALL)
        reinterpret_cast<int*>(sm.lp)[i] = __ldg(reinterpret_cast<const int*>(P.layers) + i);
    const bool attn_only = (int)blockIdx.x < P.attn_ctas;        // this CTA does nothing but attention; it lays the shared memory out its own way
    if (!attn_only) {
        const unsigned* work = P.work + (size_t)((int)blockIdx.x - P.attn_ctas) * P.work_stride;
        sm.work = P.work_smem ? work_s : work;
        if (P.work_smem) for (int i = tid; i < P.work_stride; i += DNT_ALL) work_s[i] = __ldg(work + i);
    }
    if (tid == 0) s_quit = 0;
    if (lane == 0 && warp < DNW) {
        if (!attn_only) {
            #pragma unroll
            for (int s = 0; s < 2 * DS; s++) mbar_init(&sm.bars[(s < DS ? 0 : DNW * DS - DS) + warp * DS + s], 1);
        }
        mbar_fence_init();
    }
    __syncthreads();                                  // (all nine warps; the last time)

    if (attn_only) {                                  // CTAs [0, attn_ctas): attention and nothing else
        if (warp < DNW) attn_cta_main<HD, G>(P, step0, step1, ph0, ph1, smem, sm.stage);
        return;
    }

    // jobs covered by the phase range of this launch
    auto job_of_phase = [&](int ph) -> int {          // first job at or after phase ph
        if (ph >= nph - 1) return ph >= nph ? njobs : njobs - 1;
        const int l = ph / 5, k = ph % 5;
        return 4 * l + (k == 0 ? 0 : k <= 2 ? 1 : k == 3 ? 2 : 3);
    };
    if (warp == DNW) {                                // weights depend on nothing: their stream runs ahead of all waits
        stream_weights(sm, P, lane, step1 - step0, job_of_phase(ph0), job_of_phase(ph1), &s_quit);
        return;
    }
    WarpStream ws;
    ws.init(sm, P, warp);
    pdl_launch_dependents();
    pdl_wait_prior();

    const int maxin = P.E > P.FF ? P.E : P.FF;
    int8_t* xq_s = reinterpret_cast<int8_t*>(sm.stage);
    BlockScale* xs_s = reinterpret_cast<BlockScale*>(sm.stage + maxin);
    bool ok = true, done = true, h_valid = false;                   // h_valid: this CTA's shared-memory copy of the residual stream is current
    int err_code = MI_ERR_TIMEOUT;
    const unsigned epoch = __ldcg(P.epoch_dev);
    const int pos_base = P.pos_dev ? __ldcg(P.pos_dev) : P.pos0;
    // candidates of the greedy pick: one {value, index} pair of words per CTA (and per GPU when the exchange runs in here)
    const int cand_world = P.tp.on ? P.tp.world : 1, n_cand = cand_world * ws.ggrid;
    const int my_cand = P.xo.cand + ((P.tp.on ? P.tp.rank : 0) * ws.ggrid + ws.gcta) * 4;

    // cos / sin of a position's angles come from the table made at load: the double-precision cosine and sine and their
    // argument reduction stay out of this function (as code, and as calls inside the step loop)
    auto rope_table = [&](int pos) {
        if (tid < HD) sm.cs[tid] = __ldg(P.rope_cs + (size_t)min(max(pos, 0), P.max_seq - 1) * HD + tid);
    };

#if MI_PROF
    const long long prof_c0 = clock64(); const unsigned long long prof_t0 = gtime_ns();
    if (tid == 0) s_prof_t = prof_t0;
#endif
    if (step0 < step1) rope_table(pos_base + step0);
    cta__syncthreads();
    for (int step = step0; step < step1 && ok; step++) {
        const int pos = pos_base + step;
        if (pos < 0 || pos >= P.max_seq || !lean_regime_ok(pos, P.attn_ctas)) { ok = false; err_code = MI_ERR_LIMIT; break; }   // the same on every CTA: nobody waits for anybody
        const unsigned tag0 = epoch + (unsigned)(step - step0) * (unsigned)nph + 1u;        // tag of (step, phase 0)
        if (step > step0 && ph1 != nph) { rope_table(pos); cta__syncthreads(); }     // (otherwise the previous step's lm_head phase has made the table)
        prof_mark(P, kProfStep);
        for (int ph = ph0; ph < ph1 && ok; ph++) {
            const int l = ph / 5;
            int k = ph == nph - 1 ? 5 : ph % 5;
            Pub pub;
            pub.xw = P.xw; pub.tag = tag0 + (unsigned)ph; pub.mute = ph == P.drop_phase; pub.stride = P.xo.total;
#if MI_TP
            pub.tp = &P.tp;
#endif
            const int kind = k == 0 ? JOB_QKV : k == 2 ? JOB_O : k == 3 ? JOB_GU : JOB_DOWN, kb = P.kb[kind];
            const bool half = P.half_rows >> kind & 1;
            const float* bias = k == 0 ? sm.lp[l].bqkv : nullptr;
            JobStart js;
            js.at = 0;
            if (k != 1 && k != 5) js = begin_cta_job(ws, sm.work, kind, kb, half, lane, bias);
            same_code(k);
            // One call site each for the norm prologue, the q8 prologue and the CTA job: the four per-layer GEMV
            // phases run the same instructions (they stay in the instruction cache from phase to phase) and differ
            // only in pointers and in the few lines of their epilogue.
#if MI_PROF
            if (P.hold_us && (int)blockIdx.x == P.prof_cta && (k == 0 || k == 3 || k == 5))
                for (const unsigned long long t0 = gtime_ns(); gtime_ns() - t0 < (unsigned long long)P.hold_us * 1000ull;) {}
#endif
            if (k == 0 || k == 3 || k == 5) {
                // QKV : h = (l == 0) ? embedding : h + down projection of layer l-1        (committed as h_in)
                // GU  : h = h + O projection                                                 (committed as h_mid)
                // LM  : final norm over h + last down projection
                const float* gsrc = nullptr; const unsigned long long* addw = nullptr; float* commit = nullptr; const float* nw = nullptr;
                if (k == 0 && l == 0) {
                    int tok = step < P.n_forced ? __ldg(P.in_tokens + step) : (step == step0 ? __ldcg(P.cur_token) : s_tok);
                    tok = min(max(tok, 0), P.V - 1);
                    residual_init(P, sm.h, nullptr, tok, P.E);
                    commit = P.h_in; nw = sm.lp[0].attn_norm;
                } else if (k == 0) {
                    gsrc = h_valid ? nullptr : P.h_mid; addw = xw_read(P) + P.xo.down; commit = P.h_in; nw = sm.lp[l].attn_norm;
                } else if (k == 3) {
                    gsrc = h_valid ? nullptr : P.h_in; addw = xw_read(P) + P.xo.o; commit = P.h_mid; nw = sm.lp[l].ffn_norm;
                } else {
                    gsrc = h_valid ? nullptr : P.h_mid; addw = xw_read(P) + P.xo.down; nw = P.out_norm;
                }
                if (gsrc) residual_init(P, sm.h, gsrc, 0, P.E);                 // a launch that starts in mid-step
                // the committed copy serves launches that start in mid-step (and state read-back); a launch over whole steps has no reader for it
                if (MI_LEAN && ph0 == 0 && ph1 == nph) commit = nullptr;
                ok = stage_norm_q8u<norm_chunks(HD, G)>(done, P, sm.h, addw, pub.tag - 1u, commit, nw, P.E, P.eps, sm.red, xq_s, xs_s);
                h_valid = true;
                prof_mark(P, 2 * k);
            } else if (k == 2 || k == 4) {
                if (js.at) {                                      // only CTAs that have a unit of the job consume its input
                    prof_mark(P, 2 * k);
                    ok = stage_poll_q8(done, P, xw_read(P) + (k == 2 ? P.xo.att : P.xo.act), k == 2 ? P.NH * HD : P.FF, k == 2 ? P.att_scales : P.FF / 32, pub.tag - 1u, xq_s, xs_s);
                    prof_mark(P, kProfWait);
                }
            }
            if (!ok) break;
            same_code(k);
            if (k == 1) {
                const int by = ws.gcta - P.seen_first;
                if ((unsigned)by < (unsigned)P.seen_n && tid == 0) pub.all(P.xo.att + P.NH * HD / 4 + P.NH * HD / 32 + by, 0u);        // (bystanders)
                if (pos + 1 <= kShortAttnMax && P.attn_ctas > 0) {
                    // the attention CTAs' business
                }
#if MI_LEAN == 0
                else if (pos + 1 <= kShortAttnMax) ok = attention_short<HD, G>(P, l, pos, sm.stage, pub.tag - 1u, pub);
                else ok = attention_split<HD, G>(P, l, pos, sm.stage, pub.tag - 1u, pub);
#elif MI_LEAN == 2
                else ok = attention_split<HD, G>(P, l, pos, sm.stage, pub.tag - 1u, pub);
#endif
            } else if (k != 5) {
                const int nq = P.NH * HD;
                done = run_cta_job(ws, P, sm, js, kb, k == 4 ? P.ks_down : 1, k == 3, half, lane, xq_s, xs_s, bias, pub, [&](int g, int ln, float v0, float v1, float bv) {
                    if (k == 0) {                                            // + bias, RoPE, packed q / k / v
                        const int p = g + (half ? ln & 15 : ln);      // g: the unit's first row
                        const float v = __fadd_rn(v0, bv);
                        const float partner = __shfl_xor_sync(0xffffffffu, v, 1);
                        float out = v;
                        if (p < nq + P.KVD) {                                  // q or k: rotate the (even, odd) lane pair
                            const int within = (p < nq ? p : p - nq) % HD, i = within >> 1;
                            const double c = sm.cs[i], s = sm.cs[HD / 2 + i];    // products are exact in double: one rounding each
                            if ((within & 1) == 0) out = __double2float_rn(__dsub_rn(__dmul_rn((double)v, c), __dmul_rn((double)partner, s)));
                            else out = __double2float_rn(__dadd_rn(__dmul_rn((double)partner, s), __dmul_rn((double)v, c)));
                        }
                        if (p < nq + 2 * P.KVD && (!half || ln < 16)) pub.all(P.xo.qkv + p, __float_as_uint(out));
                    } else if (k == 3) {                                     // SwiGLU of (gate, up), one q8_0 block per warp
                        const double gd = (double)v0;
                        const float a = __double2float_rn(__dmul_rn(__ddiv_rn(gd, __dadd_rn(1.0, exp_shared(-gd))), (double)v1));
                        __half dq; int sq;
                        const int qv = quant_block_warp2(a, dq, sq);         // FF is a multiple of 32: group g is block g
                        publish_q8_block<true>(pub, P.xo.act, P.xo.act + P.FF / 4, g, ln, qv, dq, sq);
                    } else if (k == 2) {
                        if (!half || ln < 16) pub.all(P.xo.o + g + ln, __float_as_uint(v0));
                    } else {
                        if (!half || ln < 16) pub.shared(P.xo.down + g + ln, __float_as_uint(v0));
                    }
                }) && done;
            } else {
                // ---- lm_head on the staged final norm, greedy argmax (lowest index wins ties)
                // Each candidate is {best value, its row, second-best value}: the runner-up gives the logit margin (top-1 minus
                // top-2) that the reference's engine reports per token (src/mega.cu:523-550, 385-392).
                Cand cd; cd.best = -INFINITY; cd.idx = 0x7fffffff; cd.second = -INFINITY;
                float* lg = P.logits ? P.logits + (long long)(step - step0) * P.logits_stride : nullptr;
                ok = run_warp_job(ws, 4 * P.L, P, lane, xq_s, xs_s, [&](int g, int ln, float v0) {
                    const int r = g * 32 + ln;
                    if (r < P.V) {
                        if (lg) lg[r] = v0;
                        // the reference's scan starts from logits[0] and moves on strict '>' (src/cpu_infer.cpp:153-154): a NaN
                        // never wins, and a NaN in row 0 is never beaten
                        const float vv = (r == 0 && v0 != v0) ? INFINITY : v0;
                        cd.add(vv, r);
                    }
                });
                cd.warp_reduce();
                cta__syncthreads();
                float* cv = reinterpret_cast<float*>(sm.red); int* ci = reinterpret_cast<int*>(sm.red) + 16; float* c2 = reinterpret_cast<float*>(sm.red) + 32;
                if (lane == 0) { cv[warp] = cd.best; ci[warp] = cd.idx; c2[warp] = cd.second; }
                cta__syncthreads();
                if (tid == 0) {
                    Cand t; t.best = cv[0]; t.idx = ci[0]; t.second = c2[0];
                    for (int w = 1; w < DNW; w++) { Cand o; o.best = cv[w]; o.idx = ci[w]; o.second = c2[w]; t.merge(o); }
                    if (kRowsCross) fence_acq_rel_gpu();                // rows of the cache written in this step (rows_ordered)
                    pub.shared(my_cand, __float_as_uint(t.best));
                    pub.shared(my_cand + 1, (unsigned)t.idx);
                    pub.shared(my_cand + 2, __float_as_uint(t.second));
                }
                // the next step's angles while the other CTAs' candidates arrive
                if (step + 1 < step1) rope_table(pos + 1);
                // every CTA makes the pick over all candidates itself (the same bits everywhere); the first GEMV CTA writes it out
                prof_mark(P, 2 * k + 1);
                cd.best = -INFINITY; cd.idx = 0x7fffffff; cd.second = -INFINITY;
                bool okc = ok;
                constexpr int CW = kRowsCross ? 7 : 6;
                for (int c0 = 0; c0 < n_cand && okc; c0 += 2 * DNT) {
                    unsigned cw[CW], valid = 0;
                    if (c0 + tid < n_cand) valid |= 7u;
                    if (c0 + DNT + tid < n_cand) valid |= 56u;
                    if (kRowsCross && c0 == 0 && tid < P.attn_ctas) valid |= 64u;
                    const unsigned long long* cb = xw_read(P) + P.xo.cand + (size_t)(c0 + tid) * 4;
                    okc = tw_poll(P, pub.tag, valid, [&](int q) { return q == 6 ? P.xw + attdone_off(P, step) + tid : cb + (q / 3) * (4 * DNT) + (q % 3); }, cw);
                    #pragma unroll
                    for (int h = 0; h < 2; h++) {
                        if (okc && (valid >> (3 * h) & 1u)) {
                            Cand o; o.best = __uint_as_float(cw[3 * h]); o.idx = (int)cw[3 * h + 1]; o.second = __uint_as_float(cw[3 * h + 2]);
                            cd.merge(o);
                        }
                    }
                }
                if (kRowsCross) fence_acq_rel_gpu();
                prof_mark(P, kProfWait);
                cd.warp_reduce();
                ok = cta__syncthreads_and(okc ? 1 : 0) != 0;       // also: cv / ci / c2 are free again
                if (lane == 0) { cv[warp] = cd.best; ci[warp] = cd.idx; c2[warp] = cd.second; }
                cta__syncthreads();
                if (tid == 0) {
                    Cand t; t.best = cv[0]; t.idx = ci[0]; t.second = c2[0];
                    for (int w = 1; w < DNW; w++) { Cand o; o.best = cv[w]; o.idx = ci[w]; o.second = c2[w]; t.merge(o); }
                    const int tok = t.idx == 0x7fffffff ? 0 : t.idx;
                    s_tok = tok;
                    if (ws.gcta == 0 && ok) {
                        const float margin = __fsub_rn(t.best, t.second);
                        const bool stopping = P.stop_token >= 0 && tok == P.stop_token && step + 1 >= P.n_forced && ph0 == 0;
                        if (P.stop_token >= 0 && P.attn_ctas > 0) pub.local(P.xo.tokw, (unsigned)tok);
                        __stcg(P.cur_token, tok); __stcg(P.best_val, t.best); P.out_tokens[step] = tok;
                        if (P.out_margins) P.out_margins[step] = margin;
                        if (P.ring.count) {
                            // the host reads along: token, margin and time of every step into mapped host memory, the count of
                            // valid entries every fourth step and at the end, after a system-scope fence (src/mega.cu:847-856)
                            const int slot = P.ring.base + (step - step0);
                            if (slot < P.ring.capacity) {
                                P.ring.tokens[slot] = tok; P.ring.margins[slot] = margin; P.ring.ns[slot] = gtime_ns();
                                if (((step - step0) & 3) == 3 || step == step1 - 1 || stopping) { __threadfence_system(); *reinterpret_cast<volatile int*>(P.ring.count) = slot + 1; }
                            }
                        }
                    }
                }
            }
            // a wait that gave up in one warp stops the whole CTA: behind an attention phase or a pick here, behind a job at the next barrier of a prologue
            if (k == 5 || (k == 1 && !(pos + 1 <= kShortAttnMax && P.attn_ctas > 0)) || ph + 1 == ph1) { ok = cta__syncthreads_and(ok && done ? 1 : 0) != 0; done = true; }
            prof_mark(P, 2 * k + 1);
        }
        // the stop rule (every CTA has made the same pick): the step that produced the stop token was the last
        if (P.stop_token >= 0 && ok && ph0 == 0 && ph1 == nph && s_tok == P.stop_token && step + 1 >= P.n_forced && step + 1 < step1) {
            break;
        }
    }
#if MI_PROF
    if (P.prof && (int)blockIdx.x == P.prof_cta) {
        if (tid == 0) { s_prof[8] = (unsigned long long)(clock64() - prof_c0); s_prof[9] = gtime_ns() - prof_t0; }     // SM cycles and nanoseconds of the launch (overwrites two phase slots)
        cta__syncthreads();
        if (tid < kProfSlots) P.prof[tid] += s_prof[tid];
    }
#endif
    // the first GEMV CTA has seen every CTA's last candidates, which descend from every attention CTA's output (or it has given
    // up after a full time budget): all CTAs have read the epoch
    if (ws.gcta == 0 && tid == 0 && (ph1 == nph || !ok))
        *P.epoch_dev = epoch + (unsigned)(step1 - step0) * (unsigned)nph + (ok ? 0u : (unsigned)nph);
    if (!ok && lane == 0) atomicMax(P.err, err_code);
    if (tid == 0) *const_cast<volatile int*>(&s_quit) = 1;      // (tiles may be on their way: an error, or the stop token)
}

}  // inline namespace
#endif  // __CUDACC__
}  // namespace mi

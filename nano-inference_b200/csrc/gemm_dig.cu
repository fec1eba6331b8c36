// q4_0 x q8_0 product of many tokens (prompts, batches of sequences) on tcgen05: the sums of the product over blocks (gemm_tok.cu) and of the GEMV, the same
// bits, without scaling anything per block.
//
// What bounds the other product is one FP64 multiplication per (row, block, token) and the instructions around it.  Here the scales move into the operands: every scale
// is an fp16 number, so within a row (token, K range) all of them are integers times one power of two, an element is an integer of 18 to 24 bits, and that is cut into
// base-256 digits: three of the weight's against three (four) planes of the token's.  The MMAs (kind::i8, exact int32 sums) run over all of K; partial
// products of equal weight 256^s share a sum, so 9 int8 products cost three MMAs of N = 3 tokens and five columns of tensor memory a token.  At the end of a unit the sums are
// put together as one integer and rounded once.  9 products at the int8 rate are 0.035 clocks of an SM per (row, block, token), the two FP64 operations 0.031; but
// the tensor core needs no issue slots beside it.  The digits hold any row whose scales lie at most 8 binades apart and any token with at most 13 (5 with three
// planes); other rows and tokens, and scales that are not finite, are summed block by block behind the main loop.  How large the integer gets: a weight is below
// 2^(14 + s) units, s the binades between its row's scales (at most 8), an activation below 2^(18 + 5) with three planes and 2^(18 + 13) with four, so K = 2^k elements sum to
// less than 2^(37 + s + k) and 2^(45 + s + k).  The former is below 2^59 for all K; where the latter is above 2^63 (s > 7 for K = 2048), sums of launches with four planes are two
// numbers.
//
// Dataflow of a CTA (one per SM, a unit is 128 rows x T <= 64 tokens x one K range):
//   copies     : one warp streams the q4_0 tiles (bulk copies, ahead of the wait for the predecessor), one the activation planes, four blocks at a time;
//   16 warps   : nibbles and scale of a block -> three digits of 32 weights per thread (= row), in registers, then with tcgen05.st into a stage of tensor
//                memory: A operands come from there, so shared memory serves the activations only.  Each of four groups has a stage of two blocks under way, so
//                that the way from a freed stage to a full one is a store and two barriers;
//   one warp   : issues the MMAs; the whole warp runs the loop, one lane issues (see there);
//   the 16 warps again at the end of a unit, when the first stages of the next one are in place.
// Measured (event time, launches back to back, each ahead of its predecessor's end): gate/up of 333 tokens (17920 x 1536) 71 us against 121 for the product over blocks, 82 with
// four planes, down (1536 x 8960) 32 / 63, batch of 64 on 22016 x 2048 31 / 46, 2048 x 11008 16 / 26, 151936 x 2048 128 / 246; it is even at 32 tokens on 22016 x 2048 (29 / 29),
// loses at 16 (28 / 19) and at 2560 x 2048 x 64 (17 / 12).  A stage of two blocks takes 620 clocks at 64 tokens, its MMAs 576;
// the rest is the start (7000 clocks until the first MMA) and the end of a unit (6000).  Tried: weights expanded weight by weight or in byte lanes with seven sums per
// token (the expansion or the tensor memory is full first), stages of one and four blocks, eight expanding warps, results through arrays in
// registers (spills): 95 to 210 us for the gate/up.  Carry additions moved to the multiplier's pipe: no change, both sides in turn on one GPU.  A fourth weight digit for
// rows of 9 to 16 binades (95 us for the gate/up, however many): half of the instantiations for rows that cost less block by block up to 2 % of them, and go over blocks from 4 % on.
#include "gemm_dig.cuh"
#include <algorithm>
#include <atomic>
#include <mutex>
#include <type_traits>

namespace mi {
namespace {

constexpr int kStepBlk = 8, kStepBytes = kStepBlk * kTileRowBytes;          // blocks per weight copy
constexpr int kRawSlots = 4, kXSlots = 3, kXStage = 4;                       // rings: weight steps; activations, of four blocks
constexpr int kStage = 2, kRing = 8;                                        // blocks per stage of weight digits; ring of barriers for the stages
constexpr int kMaxN = kDigPlanes * kDigMaxT;                                // columns of an MMA
constexpr int kXBytes = kXStage * kMaxN * 32;
constexpr int kGroups = 4, kExpWarps = 4 * kGroups, kWarps = kExpWarps + 3, kThreads = kWarps * 32;      // groups of four warps, a quarter of the 128 rows each
constexpr int kRowNone = 255;
constexpr int kMaxInfo = 4096;                                          // tokens times K ranges of a launch
constexpr int kNW = 3, kMaxSpread = 8;                                   // digits of a weight; binades between a row's scales that they hold
constexpr long long kBias = 0x808080ll;                                  // DigX::bias times this is in the sums (expand_block)

struct DigParams {
    const uint8_t* base; const uint8_t* row_exp; int groups, nb, nst, rows;     // tiled weights; nst: steps of eight blocks
    int ksg, M; const int* bad_list; int bad_rows;                              // rows without an exponent
    DigX x; TokX q8;
    const float* bias; float* y; double* part; int ldp;
    int* err;
};

struct Smem {
    static constexpr int raw = 0, x = raw + kRawSlots * 4 * kStepBytes, bars = x + kXSlots * kXBytes;
    static constexpr int n_bars = 2 * kRawSlots + 2 * kXSlots + 2 * kRing + 3;
    static constexpr int table = bars + (n_bars * 8 + 31) / 16 * 16;         // 16 bytes per warp and token of its group
    static constexpr int bytes = table + kExpWarps * (kDigMaxT / kGroups) * 16 + 256;
};

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t a, const unsigned (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(a), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
__device__ __forceinline__ void tmem_zero32(uint32_t a) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};"
                 ::"r"(a), "r"(0) : "memory");
}
// The values exist here (the compiler would compute them behind the wait that follows).
__device__ __forceinline__ void keep(unsigned (&d)[2][kNW][8]) {
    #pragma unroll
    for (int b = 0; b < 2; b++)
        #pragma unroll
        for (int j = 0; j < kNW; j++)
            asm volatile("" : "+r"(d[b][j][0]), "+r"(d[b][j][1]), "+r"(d[b][j][2]), "+r"(d[b][j][3]), "+r"(d[b][j][4]), "+r"(d[b][j][5]), "+r"(d[b][j][6]), "+r"(d[b][j][7]));
}
__device__ __forceinline__ void tmem_zero4(uint32_t a) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%1,%1,%1};" ::"r"(a), "r"(0) : "memory");
}
__device__ __forceinline__ void tmem_zero1(uint32_t a) { asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(a), "r"(0) : "memory"); }
__device__ __forceinline__ void tmem_ld1(uint32_t a, int& v) { asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v) : "r"(a)); }
__device__ __forceinline__ void tmem_ld4(uint32_t a, int (&v)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(a));
}

// Bounded wait of a whole warp that also ends when another role has given up.
__device__ __forceinline__ bool wait_or_abort(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
    unsigned long long t0 = 0;
    #pragma unroll 1
    for (unsigned i = 1;; i++) {
        if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
        if ((i & 255) == 0) {
            if (__any_sync(0xffffffffu, *abort_flag != 0)) return false;
            if (i == 256) t0 = gtime_ns();
            else if (__any_sync(0xffffffffu, gtime_ns() - t0 > kWaitBudgetNs)) { *abort_flag = 1; return false; }
        }
    }
}

// The digits of a block's 32 weights (nibble n - 8) * m in element order, base 256, each 128 too large and so unsigned (what that adds to the sums is
// subtracted at the end, DigX::bias).  m = a0 + 256 a1 (|m| < 2^19): two weights per multiplication in lanes of 16 bits, n a0 + c0 and
// n a1 + c1 + the carry of the former, where c0 + 256 c1 = 0x808080 - 8 m.
__device__ __forceinline__ void expand_block(const uint4& w, int m, unsigned (&d)[kNW][8]) {
    const unsigned ww[4] = {w.x, w.y, w.z, w.w};
    const unsigned c = (unsigned)kBias - 8u * (unsigned)m, c0 = (c & 255u) * 0x10001u, c1 = (c >> 8) * 0x10001u;
    const unsigned a0 = (unsigned)m & 255u, a1 = (unsigned)(m >> 8);
    #pragma unroll
    for (int i = 0; i < 8; i++) {
        const unsigned n = (i < 4 ? ww[i] : ww[i - 4] >> 4) & 0x0F0F0F0Fu;
        const unsigned ne = n & 0x00FF00FFu, no = __byte_perm(n, 0, 0x4341);
        const unsigned pe = ne * a0 + c0, po = no * a0 + c0;
        const unsigned se = ne * a1 + c1 + __byte_perm(pe, 0, 0x4341), so = no * a1 + c1 + __byte_perm(po, 0, 0x4341);
        d[0][i] = __byte_perm(pe, po, 0x6240); d[1][i] = __byte_perm(se, so, 0x6240); d[2][i] = __byte_perm(se, so, 0x7351);
    }
}

// acc + v * f in 64 bits
__device__ __forceinline__ long long mad_wide(int v, int f, long long acc) {
    long long r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(v), "r"(f), "l"(acc));
    return r;
}

// C consecutive blocks of a row and a token, and their part of the sum: the GEMV's terms
template <int C> struct BlkIn { uint4 w[C], xa[C], xb[C]; double x[C]; uint2 h; };
template <int C>
__device__ __forceinline__ double add_blocks(const BlkIn<C>& v, double acc) {
    #pragma unroll
    for (int i = 0; i < C; i++) {
        const unsigned w[4] = {v.w[i].x, v.w[i].y, v.w[i].z, v.w[i].w}, lo[4] = {v.xa[i].x, v.xa[i].z, v.xb[i].x, v.xb[i].z}, hi[4] = {v.xa[i].y, v.xa[i].w, v.xb[i].y, v.xb[i].w};
        int c = 0;                                                     // (n ^ 8) << 4 as int8 is 16 (n - 8): with TokX's 2^1004 the powers of two cancel
        #pragma unroll
        for (int k = 0; k < 4; k++) c = __dp4a((int)((w[k] & 0xF0F0F0F0u) ^ 0x80808080u), (int)hi[k], __dp4a((int)((w[k] << 4 & 0xF0F0F0F0u) ^ 0x80808080u), (int)lo[k], c));
        const double scale = __dmul_rn((double)__half2float(__ushort_as_half((unsigned short)((i < 2 ? v.h.x : v.h.y) >> 16 * (i & 1)))), __dmul_rn(v.x[i], 0x1p-1008));
        acc = __fma_rn(scale, (double)c, acc);
    }
    return acc;
}

// What the digits cannot hold (the main loop stores nothing there), block by block as the GEMV forms it: rows without an exponent with all tokens, all rows with tokens
// without planes.  A warp takes one K range of 32 tokens of such a row or of 32 rows of such a token; the whole grid shares these jobs, whose rows and tokens they are, and
// several warps of a CTA share a job's blocks while there are fewer than warps.  What bounds it is a chain of requests to L2 where there is little to do, then issue.
// Measured (launches back to back, us; without any / with one token / three / a tenth of the tokens / 1 % of the rows / 10 %, and the product over blocks): 17920x1536 with 333
// tokens 71.6 / 75.8 / 80.2 / 128.7 / 82.8 / 172.9, 121.3; 1536x8960 with 333 33.1 / 37.4 / 38.8 / 73.8 / 38.9 / 97.1, 62.8; 22016x2048 with 64 31.6 / 38.6 / - / 52.2 / 36.3 / 63.9, 46.6;
// 2048x11008 with 64 15.6 / 20.1 / - / 31.9 / 19.8 / -, 26.1.  All tokens out of range: 597 and 301 us of the first two.  (One thread per row and token before: 118 and 78 with
// one token, 1038 and 485 with 1 % of the rows.)  Tried: 16 rows x 8 tokens per warp on mma.sync (7 of 8 columns idle for one token: 85 and 53), units
// summed by the CTA that has them (97 with 1 % of the rows: rows are not spread evenly).
template <int KB, bool PART>
static __device__ __forceinline__ void sum_over_blocks(const DigParams& p, uint8_t* smem, bool any_tokens) {
    constexpr int C = KB < 4 ? KB : 4, S = KB / C;                     // blocks requested together, of a tile's KB
    constexpr int kWords = kMaxInfo / (32 * kExpWarps);
    double* fold = reinterpret_cast<double*>(smem);                    // [warp][lane]
    unsigned short* toks = reinterpret_cast<unsigned short*>(smem + kExpWarps * 32 * 8);      // tokens without planes: K range * M + token
    __shared__ int s_count[kExpWarps];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int n_toks = 0;
    if (any_tokens) {
        const int total = p.M * p.ksg, words = (total + 32 * kExpWarps - 1) / (32 * kExpWarps);        // 32 entries each, a run of them per warp: the same list in every CTA
        unsigned none[kWords];
        int mine = 0;
        if (warp < kExpWarps) {
            bool b[kWords];
            #pragma unroll
            for (int i = 0; i < kWords; i++) { const int at = (warp * words + i) * 32 + lane; b[i] = i < words && at < total && __ldcg(p.x.info + at) >> 8 == kDigNone; }
            #pragma unroll
            for (int i = 0; i < kWords; i++) { none[i] = __ballot_sync(0xffffffffu, b[i]); mine += __popc(none[i]); }
            if (lane == 0) s_count[warp] = mine;
        }
        __syncthreads();
        int at = 0;
        for (int k = 0; k < kExpWarps; k++) { if (k < warp) at += s_count[k]; n_toks += s_count[k]; }
        if (warp < kExpWarps)
            #pragma unroll
            for (int i = 0; i < kWords; i++) {
                if (none[i] >> lane & 1) toks[at + __popc(none[i] & ((1u << lane) - 1))] = (warp * words + i) * 32 + lane;
                at += __popc(none[i]);
            }
        __syncthreads();
    }
    const int tg = (p.M + 31) / 32, rg = (p.rows + 31) / 32, by_row = p.bad_rows * p.ksg * tg, jobs = by_row + n_toks * rg;
    int shift = 0;                                                     // 2^shift warps per job
    while (shift < 4 && jobs << (shift + 1) <= (int)gridDim.x * kExpWarps) shift++;
    #pragma unroll 1
    for (int j0 = blockIdx.x * (kExpWarps >> shift); j0 < jobs; j0 += gridDim.x * (kExpWarps >> shift)) {
        const int j = j0 + (warp >> shift), part = warp & ((1 << shift) - 1);
        const bool mine = warp < kExpWarps && j < jobs;
        int row = 0, n = 0, sp = 0;                                    // this lane's
        if (mine && j < by_row) { const int q = j / tg; n = (j - q * tg) * 32 + lane; row = __ldg(p.bad_list + q / p.ksg); sp = q % p.ksg; }
        else if (mine) { const int q = (j - by_row) / rg, e = toks[q]; row = (j - by_row - q * rg) * 32 + lane; sp = e / p.M; n = e - sp * p.M; }
        const bool has = mine && row < p.rows && n < p.M;
        double acc = 0.0;
        if (mine) {
            const int r = min(row, p.rows - 1), c = min(n, p.M - 1), b0 = sp * p.nst / p.ksg * kStepBlk, tiles = (min((sp + 1) * p.nst / p.ksg * kStepBlk, p.nb) - b0) / KB;
            const int t0 = b0 / KB + (tiles * part >> shift), t1 = b0 / KB + (tiles * (part + 1) >> shift);
            const uint8_t* w = p.base + ((size_t)(r >> 5) * p.nb + t0 * KB) * kTileRowBytes, * h = w + KB * 512 + (r & 31) * KB * 2;
            w += (r & 31) * 16;
            const unsigned* x = p.q8.q + tok_word(p.q8.J, t0 * KB, c, 0);                      // a block of a token is eight words: elements 0, 16, 4, 20, ..
            const double* d = p.q8.d + tok_scale(p.q8.J, t0 * KB, c);
            const size_t x_step = (size_t)p.q8.J * 64, d_step = (size_t)p.q8.J * 8;
            #pragma unroll 1
            for (int t = t0; t < t1; t++) {
                #pragma unroll
                for (int s = 0; s < S; s++) {
                    BlkIn<C> v;
                    #pragma unroll
                    for (int i = 0; i < C; i++) {
                        v.w[i] = __ldg(reinterpret_cast<const uint4*>(w + (s * C + i) * 512));
                        v.xa[i] = __ldcg(reinterpret_cast<const uint4*>(x)); v.xb[i] = __ldcg(reinterpret_cast<const uint4*>(x) + 1);
                        v.x[i] = __ldcg(d);
                        x += x_step; d += d_step;
                    }
                    if constexpr (C == 4) v.h = __ldg(reinterpret_cast<const uint2*>(h) + s);
                    else if constexpr (C == 2) v.h.x = __ldg(reinterpret_cast<const unsigned*>(h));
                    else v.h.x = __ldg(reinterpret_cast<const unsigned short*>(h));
                    acc = add_blocks(v, acc);
                }
                w += KB * kTileRowBytes; h += KB * kTileRowBytes;
            }
        }
        if (shift) {                                                   // (all jobs are under way then)
            if (mine) fold[warp * 32 + lane] = acc;
            __syncthreads();
            if (part) continue;
            #pragma unroll 1
            for (int k = 1; k < 1 << shift; k++) if (mine) acc = __dadd_rn(acc, fold[(warp + k) * 32 + lane]);
        }
        if (!has) continue;
        if constexpr (PART) __stcg(p.part + ((size_t)sp * p.M + n) * p.ldp + row, acc);
        else p.y[(size_t)n * p.rows + row] = __double2float_rn(acc) + (p.bias ? __ldg(p.bias + row) : 0.f);
    }
}

// TWO: sums of four planes in two parts (a form of its own: they take a tenth longer, 333 tokens on 17920 x 1536 91 us instead of 83)
template <int KB, bool PART, bool TWO>
__global__ void __launch_bounds__(kThreads, 1) gemm_dig_kernel(const __grid_constant__ DigParams p) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    uint8_t* smem = smem_raw + (0u - smem_u32(smem_raw) & 255u);          // the swizzle goes by address bits
    uint8_t* raw = smem + Smem::raw;
    uint8_t* xs = smem + Smem::x;
    uint64_t* raw_full = reinterpret_cast<uint64_t*>(smem + Smem::bars);
    uint64_t* raw_empty = raw_full + kRawSlots;
    uint64_t* x_full = raw_empty + kRawSlots;
    uint64_t* x_empty = x_full + kXSlots;
    uint64_t* full = x_empty + kXSlots;
    uint64_t* empty = full + kRing;
    uint64_t* d_full = empty + kRing;
    uint64_t* d_empty = d_full + 1;
    uint64_t* drained = d_empty + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
    __shared__ int s_abort, s_planes, s_none;
    volatile int* abort_flag = &s_abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr int wRaw = kExpWarps, wX = wRaw + 1, wMma = wX + 1;

    if (tid == 0) {
        for (int i = 0; i < kRawSlots; i++) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], kExpWarps); }
        for (int i = 0; i < kRing; i++) { mbar_init(&full[i], 4); mbar_init(&empty[i], 1); }
        for (int i = 0; i < kXSlots; i++) { mbar_init(&x_full[i], 1); mbar_init(&x_empty[i], 1); }
        mbar_init(d_full, 1); mbar_init(d_empty, kExpWarps); mbar_init(drained, 1);
        mbar_fence_init();
        s_abort = 0; s_planes = 3; s_none = 0;
    }
    if (warp == wMma) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __reduce_max_sync(0xffffffffu, *tmem_slot);           // (a reduction's result is in a uniform register, where the MMAs want it)

    // unit -> (K range, row tile, token tile), in this order: what a CTA starts with does not depend on the tokens
    struct Unit { int rt, ts, sp, k0, k1; };
    const int row_tiles = (p.groups + 3) / 4;
    auto unit = [&](int u) {
        Unit r;
        r.sp = u % p.ksg; const int v = u / p.ksg;
        r.rt = v % row_tiles; r.ts = v / row_tiles;
        r.k0 = r.sp * p.nst / p.ksg; r.k1 = (r.sp + 1) * p.nst / p.ksg;
        return r;
    };

    // the weights depend on nothing: their ring fills before the wait for the predecessor
    int raw_issued = 0, ru = blockIdx.x, rt_step = -1;
    auto raw_issue = [&](const Unit& U, int t) {                       // whole warp wRaw
        const int s = raw_issued % kRawSlots, bytes = min(kStepBlk, p.nb - t * kStepBlk) * kTileRowBytes;
        if (lane == 0) mbar_expect_tx(&raw_full[s], 4 * bytes);
        __syncwarp();
        if (lane < 4) {
            const int g = min(U.rt * 4 + lane, p.groups - 1);           // a missing row group re-reads the last one; its rows are never stored
            bulk_g2s(raw + ((size_t)s * 4 + lane) * kStepBytes, p.base + ((size_t)g * p.nb + t * kStepBlk) * kTileRowBytes, bytes, &raw_full[s]);
        }
        raw_issued++;
    };
    if (warp == wRaw) {
        const Unit U = unit(ru);
        for (rt_step = U.k0; rt_step < U.k1 && raw_issued < kRawSlots; rt_step++) raw_issue(U, rt_step);
        if (rt_step >= U.k1) { ru += gridDim.x; rt_step = -1; }
    }
    auto row_exp_of = [&](const Unit& U) { return (int)__ldg(p.row_exp + min(U.rt * 128 + (warp & 3) * 32 + lane, p.groups * 32 - 1)); };
    const int first_exp = row_exp_of(unit(blockIdx.x));
    if (warp < kExpWarps) {                                            // all sums start at zero
        #pragma unroll
        for (int c = 0; c < 512 / kGroups; c += 32) tmem_zero32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (warp >> 2) * (512 / kGroups) + c);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
    }
    pdl_launch_dependents();
    pdl_wait_prior();
    // planes in use among all tokens (one wide token costs every MMA of the launch a third more)
    for (int i = tid; i < p.M * p.ksg; i += kThreads) {
        const int v = __ldcg(p.x.info + i) >> 8;
        if (v == 4) s_planes = 4;
        else if (v == kDigNone) s_none = 1;
    }
    __syncthreads();
    tc_fence_after();
    const int planes = (int)__reduce_max_sync(0xffffffffu, (unsigned)s_planes);
    const bool two_parts = TWO && planes == 4;
    const int T = p.x.T, units = p.ksg * row_tiles * p.x.TT, N = planes == 4 ? 4 * T : dig_rows(T);
    // tensor memory: sums of weight 256^s in columns s * T .. (the MMAs of a token tile of an odd number of eights reach eight columns further), stages of weight
    // digits at the end
    const int fit = (512 - (kNW - 1) * T - N) / (kStage * kNW * 8), slots = fit >= 4 ? 4 : fit >= 2 ? 2 : 1;
    const uint32_t a_base = tmem + 512 - slots * (kStage * kNW * 8);

    if (warp < kExpWarps) {
        // ---------------- weights: nibbles and scales -> digits in registers, then in tensor memory (each of four groups of four warps takes every fourth
        // stage); and the sums of a unit -> results, while the next unit is under way
        const int q = warp & 3, wg = warp >> 2;
        const uint32_t trow = tmem + ((uint32_t)(q * 32) << 16), a_row = a_base + ((uint32_t)(q * 32) << 16);
        constexpr int G = kDigMaxT / kGroups;                          // tokens of a group of warps
        longlong2* table = reinterpret_cast<longlong2*>(smem + Smem::table) + warp * G;          // per token: what its 128s add to a sum, its exponent
        int n_done = 0;
        // what the end of a unit needs besides its sums, requested when the unit begins
        struct Ends { int u, ew, info; long long bias; float bv; };
        auto ends_of = [&](int u, int ew) {
            const Unit U = unit(u);
            const int row = U.rt * 128 + q * 32 + lane, n = U.ts * T + wg * G + lane;
            const bool has = lane < min(T - wg * G, G) && n < p.M;
            Ends e;
            e.u = u;
            e.ew = ew;
            e.info = has ? __ldcg(p.x.info + (size_t)U.sp * p.M + n) : 0;
            e.bias = has ? __ldcg(p.x.bias + (size_t)U.sp * p.M + n) : 0;
            e.bv = !PART && p.bias && row < p.rows ? __ldg(p.bias + row) : 0.f;
            return e;
        };
        auto finish = [&](const Ends& e) -> bool {
            const Unit U = unit(e.u);
            const int n0 = U.ts * T + wg * G, row = U.rt * 128 + q * 32 + lane;
            // tokens that are there and have digits, for a row that has (the others: sum_over_blocks)
            unsigned good = __ballot_sync(0xffffffffu, lane < min(min(T - wg * G, G), p.M - n0) && e.info >> 8 != kDigNone);
            if (row >= p.rows || e.ew == kRowNone) good = 0;
            if (lane < G) {                                            // (two parts: units of 2^32 and of 1)
                const int ex = e.info & 255;
                if (!two_parts) table[lane] = make_longlong2((long long)((unsigned long long)e.bias * (unsigned long long)kBias), PART ? (1023 - 50 + ex) << 20 : (127 - 50 + ex) << 23);
                else table[lane] = make_longlong2((long long)(unsigned)e.bias * kBias, (e.bias >> 32) * kBias << 8 | ex);
            }
            __syncwarp();
            if (!wait_or_abort(d_full, n_done & 1, abort_flag)) return false;
            n_done++;
            tc_fence_after();
            float* y = p.y + (size_t)n0 * p.rows + row;
            double* part = p.part + ((size_t)U.sp * p.M + n0) * p.ldp + row;
            const int mine = min(T - wg * G, G);
            if (!two_parts) {
                #pragma unroll 1
                for (int g = 0; g < mine; g += 4) {                    // (rolled: four tokens at a time fit the registers and the instruction cache)
                    const uint32_t a = trow + wg * G + g;
                    int d[kNW + 2][4];
                    unsigned high[4] = {0, 0, 0, 0};
                    if (planes == 4) {
                        tmem_ld4(a + (kNW + 2) * T, d[0]);
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        #pragma unroll
                        for (int i = 0; i < 4; i++) high[i] = (unsigned)d[0][i] << 8;
                    }
                    #pragma unroll
                    for (int i = 0; i < kNW + 2; i++) tmem_ld4(a + i * T, d[i]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    #pragma unroll
                    for (int i = 0; i < kNW + 2; i++) tmem_zero4(a + i * T);       // for the next unit
                    if (planes == 4) tmem_zero4(a + (kNW + 2) * T);
                    #pragma unroll
                    for (int i = 0; i < 4; i++) {                      // the sum is below 2^63, whatever its parts are
                        const longlong2 tok = table[g + i];
                        long long v = (long long)((unsigned long long)(high[i] + (unsigned)d[4][i]) << 32) - tok.x;
                        v = mad_wide(d[0][i], 1, v); v = mad_wide(d[1][i], 1 << 8, v); v = mad_wide(d[2][i], 1 << 16, v); v = mad_wide(d[3][i], 1 << 24, v);
                        if (good >> (g + i) & 1) {
                            if constexpr (PART) __stcg(part, __dmul_rn(__ll2double_rn(v), __hiloint2double((int)tok.y + (e.ew << 20), 0)));
                            // (times a power of two that leaves the result a normal number: the one rounding is the conversion's)
                            else *y = __fmul_rn(__ll2float_rn(v), __int_as_float((int)tok.y + (e.ew << 23))) + e.bv;
                        }
                        if constexpr (PART) part += p.ldp; else y += p.rows;
                    }
                }
            } else {
                #pragma unroll 1
                for (int t = 0; t < mine; t++) {                       // sums below 2^67 in two parts; token by token, so that its code takes no registers from the rest
                    int d[kNW + 3];
                    #pragma unroll
                    for (int i = 0; i < kNW + 3; i++) tmem_ld1(trow + wg * G + t + i * T, d[i]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    #pragma unroll
                    for (int i = 0; i < kNW + 3; i++) tmem_zero1(trow + wg * G + t + i * T);
                    const longlong2 tok = table[t];
                    long long lo = mad_wide(d[0], 1, -tok.x), hi = mad_wide(d[5], 1 << 8, (long long)d[4]) - (tok.y >> 8);
                    lo = mad_wide(d[1], 1 << 8, lo); lo = mad_wide(d[2], 1 << 16, lo); lo = mad_wide(d[3], 1 << 24, lo);
                    hi += lo >> 32;                                    // below 2^36, and the rest of lo is 0 .. 2^32 - 1: the double rounds once
                    const double v = __fma_rn((double)hi, 0x1p32, (double)(unsigned)lo);
                    const int ex = ((int)tok.y & 255) + e.ew - 50;
                    if (good >> t & 1) {
                        if constexpr (PART) __stcg(part, __dmul_rn(v, __hiloint2double((1023 + ex) << 20, 0)));
                        else *y = __fmul_rn(__double2float_rn(v), __int_as_float((127 + ex) << 23)) + e.bv;
                    }
                    if constexpr (PART) part += p.ldp; else y += p.rows;
                }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(d_empty);
            return true;
        };
        if (lane == 0) mbar_arrive(d_empty);
        int s = 0, sc0 = 0;                                            // sc0: stages of all units before
        Ends now{}, before{};
        int next_exp = first_exp;
        bool pending = false;
        uint32_t raw_phase = 0;
        bool ok = true;
        #pragma unroll 1
        for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
            const Unit U = unit(u);
            now = ends_of(u, next_exp);
            if (u + (int)gridDim.x < units) next_exp = row_exp_of(unit(u + gridDim.x));        // (its latency is not for the next unit's first block)
            int sc = sc0 + ((wg - sc0) & (kGroups - 1)), step0 = sc0;
            #pragma unroll 1
            for (int t = U.k0; t < U.k1; t++) {
                const int nblk = min(kStepBlk, p.nb - t * kStepBlk), end = step0 + (nblk + 1) / kStage;
                if (!(ok = wait_or_abort(&raw_full[s], raw_phase, abort_flag))) break;
                const uint8_t* grp = raw + ((size_t)s * 4 + q) * kStepBytes;
                #pragma unroll 1
                for (; sc < end; sc += kGroups) {
                    // the first stage of a unit goes beside the last ones of the unit before, whose sums are read then (later stages would wait for its last MMAs)
                    if (pending && sc > sc0) { if (!(ok = finish(before))) break; pending = false; }
                    unsigned d[kStage][kNW][8];
                    #pragma unroll
                    for (int b = 0; b < kStage; b++) {
                        const int k = min((sc - step0) * kStage + b, nblk - 1);
                        const uint8_t* tile = grp + k / KB * (KB * kTileRowBytes);
                        const uint4 w = *reinterpret_cast<const uint4*>(tile + (k % KB * 32 + lane) * 16);
                        const unsigned h = *reinterpret_cast<const unsigned short*>(tile + KB * 512 + (lane * KB + k % KB) * 2);
                        const int m = scale_mantissa(h) << ((scale_exponent(h) - now.ew) & 31);
                        expand_block(w, h & 0x8000u ? -m : m, d[b]);
                    }
                    keep(d);
                    // (a ring of eight barriers, whatever the number of slots: a group never falls two phases behind)
                    if (sc >= slots && !(ok = wait_or_abort(&empty[(sc - slots) % kRing], ((sc - slots) / kRing) & 1, abort_flag))) break;
                    tc_fence_after();
                    #pragma unroll
                    for (int b = 0; b < kStage; b++)
                        #pragma unroll
                        for (int j = 0; j < kNW; j++) tmem_st8(a_row + ((sc & (slots - 1)) * kStage + b) * (kNW * 8) + 8 * j, d[b][j]);
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&full[sc % kRing]);
                }
                if (!ok) break;
                step0 = end;
                __syncwarp();
                if (lane == 0) mbar_arrive(&raw_empty[s]);
                if (++s == kRawSlots) { s = 0; raw_phase ^= 1; }
            }
            sc0 = step0;
            if (ok && pending) ok = finish(before);
            before = now; pending = true;
        }
        if (ok && pending) finish(before);
    } else if (warp == wRaw) {
        bool ok = true;
        for (; ru < units && ok; ru += gridDim.x, rt_step = -1) {
            const Unit U = unit(ru);
            for (int t = rt_step < 0 ? U.k0 : rt_step; t < U.k1; t++) {
                if (raw_issued >= kRawSlots && !wait_or_abort(&raw_empty[raw_issued % kRawSlots], (raw_issued / kRawSlots & 1) ^ 1, abort_flag)) { ok = false; break; }
                raw_issue(U, t);
            }
        }
    } else if (warp == wX) {
        // ---------------- activations, four blocks at a time: one copy where three planes are in use, else the fourth one from its own place
        int issued = 0, slot = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
            const Unit U = unit(u);
            const int b1 = min(U.k1 * kStepBlk, p.nb);
            for (int b = U.k0 * kStepBlk; b < b1; b += kXStage, issued++) {
                const int nblk = min(kXStage, b1 - b);
                if (!wait_or_abort(&x_empty[slot], phase ^ 1, abort_flag)) { ok = false; break; }
                uint8_t* dst = xs + (size_t)slot * kXBytes;
                if (lane == 0) mbar_expect_tx(&x_full[slot], nblk * N * 32);
                __syncwarp();
                if (planes == 3) {
                    if (lane == 0) bulk_g2s(dst, p.x.q + dig_offset(p.x, p.nb, U.ts, b, 0, 0, 0), nblk * N * 32, &x_full[slot]);
                } else if (lane < 2 * nblk) {
                    const int k = lane >> 1, j = (lane & 1) * 3;
                    bulk_g2s(dst + (k * N + j * T) * 32, p.x.q + dig_offset(p.x, p.nb, U.ts, b + k, 0, j, 0), (j ? 1 : 3) * T * 32, &x_full[slot]);
                }
                __syncwarp();
                if (++slot == kXSlots) { slot = 0; phase ^= 1; }
            }
        }
        if (!ok && lane == 0)                                          // copies in flight target this CTA
            for (int k = max(0, issued - kXSlots); k < issued; k++) (void)mbar_wait_bounded(&x_full[k % kXSlots], (k / kXSlots) & 1);
    } else {
        // ---------------- MMAs: a digit of the weights against all planes of the tokens, into the sums from the digit's own weight up.
        // The whole warp runs the loop and one lane issues: operands of uniform code are in uniform registers already.  (A loop of one lane took
        // 100 cycles per MMA to move them there; the MMA itself takes N / 2.)
        const uint32_t idesc = (2u << 4) | (0u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
        uint32_t elected;
        asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(elected));
        auto mma = [&](uint32_t a, uint32_t x) {
            const uint64_t db = (uint64_t)((x & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)16 << 32) | (1ull << 46) | (6ull << 61);       // eight rows of 32 bytes, 32-byte swizzle
            #pragma unroll
            for (int i = 0; i < kNW; i++)
                asm volatile(
                    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, 1, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
                    ::"r"(tmem + (uint32_t)(i * T)), "r"(a + 8 * i), "l"(db), "r"(idesc) : "memory");
        };
        // the same; returns whether two barriers' phases are over, asked before the MMAs are issued and answered behind them (a wait for a barrier that is through
        // already keeps the warp for 110 clocks)
        auto mma_and_test = [&](uint32_t a, uint32_t x, uint32_t bar0, uint32_t par0, uint32_t bar1, uint32_t par1) -> uint32_t {
            const uint64_t db = (uint64_t)((x & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t)16 << 32) | (1ull << 46) | (6ull << 61);       // eight rows of 32 bytes, 32-byte swizzle
            uint32_t r;
            asm volatile(
                "{\n\t.reg .pred p, t, u;\n\tsetp.ne.b32 p, 1, 0;\n\t"
                "mbarrier.test_wait.parity.shared::cta.b64 t, [%9], %10;\n\t"
                "mbarrier.test_wait.parity.shared::cta.b64 u, [%11], %12;\n\t"
                "tcgen05.mma.cta_group::1.kind::i8 [%1], [%4], %7, %8, p;\n\t"
                "tcgen05.mma.cta_group::1.kind::i8 [%2], [%5], %7, %8, p;\n\t"
                "tcgen05.mma.cta_group::1.kind::i8 [%3], [%6], %7, %8, p;\n\t"
                "and.pred t, t, u;\n\tselp.u32 %0, 1, 0, t;\n\t}"
                : "=r"(r) : "r"(tmem), "r"(tmem + (uint32_t)T), "r"(tmem + (uint32_t)(2 * T)), "r"(a), "r"(a + 8), "r"(a + 16), "l"(db), "r"(idesc),
                  "r"(bar0), "r"(par0), "r"(bar1), "r"(par1) : "memory");
            return r;
        };
        int n_done = 0, sc = 0, xslot = 0;
        uint32_t x_phase = 0;
        bool ok = true;
        uint32_t ready = 0;                                            // the next stage's operands were seen
        for (int u = blockIdx.x; u < units && ok; u += gridDim.x, n_done++) {
            const Unit U = unit(u);
            const int b1 = min(U.k1 * kStepBlk, p.nb);
            if (!wait_or_abort(d_empty, n_done & 1, abort_flag)) { ok = false; break; }
            #pragma unroll 1
            for (int b = U.k0 * kStepBlk, g = 0; b < b1; b += kStage, g ^= 1) {
                if (!__any_sync(0xffffffffu, ready != 0) &&
                    ((g == 0 && !wait_or_abort(&x_full[xslot], x_phase, abort_flag)) || !wait_or_abort(&full[sc % kRing], (sc / kRing) & 1, abort_flag))) { ok = false; break; }
                tc_fence_after();
                const uint32_t a = a_base + (sc & (slots - 1)) * (kStage * kNW * 8), x = smem_u32(xs) + xslot * kXBytes + g * kStage * N * 32;
                const bool last = b + kStage >= b1, turn = g == 1 || last;                    // turn: the next stage begins another copy of activations
                const int ns = sc + 1, nx = turn ? (xslot + 1 == kXSlots ? 0 : xslot + 1) : xslot;
                const uint32_t np = turn && nx == 0 ? x_phase ^ 1 : x_phase;
                ready = 0;
                if (b + kStage <= b1) {
                    if (elected) {
                        mma(a, x);
                        ready = mma_and_test(a + kNW * 8, x + N * 32, smem_u32(&full[ns % kRing]), (ns / kRing) & 1, smem_u32(turn ? &x_full[nx] : &full[ns % kRing]), turn ? np : (ns / kRing) & 1);
                        tc_commit(&empty[sc % kRing]);
                        if (turn) tc_commit(&x_empty[xslot]);
                    }
                } else {
                    if (elected) { mma(a, x); tc_commit(&empty[sc % kRing]); tc_commit(&x_empty[xslot]); }
                }
                __syncwarp();
                sc = ns; xslot = nx; x_phase = np;
                if (last) break;
            }
            if (ok && elected) tc_commit(d_full);
            __syncwarp();
        }
        if (elected) tc_commit(drained);                               // tensor memory is given back below
        __syncwarp();
        (void)mbar_wait_bounded(drained, 0);
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        if (tid == 0) atomicMax(p.err, MI_ERR_TIMEOUT);
        if (warp == wRaw && lane == 0)
            for (int k = max(0, raw_issued - kRawSlots); k < raw_issued; k++) (void)mbar_wait_bounded(&raw_full[k % kRawSlots], (k / kRawSlots) & 1);
    }
    if (warp == wMma) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    }
    // (behind the loops: a call inside them, taken or not, keeps their values out of half the registers)
    if ((p.bad_rows || s_none) && !*abort_flag) sum_over_blocks<KB, PART>(p, smem, s_none);
}

// the digits of 16 elements, all planes
__device__ __forceinline__ void dig_store(const DigX& out, int nb, int tt, int b, int half, int t, const unsigned (&q)[4], int m) {
    unsigned d[4][4];
    #pragma unroll
    for (int k = 0; k < 4; k++) {
        unsigned v[4];
        dig_word(q[k], m, v);
        #pragma unroll
        for (int j = 0; j < 4; j++) d[j][k] = v[j];
    }
    #pragma unroll
    for (int j = 0; j < 4; j++)
        *reinterpret_cast<uint4*>(out.q + dig_offset(out, nb, tt, b, half, j, t)) = make_uint4(d[j][0], d[j][1], d[j][2], d[j][3]);
    if (3 * out.T + t < dig_rows(out.T))                              // rows of padding
        *reinterpret_cast<uint4*>(out.q + dig_offset(out, nb, tt, b, half, 0, 3 * out.T + t)) = make_uint4(0, 0, 0, 0);
}

// One CTA per (token, K range)
__global__ void __launch_bounds__(256) tok_digits_kernel(TokX x, int nb, int nst, DigX out, int M) {
    __shared__ DigReduce red;
    const int n = blockIdx.x, sp = blockIdx.y, ksg = gridDim.y, tid = threadIdx.x;
    const int b0 = sp * nst / ksg * kStepBlk, b1 = min((sp + 1) * nst / ksg * kStepBlk, nb);
    pdl_launch_dependents(); pdl_wait_prior();
    auto bits = [&](int b) { return (unsigned)__half_as_ushort(__float2half_rn((float)__dmul_rn(__ldcg(x.d + tok_scale(x.J, b, n)), 0x1p-1004))); };
    DigRange mine;
    for (int i = 2 * b0 + tid; i < 2 * b1; i += 256) {
        const unsigned h = bits(i >> 1);
        int sum = 0;
        #pragma unroll
        for (int k = 0; k < 4; k++) sum = __dp4a((int)__ldcg(x.q + tok_word(x.J, i >> 1, n, 16 * (i & 1) + 4 * k)), 0x01010101, sum);
        mine.add(h, sum);
    }
    const DigRange all = mine.over_cta(red);
    const int need = all.planes();
    if (tid == 0) { out.info[(size_t)sp * M + n] = all.unit() | need << 8; out.bias[(size_t)sp * M + n] = all.total(); }
    const int tt = n / out.T, t = n - tt * out.T;
    for (int i = 2 * b0 + tid; i < 2 * b1; i += 256) {               // two threads have a block's halves, a sector together
        const int b = i >> 1, half = i & 1, m = all.factor(bits(b));
        unsigned q[4];
        #pragma unroll
        for (int k = 0; k < 4; k++) q[k] = __ldcg(x.q + tok_word(x.J, b, n, 16 * half + 4 * k));
        dig_store(out, nb, tt, b, half, t, q, m);
    }
}

// SwiGLU, q8_0 and digits of one token over one K range.  What bounds it is the FP64 pipe (about 40 operations per element, an exponential and a division) as long as little is issued beside
// it: a warp has four blocks at once, four elements per lane (333 tokens of the 1.5B shape, where 2.98 million elements are 6.5 us of the pipe: 21 us; with an element
// per lane and a block per warp at a time 28).  Eight warps: 64 sequences of the 3B shape 3526 us, with sixteen 3570.  The blocks wait in shared memory for the range's exponent.
constexpr int kSwiWarps = 8;
__global__ void __launch_bounds__(kSwiWarps * 32) swiglu_digits_kernel(const float* y, TokX act, int nb, int nst, DigX out, int M) {
    __shared__ DigReduce red;
    extern __shared__ __align__(16) uint8_t smem[];                    // [block] 32 int8, then the scales
    const int n = blockIdx.x, sp = blockIdx.y, ksg = gridDim.y, tid = threadIdx.x, e = (tid & 7) * 4;
    const int b0 = sp * nst / ksg * kStepBlk, b1 = min((sp + 1) * nst / ksg * kStepBlk, nb);
    unsigned* q = reinterpret_cast<unsigned*>(smem);
    unsigned short* sc = reinterpret_cast<unsigned short*>(smem + (size_t)(b1 - b0) * 32);
    pdl_launch_dependents(); pdl_wait_prior();
    const float* row = y + (size_t)n * 64 * nb + e;
    auto fetch = [&](int b, float4& g, float4& u) {                    // (a block past the range: the last one again)
        const float4* p = reinterpret_cast<const float4*>(row + (size_t)min(b, b1 - 1) * 64);
        g = __ldcg(p); u = __ldcg(p + 8);
    };
    DigRange mine;
    float4 g = make_float4(0.f, 0.f, 0.f, 0.f), u = g;
    constexpr int S = kSwiWarps * 4;                                   // blocks of the CTA at a time
    if (b0 < b1) fetch(b0 + (tid >> 3), g, u);
    #pragma unroll 1
    for (int r = b0; r < b1; r += S) {
        const int b = r + (tid >> 3);
        const float4 gn = g, un = u;
        if (r + S < b1) fetch(b + S, g, u);
        const SwiBlock v = swiglu_block(gn, un);
        if (b < b1) {
            q[(b - b0) * 8 + (tid & 7)] = v.q;
            act.q[tok_word(act.J, b, n, e)] = v.q;
            if (e == 0) { sc[b - b0] = __half_as_ushort(v.d); act.d[tok_scale(act.J, b, n)] = tok_scale_value(v.d); mine.add(__half_as_ushort(v.d), v.sum); }
        }
    }
    const DigRange all = mine.over_cta(red);
    if (tid == 0) { out.info[(size_t)sp * M + n] = all.unit() | all.planes() << 8; out.bias[(size_t)sp * M + n] = all.total(); }
    const int tt = n / out.T, t = n - tt * out.T;
    for (int i = tid; i < 2 * (b1 - b0); i += kSwiWarps * 32) {
        const int b = i >> 1, half = i & 1, m = all.factor(sc[b]);
        const uint4 w = reinterpret_cast<const uint4*>(q)[i];
        const unsigned ww[4] = {w.x, w.y, w.z, w.w};
        dig_store(out, nb, tt, b0 + b, half, t, ww, m);
    }
}

// One warp per row
template <int KB>
__global__ void __launch_bounds__(256) row_exponents_kernel(const uint8_t* base, int groups, int nb, uint8_t* row_exp, int* found) {
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= groups * 32) return;
    int lo = 31, hi = 0;
    for (int b = lane; b < nb; b += 32) {
        const uint8_t* tile = base + ((size_t)(row >> 5) * nb + b / KB * KB) * kTileRowBytes;
        const unsigned h = __ldg(reinterpret_cast<const unsigned short*>(tile + KB * 512) + (row & 31) * KB + b % KB);
        if (h & 0x7FFFu) { lo = min(lo, scale_exponent(h)); hi = max(hi, scale_exponent(h)); }
    }
    lo = __reduce_min_sync(0xffffffffu, lo); hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane) return;
    lo = min(lo, max(hi, 1));
    row_exp[row] = hi == 31 || hi - lo > kMaxSpread ? kRowNone : lo;
    if (row_exp[row] == kRowNone) atomicAdd(found, 1);
    else if (hi - lo > found[1]) atomicMax(found + 1, hi - lo);
}

__global__ void __launch_bounds__(256) list_rows_kernel(const uint8_t* row_exp, int rows, int* list, int* count) {
    const int row = blockIdx.x * 256 + threadIdx.x;
    if (row < rows && row_exp[row] == kRowNone) list[atomicAdd(count, 1)] = row;
}

template <int KB, bool PART, bool TWO>
int launch_dig(mi_ctx* ctx, const DigParams& p, bool pdl) {
    const int units = (p.groups + 3) / 4 * p.x.TT * p.ksg;             // at least
    auto kern = gemm_dig_kernel<KB, PART, TWO>;
    static std::mutex mu;
    static std::atomic<unsigned> raised{0};                   // bit per device
    if (!(raised.load(std::memory_order_acquire) >> (ctx->device & 31) & 1u)) {
        std::lock_guard<std::mutex> hold(mu);
        MI_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem::bytes));
        raised.fetch_or(1u << (ctx->device & 31), std::memory_order_release);
    }
    MI_CUDA(ctx, launch_k(pdl, kern, dim3((unsigned)std::min(units, ctx->sm_count)), dim3(kThreads), Smem::bytes, ctx->stream, p));
    return MI_OK;
}
template <int KB>
int launch_kb(mi_ctx* ctx, const DigParams& p, bool part, bool two, bool pdl) {
    if (two) return part ? launch_dig<KB, true, true>(ctx, p, pdl) : launch_dig<KB, false, true>(ctx, p, pdl);
    return part ? launch_dig<KB, true, false>(ctx, p, pdl) : launch_dig<KB, false, false>(ctx, p, pdl);
}

}  // namespace

// Token tiles and K ranges of a product over digits, the fewest clocks by a model from measured launches: 7000 until the first MMA, 290 per block or what its MMAs take,
// 4000 and 80 per token for the end of a unit; for rows without an exponent what sum_over_blocks takes, 480 per block and round of its jobs (it decides whether a
// matrix with many such rows goes over digits at all; tokens without planes are known on the GPU only).
static double rows_cost(long long jobs, int nblk, long long ctas) {
    if (!jobs) return 0.0;
    int shift = 0;
    while (shift < 4 && jobs << (shift + 1) <= ctas * kExpWarps) shift++;
    const long long at_once = ctas * (kExpWarps >> shift);
    return 2000 + (double)((jobs + at_once - 1) / at_once) * ((nblk >> shift) + 1) * 480;
}
bool plan_gemm_dig(mi_ctx* ctx, const mi_weight* w, bool part, int M, DigPlan* out) {
    const int nst = (w->nb + kStepBlk - 1) / kStepBlk, rt = (w->groups + 3) / 4;
    const int TT = (M + kDigMaxT - 1) / kDigMaxT, T = ((M + TT - 1) / TT + 7) / 8 * 8;
    const double blk = std::max(kNW * dig_rows(T) / 2 + 30.0, 290.0);
    double best = 1e300;
    if (!w->row_exp) return false;
    for (int ksg = 1; ksg <= (part ? std::min(nst, 8) : 1); ksg++) {
        const int steps = (nst + ksg - 1) / ksg;
        if (steps * kStepBlk * 32 > 16384) continue;                   // a sum of digit products stays below 2^31 (three pairs of 255 * 128 per element)
        const long long units = (long long)rt * TT * ksg, rounds = (units + ctx->sm_count - 1) / ctx->sm_count;
        const int nblk = std::min(steps * kStepBlk, w->nb);
        const double cost = 7000 + rounds * (nblk * blk + 4000 + 80.0 * T) + rows_cost((long long)w->bad_rows * ksg * ((M + 31) / 32), nblk, std::min<long long>(units, ctx->sm_count)) + (part ? ksg * (double)M * w->rows * 16 / (ctx->sm_count * 40.0) : 0.0);
        if (cost < best) { best = cost; *out = DigPlan{T, TT, ksg, cost}; }
    }
    return best < 1e300;
}

// Where the line lies: both products' cost models, corrected by passes of 17 to 512 tokens of the 0.5B, 1.5B and 3B shapes, each timed with one product at a time over
// digits.  The block product takes a tenth more than its model says; digits of the attention's output (a launch of their own) and of SwiGLU's cost 28 clocks a token
// (333 tokens: 5 us), the lm_head over digits 15 us more than its model says.  Of 3 x 31 passes the rule loses 0.1 us a layer against the better choice
// of each product, 4.7 of 149 at most (the 3B shape's QKV at 72 tokens).
bool choose_gemm_dig(mi_ctx* ctx, const mi_weight* w, int i, int M, const GemmPlan& blocks, DigPlan* out) {
    const bool part = i == 1 || i == 3;
    return M > kMaxFusedTok && plan_gemm_dig(ctx, w, part, M, out) && out->cost + (part ? 28.0 * M : i == 4 ? 28500.0 : 0.0) < 1.1 * blocks.cost;
}

int launch_gemm_dig(mi_ctx* ctx, const mi_weight* w, const DigPlan& pl, int mode, const DigX& x, GemmParams g, bool pdl) {
    DigParams p{};
    p.base = w->dev; p.row_exp = w->row_exp; p.groups = w->groups; p.nb = w->nb; p.nst = (w->nb + kStepBlk - 1) / kStepBlk; p.rows = (int)w->rows;
    p.ksg = pl.ksg; p.M = g.M;
    int bits = 45 + w->row_spread;                                     // of a sum of one element, four planes
    for (int k = std::min((p.nst + pl.ksg - 1) / pl.ksg * kStepBlk, w->nb) * 32; k > 1; k = (k + 1) / 2) bits++;
    const bool two = bits > 63;
    p.x = x; p.q8 = g.x; p.bias = g.bias; p.y = g.y; p.part = g.part; p.ldp = g.ldp; p.err = ctx->d_err; p.bad_list = w->bad_list; p.bad_rows = w->bad_rows;
    const bool part = mode == GEMM_PART;
    if (p.M * p.ksg > kMaxInfo) return set_error(ctx, MI_ERR_LIMIT, "gemm: %d tokens in one launch", p.M);
    switch (w->kb) {
        case 8: return launch_kb<8>(ctx, p, part, two, pdl);
        case 4: return launch_kb<4>(ctx, p, part, two, pdl);
        case 2: return launch_kb<2>(ctx, p, part, two, pdl);
        default: return launch_kb<1>(ctx, p, part, two, pdl);
    }
}

int launch_tok_digits(mi_ctx* ctx, const mi_weight* w, const DigPlan& pl, const TokX& x, const DigX& out, int M, bool pdl) {
    MI_CUDA(ctx, launch_k(pdl, tok_digits_kernel, dim3(M, pl.ksg), dim3(256), 0, ctx->stream, x, w->nb, (w->nb + kStepBlk - 1) / kStepBlk, out, M));
    return MI_OK;
}

int launch_swiglu_digits(mi_ctx* ctx, const mi_weight* w, const DigPlan& pl, const float* y, const TokX& act, const DigX& out, int M, bool pdl) {
    const int nst = (w->nb + kStepBlk - 1) / kStepBlk, blocks = (nst + pl.ksg - 1) / pl.ksg * kStepBlk;        // of a range, at most
    MI_CUDA(ctx, launch_k(pdl, swiglu_digits_kernel, dim3(M, pl.ksg), dim3(kSwiWarps * 32), (size_t)blocks * 34, ctx->stream, y, act, w->nb, nst, out, M));
    return MI_OK;
}

int launch_row_exponents(mi_ctx* ctx, const mi_weight* w, uint8_t* row_exp, int* found) {
    const dim3 grid((unsigned)(w->groups * 4));
    if (w->groups == 0) return MI_OK;
    switch (w->kb) {
        case 8: row_exponents_kernel<8><<<grid, 256, 0, ctx->stream>>>(w->dev, w->groups, w->nb, row_exp, found); break;
        case 4: row_exponents_kernel<4><<<grid, 256, 0, ctx->stream>>>(w->dev, w->groups, w->nb, row_exp, found); break;
        case 2: row_exponents_kernel<2><<<grid, 256, 0, ctx->stream>>>(w->dev, w->groups, w->nb, row_exp, found); break;
        default: row_exponents_kernel<1><<<grid, 256, 0, ctx->stream>>>(w->dev, w->groups, w->nb, row_exp, found); break;
    }
    MI_CUDA(ctx, cudaGetLastError());
    return MI_OK;
}

int launch_list_rows(mi_ctx* ctx, const mi_weight* w, int* list, int* count) {
    if (w->rows > 0) list_rows_kernel<<<(unsigned)((w->rows + 255) / 256), 256, 0, ctx->stream>>>(w->row_exp, (int)w->rows, list, count);
    MI_CUDA(ctx, cudaGetLastError());
    return MI_OK;
}

}  // namespace mi

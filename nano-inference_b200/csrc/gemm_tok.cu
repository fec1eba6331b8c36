// q4_0 x q8_0 product for M tokens per weight pass (prompt chunks, drafted tokens, batches): the GEMV's sums, token by
// token the same bits, with the integer block dot products on the tensor cores.
//
// Replaces gemv_dp4a_batch<T> (reference src/cuda_infer.cu:183-222) and mma_s8 / tile_dot (reference
// src/mega.cu:197-244).
//
// What bounds it.  Every q4_0 block has a scale of its own, so an integer sum lives for K = 32 only: per (row, block,
// token) one int32 has to be scaled by dw*dx and added in double.  Measured alone, a DFMA keeps an SM sub-partition for 2.25 cycles and an
// mma.m16n8k32.s8 for 12 (four values per lane): 4.5 + 3 cycles a value, the floor of this scheme.  The rest are moves, shared-memory loads and
// unpacking.  The gate/up product of 333 tokens (17920 x 1536, tiles of 24, three warps per sub-partition) takes 13.6 cycles a value: issue active 54 %
// of the cycles, FP64 pipe 32 %, int8 MMA 15 %, so no unit by itself is full, but issued instructions and the cycles above together are 94 % of the
// time of the SMs that have work; 128 tokens (tiles of 32, two warps, the second round nine tenths full): 15 cycles, 46 / 28 / 13 %, 80 %.  Passes of 16
// tokens are as much waiting as issue (30 cycles a value at the 1.5B shape's gate/up; first tiles and staging).  So the design minimizes what is issued per value:
//   * mma.sync and not tcgen05: its operands and sums are registers.  A nibble tile becomes an A fragment with three logic
//     operations per two registers straight from a 4-byte shared-memory load, and a sum goes from the MMA into the FMA.
//     A tcgen05.kind::i8 kernel with the same scaling was built and measured beside it: its MMAs cost no issue slots, but
//     operand tiles through shared memory, sums through tensor memory, the barriers between the two and units of 128
//     rows cost more (1536 x 8960, 5 tokens: 8.0 us against 4.8; lm_head shape, 16 tokens: 85 us against 56).
//   * t = fma(dw, 2^52 + 2^31 + s, -dw (2^52 + 2^31)) = dw * s exactly, then acc = fma(dx, t, acc), the GEMV's one rounding.
//     The MMA starts from C = 2^31, so its result read as unsigned is s + 2^31 and with 0x43300000 above it is that
//     double.  Four register pairs keep the upper half for the whole kernel; a sum costs one move into a lower half.
//     (Left to itself the compiler moves both halves, half as many cycles again.)
//   * dw's fp16 bits are shifted into a double's exponent field (see TokX for the powers of two);
//   * the nibble offset costs nothing: (nibble << 4) ^ 0x80 is the signed byte 16 (n - 8).
//
// Shape of the work.  A unit is a group of 32 rows (a gate and an up group for GEMM_GU) against one token tile of up to 32 tokens over
// one K range.  Large matrices: a unit belongs to one warp (kw = 1), which goes from its first tile to its stores without
// meeting another warp.  Small ones: kw warps of a CTA share the K tiles of a unit and fold their sums through shared memory.
// Each warp streams its tiles through a ring of bulk copies that starts before the kernel waits for its predecessor (weights
// depend on nothing); the activations of the CTA's K range and token tile are staged once, or chunk by chunk where they do
// not fit.  Products of more tokens go to gemm_dig.cu where the pass's cost model says so.  With 32 rows x 32 tokens per warp an A fragment serves four MMAs and a B fragment two.  For many tokens a tcgen05 kernel with this scaling per block, of
// four roles (unpackers, MMA issuer, activation copies, scaling warps reading tensor memory) was measured as well: 17920 x 1536 with 333
// tokens 130 us against 123, 2048 x 11008 with 64 tokens 26.6 against 28; one thread issuing an MMA per 32-element block took 150 cycles
// for each, and the unpackers' issue slots are missing beside the scaling.
#include "gemm_tok.cuh"
#include <algorithm>
#include <atomic>
#include <mutex>

namespace mi {

constexpr int kRing = 2;                                     // ring slots per warp
constexpr int kStaticSmem = 64;                              // room for static shared memory
constexpr int kFoldLd = 34;                                  // doubles per token in the fold buffer: conflict-free for the MMA's layout
__host__ __device__ constexpr int tok_warps(int NT) { return NT <= 3 ? 12 : 8; }

constexpr int kStepBlk = 8;                                  // blocks per ring slot: one tile of eight blocks, or as many smaller ones (they are contiguous)
constexpr int kStepBytes = kStepBlk * kTileRowBytes;

template <int NT, bool FOLD>
struct TokSmem {
    static constexpr int W = tok_warps(NT), TB = kStepBytes, N = NT * 8;
    static constexpr int ring = W * kRing * TB;
    static constexpr int scratch = FOLD ? W * N * kFoldLd * 8 : 0;                          // partial sums of all warps
    static constexpr int bars = ((W * kRing + 1) * 8 + 15) / 16 * 16;
    static constexpr int fixed = ring + scratch + bars;
    static constexpr int x_block = NT * 256 + N * 8, x_step = kStepBlk * x_block;
};

__device__ __forceinline__ void mma_s8(int (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, const uint2& b) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b.x), "r"(b.y), "r"((int)0x80000000));
}

// One tile (32 rows, KB blocks) against NT * 8 tokens.  Lane (g = lane / 4, t = lane % 4) holds rows g + 8 i (i = 0..3) and tokens
// 2t, 2t + 1 of every token group: acc[j][2 i + c] is row g + 8 i, token 8 j + 2 t + c.
// poison: 0 + 0 * scale over all scales seen: NaN once a weight scale was not finite (its bits pass for a number here; see row_sum).
// pair: upper halves 0x43300000.
template <int KB, int NT>
__device__ __forceinline__ void tile_mma(const uint8_t* tile, const uint2* bs, const double* dxs, int lane, double (&acc)[NT][8], __half2 (&poison)[4], double (&pair)[4]) {
    const int g = lane >> 2, t = lane & 3;
    constexpr int SW = KB >= 2 ? KB / 2 : 1;
    unsigned sc[4][SW];
    #pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint8_t* sp = tile + KB * 512 + (g + 8 * i) * (KB * 2);
        if constexpr (KB == 8) { const uint4 v = *reinterpret_cast<const uint4*>(sp); sc[i][0] = v.x; sc[i][1] = v.y; sc[i][2] = v.z; sc[i][3] = v.w; }
        else if constexpr (KB == 4) { const uint2 v = *reinterpret_cast<const uint2*>(sp); sc[i][0] = v.x; sc[i][1] = v.y; }
        else if constexpr (KB == 2) sc[i][0] = *reinterpret_cast<const unsigned*>(sp);
        else sc[i][0] = *reinterpret_cast<const unsigned short*>(sp);
        #pragma unroll
        for (int k = 0; k < SW; k++) poison[i] = __hfma2(*reinterpret_cast<const __half2*>(&sc[i][k]), __half2half2(__ushort_as_half(0)), poison[i]);
    }
    #pragma unroll
    for (int k = 0; k < KB; k++) {
        unsigned lo[4], hi[4];
        double dw[4], cw[4];
        #pragma unroll
        for (int i = 0; i < 4; i++) {
            const unsigned w = *reinterpret_cast<const unsigned*>(tile + (k * 32 + g + 8 * i) * 16 + 4 * t);
            lo[i] = ((w << 4) & 0xF0F0F0F0u) ^ 0x80808080u;
            hi[i] = (w & 0xF0F0F0F0u) ^ 0x80808080u;
            const unsigned s = sc[i][k / 2];
            const unsigned dhi = (k & 1) ? (((s >> 6) & 0x01FFFC00u) | (s & 0x80000000u)) : (((s << 10) & 0x01FFFC00u) | ((s << 16) & 0x80000000u));
            dw[i] = __hiloint2double((int)dhi, 0);
            cw[i] = __dmul_rn(dw[i], -4503601774854144.0);                      // -(2^52 + 2^31) dw: exact
        }
        #pragma unroll
        for (int j = 0; j < NT; j++) {
            const uint2 b = bs[(k * NT + j) * 32 + lane];
            const double2 dx = *reinterpret_cast<const double2*>(dxs + (k * NT + j) * 8 + 2 * t);
            int d[2][4];
            mma_s8(d[0], lo[0], lo[1], hi[0], hi[1], b);
            mma_s8(d[1], lo[2], lo[3], hi[2], hi[3], b);
            #pragma unroll
            for (int h = 0; h < 2; h++)
                #pragma unroll
                for (int r = 0; r < 4; r++) {
                    const int i = 2 * h + (r >> 1);
                    asm volatile("{\n\t.reg .b32 l, u;\n\tmov.b64 {l, u}, %0;\n\tmov.b64 %0, {%1, u};\n\t}" : "+d"(pair[r]) : "r"(d[h][r]));
                    acc[j][2 * i + (r & 1)] = __fma_rn((r & 1) ? dx.y : dx.x, __fma_rn(dw[i], pair[r], cw[i]), acc[j][2 * i + (r & 1)]);
                }
        }
    }
}

// One row's sum over a warp's steps (every kw-th from t0 on, below t1) for token n, formed as the GEMV forms it.  For rows with a weight scale that is not
// finite: infinities and NaN come out as they do there.  Straight from global memory; such rows do not occur in a working
// model.  Out of line: inlined it cost 16-token passes up to 0.6 % in registers (16 sequences of the 3B shape 1968 instead of 1958 us).
template <int KB, bool ROWMAJOR>
static __device__ __noinline__ double row_sum(const GemmParams& p, int grp, int row, int n, int t0, int t1, int kw) {
    double acc = 0.0;
    #pragma unroll 1
    for (int t = t0; t < t1; t += kw) {
        #pragma unroll 1
        for (int b = t * kStepBlk; b < min((t + 1) * kStepBlk, p.nb); b++) {
            const uint8_t* tile = p.base + ((size_t)grp * p.nb + b / KB * KB) * kTileRowBytes;
            const uint4 w = __ldg(reinterpret_cast<const uint4*>(tile) + b % KB * 32 + row);
            const float dw = __half2float(__ldg(reinterpret_cast<const __half*>(tile + KB * 512) + row * KB + b % KB));
            int4 xa, xc;
            float dx;
            if constexpr (ROWMAJOR) {
                const int4* x = reinterpret_cast<const int4*>(p.xq + ((size_t)n * p.nb + b) * 32);
                xa = __ldcg(x); xc = __ldcg(x + 1);
                dx = __half2float(__ushort_as_half(__ldcg(reinterpret_cast<const unsigned short*>(p.xd) + (size_t)n * p.nb + b)));
            } else {
                auto word = [&](int e) { return (int)__ldcg(p.x.q + tok_word(p.x.J, b, n, e)); };
                xa = make_int4(word(0), word(4), word(8), word(12)); xc = make_int4(word(16), word(20), word(24), word(28));
                dx = (float)__dmul_rn(__ldcg(p.x.d + tok_scale(p.x.J, b, n)), 0x1p-1004);
            }
            acc = blk_acc(acc, dw, dx, dot_q4_block(w, xa, xc), __int2float_rn(8 * sum_x_block(xa, xc)));
        }
    }
    return acc;
}

template <int KB, int NT, int MODE, bool ROWMAJOR, bool FOLD>
__global__ void __launch_bounds__(tok_warps(NT) * 32, 1) gemm_q4_q8_tok_kernel(const __grid_constant__ GemmParams p) {
    using SM = TokSmem<NT, FOLD>;
    constexpr int W = SM::W, TB = SM::TB, N = SM::N, U = MODE == GEMM_GU ? 2 : 1;
    static_assert(FOLD || MODE == GEMM_PLAIN || MODE == GEMM_PART, "epilogues across rows work on folded sums");
    extern __shared__ __align__(128) uint8_t smem[];
    uint8_t* scratch = smem + SM::ring;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + SM::ring + SM::scratch);
    uint64_t* xbar = bars + W * kRing;
    uint2* bs = reinterpret_cast<uint2*>(smem + SM::fixed);                              // staged activations: operands of a chunk, then its scales
    double* dxs = reinterpret_cast<double*>(smem + SM::fixed + (size_t)p.kct * kStepBlk * NT * 256);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int sp = (int)(blockIdx.x % p.ksg), rest = (int)(blockIdx.x / p.ksg), c = rest % p.C, tt = rest / p.C;
    const int k0 = sp * p.nt / p.ksg, k1 = (sp + 1) * p.nt / p.ksg, nchunk = (k1 - k0 + p.kct - 1) / p.kct;      // this CTA's K range, in steps
    // the warp's row group of round r: group0 + r * gstride, while below glimit
    const int kw = FOLD ? p.kw : 1, rg = FOLD ? W / kw : W, gi = FOLD ? warp / kw : warp, part = FOLD ? warp - gi * kw : 0;
    const int group0 = FOLD ? c * rg + gi : warp * p.C + c, gstride = p.C * rg, glimit = gi < rg ? p.groups : 0;
    const int rounds = FOLD ? ((p.groups + rg - 1) / rg - c + p.C - 1) / p.C : (p.groups + p.C * W - 1) / (p.C * W);
    const int ntok = min(N, p.M - tt * N);

    uint8_t* ring = smem + (size_t)warp * kRing * TB;
    uint64_t* rbar = bars + warp * kRing;
    if (lane == 0) {
        #pragma unroll
        for (int s = 0; s < kRing; s++) mbar_init(&rbar[s], 1);
        if (warp == 0) mbar_init(xbar, 1);
        mbar_fence_init();
    }
    __syncwarp();
    // producer (lane 0), kRing tiles ahead of the consumer below: every kw-th tile of the K range, round after round
    const uint64_t policy = l2_policy_evict_first();
    int issued = 0, consumed = 0, pr = 0, pt = k0 + part;
    auto issue_one = [&]() {
        if (pr >= rounds || pt >= k1) return;                                            // done, or more warps than tiles
        const int grp = group0 + pr * gstride;
        if (grp >= glimit) { pr = rounds; return; }                                      // groups only grow: nothing follows
        const int s = issued % kRing;
        const int bytes = min(kStepBlk, p.nb - pt * kStepBlk) * kTileRowBytes;
        mbar_expect_tx(&rbar[s], bytes);
        bulk_g2s_hint(ring + (size_t)s * TB, p.base + ((size_t)grp * p.nb + pt * kStepBlk) * kTileRowBytes, bytes, &rbar[s], policy);
        issued++; pt += kw;
        if (pt >= k1) { pt = k0 + part; pr++; }
    };
    if (lane == 0) {
        #pragma unroll
        for (int s = 0; s < kRing; s++) issue_one();
    }
    pdl_launch_dependents();
    pdl_wait_prior();                                                                    // activations come from the kernel before
    __syncthreads();                                                                     // xbar is initialised

    unsigned xphase = 0;
    auto stage = [&](int b0, int nblk) {                                                 // activations of blocks b0 .. b0 + nblk
        if constexpr (ROWMAJOR) {
            // 16 bytes per thread and load (half h of block b of token n), four loads in flight; they land as four lanes' words
            const int items = nblk * NT * 16;
            for (int i0 = tid; i0 < items; i0 += 4 * W * 32) {
                int4 v[4];
                #pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int i = i0 + u * W * 32, n = tt * N + (i >> 1) % N, b = (i >> 1) / N;
                    v[u] = make_int4(0, 0, 0, 0);
                    if (i < items && n < p.M) v[u] = __ldcg(reinterpret_cast<const int4*>(p.xq + ((size_t)n * p.nb + b0 + b) * 32) + (i & 1));
                }
                #pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int i = i0 + u * W * 32, n = (i >> 1) % N, b = (i >> 1) / N;
                    if (i < items) {
                        int* dst = reinterpret_cast<int*>(bs + ((size_t)b * NT + (n >> 3)) * 32 + (n & 7) * 4) + (i & 1);
                        dst[0] = v[u].x; dst[2] = v[u].y; dst[4] = v[u].z; dst[6] = v[u].w;
                    }
                }
            }
            #pragma unroll 4
            for (int i = tid; i < nblk * N; i += W * 32) {
                const int n = tt * N + i % N, b = i / N;
                dxs[i] = n < p.M ? tok_scale_value(__ushort_as_half(__ldcg(reinterpret_cast<const unsigned short*>(p.xd) + (size_t)n * p.nb + b0 + b))) : 0.0;
            }
        } else if (warp == 0) {
            if (lane == 0) mbar_expect_tx(xbar, (unsigned)nblk * SM::x_block);
            __syncwarp();
            if (p.x.J == NT) {
                if (lane == 0) {
                    bulk_g2s(bs, p.x.q + (size_t)b0 * (NT * 64), (unsigned)nblk * (NT * 256), xbar);
                    bulk_g2s(dxs, p.x.d + (size_t)b0 * N, (unsigned)nblk * (N * 8), xbar);
                }
            } else {
                for (int b = lane; b < nblk; b += 32) {
                    bulk_g2s(bs + (size_t)b * NT * 32, p.x.q + ((size_t)(b0 + b) * p.x.J + tt * NT) * 64, NT * 256, xbar);
                    bulk_g2s(dxs + (size_t)b * N, p.x.d + ((size_t)(b0 + b) * p.x.J + tt * NT) * 8, N * 8, xbar);
                }
            }
        }
    };
    stage(k0 * kStepBlk, min(min(k0 + p.kct, k1) * kStepBlk, p.nb) - k0 * kStepBlk);
    if constexpr (ROWMAJOR) __syncthreads();
    bool ok = true, xready = ROWMAJOR;

    // register pairs whose upper half stays 0x43300000 while sums pass through the lower half (opaque, so that the
    // compiler does not rebuild the constant for every sum)
    double pair[4];
    #pragma unroll
    for (int i = 0; i < 4; i++) asm volatile("mov.b64 %0, 0x4330000000000000;" : "=d"(pair[i]));

    bool first = true;
    for (int r = 0; r < rounds; r++) {
        const int grp0 = group0 + r * gstride;
        const bool mine = grp0 < glimit;
        double acc[NT][8];
        #pragma unroll
        for (int j = 0; j < NT; j++)
            #pragma unroll
            for (int i = 0; i < 8; i++) acc[j][i] = 0.0;
        __half2 poison[4];
        #pragma unroll
        for (int i = 0; i < 4; i++) poison[i] = __half2half2(__ushort_as_half(0));
        int t = k0 + part;
        for (int ch = 0; ch < nchunk; ch++) {
            const int c0 = k0 + ch * p.kct, c1 = min(c0 + p.kct, k1);
            if (nchunk > 1 && !first) {                                              // everyone has left the previous chunk: the next one over it
                __syncthreads();
                if constexpr (!ROWMAJOR) { if (warp == 0) asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
                stage(c0 * kStepBlk, min(c1 * kStepBlk, p.nb) - c0 * kStepBlk);
                if constexpr (ROWMAJOR) __syncthreads(); else xready = false;
            }
            first = false;
            if (!xready) {
                if (ok && !mbar_wait_bounded(xbar, xphase)) ok = false;
                xphase ^= 1u; xready = true;
            }
            if (mine) {
                for (; t < c1 && ok; t += kw) {
                    const int s = consumed % kRing;
                    if (!mbar_wait_bounded(&rbar[s], (consumed / kRing) & 1)) { ok = false; break; }
                    if constexpr (KB == kStepBlk) tile_mma<KB, NT>(ring + (size_t)s * TB, bs + (size_t)(t - c0) * (KB * NT * 32), dxs + (size_t)(t - c0) * (KB * N), lane, acc, poison, pair);
                    else {
                        const int nb = min(kStepBlk, p.nb - t * kStepBlk);
                        #pragma unroll 4
                        for (int k = 0; k < nb; k += KB)
                            tile_mma<KB, NT>(ring + (size_t)s * TB + k * kTileRowBytes, bs + (size_t)((t - c0) * kStepBlk + k) * (NT * 32), dxs + (size_t)((t - c0) * kStepBlk + k) * N, lane, acc, poison, pair);
                    }
                    consumed++;
                    __syncwarp();
                    if (lane == 0) issue_one();
                }
            }
        }
        unsigned bad = 0;                                                                // bit i: row g + 8 i has such a scale among this warp's tiles
        #pragma unroll
        for (int i = 0; i < 4; i++) bad |= (unsigned)__hisnan(__hadd(__low2half(poison[i]), __high2half(poison[i]))) << i;
        // those rows' sums again, over the ones the lane has just stored: store(row of the group, token of the tile, sum)
        auto again = [&](auto store) {
            #pragma unroll 1
            for (; bad; bad &= bad - 1) {
                const int row = g + 8 * (__ffs(bad) - 1);
                #pragma unroll 1
                for (int q = 0; q < 2 * NT; q++) {
                    const int n = 8 * (q >> 1) + 2 * t4 + (q & 1);
                    if (n < ntok) store(row, n, row_sum<KB, ROWMAJOR>(p, grp0, row, tt * N + n, k0 + part, k1, kw));
                }
            }
        };
        if constexpr (!FOLD) {
            if (!mine) continue;
            // straight from the MMA's layout: lane (g, t4) has rows g + 8 i and tokens 8 j + 2 t4 + cc
            #pragma unroll
            for (int i = 0; i < 4; i++) {
                const int row = grp0 * 32 + g + 8 * i;
                const float bv = MODE == GEMM_PLAIN && p.bias && row < p.rows ? __ldg(p.bias + row) : 0.f;
                #pragma unroll
                for (int j = 0; j < NT; j++)
                    #pragma unroll
                    for (int cc = 0; cc < 2; cc++) {
                        const int n = 8 * j + 2 * t4 + cc;
                        if (n >= ntok || row >= p.rows) continue;
                        if constexpr (MODE == GEMM_PART) __stcg(p.part + ((size_t)sp * p.M + tt * N + n) * p.ldp + row, acc[j][2 * i + cc]);
                        else p.y[(size_t)(tt * N + n) * p.rows + row] = __double2float_rn(acc[j][2 * i + cc]) + bv;
                    }
            }
            if (bad) again([&](int r32, int n, double v) {
                const int row = grp0 * 32 + r32;
                if (row >= p.rows) return;
                if constexpr (MODE == GEMM_PART) __stcg(p.part + ((size_t)sp * p.M + tt * N + n) * p.ldp + row, v);
                else p.y[(size_t)(tt * N + n) * p.rows + row] = __double2float_rn(v) + (p.bias ? __ldg(p.bias + row) : 0.f);
            });
        } else {
            double* fold = reinterpret_cast<double*>(scratch);                           // [warp][token][kFoldLd]
            if (r > 0) __syncthreads();                                                  // the previous round's sums have been read
            if (gi < rg) {
                double* fw = fold + (size_t)warp * N * kFoldLd;
                #pragma unroll
                for (int j = 0; j < NT; j++)
                    #pragma unroll
                    for (int i = 0; i < 8; i++) fw[(8 * j + 2 * t4 + (i & 1)) * kFoldLd + g + 8 * (i >> 1)] = acc[j][i];
                if (bad) again([&](int row, int n, double v) { fw[n * kFoldLd + row] = v; });
            }
            __syncthreads();
            // one warp per (row group [pair], token): lane = row
            const int set0 = (c + r * p.C) * rg, units = min(rg, p.groups - set0) / U;
            int u = 0, n = warp;
            while (u < units && n >= ntok) { n -= ntok; u++; }
            #pragma unroll 1
            while (u < units) {
                const int grp = set0 + u * U, m = tt * N + n, row = grp * 32 + lane;
                const double* f0 = fold + ((size_t)u * U * kw * N + n) * kFoldLd + lane;
                double v0 = f0[0];
                for (int q = 1; q < kw; q++) v0 = __dadd_rn(v0, f0[(size_t)q * N * kFoldLd]);
                if constexpr (MODE == GEMM_GU) {
                    const double* f1 = f0 + (size_t)kw * N * kFoldLd;
                    double v1 = f1[0];
                    for (int q = 1; q < kw; q++) v1 = __dadd_rn(v1, f1[(size_t)q * N * kFoldLd]);
                    store_tok_block(p.act, grp >> 1, m, lane, swiglu(__double2float_rn(v0), __double2float_rn(v1)));
                } else if constexpr (MODE == GEMM_QKV) {
                    rope_store(p.rope, row, m, __fadd_rn(__double2float_rn(v0), __ldg(p.bias + row)));
                } else if constexpr (MODE == GEMM_PART) {
                    if (row < p.rows) __stcg(p.part + ((size_t)sp * p.M + m) * p.ldp + row, v0);
                } else {
                    if (row < p.rows) p.y[(size_t)m * p.rows + row] = __double2float_rn(v0) + (p.bias ? __ldg(p.bias + row) : 0.f);
                }
                n += W;
                while (u < units && n >= ntok) { n -= ntok; u++; }
            }
        }
    }
    if (!ok && lane == 0) {
        atomicMax(p.err, MI_ERR_TIMEOUT);
        for (int k = consumed; k < issued; k++) (void)mbar_wait_bounded(&rbar[k % kRing], (k / kRing) & 1);    // copies in flight target this CTA
    }
}

// y[m][row] = fp32(sum of the K ranges) + bias
__global__ void __launch_bounds__(256) sum_ranges_kernel(const double* part, int ranges, int rows, const float* bias, float* y) {
    const int row = blockIdx.x * 256 + threadIdx.x, m = blockIdx.y;
    pdl_launch_dependents(); pdl_wait_prior();
    if (row >= rows) return;
    const double* s = part + (size_t)m * rows + row;
    double v = __ldcg(s);
    for (int q = 1; q < ranges; q++) v = __dadd_rn(v, __ldcg(s + (size_t)q * gridDim.y * rows));
    y[(size_t)m * rows + row] = __double2float_rn(v) + (bias ? __ldg(bias + row) : 0.f);
}

// ---- host side -----------------------------------------------------------------------------------------------------

namespace {
struct SmemNeed { int ring_bars, fold, x_step; };
SmemNeed smem_need(int NT) {
    switch (NT) {
        #define MI_F(nt) case nt: return SmemNeed{TokSmem<nt, false>::fixed, TokSmem<nt, true>::fixed, TokSmem<nt, true>::x_step};
        MI_F(1) MI_F(2) MI_F(3)
        #undef MI_F
    }
    return SmemNeed{TokSmem<4, false>::fixed, TokSmem<4, true>::fixed, TokSmem<4, true>::x_step};
}
}  // namespace

// How to cut a matrix: kw warps per row group (1: warps work alone), C CTAs per (K range, token tile), ksg K ranges (only where
// the consumer adds them, GEMM_PART).  Small matrices want every sub-partition of every SM to have a tile, large ones want
// warps that never meet.  The choice is the minimum of a rough model in clocks, from the measured costs: a tile costs its blocks'
// issue slots, which the warps of a sub-partition share, the end of a unit its stores or a pass through shared memory.
int plan_gemm_tok(mi_ctx* ctx, const mi_weight* w, int mode, int M, const TokTiling& tl, GemmPlan* out) {
    const int NT = tl.NT, TT = tl.TT, W = tok_warps(NT), N = NT * 8, U = mode == GEMM_GU ? 2 : 1, ntok = std::min(M, N);
    const SmemNeed need = smem_need(NT);
    const int nt = (w->nb + kStepBlk - 1) / kStepBlk;                                     // steps of eight blocks
    const double c_blk[kMaxTokNT + 1] = {0, 121, 200, 290, 400};                          // clocks per block, two or three warps per sub-partition
    const double c_tile = kStepBlk * (c_blk[NT] + (w->kb < 8 ? 30 : 0)) + 100;
    const double c_tok = mode == GEMM_GU ? 640 : mode == GEMM_QKV ? 300 : 60;             // end of a round, per token and warp
    double best = 1e300;
    const int max_ksg = mode == GEMM_PART ? std::min(nt, 8) : 1;
    for (int ksg = 1; ksg <= max_ksg; ksg++) {
        const int ntr = (nt + ksg - 1) / ksg, cmax = std::max(1, ctx->sm_count / (ksg * TT));
        for (int v = 0; v <= W; v++) {                                                // 0: warps alone; else v warps per row group, sums through shared memory
            const bool fold = v > 0;
            const int kw = std::max(1, v), rg = W / kw;
            if (fold ? (v == 1 && U == 1) || rg % U || W / rg != kw : U == 2 || mode == GEMM_QKV) continue;   // pairs stay together; no warps idle by rounding
            const int fixed = fold ? need.fold : need.ring_bars;
            const int fit = (ctx->smem_optin - kStaticSmem - fixed) / need.x_step;
            if (fit < 1) continue;
            const int kct = std::min(ntr, fit), nchunk = (ntr + kct - 1) / kct;
            const int nsets = fold ? (w->groups + rg - 1) / rg : w->groups, C = std::min(nsets, cmax);
            const int rounds = fold ? (nsets + C - 1) / C : (nsets + C * W - 1) / (C * W), waves = (ksg * TT * C + ctx->sm_count - 1) / ctx->sm_count;
            double cost;
            if (fold) {
                const int tiles = (ntr + kw - 1) / kw, sub = (std::min(kw, ntr) * std::min(rg, w->groups) + 3) / 4;       // warps with tiles per sub-partition
                const int items = (rg / U * ntok + W - 1) / W;
                cost = rounds * (tiles * std::max(sub * c_tile, c_tile * 1.2) + 900 + 60.0 * NT + items * (c_tok + 20.0 * U * kw));
            } else {
                const int sub = (int)((nsets + (long long)C * 4 - 1) / ((long long)C * 4));                                // units of the busiest sub-partition
                cost = sub * (ntr * c_tile * (sub > 1 ? 1.0 : 1.2) + 250.0 * NT) + 300;
            }
            cost = waves * (cost + 600 + (nchunk > 1 ? rounds * nchunk * 1500.0 : 0.0)) + (mode == GEMM_PART ? ksg * (double)M * w->rows * 16 / (ctx->sm_count * 40.0) : 0.0);
            if (cost < best) {
                best = cost;
                *out = GemmPlan{NT, TT, ksg, kct, C, kw, fold, (size_t)fixed + (size_t)kct * need.x_step, cost};
            }
        }
    }
    if (best == 1e300) return set_error(ctx, MI_ERR_UNSUPPORTED, "gemm: tile depth %d does not fit the shared memory", w->kb);
    out->cost += 0.4 * TT * (double)w->groups * w->nb * kTileRowBytes / 3400.0;     // every token tile reads the weights again (3400 bytes per clock of HBM)
    // What several token tiles cost beyond that, fitted to 124 passes of 17 .. 512 tokens, prompts and batches, each timed with tiles of 16, 24 and 32
    // tokens: 0.1 us per tile, and per launch of folded units 2, 2.5 and 1.5 us (clocks here).  It decides between tilings, not between cuts.
    out->cost += 190.0 * TT;
    if (out->fold && TT > 1) out->cost += NT == 2 ? 3800 : NT == 3 ? 4750 : 2850;
    return MI_OK;
}

// The token tile of a whole pass (its products share the operand order): wide ones issue less per value and read the weights
// less often, narrow ones leave more warps per sub-partition and divide the work more evenly.  The cheapest by the products' cost model, which over
// those passes is the fastest to 0.2 % on average and 4.3 % at most.  A layer's products in us, with tiles of 16 / 24 / 32 tokens: 1.5B shape, 32 tokens
// 52 / - / 49, 333 tokens 249 / 238 / 256; 0.5B shape, 48 tokens 37 / 43 / -, 96 tokens 56 / 56 / 47; 3B shape, 64 tokens 107 / 123 / 112.
int plan_pass_products(mi_ctx* ctx, const mi_weight* const mats[5], int L, int M, int n_head, TokTiling* tiles, GemmPlan plans[5]) {
    const bool fused = M <= kMaxFusedTok;
    const int modes[5] = {fused ? GEMM_QKV : GEMM_PLAIN, GEMM_PART, fused ? GEMM_GU : GEMM_PLAIN, GEMM_PART, GEMM_PLAIN};
    double best = 1e300;
    for (int max_nt = kMaxTokNT; max_nt >= 2 && (max_nt == kMaxTokNT || !fused); max_nt--) {
        const TokTiling tl = tok_tiling(M, max_nt);
        GemmPlan p[5];
        double cost = 0.0;
        for (int i = 0; i < 5; i++) {
            const bool head = i == 4;
            const int Mi = head ? std::max(n_head, 1) : M;
            const int st = plan_gemm_tok(ctx, mats[i], modes[i], Mi, Mi == M ? tl : tok_tiling(Mi), &p[i]);
            if (st != MI_OK) return st;
            if (!head || n_head > 0) cost += (head ? 1 : L) * p[i].cost;
        }
        if (cost < best) { best = cost; *tiles = tl; std::copy(p, p + 5, plans); }
    }
    return MI_OK;
}

namespace {
template <int KB, int NT, int MODE, bool ROWMAJOR, bool FOLD>
int launch_one(mi_ctx* ctx, const GemmPlan& pl, const GemmParams& p, bool pdl) {
    auto kern = gemm_q4_q8_tok_kernel<KB, NT, MODE, ROWMAJOR, FOLD>;
    // the opt-in shared-memory size is a property of (device, kernel): set once to the most this kernel may use
    static std::mutex mu;
    static std::atomic<unsigned> raised{0};                   // bit per device
    if (!(raised.load(std::memory_order_acquire) >> (ctx->device & 31) & 1u)) {
        std::lock_guard<std::mutex> hold(mu);
        MI_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->smem_optin - kStaticSmem));
        raised.fetch_or(1u << (ctx->device & 31), std::memory_order_release);
    }
    MI_CUDA(ctx, launch_k(pdl, kern, dim3((unsigned)(pl.ksg * pl.TT * pl.C)), dim3(tok_warps(NT) * 32), pl.smem, ctx->stream, p));
    return MI_OK;
}
template <int KB, int NT, bool FOLD>
int launch_mode(mi_ctx* ctx, const GemmPlan& pl, int mode, bool rowmajor, const GemmParams& p, bool pdl) {
    if (rowmajor) {
        if constexpr (NT <= 2) return mode == GEMM_PART ? launch_one<KB, NT, GEMM_PART, true, FOLD>(ctx, pl, p, pdl) : launch_one<KB, NT, GEMM_PLAIN, true, FOLD>(ctx, pl, p, pdl);
        return set_error(ctx, MI_ERR_LIMIT, "gemm: row-major activations of more than 16 tokens");
    }
    if (mode == GEMM_PLAIN) return launch_one<KB, NT, GEMM_PLAIN, false, FOLD>(ctx, pl, p, pdl);
    if (mode == GEMM_PART) return launch_one<KB, NT, GEMM_PART, false, FOLD>(ctx, pl, p, pdl);
    if constexpr (NT * 8 <= kMaxFusedTok && FOLD) {
        if (mode == GEMM_QKV) return launch_one<KB, NT, GEMM_QKV, false, FOLD>(ctx, pl, p, pdl);
        if (mode == GEMM_GU) return launch_one<KB, NT, GEMM_GU, false, FOLD>(ctx, pl, p, pdl);
    }
    return set_error(ctx, MI_ERR_LIMIT, "gemm: mode %d for %d token groups", mode, NT);
}
template <int KB, int NT>
int launch_fold(mi_ctx* ctx, const GemmPlan& pl, int mode, bool rowmajor, const GemmParams& p, bool pdl) {
    return pl.fold ? launch_mode<KB, NT, true>(ctx, pl, mode, rowmajor, p, pdl) : launch_mode<KB, NT, false>(ctx, pl, mode, rowmajor, p, pdl);
}
template <int KB>
int launch_nt(mi_ctx* ctx, const GemmPlan& pl, int mode, bool rowmajor, const GemmParams& p, bool pdl) {
    switch (pl.NT) {
        case 1: return launch_fold<KB, 1>(ctx, pl, mode, rowmajor, p, pdl);
        case 2: return launch_fold<KB, 2>(ctx, pl, mode, rowmajor, p, pdl);
        case 3: return launch_fold<KB, 3>(ctx, pl, mode, rowmajor, p, pdl);
        default: return launch_fold<KB, 4>(ctx, pl, mode, rowmajor, p, pdl);
    }
}
}  // namespace

int launch_gemm_tok(mi_ctx* ctx, const mi_weight* w, const GemmPlan& pl, int mode, bool rowmajor, GemmParams p, bool pdl) {
    p.base = w->dev; p.groups = w->groups; p.nt = (w->nb + kStepBlk - 1) / kStepBlk; p.nb = w->nb; p.rows = (int)w->rows;
    p.ksg = pl.ksg; p.kct = pl.kct; p.C = pl.C; p.kw = pl.kw; p.err = ctx->d_err;
    switch (w->kb) {
        case 8: return launch_nt<8>(ctx, pl, mode, rowmajor, p, pdl);
        case 4: return launch_nt<4>(ctx, pl, mode, rowmajor, p, pdl);
        case 2: return launch_nt<2>(ctx, pl, mode, rowmajor, p, pdl);
        case 1: return launch_nt<1>(ctx, pl, mode, rowmajor, p, pdl);
        default: return set_error(ctx, MI_ERR_INVALID, "gemm: bad tile depth %d", w->kb);
    }
}

}  // namespace mi

using namespace mi;

extern "C" int mi_gemm_q4_q8(mi_ctx* ctx, const mi_weight* w, const int8_t* xq_dev, const uint16_t* xd_dev, int M,
                             const float* bias_dev, float* y_dev) {
    if (!ctx) return MI_ERR_INVALID;
    if (!w || !xq_dev || !xd_dev || !y_dev) return set_error(ctx, MI_ERR_INVALID, "gemm: null argument");
    if (M < 1 || M > 16) return set_error(ctx, MI_ERR_LIMIT, "gemm: M=%d tokens per pass; this entry point takes 1..16", M);
    if (((uintptr_t)xq_dev & 15) != 0) return set_error(ctx, MI_ERR_INVALID, "gemm: xq_dev must be 16-byte aligned");
    if (w->count != 1) return set_error(ctx, MI_ERR_UNSUPPORTED, "gemm: matrix stacks are not supported");
    if (w->rows == 0) return MI_OK;
    GemmPlan pl;
    int st = plan_gemm_tok(ctx, w, GEMM_PLAIN, M, tok_tiling(M), &pl);
    if (st != MI_OK) return st;
    GemmParams p{};
    p.M = M; p.xq = xq_dev; p.xd = reinterpret_cast<const __half*>(xd_dev); p.bias = bias_dev; p.y = y_dev;
    const int steps = (w->nb + kStepBlk - 1) / kStepBlk;
    if (pl.kct >= steps) return launch_gemm_tok(ctx, w, pl, GEMM_PLAIN, true, p, true);
    // The activations of all of K do not fit a CTA's staging: K ranges over the grid and a small kernel that adds them, instead of
    // staging chunk after chunk in every CTA (1536 x 8960, 16 tokens: 27.7 us that way).
    if ((st = plan_gemm_tok(ctx, w, GEMM_PART, M, tok_tiling(M), &pl)) != MI_OK) return st;
    if ((st = ensure_scratch(ctx, (size_t)pl.ksg * M * w->rows, 0)) != MI_OK) return st;
    p.part = ctx->part; p.ldp = (int)w->rows;
    if ((st = launch_gemm_tok(ctx, w, pl, GEMM_PART, true, p, true)) != MI_OK) return st;
    MI_CUDA(ctx, launch_k(true, sum_ranges_kernel, dim3((unsigned)((w->rows + 255) / 256), M), dim3(256), 0, ctx->stream, (const double*)ctx->part, pl.ksg, (int)w->rows, bias_dev, y_dev));
    return MI_OK;
}

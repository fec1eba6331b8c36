// The M-token q4_0 x q8_0 product: what the GEMM kernel (gemm_tok.cu) and the kernels around it share.
#pragma once
#include "gemv_core.cuh"

namespace mi {

// ---- activations in operand order ------------------------------------------------------------------------------------
// The B operand of mma.m16n8k32 holds, for a block of 32 elements and eight tokens, in lane 4*n + t the bytes 4t .. 4t+3
// and 16+4t .. 16+4t+3 of token n.  The kernels that quantize activations inside the M-token pass store them in exactly
// that order, so that staging is one bulk copy and an operand one 8-byte load per lane:
//     q : [block of 32][group of eight tokens, J of them][lane] 8 bytes
//     d : [block][8 J tokens] double  d * 2^1004
// Why 2^1004: the product takes the weight scale's fp16 bits into the exponent field of a double as they are, which is
// the scale times 2^-1008 (fp16 subnormals and zero included), and multiplies nibbles that are 16 times too large; the
// powers of two meet in the product and cancel: 2^1004 * 2^-1008 * 2^4 = 1.
struct TokX {
    unsigned* q; double* d; int J;
};
constexpr int kMaxTokNT = 4;                           // groups of eight tokens that one CTA of the product handles

// 32-bit word of `q` that holds elements e .. e+3 (e a multiple of four) of block b, token n
__host__ __device__ inline size_t tok_word(int J, int b, int n, int e) {
    return (((size_t)b * J + (n >> 3)) * 32 + (n & 7) * 4 + ((e & 15) >> 2)) * 2 + (e >> 4);
}
__host__ __device__ inline size_t tok_scale(int J, int b, int n) { return (size_t)b * (8 * J) + n; }

#ifdef __CUDACC__
__device__ __forceinline__ double tok_scale_value(__half d) { return __dmul_rn((double)__half2float(d), 0x1p1004); }
// quantize one block held one element per lane to q8_0 (src/cuda_infer.cu:80-89) and store it as block b of token n
__device__ __forceinline__ void store_tok_block(const TokX& x, int b, int n, int lane, float a) {
    const float am = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(a))));
    const float inv = am > 0.f ? __fdiv_rn(127.f, am) : 0.f;
    unsigned v = (unsigned)__float2int_rn(__fmul_rn(a, inv)) & 0xffu;
    v |= __shfl_down_sync(0xffffffffu, v, 1) << 8;
    v |= __shfl_down_sync(0xffffffffu, v, 2) << 16;
    if ((lane & 3) == 0) x.q[tok_word(x.J, b, n, lane)] = v;
    if (lane == 0) x.d[tok_scale(x.J, b, n)] = tok_scale_value(__float2half_rn(__fdiv_rn(am, 127.f)));
}
#endif

// ---- the product -------------------------------------------------------------------------------------------------------
enum GemmMode {
    GEMM_PLAIN = 0,    // y[m][row] = fp32(sum) + bias
    GEMM_PART = 1,     // double sums of every K range, part[range][m][row]: the kernel that consumes them adds the ranges
    GEMM_QKV = 2,      // + bias, rotary embedding; q in natural order, k and v as fp16 into the cache          (up to kMaxFusedTok tokens)
    GEMM_GU = 3        // rows come as (gate, up) groups of 32: SwiGLU, q8_0, operand order                         (up to kMaxFusedTok tokens)
};
// Up to this many tokens the rotary embedding and SwiGLU run in the product's epilogue, which saves a launch.  Each of their
// items (a warp's 32 elements of a token) is a dependent chain of 500 - 900 clocks (a double-precision exponential and
// division; the position's angles from memory), of which the product's eight warps overlap two per sub-partition: 640
// clocks per item measured.  With more tokens that is longer than a kernel of their own at full occupancy (gate/up of the 1.5B shape,
// 64 tokens: 37 us fused, 27 + 4 apart).
constexpr int kMaxFusedTok = 16;

// Rotary embedding, and where q, k and v of a token go: token n sits at position pos_arr[n] (or *pos0 + n) of cache slab slot_arr[n]
struct RopeParams {
    float* q; int nq, HD; __half* kc; __half* vc; int KVD; long long slab_stride; int layer, max_seq;
    const float* cs; const float* freq; int rows;       // angles of positions below `rows`: cos then sin [HD/2] each; frequencies for the others
    const int* pos0; const int* pos_arr; const int* slot_arr;
};
#ifdef __CUDACC__
// v: row `row` of the packed QKV vector of token n with the bias added, one row per lane (all lanes of a warp call, rows 32-aligned)
__device__ __forceinline__ void rope_store(const RopeParams& p, int row, int n, float v) {
    const float partner = __shfl_xor_sync(0xffffffffu, v, 1);
    if (row >= p.nq + 2 * p.KVD) return;
    const int pos = p.pos_arr ? __ldg(p.pos_arr + n) : __ldg(p.pos0) + n;
    const size_t slab = p.slot_arr ? (size_t)__ldg(p.slot_arr + n) * (size_t)p.slab_stride : 0;
    const size_t crow = slab + ((size_t)p.layer * p.max_seq + pos) * p.KVD;
    if (row >= p.nq + p.KVD) { p.vc[crow + (row - p.nq - p.KVD)] = __float2half_rn(v); return; }
    // q and k rows come pair-adjacent: slots 2i and 2i + 1 of a head are its dims i and i + HD / 2
    const int within0 = row < p.nq ? row : row - p.nq, head = within0 / p.HD, within = within0 - head * p.HD, i = within >> 1;
    double c, s;
    if (pos < p.rows) {
        c = (double)__ldg(p.cs + (size_t)pos * p.HD + i); s = (double)__ldg(p.cs + (size_t)pos * p.HD + p.HD / 2 + i);
    } else {
        const double th = (double)__fmul_rn((float)pos, __ldg(p.freq + i));                // fp32 angle, as src/cpu_infer.cpp:54
        c = (double)__double2float_rn(cos(th)); s = (double)__double2float_rn(sin(th));
    }
    const bool odd = within & 1;
    const float out = odd ? __double2float_rn(__dadd_rn(__dmul_rn((double)partner, s), __dmul_rn((double)v, c)))
                          : __double2float_rn(__dsub_rn(__dmul_rn((double)v, c), __dmul_rn((double)partner, s)));
    const int nat = head * p.HD + i + (odd ? p.HD / 2 : 0);
    if (row < p.nq) p.q[(size_t)n * p.nq + nat] = out;
    else p.kc[crow + nat] = __float2half_rn(out);
}
__device__ __forceinline__ float swiglu(float gate, float up) {
    const double gd = (double)gate;
    return __double2float_rn(__dmul_rn(__ddiv_rn(gd, __dadd_rn(1.0, exp(-gd))), (double)up));
}
// SwiGLU and q8_0 of one block by eight lanes of a warp, four consecutive elements each (all lanes of the warp call): the lane's four int8 values, the block's fp16 scale and the
// sum of its values.  Of what a block takes besides its 32 exponentials and divisions (reductions, one division for 127 / max and max / 127) a warp does four at once.
struct SwiBlock { unsigned q; __half d; int sum; };
__device__ __forceinline__ SwiBlock swiglu_block(float4 g, float4 u) {
    const float a[4] = {swiglu(g.x, u.x), swiglu(g.y, u.y), swiglu(g.z, u.z), swiglu(g.w, u.w)};
    unsigned am = 0;                                       // over the bits: a NaN counts as the largest
    #pragma unroll
    for (int i = 0; i < 4; i++) am = max(am, __float_as_uint(fabsf(a[i])));
    #pragma unroll
    for (int o = 1; o < 8; o <<= 1) am = max(am, __shfl_xor_sync(0xffffffffu, am, o));
    const float m = __uint_as_float(am);
    const bool odd = threadIdx.x & 1;
    const float r = __fdiv_rn(odd ? m : 127.f, odd ? 127.f : m), other = __shfl_xor_sync(0xffffffffu, r, 1), inv = m > 0.f ? (odd ? other : r) : 0.f;
    SwiBlock b;
    b.d = __float2half_rn(odd ? r : other);
    b.q = 0;
    #pragma unroll
    for (int i = 0; i < 4; i++) b.q |= ((unsigned)__float2int_rn(__fmul_rn(a[i], inv)) & 0xffu) << (8 * i);
    b.sum = __dp4a((int)b.q, 0x01010101, 0);
    #pragma unroll
    for (int o = 1; o < 8; o <<= 1) b.sum += __shfl_xor_sync(0xffffffffu, b.sum, o);
    return b;
}
#endif

struct GemmParams {
    const uint8_t* base; int groups, nt, nb, rows;      // tiled weights; nt: steps of eight blocks
    int ksg, kct, C, kw;                                // K ranges of the grid; steps per staged chunk; CTAs per (range, token tile); warps that share a unit's steps
    int M;                                              // tokens
    TokX x;                                             // activations in operand order, or
    const int8_t* xq; const __half* xd;                 // row-major: [M][nb*32], [M][nb]
    const float* bias; float* y;
    double* part; int ldp;                              // part[(range * M + m) * ldp + row]
    RopeParams rope;                                    // GEMM_QKV
    TokX act;                                           // GEMM_GU
    int* err;
};

// Token tiles of a pass over M tokens: TT tiles of NT groups of eight; operand buffers hold J = NT * TT groups per block.
struct TokTiling { int NT, TT; int J() const { return NT * TT; } };
inline TokTiling tok_tiling(int M, int max_nt = kMaxTokNT) {
    const int J = (M + 7) / 8, TT = (J + max_nt - 1) / max_nt;
    return TokTiling{(J + TT - 1) / TT, TT};
}
// How a launch over one matrix and M tokens is cut (see plan_gemm_tok).
struct GemmPlan { int NT, TT, ksg, kct, C, kw; bool fold; size_t smem; double cost; };
int plan_gemm_tok(mi_ctx* ctx, const mi_weight* w, int mode, int M, const TokTiling& tiles, GemmPlan* out);
// The products of a pass of M tokens over L layers, QKV, O, gate/up, down (mats: those of one layer) and the lm_head over the last n_head of them (0: none)
int plan_pass_products(mi_ctx* ctx, const mi_weight* const mats[5], int L, int M, int n_head, TokTiling* tiles, GemmPlan plans[5]);
int launch_gemm_tok(mi_ctx* ctx, const mi_weight* w, const GemmPlan& plan, int mode, bool rowmajor, GemmParams p, bool pdl);

}  // namespace mi

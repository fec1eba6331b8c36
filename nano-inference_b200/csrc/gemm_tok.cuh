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
    GEMM_QKV = 2,      // + bias, rotary embedding; q in natural order, k and v as fp16 into the cache
    GEMM_GU = 3        // rows come as (gate, up) groups of 32: SwiGLU, q8_0, operand order
};

struct GemmParams {
    const uint8_t* base; int groups, nt, nb, rows;      // tiled weights
    int ksg, kct, C, kw;                                // K ranges of the grid; tiles per staged chunk; CTAs per (range, token tile); warps that share a unit's K tiles
    int M;                                              // tokens
    TokX x;                                             // activations in operand order, or
    const int8_t* xq; const __half* xd;                 // row-major: [M][nb*32], [M][nb]
    const float* bias; float* y;
    double* part; int ldp;                              // part[(range * M + m) * ldp + row]
    // GEMM_QKV
    float* q; int nq, HD; __half* kc; __half* vc; int KVD; long long slab_stride; int layer, max_seq;
    const float* rope_cs; const float* rope_freq; int rope_rows;
    const int* pos0; const int* pos_arr; const int* slot_arr;
    TokX act;                                           // GEMM_GU
    int* err;
};

// Token tiles of a pass over M tokens: TT tiles of NT groups of eight; operand buffers hold J = NT * TT groups per block.
struct TokTiling { int NT, TT; int J() const { return NT * TT; } };
inline TokTiling tok_tiling(int M) {
    const int J = (M + 7) / 8, TT = (J + kMaxTokNT - 1) / kMaxTokNT;
    return TokTiling{(J + TT - 1) / TT, TT};
}
// How a launch over one matrix and M tokens is cut (see plan_gemm_tok).
struct GemmPlan { int NT, TT, ksg, kct, C, kw; size_t smem; };
int plan_gemm_tok(mi_ctx* ctx, const mi_weight* w, int mode, int M, GemmPlan* out);
int launch_gemm_tok(mi_ctx* ctx, const mi_weight* w, const GemmPlan& plan, int mode, bool rowmajor, GemmParams p, bool pdl);

}  // namespace mi

// The q4_0 x q8_0 product on whole-K integer sums (gemm_dig.cu): what its kernels and the passes around them share.
#pragma once
#include "gemm_tok.cuh"

namespace mi {

// Activations as digits.  A token's element is xq * dx with dx an fp16 scale: an integer X = xq * (dx / 2^ex) times 2^ex, with ex the
// smallest exponent among the blocks of one K range, cut into four balanced base-256 digits (planes).
//     q    : [token tile of T][block of 32][row = plane * T + token, planes 0 .. 2, padded to a multiple of 16 rows] 32 bytes: the MMA's operand with the
//            32-byte swizzle (the halves of rows 4 .. 7 of eight change places); behind all of it plane 3 as [token tile][block][token].  A token's block is a
//            whole sector: without the swizzle it is two halves of sectors, which it took SwiGLU 31 us to write for 333 tokens of the 1.5B shape.
//     info : [K range][token] ex | planes in use << 8 (3 or 4; kDigNone: the digits cannot hold it, see sum_over_blocks)
//     bias : [K range][token] sum of X
struct DigX { uint8_t* q; int* info; long long* bias; int T, TT; };
constexpr int kDigPlanes = 4, kDigNone = 255, kDigMaxT = 64;                          // tokens of a tile
__host__ __device__ inline int dig_rows(int T) { return (3 * T + 15) / 16 * 16; }
// where 16 elements (half 0 or 1 of a block) of a token of a tile are
__host__ __device__ inline size_t dig_offset(const DigX& x, int nb, int tt, int b, int half, int plane, int t) {
    const size_t at = (size_t)tt * nb + b, row = plane < 3 ? at * dig_rows(x.T) + plane * x.T + t : (size_t)x.TT * nb * dig_rows(x.T) + at * x.T + t;
    return row * 32 + (half ^ (t >> 2 & 1)) * 16;
}
inline size_t dig_bytes(int nb, int tokens) { return (size_t)nb * 2 * 16 * (4 * (tokens + kDigMaxT) + 8 * (tokens / kDigMaxT + 1)); }   // room for any tiling of so many tokens
#ifdef __CUDACC__
// fp16 bits of a scale as mantissa * 2^(exponent - 25)
__device__ __forceinline__ int scale_exponent(unsigned h) { return max((int)(h >> 10 & 31u), 1); }
__device__ __forceinline__ int scale_mantissa(unsigned h) { return (int)(h & 1023u) + ((h & 0x7C00u) ? 1024 : 0); }
// the four balanced digits of four int8 values times m, a word of four bytes per plane
__device__ __forceinline__ void dig_word(unsigned q, int m, unsigned (&d)[4]) {
    unsigned v[4];
    #pragma unroll
    for (int j = 0; j < 4; j++) v[j] = (unsigned)((int)(int8_t)(q >> (8 * j)) * m) + 0x80808080u;
    const unsigned a = __byte_perm(v[0], v[1], 0x5140), c = __byte_perm(v[2], v[3], 0x5140), e = __byte_perm(v[0], v[1], 0x7362), f = __byte_perm(v[2], v[3], 0x7362);
    d[0] = __byte_perm(a, c, 0x5410) ^ 0x80808080u; d[1] = __byte_perm(a, c, 0x7632) ^ 0x80808080u;
    d[2] = __byte_perm(e, f, 0x5410) ^ 0x80808080u; d[3] = __byte_perm(e, f, 0x7632) ^ 0x80808080u;
}
// What a token's digits over a K range need to know of its scales: smallest and largest exponent, the sum of the elements in units of 2^-24 times the smallest scale's
struct DigReduce { int lo[32], hi[32]; long long sum[32]; };
struct DigRange {
    int lo = 31, hi = 0; long long sum = 0;
    // part of a block with scale bits h, whose int8 values add up to s
    __device__ __forceinline__ void add(unsigned h, int s) {
        if (!(h & 0x7FFFu)) return;
        const int e = scale_exponent(h);
        lo = min(lo, e); hi = max(hi, e);
        sum += (long long)(s * scale_mantissa(h)) << (e - 1);
    }
    __device__ __forceinline__ DigRange over_cta(DigReduce& red) const {                 // all threads of the CTA call
        DigRange r;
        r.lo = __reduce_min_sync(0xffffffffu, lo); r.hi = __reduce_max_sync(0xffffffffu, hi);
        long long s = sum;
        #pragma unroll
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
        if (lane == 0) { red.lo[warp] = r.lo; red.hi[warp] = r.hi; red.sum[warp] = s; }
        __syncthreads();
        r.lo = __reduce_min_sync(0xffffffffu, lane < nw ? red.lo[lane] : 31); r.hi = __reduce_max_sync(0xffffffffu, lane < nw ? red.hi[lane] : 0);
        s = lane < nw ? red.sum[lane] : 0;
        #pragma unroll
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        r.sum = s;
        return r;
    }
    __device__ __forceinline__ int planes() const { return hi == 31 || hi - lo > 13 ? kDigNone : hi - lo > 5 ? 4 : 3; }
    __device__ __forceinline__ int unit() const { return min(lo, max(hi, 1)); }
    __device__ __forceinline__ long long total() const { return planes() == kDigNone ? 0 : sum >> (unit() - 1); }
    __device__ __forceinline__ int factor(unsigned h) const { return planes() == kDigNone ? 0 : scale_mantissa(h) << ((scale_exponent(h) - unit()) & 31); }
};
#endif

// How a product of M tokens is cut: token tiles, K ranges.
struct DigPlan { int T, TT, ksg; double cost; };
bool plan_gemm_dig(mi_ctx* ctx, const mi_weight* w, bool part, int M, DigPlan* out);
// Whether product i of a pass (0 QKV, 1 O, 2 gate/up, 3 down, 4 lm_head) over M tokens goes over digits, and how: `blocks` is the plan it has otherwise.
bool choose_gemm_dig(mi_ctx* ctx, const mi_weight* w, int i, int M, const GemmPlan& blocks, DigPlan* out);
// y = fp32(sum) + bias (GEMM_PLAIN), or double sums per K range (GEMM_PART); x: the digits, p.x: the same activations as q8_0
int launch_gemm_dig(mi_ctx* ctx, const mi_weight* w, const DigPlan& pl, int mode, const DigX& x, GemmParams p, bool pdl);
int launch_tok_digits(mi_ctx* ctx, const mi_weight* w, const DigPlan& pl, const TokX& x, const DigX& out, int M, bool pdl);
// The same behind SwiGLU: rows of y come as (gate, up) groups of 32, w is the matrix that takes its result; act: the result as q8_0
int launch_swiglu_digits(mi_ctx* ctx, const mi_weight* w, const DigPlan& pl, const float* y, const TokX& act, const DigX& out, int M, bool pdl);
// Exponents of a matrix's rows, for the product's weight digits: row_exp[groups * 32]; found (zeros before): how many have none, the most binades between the scales of another.
int launch_row_exponents(mi_ctx* ctx, const mi_weight* w, uint8_t* row_exp, int* found);
// The rows that have none, in any order; *count: zero before
int launch_list_rows(mi_ctx* ctx, const mi_weight* w, int* list, int* count);

}  // namespace mi

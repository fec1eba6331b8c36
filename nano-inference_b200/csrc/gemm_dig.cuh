// The q4_0 x q8_0 product on whole-K integer sums (gemm_dig.cu): what its kernels and the passes around them share.
#pragma once
#include "gemm_tok.cuh"

namespace mi {

// Activations as digits.  A token's element is xq * dx with dx an fp16 scale: an integer X = xq * (dx / 2^ex) times 2^ex, with ex the
// smallest exponent among the blocks of one K range, cut into four balanced base-256 digits (planes).
//     q    : [token tile of T][block of 32][half of 16 elements][row = plane * T + token, planes 0 .. 2, padded to a multiple of 16 rows] 16 bytes: the MMA's operand;
//            behind all of it plane 3 as [token tile][block][half][token]
//     info : [K range][token] ex | planes in use << 8 (3 or 4; kDigNone: the digits cannot hold it, see row_sum_dig)
//     bias : [K range][token] sum of X
struct DigX { uint8_t* q; int* info; long long* bias; int T, TT; };
constexpr int kDigPlanes = 4, kDigNone = 255, kDigMaxT = 64;                          // tokens of a tile
__host__ __device__ inline int dig_rows(int T) { return (3 * T + 15) / 16 * 16; }
__host__ __device__ inline size_t dig_offset(const DigX& x, int nb, int tt, int b, int half, int plane, int t) {
    const size_t at = ((size_t)tt * nb + b) * 2 + half;
    return plane < 3 ? (at * dig_rows(x.T) + plane * x.T + t) * 16 : ((size_t)x.TT * nb * 2 * dig_rows(x.T) + at * x.T + t) * 16;
}
inline size_t dig_bytes(int nb, int tokens) { return (size_t)nb * 2 * 16 * (4 * (tokens + kDigMaxT) + 8 * (tokens / kDigMaxT + 1)); }   // room for any tiling of so many tokens
// How a product of M tokens is cut: token tiles, K ranges.
struct DigPlan { int T, TT, ksg; double cost; };
bool plan_gemm_dig(mi_ctx* ctx, const mi_weight* w, bool part, int M, DigPlan* out);
// y = fp32(sum) + bias (GEMM_PLAIN), or double sums per K range (GEMM_PART); x: the digits, p.x: the same activations as q8_0
int launch_gemm_dig(mi_ctx* ctx, const mi_weight* w, const DigPlan& pl, int mode, const DigX& x, GemmParams p, bool pdl);
int launch_tok_digits(mi_ctx* ctx, const mi_weight* w, const DigPlan& pl, const TokX& x, const DigX& out, int M, bool pdl);
// Exponents of a matrix's rows, for the product's weight digits: row_exp[groups * 32]; *wide: mi_weight::wide.
int launch_row_exponents(mi_ctx* ctx, const mi_weight* w, uint8_t* row_exp, int* wide);

}  // namespace mi

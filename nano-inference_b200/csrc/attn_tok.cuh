// Attention of the M-token pass and of the stand-alone entry point (attn_tok.cu).
#pragma once
#include "gemm_tok.cuh"

namespace mi {

struct AttnParams {
    const float* q;                         // [M][NH * HD] fp32, natural dimension order
    const __half* kc; const __half* vc;     // [layer][max_seq][KVD] (+ slab)
    int M, NH, NKV, HD, KVD, layer, max_seq;
    const int* pos0; int pos0_val;          // query i sits at (pos0 ? *pos0 : pos0_val) + i, or
    const int* pos_arr; const int* slot_arr; long long slab_stride;     // at pos_arr[i] of cache slab slot_arr[i]
    float* out;                             // [M][NH * HD] fp32
    TokX x;                                 // optional: the same as q8_0 in operand order
    double* part;                           // [M][NH][nch][HD + 2] when nch > 1: chunk sums, maximum, denominator
    int nch;                                // chunks per causal range
    int qb;                                 // queries per CTA
    int early;                              // the cache rows below the first query's position may be read before the kernels ahead have finished
};
// the cut for M queries whose longest causal range has about lp_max positions (ragged: every query has a sequence of its own)
struct AttnPlan { int qb, nch; size_t part_doubles; };
AttnPlan plan_attn_tok(const mi_ctx* ctx, int NH, int NKV, int HD, int M, int lp_max, bool ragged);
size_t attn_part_max(const mi_ctx* ctx, int NH, int NKV, int HD);       // doubles that any plan for these heads needs
int launch_attn_tok(mi_ctx* ctx, AttnParams p, const AttnPlan& plan, bool pdl);

}  // namespace mi

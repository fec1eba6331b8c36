// Split-KV causal attention with grouped queries for M queries over the fp16 cache: the M-token pass (prompt chunks, drafted
// tokens, batches) and mi_attn_splitkv.
//
// Replaces attn_partial + attn_combine (reference src/cuda_infer.cu:650-702) and mega's attention + combine
// (src/mega.cu:414-521, 705-741).  Scores are double dot products rounded to fp32 once and scaled by 1/sqrt(HD) in fp32; weights,
// denominator and weighted sum are double, as everywhere in this library.
//
// What bounds it: the FP64 pipe (64 FMAs per clock and SM), 2 HD FMAs per (query, head, position); the cache itself is a few
// microseconds of HBM time.  So both products run as FP64 MMAs (mma.m8n8k4.f64: the pipe's full rate from one issue slot per
// 256 FMAs, where the scalar code this replaces spent more slots on fp16 -> double conversions and broadcast loads than on FMAs),
// and the rows of an MMA are (query, head) pairs that share a kv head: a K or V element is converted once for up to
// 4 queries x all heads of the group.
//
// A CTA has qb queries of one kv head and one chunk of their positions, and walks it in steps of 64 (one query: 128) positions:
//   scores   warp = every 8th group of 8 positions, all dims; q waits in shared memory as doubles in the order the MMA reads it;
//   weights  one warp per row: running maximum, exp, sum; stored in MMA order;
//   values   warp = HD/8 dims, all positions.
// K and V rows come through shared memory by asynchronous copies, the K rows of the next step while this step's weights and
// values are worked on, its V rows during the next scores (fetched by the lanes that use them, they left each warp waiting
// 7 of 12 cycles per instruction).  Two CTAs share an SM, so that one's exponentials run beside the other's MMAs.  With
// several chunks per range the CTAs leave {sum, maximum, denominator} per row and attn_tok_merge folds them against their
// common maximum; with one chunk the CTA finishes.  The number of chunks comes from the host and only sets how a range is
// cut, so a captured launch stays valid for any position.
#include "attn_tok.cuh"
#include <algorithm>
#include <atomic>
#include <mutex>

namespace mi {

constexpr int kAT = 256, kAW = kAT / 32;          // threads, warps
constexpr int kMaxQB = 4;                         // queries per CTA
__host__ __device__ constexpr int attn_row_tiles(int G, int QB) { return (G * QB + 7) / 8; }

template <int HD, int RT> struct AttnSmem {
    static constexpr int R = RT * 8, SUB = RT == 1 ? 128 : 64;       // rows; positions per step
    static constexpr int SCL = SUB + 4;                              // floats per row of scores
    // bytes per K and V row: a lane's 16 bytes of K (eight lanes: two rows x 64 bytes) and its 4 bytes of V (four rows x 32
    // bytes) meet no bank twice
    static constexpr int KLD = 2 * HD + 64, VLD = 2 * HD + 32;
    static constexpr int q = 0, wt = q + R * HD * 8, k = wt + R * SUB * 8, v = k + SUB * KLD, sc = v + SUB * VLD, st = sc + R * SCL * 4;
    static constexpr int bytes = st + R * 3 * 8;
};

__device__ __forceinline__ void cp16(void* dst, const void* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory"); }
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}
__device__ __forceinline__ double half_lo(unsigned w) { return (double)__half2float(__ushort_as_half((unsigned short)(w & 0xffffu))); }
__device__ __forceinline__ double half_hi(unsigned w) { return (double)__half2float(__ushort_as_half((unsigned short)(w >> 16))); }

// Four consecutive dims e .. e+3 of one (token, head): fp32 out, and q8_0 over the eight threads that share a 32-dim block
__device__ __forceinline__ void attn_emit(const AttnParams& p, int token, int e, float4 v) {
    *reinterpret_cast<float4*>(p.out + (size_t)token * p.NH * p.HD + e) = v;
    if (!p.x.q) return;                            // uniform
    // the maximum over the bits, as in the single-token kernel: a NaN counts as the largest
    unsigned am = max(max(__float_as_uint(fabsf(v.x)), __float_as_uint(fabsf(v.y))), max(__float_as_uint(fabsf(v.z)), __float_as_uint(fabsf(v.w))));
    const unsigned mask = 0xffu << (threadIdx.x & 24);               // a block's eight threads, all here or none
    am = max(am, __shfl_xor_sync(mask, am, 1));
    am = max(am, __shfl_xor_sync(mask, am, 2));
    am = max(am, __shfl_xor_sync(mask, am, 4));
    const float a = __uint_as_float(am);
    const float inv = a > 0.f ? __fdiv_rn(127.f, a) : 0.f;
    const unsigned q = ((unsigned)__float2int_rn(__fmul_rn(v.x, inv)) & 0xffu) | (((unsigned)__float2int_rn(__fmul_rn(v.y, inv)) & 0xffu) << 8) |
                       (((unsigned)__float2int_rn(__fmul_rn(v.z, inv)) & 0xffu) << 16) | ((unsigned)__float2int_rn(__fmul_rn(v.w, inv)) << 24);
    p.x.q[tok_word(p.x.J, e >> 5, token, e & 31)] = q;
    if ((e & 31) == 0) p.x.d[tok_scale(p.x.J, e >> 5, token)] = tok_scale_value(__float2half_rn(__fdiv_rn(a, 127.f)));
}

template <int HD, int G, int QB>
__global__ void __launch_bounds__(kAT, 2) attn_tok_kernel(const __grid_constant__ AttnParams p) {
    constexpr int RT = attn_row_tiles(G, QB), ROWS = G * QB;
    using SM = AttnSmem<HD, RT>;
    constexpr int R = SM::R, SUB = SM::SUB, SCL = SM::SCL;
    constexpr int NTW = HD >= 64 ? HD / 64 : 1;     // 8-dim tiles per warp in the value product
    constexpr int VW = HD / 8 / NTW;                // warps that have some
    constexpr int CH = RT == 1 ? 2 : 1;             // accumulator chains per row tile in the value product
    extern __shared__ __align__(128) uint8_t smem[];
    double* qs = reinterpret_cast<double*>(smem + SM::q);             // [dim of a lane][row tile][lane]
    double* wt = reinterpret_cast<double*>(smem + SM::wt);            // [SUB / 4][row tile][lane]
    uint8_t* ks = smem + SM::k; uint8_t* vs = smem + SM::v;          // [SUB] rows
    float* sc = reinterpret_cast<float*>(smem + SM::sc);             // [R][SCL]
    double* rm = reinterpret_cast<double*>(smem + SM::st);           // [R] running maximum
    double* rl = rm + R;                                             // [R] denominator
    double* rf = rl + R;                                             // [R] rescale factor of this step
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int nqb = (p.M + QB - 1) / QB;
    // later queries have longer ranges: they go first
    const int ch = (int)(blockIdx.x % p.nch), rest = (int)(blockIdx.x / p.nch), kvh = rest % p.NKV, q0 = (nqb - 1 - rest / p.NKV) * QB;
    const int nq = min(QB, p.M - q0);
    pdl_launch_dependents();
    if (!p.early) pdl_wait_prior();
    const int posq0 = p.pos_arr ? __ldg(p.pos_arr + q0) : (p.pos0 ? __ldg(p.pos0) : p.pos0_val) + q0;      // position of query q0; the CTA's others follow (QB > 1: one sequence)
    const size_t base = (p.slot_arr ? (size_t)__ldg(p.slot_arr + q0) * (size_t)p.slab_stride : 0) + (size_t)p.layer * p.max_seq * p.KVD + (size_t)kvh * HD;
    const int Lp = posq0 + nq;                      // positions the last query sees
    const int p0 = (int)((long long)Lp * ch / p.nch), p1 = (int)((long long)Lp * (ch + 1) / p.nch);
    auto copy_range = [&](uint8_t* dst, int ld, const __half* src, int b0, int lo, int hi) {  // rows lo .. hi of the step at b0, 16 bytes per thread and copy
        for (int i = tid; i < (hi - lo) * (HD / 8); i += kAT) {
            const int r = i / (HD / 8) + lo - b0, c = i % (HD / 8);
            cp16(dst + r * ld + c * 16, src + base + (size_t)(b0 + r) * p.KVD + c * 8);
        }
    };
    auto copy_rows = [&](uint8_t* dst, int ld, const __half* src, int b0) { copy_range(dst, ld, src, b0, b0, min(b0 + SUB, p1)); cp_commit(); };
    // In a pass the rows of earlier positions have been there since before it began: they are requested before the kernel waits
    // for the projection, and the rows that it writes after that.
    const int step1 = min(p0 + SUB, p1), fresh = p.early ? min(max(p.pos_arr ? posq0 : posq0 - q0, p0), step1) : p0;
    if (p.early) {
        if (p0 < fresh) { copy_range(ks, SM::KLD, p.kc, p0, p0, fresh); copy_range(vs, SM::VLD, p.vc, p0, p0, fresh); }
        pdl_wait_prior();
    }
    if (p0 < p1) {
        copy_range(ks, SM::KLD, p.kc, p0, fresh, step1); cp_commit();
        copy_range(vs, SM::VLD, p.vc, p0, fresh, step1); cp_commit();
    }
    // q into the order the MMA reads it: lane (row, t) takes the 16-byte pieces t, t + 4, .. of a row: its dim s is 8 (4 (s / 8) + t) + s % 8
    for (int i = tid; i < R * HD; i += kAT) {
        const int d = i % HD, row = i / HD, qi = row / G, h = row - qi * G, tt = (d >> 3) & 3, s = (d >> 5) * 8 + (d & 7);
        const float v = row < ROWS && qi < nq ? __ldcg(p.q + (size_t)(q0 + qi) * p.NH * HD + (size_t)(kvh * G + h) * HD + d) : 0.f;
        qs[(s * RT + (row >> 3)) * 32 + (row & 7) * 4 + tt] = (double)v;
    }
    for (int i = tid; i < R; i += kAT) { rm[i] = -INFINITY; rl[i] = 0.0; }
    const float inv = __fdiv_rn(1.f, __fsqrt_rn((float)HD));
    double o[CH][RT][NTW][2];
    #pragma unroll
    for (int c = 0; c < CH; c++)
        #pragma unroll
        for (int r = 0; r < RT; r++)
            #pragma unroll
            for (int n = 0; n < NTW; n++) o[c][r][n][0] = o[c][r][n][1] = 0.0;

    for (int b0 = p0; b0 < p1; b0 += SUB) {
        const int np = min(SUB, p1 - b0);
        cp_wait<1>();                               // the K rows (the V rows were requested after them)
        __syncthreads();
        // ---- scores
        #pragma unroll 1
        for (int t = warp; t * 8 < np; t += kAW) {
            const uint8_t* kr = ks + min(t * 8 + g, np - 1) * SM::KLD + t4 * 16;
            double c[RT][2][2];                     // two chains per row tile
            #pragma unroll
            for (int r = 0; r < RT; r++) c[r][0][0] = c[r][0][1] = c[r][1][0] = c[r][1][1] = 0.0;
            #pragma unroll
            for (int i = 0; i < HD / 32; i++) {
                const uint4 kw = *reinterpret_cast<const uint4*>(kr + i * 64);
                const unsigned w[4] = {kw.x, kw.y, kw.z, kw.w};
                #pragma unroll
                for (int e = 0; e < 4; e++) {
                    const double k0 = half_lo(w[e]), k1 = half_hi(w[e]);
                    const double* a = qs + (size_t)((i * 8 + e * 2) * RT) * 32 + lane;
                    #pragma unroll
                    for (int r = 0; r < RT; r++) { dmma(c[r][0], a[r * 32], k0); dmma(c[r][1], a[(RT + r) * 32], k1); }
                }
            }
            #pragma unroll
            for (int r = 0; r < RT; r++)
                #pragma unroll
                for (int e = 0; e < 2; e++) {
                    const int row = 8 * r + g, pp = t * 8 + 2 * t4 + e, qi = row / G;
                    const float s = __fmul_rn(__double2float_rn(__dadd_rn(c[r][0][e], c[r][1][e])), inv);
                    sc[row * SCL + pp] = b0 + pp < p1 && b0 + pp <= posq0 + qi ? s : -INFINITY;
                }
        }
        __syncthreads();
        if (b0 + SUB < p1) copy_rows(ks, SM::KLD, p.kc, b0 + SUB); else cp_commit();
        // ---- weights: one warp per row
        #pragma unroll 1
        for (int row = warp; row < ROWS; row += kAW) {
            float s[SUB / 32], m = -INFINITY;
            #pragma unroll
            for (int i = 0; i < SUB / 32; i++) { s[i] = lane + 32 * i < np ? sc[row * SCL + lane + 32 * i] : -INFINITY; m = fmaxf(m, s[i]); }
            #pragma unroll
            for (int q = 16; q; q >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, q));
            const double mo = rm[row], mn = fmax(mo, (double)m);
            double l = 0.0;
            #pragma unroll
            for (int i = 0; i < SUB / 32; i++) {
                const double w = s[i] == -INFINITY ? 0.0 : exp((double)s[i] - mn);
                const int pp = lane + 32 * i;
                wt[((pp >> 2) * RT + (row >> 3)) * 32 + (row & 7) * 4 + (pp & 3)] = w;
                l = __dadd_rn(l, w);
            }
            #pragma unroll
            for (int q = 16; q; q >>= 1) l = __dadd_rn(l, __shfl_xor_sync(0xffffffffu, l, q));
            if (lane == 0) {
                const double f = mo == mn ? 1.0 : mo == -INFINITY ? 0.0 : exp(mo - mn);        // 1 while the maximum stands (and while there is none)
                rf[row] = f; rm[row] = mn; rl[row] = __fma_rn(rl[row], f, l);
            }
        }
        cp_wait<1>();                               // the V rows
        __syncthreads();
        // ---- values
        if (warp < VW) {
            if (b0 > p0) {
                #pragma unroll
                for (int r = 0; r < RT; r++) {
                    const double f = 8 * r + g < ROWS ? rf[8 * r + g] : 1.0;
                    #pragma unroll
                    for (int c = 0; c < CH; c++)
                        #pragma unroll
                        for (int n = 0; n < NTW; n++) { o[c][r][n][0] = __dmul_rn(o[c][r][n][0], f); o[c][r][n][1] = __dmul_rn(o[c][r][n][1], f); }
                }
            }
            const uint8_t* vr = vs + (warp * (8 * NTW) + g * NTW) * 2;
            #pragma unroll 4
            for (int s = 0; s * 4 < np; s++) {
                const uint8_t* v = vr + min(s * 4 + t4, np - 1) * SM::VLD;
                unsigned vw;
                if constexpr (NTW == 2) vw = *reinterpret_cast<const unsigned*>(v); else vw = *reinterpret_cast<const unsigned short*>(v);
                const double v0 = half_lo(vw), v1 = NTW == 2 ? half_hi(vw) : 0.0;
                const double* a = wt + (size_t)(s * RT) * 32 + lane;
                #pragma unroll
                for (int r = 0; r < RT; r++) {
                    const double w = a[r * 32];
                    if constexpr (CH == 2) {
                        if (s & 1) { dmma(o[1][r][0], w, v0); if constexpr (NTW == 2) dmma(o[1][r][NTW - 1], w, v1); }
                        else { dmma(o[0][r][0], w, v0); if constexpr (NTW == 2) dmma(o[0][r][NTW - 1], w, v1); }
                    } else {
                        dmma(o[0][r][0], w, v0);
                        if constexpr (NTW == 2) dmma(o[0][r][NTW - 1], w, v1);
                    }
                }
            }
        }
        __syncthreads();                            // scores, weights and V rows may be written again
        if (b0 + SUB < p1) copy_rows(vs, SM::VLD, p.vc, b0 + SUB);
    }
    if constexpr (CH == 2) {
        #pragma unroll
        for (int r = 0; r < RT; r++)
            #pragma unroll
            for (int n = 0; n < NTW; n++) { o[0][r][n][0] = __dadd_rn(o[0][r][n][0], o[1][r][n][0]); o[0][r][n][1] = __dadd_rn(o[0][r][n][1], o[1][r][n][1]); }
    }
    // ---- the chunk's rows
    if (p.nch > 1) {
        if (warp < VW) {
            #pragma unroll
            for (int r = 0; r < RT; r++) {
                const int row = 8 * r + g, qi = row / G, h = row - qi * G;
                if (row >= ROWS || qi >= nq) continue;
                double* gp = p.part + (((size_t)(q0 + qi) * p.NH + kvh * G + h) * p.nch + ch) * (HD + 2);
                #pragma unroll
                for (int n = 0; n < NTW; n++)
                    #pragma unroll
                    for (int e = 0; e < 2; e++) __stcg(gp + warp * (8 * NTW) + (2 * t4 + e) * NTW + n, o[0][r][n][e]);
            }
        }
        for (int row = tid; row < ROWS; row += kAT) {
            const int qi = row / G, h = row - qi * G;
            if (qi >= nq) continue;
            double* gp = p.part + (((size_t)(q0 + qi) * p.NH + kvh * G + h) * p.nch + ch) * (HD + 2) + HD;
            __stcg(gp, rm[row]); __stcg(gp + 1, rl[row]);
        }
        return;
    }
    float* of = reinterpret_cast<float*>(qs);       // [row][HD] fp32 (q is not needed any more)
    if (warp < VW) {
        #pragma unroll
        for (int r = 0; r < RT; r++) {
            if (8 * r + g >= ROWS) continue;
            const double l = rl[8 * r + g];
            #pragma unroll
            for (int n = 0; n < NTW; n++)
                #pragma unroll
                for (int e = 0; e < 2; e++) of[(8 * r + g) * HD + warp * (8 * NTW) + (2 * t4 + e) * NTW + n] = __double2float_rn(__ddiv_rn(o[0][r][n][e], l));
        }
    }
    __syncthreads();
    for (int i = tid; i < nq * G * (HD / 4); i += kAT) {              // a multiple of 8 items: the threads of a 32-dim block stay together
        const int row = i / (HD / 4), d = (i - row * (HD / 4)) * 4, qi = row / G, h = row - qi * G;
        attn_emit(p, q0 + qi, (kvh * G + h) * HD + d, *reinterpret_cast<const float4*>(of + row * HD + d));
    }
}

// Fold the chunks of one (query, head) against their common maximum.  What bounds it is latency (a launch, one trip to the L2, an
// exponential, a division), so nothing waits for anything it need not: the first eight chunks of a warp are requested before the
// maxima are known.  WPH warps share a head: all eight of a CTA where there are many chunks, one where there are few (and
// mostly many queries: a CTA per head would be idle but for a warp or two, 333 queries of 12 heads took 22 us).  Lane = the dims lane,
// lane + 32, ...  (A CTA per kv head that read maxima, factors and then all chunks in turn took 6.8 us for 5 queries and 29
// chunks, as long as the chunks themselves.)
template <int HD, int WPH>
__global__ void __launch_bounds__(kAT) attn_tok_merge(const __grid_constant__ AttnParams p) {
    constexpr int D = HD / 32, U = 8;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = warp % WPH, nch = p.nch;
    const int item = blockIdx.x * (kAW / WPH) + warp / WPH, token = item / p.NH, head = item - token * p.NH;
    pdl_launch_dependents();
    pdl_wait_prior();
    if (WPH == 1 && token >= p.M) return;
    const double* gp = p.part + (size_t)item * nch * (HD + 2);
    const int mine = (nch - sub + WPH - 1) / WPH;                    // chunks sub, sub + WPH, ..
    const double* own = gp + (size_t)sub * (HD + 2);
    constexpr size_t stride = (size_t)WPH * (HD + 2);
    auto fetch = [&](double (&v)[U][D], int i0) {
        #pragma unroll
        for (int u = 0; u < U; u++)
            #pragma unroll
            for (int d = 0; d < D; d++) v[u][d] = i0 + u < mine ? __ldcg(own + (size_t)(i0 + u) * stride + 32 * d + lane) : 0.0;
    };
    double v[U][D], o[D], l = 0.0, m = -INFINITY;
    #pragma unroll
    for (int d = 0; d < D; d++) o[d] = 0.0;
    fetch(v, 0);
    for (int c = lane; c < nch; c += 32) m = fmax(m, __ldcg(gp + (size_t)c * (HD + 2) + HD));
    #pragma unroll
    for (int q = 16; q; q >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, q));
    for (int b = 0; b < mine; b += 32) {                             // lane i prepares the factor of the i-th
        double f_l = 0.0;
        if (b + lane < mine) {
            const double* s = own + (size_t)(b + lane) * stride + HD;
            const double mc = __ldcg(s);
            f_l = mc == -INFINITY ? 0.0 : exp(mc - m);
            l = __fma_rn(__ldcg(s + 1), f_l, l);
        }
        for (int i0 = b; i0 < min(mine, b + 32); i0 += U) {
            if (i0 > 0) fetch(v, i0);
            #pragma unroll
            for (int u = 0; u < U; u++) {
                const double f = __shfl_sync(0xffffffffu, f_l, (i0 + u) & 31);
                if (i0 + u < mine) {
                    #pragma unroll
                    for (int d = 0; d < D; d++) o[d] = __fma_rn(v[u][d], f, o[d]);
                }
            }
        }
    }
    #pragma unroll
    for (int q = 16; q; q >>= 1) l = __dadd_rn(l, __shfl_xor_sync(0xffffffffu, l, q));
    auto emit = [&](int block, float y) {                            // 32 dims, one per lane
        const int e = head * HD + block * 32;
        p.out[(size_t)token * p.NH * HD + e + lane] = y;
        if (p.x.q) store_tok_block(p.x, e >> 5, token, lane, y);
    };
    if constexpr (WPH == 1) {
        float y[D];
        #pragma unroll
        for (int d = 0; d < D; d++) y[d] = __double2float_rn(__ddiv_rn(o[d], l));
        #pragma unroll
        for (int d = 0; d < D; d++) emit(d, y[d]);
    } else {
        static_assert(WPH == kAW, "a CTA per head");
        __shared__ double red[kAW][HD], den[kAW];
        #pragma unroll
        for (int d = 0; d < D; d++) red[warp][32 * d + lane] = o[d];
        if (lane == 0) den[warp] = l;
        __syncthreads();
        if (warp >= D) return;
        double s = red[0][warp * 32 + lane], dn = den[0];
        #pragma unroll
        for (int w = 1; w < kAW; w++) { s = __dadd_rn(s, red[w][warp * 32 + lane]); dn = __dadd_rn(dn, den[w]); }
        emit(warp, __double2float_rn(__ddiv_rn(s, dn)));
    }
}

// ---- host side -----------------------------------------------------------------------------------------------------

// Queries per CTA and chunks per range: the cheapest by a rough model in microseconds, from times of whole passes (three head shapes,
// 1 .. 16 queries behind 0 .. 32700 positions, prompts of 17 .. 512 tokens behind 0 .. 16000, batches of 2 .. 64; attention's share of a layer).
// A CTA costs its start and end and a time per position, which grows with the row tiles of its MMAs and with the CTAs that share its SM:
//     one row tile (one query), alone / two on an SM / each of more: 0.032 / 0.052 / 0.026 us per position at head_dim 128
//     (HD = 64, where three fit an SM: 0.022 / 0.045 / 0.016); three or four row tiles (four queries): 0.051 each (0.032), 0.59 of that alone.
// (Up to half as many CTAs as SMs are alone; more meet on the SMs that the projection before them leaves first.)  The merge is a launch of about 5.
// So four queries share a CTA where one per CTA would begin another wave, or where the FP64 pipe is what counts and the row tiles are fuller that way (6 heads:
// 24 of 24 rows instead of 6 of 8), and a range is cut from about 200 positions on.  Passes of the 1.5B shape, ms: 16 tokens at 8100 2.35 with four queries
// per CTA, 2.66 with one; 8 at 2000 1.39 and 1.15; prompt of 96 at 4000 6.1 and 9.0, of 333 10.3 and 9.9 at 500; one token at 300 1.02 cut in five,
// 1.12 in one chunk, at 60 1.00 and 0.90.  The rule finds the best of the four choices to 0.2 % on average and 5 % at most over
// those measurements; the thresholds before it (four queries from M x range = 16384 on, one chunk up to 320) lost 3.6 % on average and up to 54 %.
static double attn_cost_us(int sms, int HD, int G, int qb, int ctas, int nch, int range, int shorter) {
    const int rt = attn_row_tiles(G, qb), k = ctas <= sms / 2 ? 1 : std::max(2, (ctas + sms - 1) / sms);
    const double two = rt == 1 ? 0.038 + 0.00011 * HD : rt * (0.012 + 0.000305 * HD), alone = rt == 1 ? 0.012 + 0.000156 * HD : 0.59 * two,
                 many = rt == 1 ? 0.005 + 0.000164 * HD : 0.5 * two, start = qb == 1 ? 2.0 : 5.5;
    const double positions = (range - 0.5 * shorter * (1.0 - 1.0 / k)) / nch;             // earlier queries of a prompt see fewer, by up to `shorter`
    return start * std::max(1.0, 0.5 * k) + positions * (k == 1 ? alone : k == 2 ? two : k * many) + (nch > 1 ? 4.5 + 0.02 * nch : 0.0);
}
// No chunk is shorter than 64 positions, and no more than two CTAs per SM are made by cutting.
AttnPlan plan_attn_tok(const mi_ctx* ctx, int NH, int NKV, int HD, int M, int lp_max, bool ragged) {
    AttnPlan a{1, 1, 0};
    double best = 1e300;
    for (int qb = 1; qb <= (ragged || M == 1 ? 1 : kMaxQB); qb += kMaxQB - 1) {
        const int units = NKV * ((M + qb - 1) / qb), most = std::max(1, std::min((lp_max + 63) / 64, 2 * ctx->sm_count / units));
        for (int nch = 1; nch <= most; nch += std::max(1, most - 1)) {                    // one, and as many as may be
            const double us = attn_cost_us(ctx->sm_count, HD, NH / NKV, qb, units * nch, nch, lp_max, ragged ? 0 : M);
            if (us < best) { best = us; a.qb = qb; a.nch = nch; }
        }
    }
    a.part_doubles = a.nch > 1 ? (size_t)M * NH * a.nch * (HD + 2) : 0;
    return a;
}

// with more than one chunk there are at most two CTAs per SM, of at most kMaxQB queries of one group each
size_t attn_part_max(const mi_ctx* ctx, int NH, int NKV, int HD) { return (size_t)kMaxQB * (NH / NKV) * 2 * ctx->sm_count * (HD + 2); }

namespace {
template <int HD, int G, int QB>
int launch_qb(mi_ctx* ctx, const AttnParams& p, bool pdl) {
    constexpr int smem = AttnSmem<HD, attn_row_tiles(G, QB)>::bytes;
    auto kern = attn_tok_kernel<HD, G, QB>;
    static std::mutex mu;
    static std::atomic<unsigned> raised{0};                   // bit per device: opt-in shared memory set
    if (!(raised.load(std::memory_order_acquire) >> (ctx->device & 31) & 1u)) {
        std::lock_guard<std::mutex> hold(mu);
        MI_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        raised.fetch_or(1u << (ctx->device & 31), std::memory_order_release);
    }
    const int units = p.NKV * ((p.M + QB - 1) / QB);
    MI_CUDA(ctx, launch_k(pdl, kern, dim3(units * p.nch), dim3(kAT), smem, ctx->stream, p));
    if (p.nch > 2 * kAW) MI_CUDA(ctx, launch_k(pdl, attn_tok_merge<HD, kAW>, dim3(p.NH * p.M), dim3(kAT), 0, ctx->stream, p));
    else if (p.nch > 1) MI_CUDA(ctx, launch_k(pdl, attn_tok_merge<HD, 1>, dim3((p.NH * p.M + kAW - 1) / kAW), dim3(kAT), 0, ctx->stream, p));
    return MI_OK;
}
}  // namespace

int launch_attn_tok(mi_ctx* ctx, AttnParams p, const AttnPlan& plan, bool pdl) {
    p.qb = plan.qb; p.nch = plan.nch;
    const int G = p.NH / p.NKV;
    #define MI_A(hd, g) if (p.HD == hd && G == g) return plan.qb == 1 ? launch_qb<hd, g, 1>(ctx, p, pdl) : launch_qb<hd, g, kMaxQB>(ctx, p, pdl);
    MI_A(32, 2) MI_A(64, 2) MI_A(64, 7) MI_A(128, 6) MI_A(128, 8)
    #undef MI_A
    return set_error(ctx, MI_ERR_UNSUPPORTED, "attention: head_dim %d with %d query heads per kv head is not instantiated", p.HD, G);
}

}  // namespace mi

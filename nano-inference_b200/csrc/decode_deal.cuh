// How the matrices of a layer are dealt over the CTAs of the decode kernel that carry GEMV units: host arithmetic alone, without CUDA.
#pragma once
#include <algorithm>
#include <cstdint>

namespace mi {

constexpr int DNW = 8;            // warps per CTA that compute
constexpr int DNT = DNW * 32;     // their threads
constexpr int kMaxKSplit = 4;     // cross-CTA K-splits of the down projection
constexpr int kBatchUnits = 4;    // units of a job that a CTA works on at once: all it has, on the shapes of the range builds (lean_shape)

enum JobKind { JOB_QKV = 0, JOB_O = 1, JOB_GU = 2, JOB_DOWN = 3, JOB_LM = 4 };

struct Job {               // a tiled matrix and how it is dealt over the grid
    const uint8_t* base;   // tiled weights
    int groups;            // unit groups; one unit group = nacc consecutive 32-row groups
    int nt, ks, nb, kb, nacc, kind;
    bool half;             // units of half a row group
    int n_units;           // groups * ks, or groups * 2
    int rot;               // CTA (per-layer jobs) that gets unit 0
    int wrot;              // warp that gets tile 0 of a batch
    int g_off;             // first unit group this GPU owns (tensor parallelism; base points at it, groups counts the owned ones)
};

// rows (in groups) of a sharded matrix that GPU `rank` of `world` owns
inline void tp_share(int groups, int rank, int world, int* begin, int* end) {
    *begin = (int)((long long)groups * rank / world);
    *end = (int)((long long)groups * (rank + 1) / world);
}

// Cross-CTA K-split of a per-layer job.  A job whose result feeds an in-phase epilogue
// (QKV: bias + RoPE; gate/up: SwiGLU + q8_0) is never split across CTAs: its eight warps
// already share every unit, and so is the O projection.  The down projection has few row groups
// of many tiles; where halves of them give every CTA a unit at most they are dealt (Job::half), which needs no
// exchange (1.5B shape, us per token: two K ranges 573, whole groups 556, halves 549; a split's second hop is longer than two more rounds of tiles).  Else it is
// split until every CTA has a unit; the CTA of split 0 collects the other splits' partial sums (see run_cta_job).
inline int plan_ks(int kind, int groups, int nt, int kb, int grid) {
    if (kind != JOB_DOWN || (kb >= 4 && 2 * groups <= grid)) return 1;
    int ks = grid / std::max(groups, 1);
    return std::max(1, std::min(std::min(ks, nt), kMaxKSplit));
}

// A matrix of `groups` unit groups, nb blocks wide, on `grid` CTAs (base and wrot are the caller's).  force_ks: tuning knob, 0: none.
inline Job deal_job(int kind, int groups, int nb, int kb, int nacc, int grid, int rank, int world, int force_ks = 0) {
    Job jb{};
    jb.nb = nb; jb.kb = kb; jb.nt = nb / kb; jb.nacc = nacc; jb.kind = kind;
    // tensor parallelism: this GPU owns a contiguous range of the job's unit groups (rows); every GPU holds the
    // whole matrix but streams only its rows.  The K-split is planned from the largest share so that all GPUs
    // lay the partial sums out identically.
    // The QKV and O projections (a tenth of a layer's bytes) are the exception: every GPU computes all their rows,
    // so that attention and the O projection need no exchange at all.
    const bool replicated = kind == JOB_QKV || kind == JOB_O;
    int g0 = 0, g1 = groups;
    if (!replicated) tp_share(groups, rank, world, &g0, &g1);
    jb.g_off = g0; jb.groups = g1 - g0;
    jb.ks = plan_ks(kind, replicated ? groups : (groups + world - 1) / world, jb.nt, kb, grid);
    if (force_ks) jb.ks = std::max(1, std::min(std::min(force_ks, jb.nt), kMaxKSplit));
    if (jb.ks >= grid) jb.ks = std::max(1, grid - 1);       // the CTAs of a row group's splits must be distinct
    // units of half a row group where that leaves no CTA with two of them; pairs of groups (gate/up) stay whole, as q8_0 blocks of their result
    jb.half = nacc == 1 && jb.ks == 1 && kind != JOB_LM && kb >= 4 && 2 * jb.groups <= grid;
    jb.n_units = jb.groups * (jb.half ? 2 : jb.ks);
    // Every layer is dealt alike, so that the kernel needs one list per CTA.  Gate/up is dealt from the first CTA on and QKV from the last one back, so that as many CTAs as
    // possible have a unit of one of the two (see bystanders).  Where the down projection is split, the CTAs that fold the splits publish last, so they are the first
    // ones (unit order: split by split), and the job that follows them, QKV, is far from them; and O goes with it (each job from where the one before it
    // stopped: 3B shape 827 us per token instead of 817, 1.5B and 0.5B 1 % less).
    jb.rot = kind == JOB_QKV || kind == JOB_O ? std::max(0, grid - jb.n_units) : 0;
    return jb;
}

// first unit of a per-layer job that `cta` has (no fewer than n_units: none); the others follow `grid` apart
inline int first_unit(const Job& jb, int cta, int grid) {
    const int r = jb.rot % grid;
    return cta >= r ? cta - r : cta + grid - r;
}

// the most units of the job that a CTA has
inline int most_units(const Job& jb, int grid) { return (jb.n_units + grid - 1) / grid; }

// Shapes the context-range builds take: they hold one variant of each prologue and of the tile loop and no call to the others, and one batch of units per CTA and job
// (a full grid deals these shapes at most 455 units to 130 CTAs; with three units per batch a feed-forward width of 14336 had some of four, ran the general
// build and took 410 us per token for 12 layers where the range build takes 288).  On a smaller grid (MINFER_GRID) more than kBatchUnits units per CTA mean the general build.
// 1: embedding widths of 1025 to 2048 with tiles of 8 blocks; 2: of 513 to 1024 with tiles of 8 or 4 blocks (the small builds,
// MI_SMALL: 370 us per token at the 0.5B shape where the general build, whose loop spills, takes 430; 1.5B 520 and 772, 3B 794 and 1089); 0: neither.
inline int lean_shape(int E, int FF, int NQ) {
    auto kb = [&](int k) { return (E / 32) % k == 0 && (FF / 32) % k == 0 && (NQ / 32) % k == 0; };
    auto np = [](int n) { return (n / 8 + (n / 32 + 1) / 2 + DNT - 1) / DNT; };          // pairs of words of a q8_0 vector per thread
    if (np(FF) > 8 || np(NQ) > 8) return 0;
    return E > 1024 && E <= 2048 && kb(8) ? 1 : E > 512 && E <= 1024 && kb(4) ? 2 : 0;
}

// The CTAs with neither a gate/up nor a QKV unit, which the units just dealt leave in one run [*first, *first + *n).  They read the residual stream's words in every layer
// like all others, but nothing they hand on keeps those words from being written again: they publish a word of their own instead (XwLayout::att).
inline void bystanders(const Job& qkv, const Job& gu, int grid, int* first, int* n) {
    *first = std::min(gu.n_units, grid);
    *n = std::max(0, grid - std::min(qkv.n_units, grid) - *first);
}

}  // namespace mi

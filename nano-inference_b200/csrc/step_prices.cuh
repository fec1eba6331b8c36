// What a step of the speculation loop costs, for host code.
#pragma once
#include <algorithm>

namespace mi {

// Running averages of the device time of single-token steps and of M-token passes, by M; an M not yet seen is priced from the nearest seen one along the
// measured shape of the pass.
class StepPrices {
public:
    static constexpr int kMaxPass = 16;

    void learn_step(float ms) { learn(step, ms); }
    void learn_pass(int M, float ms) { learn(pass[M], ms); }

    // time of a pass of M tokens behind `pos` positions, 0 while nothing is known
    float pass_ms(int M, int pos) const {
        if (pass[M] > 0.f) return pass[M];
        for (int d = 1; d <= kMaxPass; d++)
            for (int q : {M - d, M + d})
                if (q >= 1 && q <= kMaxPass && pass[q] > 0.f) return pass[q] * shape(M, pos) / shape(q, pos);
        return 0.f;
    }
    // the number K <= kmax of drafted tokens that gives most tokens per time when each is accepted with probability `alpha`; 0: a plain step
    int best_draft(float alpha, int kmax, int pos) const {
        if (step <= 0.f) return 0;                                    // nothing to compare with yet: take a plain step and measure it
        int best = 0;
        float rate = 1.f / step, pw = alpha;
        for (int K = 1; K <= kmax; K++) {
            pw *= alpha;                                              // alpha^(K+1)
            const float ms = pass_ms(K + 1, pos);
            if (ms <= 0.f) continue;
            const float expect = alpha < 0.999f ? (1.f - pw) / (1.f - alpha) : (float)(K + 1);
            if (expect / ms > rate) { rate = expect / ms; best = K; }
        }
        return best;
    }
    bool knows_step() const { return step > 0.f; }

    // Time of a pass against one of 8 tokens at the beginning: the products work on groups of eight tokens (flat up to 8, a step to 9), the
    // attention on tokens x positions, in one chunk up to 160 positions.  Fitted to the three model shapes at 60 .. 8192 positions, M = 1 .. 16:
    // between any two M 14 % off at most up to 2000 positions, 20 % at 8192.
    static float shape(int M, int pos) {
        return (M <= 8 ? 0.91f + 0.011f * M : 1.07f + 0.0145f * M) + (pos > 160 ? 0.1f : 0.f) + 9e-6f * M * pos;
    }

private:
    static void learn(float& avg, float ms) { if (ms > 0.f) avg = avg > 0.f ? 0.8f * avg + 0.2f * ms : ms; }
    float step = 0.f, pass[kMaxPass + 1] = {0.f};
};

}  // namespace mi

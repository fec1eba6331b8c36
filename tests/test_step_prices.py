"""The speculation loop's prices (csrc/step_prices.cuh), compiled for the host, against measured times of single-token steps and of M-token passes."""
import subprocess
from pathlib import Path

SRC = Path(__file__).resolve().parent.parent / "nano-inference_b200" / "csrc"

# model shape, position, ms of a single-token step, ms of a pass of M = 1 .. 16 tokens on a B200
MEASURED = [
    ("0.5b", 60, 0.441, [0.606, 0.611, 0.612, 0.612, 0.626, 0.628, 0.639, 0.644, 0.771, 0.776, 0.777, 0.775, 0.835, 0.835, 0.836, 0.841]),
    ("0.5b", 500, 0.554, [0.695, 0.710, 0.716, 0.714, 0.724, 0.718, 0.732, 0.743, 0.859, 0.862, 0.871, 0.869, 0.936, 0.950, 0.956, 0.952]),
    ("0.5b", 2000, 0.57, [0.690, 0.702, 0.717, 0.729, 0.773, 0.792, 0.797, 0.814, 0.964, 1.008, 1.026, 1.033, 1.092, 1.119, 1.130, 1.128]),
    ("0.5b", 8192, 0.646, [0.800, 0.829, 0.914, 0.947, 1.042, 1.093, 1.108, 1.113, 1.443, 1.418, 1.417, 1.420, 1.586, 1.584, 1.583, 1.586]),
    ("1.5b", 60, 0.602, [0.890, 0.900, 0.893, 0.894, 0.943, 0.955, 0.959, 0.966, 1.130, 1.135, 1.141, 1.148, 1.187, 1.188, 1.195, 1.199]),
    ("1.5b", 500, 0.73, [1.038, 1.072, 1.047, 1.040, 1.084, 1.123, 1.123, 1.130, 1.297, 1.304, 1.252, 1.262, 1.335, 1.342, 1.368, 1.352]),
    ("1.5b", 2000, 0.757, [1.005, 1.039, 1.014, 1.029, 1.094, 1.108, 1.119, 1.148, 1.404, 1.450, 1.462, 1.489, 1.543, 1.580, 1.599, 1.600]),
    ("1.5b", 8192, 0.875, [1.104, 1.159, 1.230, 1.286, 1.427, 1.502, 1.674, 1.670, 2.028, 2.043, 2.046, 2.073, 2.296, 2.302, 2.322, 2.338]),
    ("3b", 60, 0.891, [1.430, 1.415, 1.406, 1.400, 1.484, 1.498, 1.502, 1.503, 1.853, 1.869, 1.889, 1.894, 1.959, 1.964, 1.974, 1.976]),
    ("3b", 500, 1.074, [1.616, 1.605, 1.598, 1.592, 1.699, 1.707, 1.713, 1.706, 1.999, 2.005, 2.023, 2.039, 2.172, 2.189, 2.192, 2.198]),
    ("3b", 2000, 1.143, [1.565, 1.569, 1.582, 1.584, 1.676, 1.696, 1.701, 1.735, 2.250, 2.330, 2.331, 2.390, 2.433, 2.486, 2.514, 2.512]),
    ("3b", 8192, 1.308, [1.713, 1.732, 1.829, 1.891, 2.100, 2.209, 2.329, 2.444, 3.063, 3.186, 3.251, 3.405, 3.545, 3.696, 3.911, 3.907]),
]

PROGRAM = r"""
#include "step_prices.cuh"
#include <cstdio>
#include <cmath>
int main() {
    int pos; double step, t[17];
    while (std::scanf("%d %lf", &pos, &step) == 2) {
        for (int M = 1; M <= 16; M++) if (std::scanf("%lf", t + M) != 1) return 2;
        double worst = 0, loss = 0;
        for (int q = 1; q <= 16; q++) {                       // one M known: every other is priced from it
            mi::StepPrices p;
            if (p.best_draft(0.9f, 15, pos) != 0) return 3;    // nothing known: a plain step
            p.learn_pass(q, (float)t[q]); p.learn_step((float)step);
            for (int M = 1; M <= 16; M++) worst = std::fmax(worst, std::fabs(p.pass_ms(M, pos) / t[M] - 1));
            if (std::fabs(p.pass_ms(q, pos) / t[q] - 1) > 1e-6) return 4;
            for (float a : {0.1f, 0.3f, 0.5f, 0.7f, 0.9f, 1.0f}) {
                auto rate = [&](int K) { double e = 0, w = 1; for (int k = 0; k <= K; k++) { e += w; w *= a; } return K == 0 ? 1 / step : e / t[K + 1]; };
                double best = 0;
                for (int K = 0; K <= 15; K++) best = std::fmax(best, rate(K));
                loss = std::fmax(loss, 1 - rate(p.best_draft(a, 15, pos)) / best);
            }
        }
        std::printf("%d %f %f\n", pos, worst, loss);
    }
    return 0;
}
"""


def test_passes_not_seen_yet_are_priced_along_the_measured_shape(tmp_path):
    src = tmp_path / "prices.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "prices"
    subprocess.run(["g++", "-O2", "-Wall", "-std=c++17", "-I", str(SRC), "-o", str(exe), str(src)], check=True)
    text = "\n".join(" ".join(map(str, [pos, step, *t])) for _, pos, step, t in MEASURED)
    r = subprocess.run([str(exe)], input=text, capture_output=True, text=True)
    assert r.returncode == 0, r
    lines = [l.split() for l in r.stdout.split("\n") if l]
    assert len(lines) == len(MEASURED)
    for pos, worst, loss in lines:
        assert float(worst) < (0.15 if int(pos) <= 2000 else 0.21), lines
        assert float(loss) < 0.16, lines                      # tokens per time lost to a wrong price

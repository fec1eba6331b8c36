"""The norms' division by a known divisor (csrc/div_known.cuh) is the division: compiled for the host and compared with `/`, bit by bit."""
import subprocess
from pathlib import Path

SRC = Path(__file__).resolve().parent.parent / "nano-inference_b200" / "csrc"

PROGRAM = r"""
#include "div_known.cuh"
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>

static uint64_t bits(double x) { uint64_t b; std::memcpy(&b, &x, 8); return b; }
static long wrong = 0;
static void check(double a, int n) {
    const double b = n, y = 1.0 / b, got = mi::div_known(a, b, y), want = a / b;
    if (bits(got) != bits(want) && !(got != got && want != want) && wrong++ < 5) std::printf("%a / %d: %a instead of %a\n", a, n, got, want);
}
int main() {
    std::mt19937_64 rng(1);
    for (int n = 32; n <= 8192; n += 32) {                                     // every embedding width a model may have
        for (double a : {0.0, 1.0, (double)n, HUGE_VAL, std::nan("")}) check(a, n);
        for (int i = 0; i < 4000; i++) {                                        // any exponent a sum of squares of fp32 values can have
            double m = 1.0 + (double)(rng() >> 12) * 0x1p-52;
            check(std::ldexp(m, (int)(rng() % 568) - 298), n);
        }
        for (int i = 0; i < 1000; i++) {                                        // next to exact quotients and to the middles between them
            const double q = 1.0 + (double)(rng() >> 12) * 0x1p-52, a = q * n;
            check(a, n); check(std::nextafter(a, 0.0), n); check(std::nextafter(a, HUGE_VAL), n);
        }
    }
    std::printf("%ld wrong\n", wrong);
    return wrong != 0;
}
"""


def test_the_norms_division_is_the_division(tmp_path):
    src = tmp_path / "div.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "div"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma", "-x", "c++", "-I", str(SRC), "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout

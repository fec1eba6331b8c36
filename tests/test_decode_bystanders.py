"""CTAs of the decode kernel that have a unit neither of QKV nor of gate/up: the list that the host makes of them against the units as dealt
(csrc/decode_deal.cuh), and a run in which one of them is far behind the others."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

import gguf_util as gu

SRC = Path(__file__).resolve().parent.parent / "nano-inference_b200" / "csrc"

PROGRAM = r"""
#include "decode_deal.cuh"
#include <cstdio>
int main() {
    int E, FF, NQ, KVD, grid, rank, world;
    while (std::scanf("%d %d %d %d %d %d %d", &E, &FF, &NQ, &KVD, &grid, &rank, &world) == 7) {
        auto kb = [](int cols) { const int nb = cols / 32; return nb % 8 == 0 ? 8 : nb % 4 == 0 ? 4 : nb % 2 == 0 ? 2 : 1; };
        auto job = [&](int kind, int groups, int cols) { return mi::deal_job(kind, groups, cols / 32, kb(cols), kind == mi::JOB_GU ? 2 : 1, grid, rank, world); };
        const mi::Job jobs[4] = {job(mi::JOB_QKV, (NQ + 2 * KVD + 31) / 32, E), job(mi::JOB_O, E / 32, NQ), job(mi::JOB_GU, FF / 32, E), job(mi::JOB_DOWN, E / 32, FF)};
        int first, n;
        mi::bystanders(jobs[mi::JOB_QKV], jobs[mi::JOB_GU], grid, &first, &n);
        std::printf("%d %d", first, n);
        for (int cta = 0; cta < grid; cta++) {
            int has = 0;
            for (const mi::Job& jb : jobs) has |= mi::first_unit(jb, cta, grid) < jb.n_units ? 1 << jb.kind : 0;
            std::printf(" %d", has);
        }
        std::printf("\n");
    }
}
"""

# embedding, feed-forward, query heads, kv heads
SHAPES = [(896, 4864, 14, 2), (1536, 8960, 12, 2), (2048, 11008, 16, 2), (2048, 14336, 16, 2), (3584, 18944, 28, 4), (512, 2048, 8, 4), (128, 352, 4, 2), (64, 32, 2, 1)]


def test_every_cta_that_reads_the_residual_stream_holds_its_writers_back(tmp_path):
    (tmp_path / "deal.cpp").write_text(PROGRAM)
    exe = tmp_path / "deal"
    subprocess.run(["g++", "-O2", "-Wall", "-std=c++17", "-I", str(SRC), "-o", str(exe), str(tmp_path / "deal.cpp")], check=True)
    cases = [(E, FF, E, kv * (E // heads), grid, rank, world) for E, FF, heads, kv in SHAPES for grid in (148, 140, 136, 134, 100, 24, 3) for world in (1, 2, 4, 8) for rank in {0, world - 1}]
    r = subprocess.run([str(exe)], input="\n".join(" ".join(map(str, c)) for c in cases), capture_output=True, text=True, check=True)
    some = 0
    for case, line in zip(cases, r.stdout.splitlines(), strict=True):
        first, n, *has = map(int, line.split())
        without = [cta for cta, kinds in enumerate(has) if not kinds & 0b101]      # no QKV (bit 0), no gate/up (bit 2)
        assert without == list(range(first, first + n)), case
        some += n > 0
    assert some > 20
    # their words, behind the attention output's scales, are awaited by whoever computes the O projection
    kernel = (SRC / "decode_kernel.cuh").read_text()
    assert "pub.all(P.xo.att + P.NH * HD / 4 + P.NH * HD / 32 + by, 0u)" in kernel and "k == 2 ? P.att_scales :" in kernel


# 24 of 134 CTAs without a unit of QKV or gate/up (110 of 148 without attention CTAs): one of them comes 200 us late to every read of the residual stream's
# words, where a layer takes some 20.  Dedicated attention, across its range, long-range attention
@pytest.mark.gpu
@pytest.mark.parametrize("attn_ctas,cta", [(14, 14 + 38), (14, 14 + 61), (0, 38), (0, 75)])
@pytest.mark.parametrize("pos", [20, 253, 700])
def test_a_late_cta_without_units_misses_nothing(ctx, pkg, tmp_path, monkeypatch, attn_ctas, cta, pos):
    import torch
    if ctx.sm_count != 148:
        pytest.skip("the CTAs without units are listed for 148 SMs")
    monkeypatch.setenv("MINFER_PROFILE", "1")
    if not attn_ctas:
        monkeypatch.setenv("MINFER_ATTN_CTAS", "0")
    args = dict(layers=3, embd=896, ff=1216, heads=14, kv_heads=2, vocab=700)
    path = gu.make_synthetic(tmp_path / "m.gguf", "tiny", seed=9, extra=[a for k, v in args.items() for a in (f"--{k.replace('_', '-')}", v)])
    n, out = 6, []
    seq = [int(t) for t in np.random.default_rng(pos).integers(0, 700, n)]
    for us in (0, 200):
        m = pkg.Model(ctx, path, pos + n)
        gen = torch.Generator(device="cuda").manual_seed(pos)
        for name in ("kcache", "vcache"):
            m.state_tensor(name).view(torch.float16).normal_(generator=gen)
        torch.cuda.synchronize()
        m.debug_hold(cta, us)
        lg = torch.zeros((n, 700), device="cuda")
        ids, ms = m.decode(seq, n, pos, lg)
        ctx.sync()
        assert ms >= n * (2 * args["layers"] + 1) * us * 1e-3          # (it was late)
        out.append((ids, lg.clone()))
        m.free()
    assert out[0][0] == out[1][0]
    assert torch.equal(out[0][1].view(torch.int32), out[1][1].view(torch.int32))

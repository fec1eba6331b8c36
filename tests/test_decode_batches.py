"""Units of a job that a CTA of the decode kernel works on at once: the context-range builds hold one such batch (csrc/decode_deal.cuh), so all shapes they are
chosen for have to fit it; and runs with two to four units per batch, and with several batches, against the M-token pass."""
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
    int E, FF, NQ, KVD, grid, most = 0, shapes = 0;
    while (std::scanf("%d %d %d %d %d", &E, &FF, &NQ, &KVD, &grid) == 5) {
        if (!mi::lean_shape(E, FF, NQ)) continue;
        auto kb = [](int cols) { const int nb = cols / 32; return nb % 8 == 0 ? 8 : nb % 4 == 0 ? 4 : nb % 2 == 0 ? 2 : 1; };
        auto units = [&](int kind, int groups, int cols) { return mi::most_units(mi::deal_job(kind, groups, cols / 32, kb(cols), kind == mi::JOB_GU ? 2 : 1, grid, 0, 1), grid); };
        for (int u : {units(mi::JOB_QKV, (NQ + 2 * KVD) / 32, E), units(mi::JOB_O, E / 32, NQ), units(mi::JOB_GU, FF / 32, E), units(mi::JOB_DOWN, E / 32, FF)}) most = std::max(most, u);
        shapes++;
    }
    std::printf("%d %d %d\n", shapes, most, mi::kBatchUnits);
}
"""


def test_every_shape_of_the_range_builds_is_one_batch(tmp_path):
    (tmp_path / "deal.cpp").write_text(PROGRAM)
    exe = tmp_path / "deal"
    subprocess.run(["g++", "-O2", "-Wall", "-std=c++17", "-I", str(SRC), "-o", str(exe), str(tmp_path / "deal.cpp")], check=True)
    cases = []
    for HD, G in ((64, 2), (64, 7), (128, 6), (128, 8)):               # the head shapes there are kernels for, but the smallest
        for kv in range(1, 17):
            E, heads = HD * G * kv, G * kv
            ctas = heads // (2 if G % 2 == 0 and G > 2 else 1)         # set aside for attention, where the grid can spare them
            grid = 148 - (ctas if ctas * 8 <= 148 else 0)
            cases += [(E, FF, E, HD * kv, grid) for FF in range(128, 16385, 128)]
    r = subprocess.run([str(exe)], input="\n".join(" ".join(map(str, c)) for c in cases), capture_output=True, text=True, check=True)
    shapes, most, batch = map(int, r.stdout.split())
    assert shapes > 200 and most <= batch


# units per CTA of gate/up: four and three on the short- and the long-range build, the same on a smaller grid, and six (two batches, general build)
@pytest.mark.gpu
@pytest.mark.parametrize("grid,shape", [(148, dict(embd=2048, ff=14336, heads=16, kv_heads=2)), (100, dict(embd=1536, ff=8960, heads=12, kv_heads=2)), (60, dict(embd=1536, ff=8960, heads=12, kv_heads=2))])
@pytest.mark.parametrize("pos", [0, 300])
def test_batches_of_several_units(ctx, pkg, tmp_path, monkeypatch, grid, shape, pos):
    import torch
    monkeypatch.setenv("MINFER_GRID", str(grid))
    args = dict(shape, layers=2, vocab=700)
    path = gu.make_synthetic(tmp_path / "m.gguf", "tiny", seed=2, extra=[a for k, v in args.items() for a in (f"--{k.replace('_', '-')}", v)])
    m = pkg.Model(ctx, path, pos + 6)
    gen = torch.Generator(device="cuda").manual_seed(grid)
    for name in ("kcache", "vcache"):
        m.state_tensor(name).view(torch.float16).normal_(generator=gen)
    torch.cuda.synchronize()
    seq = [int(t) for t in np.random.default_rng(grid).integers(0, 700, 6)]
    one, many = (torch.zeros((6, 700), device="cuda") for _ in range(2))
    ids, _ = m.decode(seq, 6, pos, one)
    want, _ = m.verify(seq, pos, many)
    ctx.sync()
    assert torch.equal(one.view(torch.int32), many.view(torch.int32))
    assert list(ids) == list(want)
    m.free()

"""Every build of the decode kernel that runs has an instrumented one (MINFER_PROFILE), for the same range and shapes, with the same bits."""
import re
from pathlib import Path

import numpy as np
import pytest

import gguf_util as gu

CSRC = Path(__file__).resolve().parent.parent / "nano-inference_b200" / "csrc"


def settings(text):
    lean, small = (re.search(rf"#define {d} (\d)", text) for d in ("MI_LEAN", "MI_SMALL"))
    return int(lean[1]) if lean else 0, int(small[1]) if small else 0, tuple(sorted(re.findall(r"MI_PICK\((\d+), (\d+)\)", text)))


def test_every_range_build_has_an_instrumented_twin():
    plain, prof = {}, {}
    for f in CSRC.glob("decode_*.cu"):
        text = f.read_text()
        if "MI_TP 1" in text or "decode_kernel.cuh" not in text:
            continue
        (prof if "#define MI_PROF 1" in text else plain)[settings(text)] = re.search(r"const void\* (\w+)\(", text)[1]
    assert len(plain) == 4 and all(s in prof for s in plain), (plain, prof)
    dispatch = (CSRC / "decode.cu").read_text()
    branch = dispatch[dispatch.index("} else if (P.prof) {"):dispatch.index("#define MI_PICK", dispatch.index("} else if (P.prof) {"))]
    for name in [*plain.values(), *(prof[s] for s in plain)]:
        assert name + "(m->HD" in branch, name


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [dict(embd=896, ff=1216, heads=14), dict(embd=1536, ff=1024, heads=12), dict(embd=128, ff=352, heads=4)])
@pytest.mark.parametrize("pos", [20, 250, 700])
def test_instrumented_builds_give_the_same_bits(ctx, pkg, tmp_path, monkeypatch, shape, pos):
    import torch
    args = dict(shape, layers=2, kv_heads=2, vocab=700)
    path = gu.make_synthetic(tmp_path / "m.gguf", "tiny", seed=4, extra=[a for k, v in args.items() for a in (f"--{k.replace('_', '-')}", v)])
    n, out = 12, []
    seq = [int(t) for t in np.random.default_rng(pos).integers(0, 700, n)]
    for profiled in (False, True):
        if profiled:
            monkeypatch.setenv("MINFER_PROFILE", "1")
        m = pkg.Model(ctx, path, pos + n)
        gen = torch.Generator(device="cuda").manual_seed(pos)
        for name in ("kcache", "vcache"):
            m.state_tensor(name).view(torch.float16).normal_(generator=gen)
        torch.cuda.synchronize()
        lg = torch.zeros((n, 700), dtype=torch.float32, device="cuda")
        ids, _ = m.decode(seq, n, pos, lg)
        ctx.sync()
        out.append((ids, lg.clone()))
        marks = m.state("profile", np.uint64, 32)
        assert (marks[[12, 18, 19]] > 0).all() == profiled
        m.free()
    assert out[0][0] == out[1][0]
    assert torch.equal(out[0][1].view(torch.int32), out[1][1].view(torch.int32))

"""How the decode kernel's matrices are dealt over the grid: half row groups, whole ones, K ranges, several units per CTA in one batch and in more.  Each against the M-token
pass, which is cut without regard to any of it, as bits; and SwiGLU with digits where its blocks do not fill the CTA's rounds."""
import numpy as np
import pytest

import gguf_util as gu

pytestmark = pytest.mark.gpu


def model_file(tmp_path, **shape):
    args = dict(dict(layers=2, kv_heads=2, vocab=700), **shape)
    return gu.make_synthetic(tmp_path / "m.gguf", "tiny", seed=6, extra=[a for k, v in args.items() for a in (f"--{k.replace('_', '-')}", v)])


# (tiles of 4, 8 and, in the down projection, 2 and 1 blocks).  148: halves, or K ranges where tiles are shallow; 100: whole groups of 1536 rows; 24: up to three units per CTA;
# 16: more, in several batches (fewer CTAs than query heads the kernel has never taken)
@pytest.mark.parametrize("shape", [dict(embd=896, ff=1216, heads=14), dict(embd=1536, ff=2048, heads=12), dict(embd=2048, ff=2816, heads=16), dict(embd=128, ff=352, heads=4)])
@pytest.mark.parametrize("grid", [148, 100, 24, 16])
@pytest.mark.parametrize("pos", [0, 300])
def test_every_dealing_gives_the_pass_s_logits(ctx, pkg, tmp_path, monkeypatch, shape, grid, pos):
    import torch
    monkeypatch.setenv("MINFER_GRID", str(grid))
    m = pkg.Model(ctx, model_file(tmp_path, **shape), pos + 12)
    gen = torch.Generator(device="cuda").manual_seed(grid)
    for name in ("kcache", "vcache"):
        m.state_tensor(name).view(torch.float16).normal_(generator=gen)
    torch.cuda.synchronize()
    seq = [int(t) for t in np.random.default_rng(grid).integers(0, 700, 12)]
    one, many = (torch.zeros((12, 700), device="cuda") for _ in range(2))
    ids, _ = m.decode(seq, 12, pos, one)
    want, _ = m.verify(seq, pos, many)
    ctx.sync()
    assert torch.equal(one.view(torch.int32), many.view(torch.int32))
    assert list(ids) == list(want)
    m.free()


# blocks: 1, one less and one more than the 32 that a CTA has at a time, two rounds, a ragged third
@pytest.mark.parametrize("blocks", [1, 31, 33, 64, 71])
@pytest.mark.parametrize("n", [17, 40])
def test_swiglu_of_any_number_of_blocks(ctx, pkg, tmp_path, blocks, n):
    import torch
    path = model_file(tmp_path, embd=256, ff=32 * blocks, heads=4)
    tokens = np.random.default_rng(blocks).integers(0, 700, n).astype(np.int32)
    caches, last = [], []
    for which in (-1, 1):                                  # the product over blocks; over digits
        m = pkg.Model(ctx, path, n + 1)
        m.debug_products(which)
        m.prefill(tokens)
        lg = torch.zeros((1, 700), device="cuda")
        m.decode([int(tokens[0])], 1, n, lg)
        ctx.sync()
        caches.append([m.state_tensor(k).clone() for k in ("kcache", "vcache")])
        last.append(lg.clone())
        m.free()
    assert torch.equal(last[0].view(torch.int32), last[1].view(torch.int32))
    assert all(torch.equal(a, b) for a, b in zip(*caches))

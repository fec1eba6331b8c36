"""Passes of more than 16 tokens: the product over whole-K digit sums gives what the product over blocks gives, bit for bit, at the edges of its tiles and for
scales that its digits hold with three planes, with four, or not at all."""
import numpy as np
import pytest

import gguf_util as gu

pytestmark = pytest.mark.gpu


def patch(path, name, edit, dtype):
    r = gu.GgufReader(path)
    _, _, off, nbytes = r.tensors[name]
    raw = r.tensor_bytes(name)
    _, rows, cols = r.shape(name)
    edit(raw.view(np.float32) if dtype == "f32" else raw.reshape(rows, cols // 32, 18)[:, :, :2].view(np.uint16)[:, :, 0])
    with open(path, "r+b") as f:
        f.seek(off)
        f.write(raw.tobytes())


def lower(d, binades):
    """fp16 scales `binades` powers of two smaller (zero where that is below the smallest normal number)"""
    e = (d >> 10) & 31
    return np.where(e > binades, d - (binades << 10), d & 0x8000).astype(np.uint16)


def same(ctx, pkg, path, n, V):
    """Prompt pass of n tokens, then a batch of min(n, 64) sequences: caches and logits of both products"""
    import torch
    seq = [int(t) for t in np.random.default_rng(n).integers(0, V, n)]
    kept = []
    for which in (-1, 1):
        m = pkg.Model(ctx, path, n + 1)
        m.debug_products(which)
        out = [m.prefill(seq, 0)[0]]
        for name in ("kcache", "vcache"):
            out.append(m.state_tensor(name).cpu().numpy().copy())
        B = min(n, 64)
        b = pkg.Batch(m, B, 4)
        logits = torch.zeros((B, V), device="cuda")
        for p in range(2):                                   # (the second step of a kind runs as a graph)
            out.append(list(b.step(seq[:B], list(range(B)), [p] * B, logits)[0]))
            out.append(logits.cpu().numpy().copy())
        b.free(); m.free()
        kept.append(out)
    for i, (x, y) in enumerate(zip(*kept)):
        assert np.array_equal(np.asarray(x), np.asarray(y), equal_nan=np.asarray(x).dtype.kind == "f"), i
    assert any(np.any(np.asarray(x) != 0) for x in kept[0][1:3])


# matrices of 6, 10, 12, 14, 16 and 11, 43 blocks per row (tile depths 2, 2, 4, 2, 8 and 1: whole steps, a step of one stage, an odd last block), row counts off the
# tile of 128; tokens: one tile of every width, an odd number of eights, several tiles, the longest pass
@pytest.mark.parametrize("embd,ff", [(192, 352), (320, 1376), (384, 256), (448, 736), (512, 1024)])
@pytest.mark.parametrize("n", [17, 24, 40, 56, 64, 65, 130, 512])
def test_digit_product_equals_block_product(ctx, pkg, tmp_path, embd, ff, n):
    path = gu.make_synthetic(tmp_path / "m.gguf", "tiny", seed=embd + n, extra=["--layers", 2, "--embd", embd, "--heads", embd // 32, "--kv-heads", embd // 64, "--ff", ff, "--vocab", 700])
    same(ctx, pkg, path, n, 700)


# how many binades a row's weight scales, or a token's activation scales, lie apart: three and four digits, and more than the digits hold (rows and tokens
# summed block by block); not finite
@pytest.mark.parametrize("weights", [0, 8, 9, 14, 17, 25, "inf"])
@pytest.mark.parametrize("acts", [0, 5, 7, 12, 16, "inf"])
def test_scales_far_apart(ctx, pkg, tmp_path, weights, acts):
    path = gu.make_synthetic(tmp_path / "m.gguf", "tiny", seed=5, std=2.0, extra=["--layers", 2, "--embd", 256, "--heads", 8, "--kv-heads", 4, "--ff", 512, "--vocab", 400])
    if weights:
        for name in ("blk.0.attn_q.weight", "blk.0.ffn_gate.weight", "blk.1.ffn_down.weight", "blk.0.attn_output.weight"):
            def edit(d):
                if weights == "inf":
                    d[3, 1] = 0x7C00
                else:
                    d[3::50, 1] = lower(d[3::50, 1], weights)
                    d[7, :] = 0                                  # a row of zeros
            patch(path, name, edit, "q4")
    if acts:
        def edit(w):
            w[32:64] = np.inf if acts == "inf" else w[32:64] * 2.0 ** -acts
        patch(path, "blk.1.ffn_norm.weight" if acts == "inf" else "blk.0.ffn_norm.weight", edit, "f32")
        if acts != "inf":
            patch(path, "blk.1.attn_norm.weight", edit, "f32")
    same(ctx, pkg, path, 40, 400)


# the shapes it is meant for, by cost
@pytest.mark.parametrize("preset,n", [("1.5b", 333), ("0.5b", 200), ("3b", 64)])
def test_digit_product_on_model_shapes(ctx, pkg, tmp_path, preset, n):
    path = gu.make_synthetic(tmp_path / "m.gguf", preset, seed=2, extra=["--layers", 1, "--vocab", 1500])
    same(ctx, pkg, path, n, 1500)

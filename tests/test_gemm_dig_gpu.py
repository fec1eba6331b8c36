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


def rewrite(path, **tensors):
    """tensors: name with _ for . -> edit(fp16 scale bits [rows, blocks], nibbles [rows, blocks, 16]) of a q4_0 matrix, or edit(values) of an fp32 vector"""
    r = gu.GgufReader(path)
    with open(path, "r+b") as f:
        for name, edit in tensors.items():
            name = name.replace("__", ".")
            typ, rows, cols = r.shape(name)
            raw = r.tensor_bytes(name)
            if typ == 0:
                edit(raw.view(np.float32))
            else:
                q = raw.reshape(rows, cols // 32, 18)
                d, n = np.ascontiguousarray(q[:, :, :2]).view(np.uint16)[:, :, 0], q[:, :, 2:]
                edit(d, n)
                q[:, :, :2] = d[:, :, None].view(np.uint8)
            f.seek(r.tensors[name][2])
            f.write(raw.tobytes())


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


# The widest rows against the widest tokens that the digits hold: all blocks at the top of the range but one at its bottom, sums of one sign (every weight -8 or 7, every
# activation the block's largest) and random ones.  The integer sum of such a row passes 2^63 (8 binades; with 7 at up to 2048 elements and 5 at 8192 it stays just
# below).  Both products round a sum that wide to 53 bits on the way, the block product at every addition, this one once; what is compared is the fp32 value.
def top_but_one(d, low, spread):
    """exponent fields low + spread, one block of a row low; signs and mantissas as they are"""
    d[:] = (d & 0x83FF) | ((low + spread) << 10)
    d[:, 5] = (d[:, 5] & 0x83FF) | (low << 10)


@pytest.mark.parametrize("spread", [5, 7, 8, 16])
@pytest.mark.parametrize("signs", ["one", "random"])
@pytest.mark.parametrize("embd", [1536, 2048, 8192])
@pytest.mark.parametrize("n", [24, 40, 56, 64])
def test_sums_beyond_64_bits(ctx, pkg, tmp_path, spread, signs, embd, n):
    """lm_head on the embedding itself (the layer adds nothing)"""
    path = gu.make_synthetic(tmp_path / "m.gguf", "tiny", seed=3, std=0.5, extra=["--layers", 1, "--embd", embd, "--heads", embd // 128, "--kv-heads", 8 if embd > 2048 else 2, "--ff", 256, "--vocab", 600, "--untied"])

    def nothing(d, q):
        d[:] = 0

    def head(d, q):
        d[:] = d & 0xFF00 | 0xFF if signs == "random" else 0x03FF
        top_but_one(d, 1, spread)
        if signs == "one":
            q[::2], q[1::2] = 0x00, 0xFF                                  # -8 throughout, 7 throughout

    def embedding(d, q):
        d &= 0x7FFF
        if signs == "one":
            d[:], q[:] = 0x3800, 0xFF

    def norm(w):
        w[:] = 127 * 1.999 if signs == "one" else 30.0                    # block scales of about 2^0 and 2^-13
        w[32 * 9:32 * 10] *= 2.0 ** -13

    rewrite(path, blk__0__attn_output__weight=nothing, blk__0__ffn_down__weight=nothing, output__weight=head, token_embd__weight=embedding, output_norm__weight=norm)
    same(ctx, pkg, path, n, 600)


@pytest.mark.parametrize("spread", [8, 16])
@pytest.mark.parametrize("signs", ["one", "random"])
@pytest.mark.parametrize("embd,ff,n", [(512, ff, n) for ff in (1536, 8960, 16384) for n in (24, 40, 64, 120)] + [(2048, 16384, 512)])       # (the last: all of K in one range)
def test_sums_beyond_64_bits_over_ranges(ctx, pkg, tmp_path, spread, signs, embd, ff, n):
    """down projection: one gate for all, so that SwiGLU's result is that gate times the up rows"""
    path = gu.make_synthetic(tmp_path / "m.gguf", "tiny", seed=4, std=0.5, extra=["--layers", 1, "--embd", embd, "--heads", embd // 64, "--kv-heads", embd // 128, "--ff", ff, "--vocab", 600])

    def nothing(d, q):
        d[:] = 0

    def gate(d, q):
        d[:], q[:] = 0x2800, 0xFF                                         # 512 * 7 / 32 = 112 for an input of ones

    def up(d, q):
        if signs == "one":
            q[:] = 0xFF
            d[:] = 0x1400                                                 # 2^-10
        else:
            d[:] = d & 0x8000 | 0x2C00                                    # 2^-4
        low = np.arange(ff) // 32 % 8 == 3                                # every eighth block 13 binades below: one in each K range at least
        d[low] = d[low] & 0x8000 | (2 if signs == "one" else 128)

    def down(d, q):
        d[:] = d & 0xFF00 | 0xFF if signs == "random" else 0x03FF
        top_but_one(d, 1, spread)
        for b in range(5, ff // 32, 48):
            d[:, b] = d[:, 5]
        if signs == "one":
            q[::2], q[1::2] = 0x00, 0xFF

    def embedding(d, q):
        if signs == "one":
            d[:], q[:] = 0x3800, 0xFF

    def ones(w):
        w[:] = 1.0

    rewrite(path, blk__0__attn_output__weight=nothing, blk__0__ffn_gate__weight=gate, blk__0__ffn_up__weight=up, blk__0__ffn_down__weight=down, blk__0__ffn_norm__weight=ones,
            **({"token_embd__weight": embedding, "output__weight": embedding} if signs == "one" else {}))
    same(ctx, pkg, path, n, 600)


# Some rows and some tokens out of the digits' range, the rest within: one of each, a half, several rounds of the warps that sum them, all; every tile depth
@pytest.mark.parametrize("embd,ff", [(192, 352), (320, 1376), (384, 256), (512, 1024)])
@pytest.mark.parametrize("n,rows,tokens", [(20, 1, 0), (40, 0, 1), (64, 1, 1), (64, 9, 0), (64, 70, 3), (64, 0, 7), (65, 17, 20), (130, 400, 33), (24, 2, 24)])
def test_rows_and_tokens_out_of_range(ctx, pkg, tmp_path, embd, ff, n, rows, tokens):
    V = 600
    path = gu.make_synthetic(tmp_path / "m.gguf", "tiny", seed=embd + n, std=2.0, extra=["--layers", 2, "--embd", embd, "--heads", embd // 32, "--kv-heads", embd // 64, "--ff", ff, "--vocab", V, "--untied"])
    rng = np.random.default_rng(n + rows)

    def wide(d, q):
        r = rng.permutation(len(d))[:rows]
        d[r, -1] = lower(d[r, -1], 12)

    def embedding(d, q):                                              # the tokens that `same` draws last
        ids = np.random.default_rng(n).integers(0, V, n)[n - tokens:] if tokens else []
        for t in ids:
            d[t] += 4 << 10
            d[t, 1] = d[t, 1] & 0x8000 | 1 << 10

    def norm(w):
        w[:] = 200.0                                                  # the largest blocks' scales are above one, so that 2^-14 of them is not subnormal

    rewrite(path, token_embd__weight=embedding, blk__0__attn_norm__weight=norm, blk__0__ffn_norm__weight=norm, output_norm__weight=norm,
            **{t: wide for t in ("blk__0__attn_q__weight", "blk__0__attn_output__weight", "blk__1__ffn_up__weight", "blk__0__ffn_down__weight", "output__weight")})
    same(ctx, pkg, path, n, V)


# What is out of range must not cost more than the product over blocks: one token of a pass whose normed inputs are, and 1 % of every matrix's rows
@pytest.mark.parametrize("preset,n", [("1.5b", 333), ("3b", 64)])
@pytest.mark.parametrize("what", ["token", "rows"])
def test_time_of_passes_out_of_range(ctx, pkg, tmp_path, preset, n, what):
    std = 0.02 if what == "token" else 64.0
    path = gu.make_synthetic(tmp_path / "m.gguf", preset, seed=6, std=std, extra=["--layers", 3, "--vocab", 1500, "--untied"])

    def nothing(d, q):
        d[:] = 0

    def embedding(d, q):
        d[7] += 4 << 10
        d[7, 1] = d[7, 1] & 0x8000 | 1 << 10

    def wide(d, q):
        d[::100, 1] = lower(d[::100, 1], 18)

    def norm(w):
        w[:] = 4.0 / std

    rewrite(path, **{f"blk__{l}__{t}__weight": norm for l in range(3) for t in ("attn_norm", "ffn_norm")})
    if what == "token":                                               # (layers that add nothing: the norms see the embedding)
        rewrite(path, token_embd__weight=embedding, **{f"blk__{l}__{t}__weight": nothing for l in range(3) for t in ("attn_output", "ffn_down")})
    else:
        rewrite(path, **{f"blk__{l}__{t}__weight": wide for l in range(3) for t in ("attn_q", "attn_output", "ffn_gate", "ffn_up", "ffn_down")})
    m = pkg.Model(ctx, path, 400)
    seq = [7 if i == 10 else 8 + i for i in range(n)]
    ms = {}
    for which in (-1, 0):
        m.debug_products(which)
        if n > 64:
            ms[which] = min(m.prefill(seq, 0)[1] for _ in range(12))
        else:
            b = pkg.Batch(m, n, 8)
            ms[which] = min(b.step(seq, list(range(n)), [3] * n)[1] for _ in range(12))
            b.free()
    m.free()
    print(ms)
    assert ms[0] < 1.03 * ms[-1], ms

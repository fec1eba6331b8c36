"""Every product, attention and pass variant at the sizes where it can go wrong: the edges of its tiles, the remainders, the
smallest and largest of its range.  Products against the CPU oracle and, token by token, the GEMV; passes of many tokens against
the single-token decode kernel, as bits."""
import numpy as np
import pytest

import gguf_util as gu
import oracle_util as ou

pytestmark = pytest.mark.gpu


def rel_err(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-30))


def product_inputs(ctx, rows, cols, M):
    import torch
    rng = np.random.default_rng(rows * 7 + cols + M)
    raw = ou.quantize_q4_0((rng.standard_normal((rows, cols), dtype=np.float32) * 0.02))
    X = rng.standard_normal((M, cols), dtype=np.float32)
    w = ctx.upload_q4_0(raw, rows, cols)
    xq = torch.empty((M, cols), dtype=torch.int8, device="cuda")
    xd = torch.empty((M, cols // 32), dtype=torch.float16, device="cuda")
    ctx.quant_q8(torch.from_numpy(X).cuda(), xq, xd, n=cols, M=M)
    return raw, X, w, xq, xd


def gemv(ctx, w, xq, xd, rows):
    import torch
    y = torch.full((rows,), float("nan"), dtype=torch.float32, device="cuda")
    ctx.gemv_q4_q8(w, xq, xd, y)
    ctx.sync()
    return y.cpu().numpy()


# columns / 32: odd (tiles of one block), 2 mod 4, 4 mod 8, multiples of 8; fewer tiles than warps, as many, more; the most columns.
# Rows: a single one, a ragged group, and enough groups for the streaming kernel (the last two).
@pytest.mark.parametrize("rows,nb", [(1, 1), (33, 7), (64, 71), (31, 10), (96, 34), (257, 12), (33, 100), (32, 8), (255, 56), (100, 64), (33, 200), (64, 343), (65, 344),
                                     (75800, 9), (75777, 24)])
def test_gemv_matches_the_oracle(ctx, rows, nb):
    raw, X, w, xq, xd = product_inputs(ctx, rows, nb * 32, 1)
    eq, ed = ou.quant_q8(X[0])
    got = gemv(ctx, w, xq[0], xd[0], rows)
    assert np.array_equal(got, ou.gemv_q4_q8(raw, rows, nb * 32, eq, ed))


# depths whose activations fit one staging and depths that do not (K ranges and a second kernel), every tile depth, a last step
# of fewer than eight blocks, token groups of eight full and ragged
@pytest.mark.parametrize("rows,nb", [(33, 1), (40, 43), (96, 90), (777, 68), (1000, 344), (65, 343), (2049, 280)])
@pytest.mark.parametrize("M", [3, 8, 9, 16])
def test_m_token_product_equals_gemv(ctx, rows, nb, M):
    import torch
    raw, X, w, xq, xd = product_inputs(ctx, rows, nb * 32, M)
    bias = torch.randn(rows, device="cuda")
    Y = torch.full((M, rows), float("nan"), dtype=torch.float32, device="cuda")
    ctx.gemm_q4_q8(w, xq, xd, M, Y, bias=bias)
    ctx.sync()
    for m in (0, M // 2, M - 1):
        y = torch.empty(rows, dtype=torch.float32, device="cuda")
        ctx.gemv_q4_q8(w, xq[m], xd[m], y, bias=bias)
        ctx.sync()
        assert np.array_equal(Y[m].cpu().numpy(), y.cpu().numpy()), f"token {m}"


def attention_f64(q, K, V, n_head, n_kv, hd, pos):
    out = np.zeros(n_head * hd)
    for h in range(n_head):
        c = slice(h // (n_head // n_kv) * hd, (h // (n_head // n_kv) + 1) * hd)
        s = K[:pos + 1, c].astype(np.float64) @ q[h * hd:(h + 1) * hd].astype(np.float64)
        s = (s.astype(np.float32) * np.float32(1.0 / np.sqrt(np.float32(hd)))).astype(np.float64)
        w = np.exp(s - s.max())
        out[h * hd:(h + 1) * hd] = (w @ V[:pos + 1, c].astype(np.float64)) / w.sum()
    return out


# one chunk and several, ranges that end at, before and behind a step of 64 or 128 positions, blocks of four queries full and ragged
@pytest.mark.parametrize("n_head,n_kv,hd", [(16, 2, 128), (12, 2, 128), (7, 1, 64), (4, 2, 64), (2, 1, 32)])
@pytest.mark.parametrize("pos0,M", [(0, 2), (62, 3), (63, 1), (127, 5), (300, 16), (319, 1), (320, 7), (511, 2), (2047, 13)])
def test_attention_of_several_queries(ctx, n_head, n_kv, hd, pos0, M):
    import torch
    g = torch.Generator(device="cuda").manual_seed(pos0 + M + hd)
    K, V = (torch.randn((pos0 + M, n_kv * hd), generator=g, device="cuda").half() for _ in range(2))
    q = torch.randn((M, n_head * hd), generator=g, device="cuda") * 3
    out = torch.zeros_like(q)
    ctx.attn_splitkv(q, K.view(torch.int16), V.view(torch.int16), n_head, n_kv, hd, pos0, M, out)
    ctx.sync()
    for i in (0, M // 2, M - 1):
        want = attention_f64(q[i].cpu().numpy(), K.cpu().numpy(), V.cpu().numpy(), n_head, n_kv, hd, pos0 + i)
        assert rel_err(out[i].cpu().numpy(), want) < 1e-5, f"query {i}"


def model(tmp_path, preset, **sizes):
    extra = [a for k, v in sizes.items() for a in (f"--{k.replace('_', '-')}", v)]
    path = gu.make_synthetic(tmp_path / "m.gguf", preset, seed=11, extra=extra)
    return path, gu.GgufReader(path).config()["n_vocab"]


# embedding widths with tiles of one, two, four and eight blocks; two kv heads, and one (seven query heads per CTA group)
SHAPES = [dict(layers=2, embd=128, ff=352, heads=4, kv_heads=2, vocab=500), dict(layers=2, embd=896, ff=1216, heads=14, kv_heads=2, vocab=700)]


# token tiles of one and several groups, the last of the fused epilogues and the first of the separate ones, the largest pass, and two passes
@pytest.mark.parametrize("shape", range(len(SHAPES)))
@pytest.mark.parametrize("n", [1, 15, 16, 17, 32, 33, 65, 512, 513])
def test_prompt_passes_leave_the_state_that_decoding_leaves(ctx, pkg, tmp_path, shape, n):
    import torch
    path, V = model(tmp_path, "tiny", **SHAPES[shape])
    seq = [int(t) for t in np.random.default_rng(n).integers(0, V, n)]
    a, b = pkg.Model(ctx, path, n + 8), pkg.Model(ctx, path, n + 8)
    want, _ = a.decode(seq, n, 0)
    first, _ = b.prefill(seq, 0, chunk=16)
    assert first == want[-1]
    for name in ("kcache", "vcache"):
        assert torch.equal(a.state_tensor(name), b.state_tensor(name)), name
    la, lb = (torch.zeros((5, V), dtype=torch.float32, device="cuda") for _ in range(2))
    assert a.decode([first], 5, n, la)[0] == b.decode([first], 5, n, lb)[0]
    ctx.sync()
    assert torch.equal(la.view(torch.int32), lb.view(torch.int32))
    a.free(); b.free()


# the last and first sizes of the fused and the wide pass, a full pass, and a batch of two passes
@pytest.mark.parametrize("n", [2, 16, 17, 64, 65])
def test_batches_of_every_pass_size(ctx, pkg, tmp_path, n):
    import torch
    path, V = model(tmp_path, "tiny", **SHAPES[0])
    rng = np.random.default_rng(n)
    m = pkg.Model(ctx, path, 32)
    bt = pkg.Batch(m, n, 32)
    first = [int(t) for t in rng.integers(0, V, n)]
    lg = torch.zeros((n, V), dtype=torch.float32, device="cuda")
    t1, _ = bt.step(first, list(range(n)), [0] * n)
    t2, _ = bt.step(t1, list(range(n)), [1] * n, lg)
    for i in (0, n // 2, n - 1):
        ref = torch.zeros((2, V), dtype=torch.float32, device="cuda")
        assert m.decode([first[i]], 2, 0, ref)[0] == [t1[i], t2[i]], f"sequence {i}"
        ctx.sync()
        assert torch.equal(lg[i].view(torch.int32), ref[1].view(torch.int32)), f"sequence {i}"
    bt.free(); m.free()


# decoding across the change of attention kernel and of its chunks, on the builds for narrow and for wide models (and the general
# one), against passes of several tokens over the same cache
@pytest.mark.parametrize("shape", [SHAPES[0], SHAPES[1], dict(layers=1, embd=896, ff=1216, heads=14, kv_heads=2, vocab=700),
                                   dict(layers=2, embd=1536, ff=1024, heads=12, kv_heads=2, vocab=700), dict(layers=2, embd=2048, ff=1024, heads=16, kv_heads=2, vocab=700)])
@pytest.mark.parametrize("pos", [30, 248, 1500, 4733])
def test_decode_around_its_attention_ranges(ctx, pkg, tmp_path, shape, pos):
    import torch
    path, V = model(tmp_path, "tiny", **shape)
    n = 14
    m = pkg.Model(ctx, path, pos + n)
    gen = torch.Generator(device="cuda").manual_seed(pos)
    for name in ("kcache", "vcache"):
        m.state_tensor(name).view(torch.float16).normal_(generator=gen)
    torch.cuda.synchronize()
    seq = [int(t) for t in np.random.default_rng(pos).integers(0, V, n)]
    a, b = (torch.zeros((n, V), dtype=torch.float32, device="cuda") for _ in range(2))
    want, _ = m.verify(seq, pos, a)
    got, _ = m.decode(seq, n, pos, b)
    ctx.sync()
    assert got == want
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    m.free()


def test_arguments_of_the_per_matrix_calls(ctx, pkg):
    """Tensors and addresses are taken alike; wrong ones raise."""
    import torch
    raw, X, w, xq, xd = product_inputs(ctx, 64, 64, 2)
    y = torch.zeros((2, 64), device="cuda")
    ctx.gemv_q4_q8(w, xq[0], xd[0], y[0])
    ctx.gemv_q4_q8(w, xq[0].data_ptr(), xd[0].data_ptr(), y[1].data_ptr())
    ctx.sync()
    assert torch.equal(y[0], y[1])
    with pytest.raises(pkg.MinferError):
        ctx.quant_q8(None, xq, xd, n=64, M=1)
    with pytest.raises((TypeError, AttributeError)):
        ctx.quant_q8("not a tensor", xq, xd, n=64, M=1)

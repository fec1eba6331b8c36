"""Infinite and NaN scales of weights and activations: the M-token product gives what the GEMV gives, and the M-token pass what decoding gives."""
import numpy as np
import pytest

import gguf_util as gu
import oracle_util as ou

pytestmark = pytest.mark.gpu

INF, NINF, NAN, MAX = 0x7C00, 0xFC00, 0x7E01, 0x7BFF       # fp16 bits


def scales(raw, rows, nb):
    return raw.reshape(rows, nb, 18)[:, :, :2].view(np.uint16)[:, :, 0]


# products without and with a K split (kernel and cut), tile depths 1, 2, 4, 8, warps alone and in groups; a ragged last group and token group
@pytest.mark.parametrize("rows,nb", [(33, 7), (70, 34), (100, 12), (257, 48), (65, 344), (40000, 8)])
@pytest.mark.parametrize("M", [2, 9, 16])
def test_products_with_scales_that_are_not_finite(ctx, rows, nb, M):
    import torch
    rng = np.random.default_rng(rows + nb + M)
    raw = ou.quantize_q4_0((rng.standard_normal((rows, nb * 32), dtype=np.float32) * 0.02))
    d = scales(raw, rows, nb)
    d[0, 0] = INF
    d[1, nb - 1] = NINF
    d[2, nb // 2] = NAN
    d[3, 0], d[3, nb - 1] = INF, NINF
    d[4, 0], d[4, nb - 1] = INF, INF
    d[5, :] = INF
    d[6, nb // 2] = MAX                                    # the largest finite one
    d[rows - 1, nb - 1] = INF
    raw.reshape(rows, nb, 18)[7, 0, 2:] = 0x88             # nibbles 8: a block of zeros, with an infinite scale
    d[7, 0] = INF
    w = ctx.upload_q4_0(raw, rows, nb * 32)
    xq = torch.from_numpy(rng.integers(-127, 128, (M, nb * 32), dtype=np.int8)).cuda()
    xd = (rng.random((M, nb), dtype=np.float32) * 0.1).astype(np.float16)
    xd[0, 0] = 0.0                                         # infinity * 0
    xd[M - 1, nb - 1] = np.inf
    if M > 2:
        xd[1, 0] = np.nan
    xd = torch.from_numpy(xd).cuda()
    xq[M // 2, :32] = 0
    bias = torch.from_numpy(rng.standard_normal(rows).astype(np.float32)).cuda()
    Y = torch.zeros((M, rows), device="cuda")
    ctx.gemm_q4_q8(w, xq, xd, M, Y, bias=bias)
    for m in range(M):
        y = torch.zeros(rows, device="cuda")
        ctx.gemv_q4_q8(w, xq[m], xd[m], y, bias=bias)
        ctx.sync()
        got, want = Y[m].cpu().numpy(), y.cpu().numpy()
        assert np.array_equal(got, want, equal_nan=True), (m, np.flatnonzero(~((got == want) | (np.isnan(got) & np.isnan(want))))[:5])
        if m not in (0, 1, M - 1, M // 2):
            assert np.isinf(want[[0, 1]]).all() and np.isnan(want[2]) and np.isfinite(want[6])
    w.free()


def patched(path, name, edit):
    r = gu.GgufReader(path)
    _, _, off, nbytes = r.tensors[name]
    typ, rows, cols = r.shape(name)
    raw = r.tensor_bytes(name)
    edit(scales(raw, rows, cols // 32))
    with open(path, "r+b") as f:
        f.seek(off)
        f.write(raw.tobytes())


# rows of the vocabulary whose logits are infinite or NaN (products with and without a fold, 5 and 33 tokens); a gate row that puts an infinity into every
# token's activation, and a value row that puts one into the cache
@pytest.mark.parametrize("where", ["vocabulary", "gate", "value"])
@pytest.mark.parametrize("n", [5, 33])
def test_passes_with_scales_that_are_not_finite(ctx, pkg, tmp_path, where, n):
    import torch
    path = gu.make_synthetic(tmp_path / "m.gguf", "tiny", seed=3, extra=["--vocab", 3000])
    if where == "vocabulary":
        def edit(d):
            d[2000, 0], d[2500, 1], d[2999, 0] = INF, NINF, NAN
        patched(path, "output.weight", edit)
    else:
        def edit(d):
            d[5, 0] = INF
        patched(path, "blk.1.ffn_gate.weight" if where == "gate" else "blk.0.attn_v.weight", edit)
    a, b = pkg.Model(ctx, path, n + 2), pkg.Model(ctx, path, n + 2)
    seq = [int(t) for t in np.random.default_rng(n).integers(0, 1900, n)]
    la, lb = (torch.zeros((n, 3000), device="cuda") for _ in range(2))
    want, _ = a.decode(seq, n, 0, la)
    if n <= 16:
        got, _ = b.verify(seq, 0, lb)
        ctx.sync()
        assert got == want
        assert np.array_equal(la.cpu().numpy(), lb.cpu().numpy(), equal_nan=True)
        if where == "vocabulary":
            assert torch.isinf(la).any() and torch.isnan(la).any()
    else:
        last, _ = b.prefill(seq, 0)
        assert last == want[-1]
    for name in ("kcache", "vcache"):
        ka, kb = (m.state_tensor(name).view(torch.float16).cpu().numpy() for m in (a, b))
        assert np.array_equal(ka, kb, equal_nan=True), name
    a.free(); b.free()

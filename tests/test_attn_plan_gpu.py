"""The ways in which the attention of the M-token pass is cut (queries per CTA, chunks per range), where one gives way to the next."""
import numpy as np
import pytest

import gguf_util as gu
from test_kernel_edges_gpu import attention_f64, rel_err

pytestmark = pytest.mark.gpu


# one chunk and several (about 200 positions), ranges whose last chunk is ragged, one and four queries per CTA, the last block of four full and ragged
@pytest.mark.parametrize("n_head,n_kv,hd", [(16, 2, 128), (12, 2, 128), (14, 2, 64), (4, 2, 64), (2, 1, 32)])
@pytest.mark.parametrize("pos0,M", [(199, 1), (222, 3), (8190, 16), (8190, 13), (20001, 14), (32741, 5)])
def test_attention_of_every_cut(ctx, n_head, n_kv, hd, pos0, M):
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


# passes that fill the machine in different ways behind a context, against passes of one token: the same bits.  pos: around the ranges that captured passes
# are planned for (160, 512); behind 2000 and 5000 positions 96 tokens share CTAs in fours
@pytest.mark.parametrize("shape", [dict(embd=896, heads=14), dict(embd=1536, heads=12), dict(embd=2048, heads=16)])
@pytest.mark.parametrize("pos,n", [(150, 16), (158, 3), (505, 14), (2000, 96), (5000, 97), (100, 333)])
def test_passes_behind_a_context(ctx, pkg, tmp_path, shape, pos, n):
    import torch
    args = dict(shape, layers=2, ff=1024, kv_heads=2, vocab=700)
    extra = [a for k, v in args.items() for a in (f"--{k.replace('_', '-')}", v)]
    path = gu.make_synthetic(tmp_path / "m.gguf", "tiny", seed=11, extra=extra)
    a, b = pkg.Model(ctx, path, pos + n), pkg.Model(ctx, path, pos + n)
    gen = torch.Generator(device="cuda").manual_seed(pos)
    for name in ("kcache", "vcache"):
        a.state_tensor(name).view(torch.float16).normal_(generator=gen)
        b.state_tensor(name).copy_(a.state_tensor(name))
    torch.cuda.synchronize()
    seq = [int(t) for t in np.random.default_rng(pos).integers(0, 700, n)]
    want, _ = a.decode(seq, n, pos)
    if n <= 16:
        for _ in range(3):                            # plain, captured, replayed
            got, _ = b.verify(seq, pos)
            assert got == want
    else:
        last, _ = b.prefill(seq, pos)
        assert last == want[-1]
    for name in ("kcache", "vcache"):
        assert torch.equal(a.state_tensor(name), b.state_tensor(name)), name
    a.free(); b.free()


def test_captured_without_scratch(pkg):
    """A first call inside a stream capture, at a length that is cut elsewhere, allocates nothing."""
    import torch
    n_head, n_kv, hd, n = 12, 2, 128, 300
    K, V = (torch.randn((n, n_kv * hd), device="cuda").half() for _ in range(2))
    q = torch.randn((1, n_head * hd), device="cuda")
    out, ref = torch.zeros_like(q), torch.zeros_like(q)
    c = pkg.Context(0)
    c.use_torch_stream()
    c.attn_splitkv(q, K.view(torch.int16), V.view(torch.int16), n_head, n_kv, hd, 20, 1, out)         # the kernel is there, no scratch is
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        c.use_torch_stream()
        c.attn_splitkv(q, K.view(torch.int16), V.view(torch.int16), n_head, n_kv, hd, n - 1, 1, out)
    out.zero_()
    g.replay()
    c.use_torch_stream()
    c.attn_splitkv(q, K.view(torch.int16), V.view(torch.int16), n_head, n_kv, hd, n - 1, 1, ref)
    c.sync()
    assert rel_err(out[0].cpu().numpy(), attention_f64(q[0].cpu().numpy(), K.cpu().numpy(), V.cpu().numpy(), n_head, n_kv, hd, n - 1)) < 1e-5
    assert torch.equal(out, ref)
    del g
    c.close()

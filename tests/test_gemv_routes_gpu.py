"""The GEMV on both sides of every line between its two kernels (csrc/gemv.cu, stream_whole): the folded one, the streaming one with whole row groups,
and the streaming one in the K-split forms give the same bits, for single matrices and stacks, and the oracle's."""
import numpy as np
import pytest

import oracle_util as ou

pytestmark = pytest.mark.gpu


def random_q4(rng, blocks):
    raw = rng.integers(0, 256, (blocks, 18), dtype=np.uint8)
    raw[:, :2] = (rng.standard_normal(blocks) * 0.01).astype(np.float16).view(np.uint8).reshape(blocks, 2)
    return raw.reshape(-1)


# row groups (a last one of a single row) around 4, 8, 10 2/3, 14 and 16 per SM of 148; columns / 32 on both sides of eight and of 24 steps, whole and
# ragged steps, tile depths 1, 2, 4 and 8
@pytest.mark.parametrize("groups", [592, 593, 1184, 1185, 1577, 1579, 2071, 2072, 2368])
@pytest.mark.parametrize("nb", [33, 64, 66, 184, 188])
def test_every_route_gives_the_same_bits(ctx, groups, nb):
    import torch
    rng = np.random.default_rng(groups * 1000 + nb)
    rows, cols = groups * 32 - 31, nb * 32
    raw = random_q4(rng, rows * nb)
    w = ctx.upload_q4_0(raw, rows, cols)
    x = torch.from_numpy(rng.standard_normal(cols).astype(np.float32)).cuda()
    xq, xd = torch.empty(cols, dtype=torch.int8, device="cuda"), torch.empty(nb, dtype=torch.float16, device="cuda")
    ctx.quant_q8(x, xq, xd)
    bias = torch.from_numpy(rng.standard_normal(rows).astype(np.float32)).cuda()
    out = []
    for kw in (dict(), dict(ksplit=1), dict(ksplit=3), dict(variant=3)):
        y = torch.full((rows,), float("nan"), device="cuda")
        ctx.gemv_q4_q8(w, xq, xd, y, bias=bias, **kw)
        ctx.sync()
        out.append(y.cpu().numpy())
    for y in out[1:]:
        assert np.array_equal(out[0], y)
    pick = rng.choice(rows, 40, replace=False)
    pick[0], pick[1] = 0, rows - 1
    sel = np.ascontiguousarray(raw.reshape(rows, nb * 18)[pick]).reshape(-1)
    want = ou.gemv_q4_q8(sel, pick.size, cols, xq.cpu().numpy(), xd.cpu().numpy().view(np.uint16)) + bias.cpu().numpy()[pick]
    assert np.array_equal(out[0][pick], want)
    w.free()


@pytest.mark.parametrize("groups,count,nb", [(296, 2, 72), (197, 3, 72), (100, 20, 48), (100, 21, 48), (1, 600, 96)])
def test_stacks_take_the_same_lines(ctx, groups, count, nb):
    import torch
    rng = np.random.default_rng(groups + count)
    rows, cols = groups * 32 - 5, nb * 32
    raw = random_q4(rng, count * rows * nb)
    w = ctx.upload_q4_0(raw, rows, cols, count)
    x = torch.from_numpy(rng.standard_normal(cols).astype(np.float32)).cuda()
    xq, xd = torch.empty(cols, dtype=torch.int8, device="cuda"), torch.empty(nb, dtype=torch.float16, device="cuda")
    ctx.quant_q8(x, xq, xd)
    a, b = (torch.full((count, rows), float("nan"), device="cuda") for _ in range(2))
    ctx.gemv_q4_q8(w, xq, xd, a)
    ctx.gemv_q4_q8(w, xq, xd, b, ksplit=2)
    ctx.sync()
    assert torch.equal(a, b) and not torch.isnan(a).any()
    w.free()

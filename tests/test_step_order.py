"""Rows of the KV cache that one CTA of the decode kernel writes and another reads in the next step: the order comes from fences at the
greedy pick.  A missing fence shows in no result on this hardware, so the CPU test looks at the source; the GPU test runs the
cases in which every kind of CTA writes rows that every other kind reads."""
import re
from pathlib import Path

import numpy as np
import pytest

import gguf_util as gu

KERNEL = Path(__file__).resolve().parent.parent / "nano-inference_b200" / "csrc" / "decode_kernel.cuh"


def in_order(text, *patterns):
    at = 0
    for p in patterns:
        m = re.search(p, text[at:])
        assert m, f"{p} not found after {text[max(0, at - 80):at]!r}"
        at += m.end()


def test_rows_of_a_step_are_ordered_before_the_next_step():
    src = re.sub(r"//[^\n]*", "", KERNEL.read_text())
    pick = src[src.index("run_warp_job(ws, 4 * P.L"):src.index("s_tok = tok;")]
    # a GEMV CTA: release before its candidate, all candidates and the attention CTAs' words polled, acquire, barrier
    in_order(pick, r"__syncthreads\(\)", r"fence_acq_rel_gpu\(\)", r"pub\.shared\(my_cand", r"tw_poll\(", r"attdone_off", r"fence_acq_rel_gpu\(\)", r"__syncthreads_and\(")
    # an attention CTA: acquire before the layers of a step, release behind them
    main = src[src.index("attn_cta_main(const DecodeParams"):src.index("decode_kernel(const __grid_constant__")]
    in_order(main, r"rows_ordered\(P, tag0 - 1u, step - 1\)", r"for \(int l =", r"attention_split", r"fence_acq_rel_gpu\(\)", r"tw_st\(P\.xw \+ attdone_off")
    wait = src[src.index("bool rows_ordered("):src.index("attn_cta_main(const DecodeParams")]
    in_order(wait, r"tw_poll\(", r"fence_acq_rel_gpu\(\)", r"__syncthreads_and\(")
    # a chunk: its stores, a barrier, and a fence in the threads that announce them
    split = src[src.index("bool attention_split("):src.index("bool attention_short(")]
    in_order(split, r"P\.attn_part", r"__syncthreads\(\)", r"fence_acq_rel_gpu\(\)", r"pub\.local\(P\.xo\.attm", r"tw_poll\(", r"fence_acq_rel_gpu\(\)", r"__ldcg\(gp")


# 14 attention CTAs: with 9 to 13 chunks per kv head one of them writes the first kv head's rows; one layer: the rows of the step before are the next
# thing that is read; across 256 positions in one launch (stop rule) and in two; without attention CTAs
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [dict(layers=1, embd=896, ff=1216, heads=14, kv_heads=2), dict(layers=2, embd=896, ff=1216, heads=14, kv_heads=2),
                                   dict(layers=2, embd=1536, ff=1024, heads=12, kv_heads=2), dict(layers=1, embd=128, ff=352, heads=4, kv_heads=2)])
@pytest.mark.parametrize("pos,n,stop", [(240, 60, False), (240, 60, True), (380, 70, False)])
@pytest.mark.parametrize("attn_ctas", [True, False])
def test_long_runs_equal_single_steps(ctx, pkg, tmp_path, monkeypatch, shape, pos, n, stop, attn_ctas):
    import torch
    if not attn_ctas:
        monkeypatch.setenv("MINFER_ATTN_CTAS", "0")
    extra = [a for k, v in dict(shape, vocab=700).items() for a in (f"--{k.replace('_', '-')}", v)]
    path = gu.make_synthetic(tmp_path / "m.gguf", "tiny", seed=5, extra=extra)
    a, b = pkg.Model(ctx, path, pos + n), pkg.Model(ctx, path, pos + n)
    gen = torch.Generator(device="cuda").manual_seed(pos)
    for name in ("kcache", "vcache"):
        a.state_tensor(name).view(torch.float16).normal_(generator=gen)
        b.state_tensor(name).copy_(a.state_tensor(name))
    torch.cuda.synchronize()
    seq = [int(t) for t in np.random.default_rng(pos).integers(0, 700, n)]
    if stop:
        a.set_stop_token(699)                       # forced tokens are never the stop token's step: the run stays one launch
    la, lb = (torch.zeros((n, 700), dtype=torch.float32, device="cuda") for _ in range(2))
    got, _ = a.decode(seq, n, pos, la)
    want = []
    for i in range(n):                              # one call per token
        t, _ = b.decode([seq[i]], 1, pos + i, lb[i:i + 1])
        want += t
    ctx.sync()
    assert got == want
    assert torch.equal(la.view(torch.int32), lb.view(torch.int32))
    for name in ("kcache", "vcache"):
        assert torch.equal(a.state_tensor(name), b.state_tensor(name)), name
    a.free(); b.free()

"""What this library is used for, as cases whose speed is measured.

Every case is one pass through the public entry points of the package, on the model shapes and matrix sizes of the
benchmark configurations (Qwen2.5 0.5B / 1.5B / 3B shapes, all-q4_0 weights, q8_0 activations, fp16 KV cache).
Weights play the part of a checkpoint: a file written once per shape by the package's own synthetic-model writer.
Prompts, tokens, activations and cached keys and values come from the seed of the case.
"""
from __future__ import annotations

import math
import os
import subprocess
import tempfile
from pathlib import Path

import numpy as np
import torch

import __graft_entry__

SHAPES = {   # layers, embedding, feed-forward, query heads, kv heads, head dim
    "0.5b": (24, 896, 4864, 14, 2, 64),
    "1.5b": (28, 1536, 8960, 12, 2, 128),
    "3b": (36, 2048, 11008, 16, 2, 128),
}
VOCAB = 151936


def listed():
    return [
        # one projection of a host program that owns the layer loop: the key / value rows, the smallest matrix of the sweep
        dict(name="gemv kv 256x1536", kind="gemv", rows=256, cols=1536),
        # and a feed-forward matrix of the largest shape
        dict(name="gemv ffn 11008x2048", kind="gemv", rows=11008, cols=2048),
        # a few drafted tokens through one matrix, an odd number of them
        dict(name="gemm ffn 8960x1536 M7", kind="gemm", rows=8960, cols=1536, M=7),
        # attention of a host program over its own cache: eight drafted tokens behind a long context
        dict(name="attn 12/2x128 8100+8", kind="attn", shape="1.5b", pos=8100, M=8),
        # one token per call with the logits left on the GPU for the caller's sampler
        dict(name="decode 1.5b 1 token", kind="decode", shape="1.5b", pos=100, prompt=1, steps=1, logits=True),
        # a reply: the benchmark's headline, greedy tokens after a 64-token prompt
        dict(name="decode 1.5b 64 tokens", kind="decode", shape="1.5b", pos=64, prompt=1, steps=64, logits=False),
        # a reply behind a long document
        dict(name="decode 1.5b at 8192", kind="decode", shape="1.5b", pos=8192, prompt=1, steps=8, logits=False),
        # the small model from an empty cache: prompt and reply in one call
        dict(name="decode 0.5b 16+32", kind="decode", shape="0.5b", pos=0, prompt=16, steps=47, logits=False),
        # a prompt read in, not a multiple of anything
        dict(name="prefill 1.5b 333", kind="prefill", shape="1.5b", tokens=333),
        # drafted tokens scored in one pass, logits wanted
        dict(name="verify 1.5b M5 at 2000", kind="verify", shape="1.5b", pos=2000, M=5),
        # serving: sequences of different lengths decoded together
        dict(name="batch 3b x16", kind="batch", shape="3b", n=16, ctx=100),
        dict(name="batch 3b x64", kind="batch", shape="3b", n=64, ctx=40),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(("gemv", "gemm", "attn", "decode", "prefill", "verify", "batch"))
        shape = rng.choice(sorted(SHAPES))
        if kind in ("gemv", "gemm"):
            case = dict(kind=kind, rows=_log(rng, 256, VOCAB), cols=32 * _log(rng, 28, 344))
            if kind == "gemm":
                case["M"] = rng.randint(2, 16)
            if case["rows"] * case["cols"] > VOCAB * 2048:
                continue
        elif kind == "attn":
            case = dict(kind=kind, shape=shape, pos=_log(rng, 16, 32700), M=rng.randint(1, 16))
        elif kind == "decode":
            steps = _log(rng, 1, 64)
            case = dict(kind=kind, shape=shape, pos=_log(rng, 1, 32000), prompt=rng.randint(1, min(steps, 16)), steps=steps,
                        logits=steps <= 4 and rng.random() < 0.5)
        elif kind == "prefill":
            case = dict(kind=kind, shape=shape, tokens=_log(rng, 8, 512))
        elif kind == "verify":
            case = dict(kind=kind, shape=shape, pos=_log(rng, 1, 32000), M=rng.randint(1, 16))
        else:
            n = _log(rng, 2, 64)
            case = dict(kind=kind, shape=shape, n=n, ctx=_log(rng, 4, 100 if n <= 16 else 40))
        if _cost(case) <= most:
            return case


# ---- what a program has in hand before the call -----------------------------------------------------------------


class _State:
    pass


_kept = {}


def _package():
    return __graft_entry__.load_package()


def _context(torch_stream):
    """Models run on the library's own stream, single kernels on the stream of the tensors they work on."""
    if torch_stream not in _kept:
        ctx = _package().Context(0)
        if torch_stream:
            ctx.use_torch_stream()
        _kept[torch_stream] = ctx
    return _kept[torch_stream]


def _checkpoint(shape):
    """Path of the model file of a shape, written when it is not there yet."""
    folder = Path(tempfile.gettempdir()) / f"minfer_b200_models_{os.getuid()}"
    folder.mkdir(exist_ok=True)
    path = folder / f"{shape}.gguf"
    if not path.exists():
        part = folder / f"{shape}.{os.getpid()}.part"
        subprocess.run([str(_package().BIN_DIR / "gguf_synth"), str(part), "--preset", shape, "--seed", "1"], check=True,
                       stdout=subprocess.DEVNULL, stderr=subprocess.DEVNULL)
        os.replace(part, path)
    return path


class _Cache:
    """A model's keys or values as an array that keeps the model, which owns the memory, alive."""

    def __init__(self, model, name, shape):
        self.model = model
        data = model.state_tensor(name).data_ptr()
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f2", "data": (data, False), "version": 3, "strides": None}


def _model(s, shape, max_seq):
    s.model = _package().Model(_context(False), _checkpoint(shape), max_seq)
    L, kvd = SHAPES[shape][0], SHAPES[shape][4] * SHAPES[shape][5]
    s.cache = [torch.as_tensor(_Cache(s.model, n, (L, max_seq, kvd)), device="cuda") for n in ("kcache", "vcache")]


def _fill(s, pos, gen):
    """Keys and values of the `pos` positions that are cached already."""
    for c in s.cache:
        for layer in c:
            layer[:pos].normal_(generator=gen)


def _written(s, first, count):
    """The rows of the cache that a pass adds."""
    s.rows = [c[:, first:first + count] for c in s.cache]


def _matrix(gen, rows, cols):
    """Normal weights of std 0.02 as q4_0 blocks (ggml's rule: scale = signed largest value / -8), in the device layout."""
    raw = torch.empty((rows, cols // 32, 18), dtype=torch.uint8, device="cuda")
    step = max(1, (1 << 26) // cols)
    for r in range(0, rows, step):
        n = min(step, rows - r)
        x = torch.empty((n, cols // 32, 32), device="cuda").normal_(0.0, 0.02, generator=gen)
        d = x.gather(2, x.abs().argmax(2, keepdim=True)) / -8
        q = (x / torch.where(d == 0, torch.ones_like(d), d) + 8.5).clamp_(0, 15).to(torch.uint8)
        raw[r:r + n, :, :2] = d.to(torch.float16).view(torch.uint8)
        raw[r:r + n, :, 2:] = q[:, :, :16] | (q[:, :, 16:] << 4)
    return _context(True).repack_q4_0_dev(raw, rows, cols)


def prepare(case, seed):
    s = _State()
    s.case = case
    s.kind = kind = case["kind"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    if kind in ("gemv", "gemm"):
        M, rows, cols = case.get("M", 1), case["rows"], case["cols"]
        s.ctx = _context(True)
        s.w = _matrix(gen, rows, cols)
        s.M = M
        s.x = torch.empty((M, cols), device="cuda").normal_(generator=gen)
        s.xq = torch.empty((M, cols), dtype=torch.int8, device="cuda")
        s.xd = torch.empty((M, cols // 32), dtype=torch.float16, device="cuda")
        s.y = torch.empty((M, rows), device="cuda")
    elif kind == "attn":
        _, _, _, heads, kv, hd = SHAPES[case["shape"]]
        s.ctx = _context(True)
        s.heads, s.kv, s.hd = heads, kv, hd
        s.q = torch.empty((case["M"], heads * hd), device="cuda").normal_(generator=gen)
        s.k, s.v = (torch.empty((case["pos"] + case["M"], kv * hd), dtype=torch.float16, device="cuda").normal_(generator=gen) for _ in range(2))
        s.out = torch.empty_like(s.q)
    elif kind == "decode":
        s.tokens = rng.integers(0, VOCAB, case["prompt"]).astype(np.int32)
        _model(s, case["shape"], case["pos"] + case["steps"])
        _fill(s, case["pos"], gen)
        _written(s, case["pos"], case["steps"])
        s.logits = torch.empty((case["steps"], VOCAB), device="cuda") if case["logits"] else None
    elif kind == "prefill":
        s.tokens = rng.integers(0, VOCAB, case["tokens"]).astype(np.int32)
        _model(s, case["shape"], case["tokens"] + 1)
        _written(s, 0, case["tokens"])
    elif kind == "verify":
        s.tokens = rng.integers(0, VOCAB, case["M"]).astype(np.int32)
        _model(s, case["shape"], case["pos"] + case["M"])
        _fill(s, case["pos"], gen)
        _written(s, case["pos"], case["M"])
        s.logits = torch.empty((case["M"], VOCAB), device="cuda")
    else:
        n, ctx = case["n"], case["ctx"]
        s.model = _package().Model(_context(False), _checkpoint(case["shape"]), 1)
        s.batch = _package().Batch(s.model, n, ctx + 1)
        length = [ctx] + [int(v) for v in rng.integers(1, ctx + 1, n - 1)]
        text = rng.integers(0, VOCAB, (n, ctx + 1)).astype(np.int32)
        for p in range(ctx):                              # the sequences' own prompts, a token of each per step
            live = [i for i in range(n) if p < length[i]]
            s.batch.step(text[live, p], live, [p] * len(live))
        s.tokens, s.slots, s.positions = [int(text[i, length[i]]) for i in range(n)], list(range(n)), length
        s.logits = torch.empty((n, VOCAB), device="cuda")
    return s


# ---- the call -----------------------------------------------------------------------------------------------------


def run(s):
    case, kind = s.case, s.kind
    if kind == "gemv":
        s.ctx.quant_q8(s.x, s.xq, s.xd)
        s.ctx.gemv_q4_q8(s.w, s.xq, s.xd, s.y)
        return s.y, s.xq, s.xd
    if kind == "gemm":
        s.ctx.quant_q8(s.x, s.xq, s.xd, M=s.M)
        s.ctx.gemm_q4_q8(s.w, s.xq, s.xd, s.M, s.y)
        return s.y, s.xq, s.xd
    if kind == "attn":
        s.ctx.attn_splitkv(s.q, s.k, s.v, s.heads, s.kv, s.hd, case["pos"], case["M"], s.out)
        return s.out
    if kind == "decode":
        tokens, _ = s.model.decode(s.tokens, case["steps"], case["pos"], s.logits)
        if s.logits is not None:
            return np.array(tokens), s.logits, s.rows
        return np.array(tokens), s.model.margins(case["steps"]), s.rows
    if kind == "prefill":
        last, _ = s.model.prefill(s.tokens)
        return last, s.rows
    if kind == "verify":
        tokens, _ = s.model.verify(s.tokens, case["pos"], s.logits)
        return np.array(tokens), s.logits, s.rows
    tokens, _ = s.batch.step(s.tokens, s.slots, s.positions, s.logits)
    return np.array(tokens), s.logits


# ---- what a pass cannot do without ----------------------------------------------------------------------------------


def _shape_work(shape):
    """(weights of the layers, of the lm_head, cache bytes per position, attention flops per query and position)"""
    L, E, FF, H, KV, HD = SHAPES[shape]
    kvd = KV * HD
    return L * (2 * E * E + 2 * E * kvd + 3 * E * FF), VOCAB * E, 4 * L * kvd, 4 * L * H * HD


def work(case):
    kind = case["kind"]
    if kind in ("gemv", "gemm"):
        M, rows, cols = case.get("M", 1), case["rows"], case["cols"]
        return dict(bytes=rows * cols / 32 * 18 + M * (cols * 4 + cols / 32 * 34 + rows * 4), flops=2.0 * M * rows * cols)
    body, head, kv_bytes, att = _shape_work(case["shape"])
    if kind == "attn":
        _, _, _, heads, kv, hd = SHAPES[case["shape"]]
        M, pos = case["M"], case["pos"]
        return dict(bytes=(pos + M) * kv * hd * 4 + 2 * M * heads * hd * 4, flops=4.0 * heads * hd * sum(pos + i + 1 for i in range(M)))
    weights = (body + head) / 32 * 18
    if kind == "decode":
        ranges = [case["pos"] + i + 1 for i in range(case["steps"])]
        logits = 4 * VOCAB if case["logits"] else 0
        return dict(bytes=sum(weights + kv_bytes * r + logits for r in ranges), flops=sum(2.0 * (body + head) + att * r for r in ranges))
    if kind == "prefill":                                  # the lm_head is needed behind the last token only
        n = case["tokens"]
        return dict(bytes=weights + kv_bytes * n, flops=2.0 * (body * n + head) + att * n * (n + 1) / 2)
    if kind == "verify":
        M, pos = case["M"], case["pos"]
        return dict(bytes=weights + kv_bytes * (pos + M) + 4 * VOCAB * M, flops=2.0 * (body + head) * M + att * sum(pos + i + 1 for i in range(M)))
    n, ctx = case["n"], case["ctx"]
    return dict(bytes=weights + n * (kv_bytes * ctx / 2 + 4 * VOCAB), flops=n * (2.0 * (body + head) + att * ctx / 2))


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def tolerance(case):
    if case["kind"] in ("gemv", "gemm", "attn"):            # sums of exact products, fp32 results
        return dict(rel=1e-5)
    # whole models: an activation that lies on the edge of two int8 values moves the logits by about this much
    return dict(rel=1e-3, differ=0.01)

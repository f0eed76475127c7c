"""Timed cases of the framework: what its users run, through its public entry points.

A case is a plain dict:

  entry     "rope"    TiledSwaRope2D.apply: rotation and attention as one op on [B,H,N,d] tensors
            "packed"  TiledSwaPackedQKV.apply: the same between two projections, packed [B,N,3,H,d] in, [B,N,H*d] out
            "plain"   TiledSwa.apply (training) / tiled_swa_fwd (inference): attention without rotation
            "module"  FusedInplaceRotaryPositionEncoding2D on q and on k, then tiled_swa_fwd: the reference's own call
                      sequence, inference
  train     forward and backward (gradients of every input) or forward only
  dtype     "bf16", "fp16" or "fp32"
  B, H      batch and heads
  th, tw    grid of cells; b tokens per cell, N = th * tw * b
  wr, wc    window half sizes in cells: a token sees (2 wr + 1) x (2 wc + 1) cells, cut at the border
  dqk, dv   head dims
  rdim      rotated pairs per axis: the first 4 * rdim dims of q and k are rotated (0 with entry "plain")
  drop      share of tokens whose index is missing (-1: not rotated)
"""
import math
import random

import torch

import dl_templates_b200 as swa

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _case(name, entry, train, dtype, B, H, th, tw, wr, wc, dqk, dv, rdim=0, drop=0.0, b=1):
    c = dict(entry=entry, train=train, dtype=dtype, B=B, H=H, th=th, tw=tw, b=b, wr=wr, wc=wc, dqk=dqk, dv=dv, rdim=rdim,
             drop=drop)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # the smallest training step there is (configuration 1 of the benchmark, fp32): launches and host work
        _case("train_tiny_fp32_16x16", "rope", True, "fp32", 1, 2, 16, 16, 3, 3, 32, 32, rdim=8),
        # one small image through one layer at inference: latency of a single call
        _case("infer_small_24x24", "rope", False, "bf16", 1, 8, 24, 24, 3, 3, 64, 64, rdim=16),
        # batched inference (configuration 2)
        _case("infer_64x64_w13", "rope", False, "bf16", 4, 8, 64, 64, 6, 6, 64, 64, rdim=16),
        # a training step of a vision backbone at stage resolution, some tokens without a position (configuration 3)
        _case("train_56x56_w7_fp16", "rope", True, "fp16", 8, 12, 56, 56, 3, 3, 64, 64, rdim=16, drop=0.1),
        # wider values than keys, half of the dims rotated (configuration 4)
        _case("train_128x128_w15_dv128", "rope", True, "bf16", 4, 8, 128, 128, 7, 7, 64, 128, rdim=8),
        # the headline workload at a full GPU's batch
        _case("train_128x128_w13_bh256", "rope", True, "bf16", 16, 16, 128, 128, 6, 6, 64, 64, rdim=16),
        # one GPU's share of the largest configuration (256 x 256 tokens, 31 x 31 window, head dim 128)
        _case("train_256x256_w31_d128", "rope", True, "bf16", 2, 16, 256, 256, 15, 15, 128, 128, rdim=32),
        # a transformer block on a ragged grid between its two projections, packed tensors
        _case("train_packed_45x77_w9", "packed", True, "bf16", 2, 12, 45, 77, 4, 4, 64, 64, rdim=16),
        # the shape of the reference's own harness: cells of 16 tokens, head dim 32, no rotation
        _case("train_cells16_d32", "plain", True, "fp16", 4, 8, 16, 16, 1, 1, 32, 32, b=16),
        # full-precision training of a small model
        _case("train_fp32_40x40_w9", "rope", True, "fp32", 2, 4, 40, 40, 4, 4, 64, 64, rdim=16),
        # the reference's call sequence at inference: rotate q and k in place, then attend
        _case("infer_module_48x80_w11", "module", False, "bf16", 2, 16, 48, 80, 5, 5, 64, 64, rdim=16),
        # a head dim that is no multiple of 32, odd grid
        _case("train_33x47_d80", "rope", True, "fp16", 2, 8, 33, 47, 5, 5, 80, 80, rdim=16),
    ]


def _pairs_1d(n, reach):
    """Cell pairs (i, j) with |i - j| <= reach on a line of n cells."""
    return sum(min(n - 1, i + reach) - max(0, i - reach) + 1 for i in range(n))


def _flops(c):
    """Multiply-adds (x2) over the pairs of tokens that see each other, the window cut at the border: forward S and O;
    backward S, dP, dV, dQ, dK."""
    pairs = c["B"] * c["H"] * _pairs_1d(c["th"], c["wr"]) * _pairs_1d(c["tw"], c["wc"]) * c["b"] * c["b"]
    fwd = 2.0 * pairs * (c["dqk"] + c["dv"])
    return fwd + (2.0 * pairs * (3 * c["dqk"] + 2 * c["dv"]) if c["train"] else 0.0)


def work(case):
    rows = case["B"] * case["H"] * case["th"] * case["tw"] * case["b"]
    e = 4 if case["dtype"] == "fp32" else 2
    dqk, dv = case["dqk"], case["dv"]
    elems = rows * (2 * dqk + 2 * dv)                                # q, k, v in, o out
    if case["entry"] == "module":
        elems += rows * 2 * dqk                                      # q and k are written back rotated
    if case["train"]:
        elems += rows * (dv + 2 * dqk + dv)                          # do in; dq, dk, dv out
    extra = 0
    if case["rdim"]:
        extra = 4 * case["th"] * case["tw"] * case["b"] + 8 * case["rdim"] * (case["th"] + case["tw"] * case["b"])
    return {"bytes": e * elems + extra, "flops": _flops(case)}


def tolerance(case):
    # fp32: 32-bit sums.  16-bit: P and dS are rounded to the input type before they are contracted, and so are the outputs
    return {"rel": {"fp32": 1e-5, "fp16": 2e-3, "bf16": 1e-2}[case["dtype"]]}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    """Another case of the same ranges: every entry, type, direction, head dim, window and grid the listed ones stand for."""
    while True:
        entry = rng.choice(["rope", "rope", "rope", "packed", "plain", "module"])
        dtype = rng.choice(["bf16", "bf16", "bf16", "fp16", "fp16", "fp32"])
        train = entry != "module" and rng.random() < 0.7
        b = 1 if rng.random() < 0.75 else rng.choice([2, 4, 16])
        th, tw = _log_int(rng, 12, 192), _log_int(rng, 12, 192)
        if b > 1:
            th, tw = max(6, th // 4), max(6, tw // (2 * b))
        wr = rng.randint(1, 2) if b == 16 else rng.randint(1, 7) if rng.random() < 0.8 else rng.randint(8, 15)
        wc = wr if b == 1 and rng.random() < 0.8 else rng.randint(1, max(1, min(7, 24 // b)))
        if max(wr, wc) > 7 and b > 1:
            continue
        dqk = rng.choice([64] * 6 + [128] * 3 + [32, 32, 96, 96, 80, 48])
        dv = dqk if entry == "packed" or rng.random() < 0.8 else rng.choice([32, 64, 128])
        rdim = 0 if entry == "plain" else rng.choice([r for r in (8, 16, 32) if 4 * r <= dqk])
        drop = rng.choice([0.0, 0.0, 0.1]) if rdim else 0.0
        B, H = _log_int(rng, 1, 16), rng.choice([1, 2, 3, 4, 6, 8, 12, 16])
        c = _case(None, entry, train, dtype, B, H, th, tw, wr, wc, dqk, dv, rdim, drop, b)
        w = work(c)
        most = (3e9, 1.5e9) if dtype == "fp32" else (1.2e12, 2.4e9)     # never above the largest listed case's cost
        if w["flops"] <= most[0] and w["bytes"] <= most[1]:
            return c


class State:
    """What a program keeps around the op: inputs, the rotation's index and tables, the window."""


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    dtype = DTYPES[case["dtype"]]
    B, H, b, th, tw = case["B"], case["H"], case["b"], case["th"], case["tw"]
    N = th * tw * b
    g = torch.Generator(device=dev).manual_seed(seed)

    def normal(*shape):
        return torch.randn(shape, generator=g, device=dev, dtype=dtype)

    s = State()
    s.entry, s.train = case["entry"], case["train"]
    s.win = (b, th, tw, case["wr"], case["wc"], case["dqk"] ** -0.5)
    if s.entry == "packed":
        s.qkv = normal(B, N, 3, H, case["dqk"]).requires_grad_(s.train)
        s.do = normal(B, N, H * case["dv"]) if s.train else None
    else:
        s.q, s.k = (normal(B, H, N, case["dqk"]) for _ in range(2))
        s.v = normal(B, H, N, case["dv"])
        s.do = normal(B, H, N, case["dv"]) if s.train else None
        for t in (s.q, s.k, s.v):
            t.requires_grad_(s.train)
    s.rope, s.module = (None, None, None), None
    if case["rdim"]:
        idx = swa.FusedInplaceRotaryPositionEncoding2D.encode_idx(th, tw * b).to(dev)
        if case["drop"]:
            idx[torch.rand((N,), generator=g, device=dev) < case["drop"]] = -1
        s.module = swa.FusedInplaceRotaryPositionEncoding2D(2 * case["rdim"], th, tw * b).to(dev)
        s.rope = (idx, s.module.row_buffer.cs_components, s.module.col_buffer.cs_components)
    return s


def run(s):
    if s.entry == "module":
        with torch.no_grad():
            q, k = s.module(s.q, s.rope[0]), s.module(s.k, s.rope[0])
            return swa.tiled_swa_fwd(q, k, s.v, *s.win), q, k
    if s.entry == "packed":
        inputs, call = (s.qkv,), lambda: swa.TiledSwaPackedQKV.apply(s.qkv, *s.rope, *s.win)
    elif s.entry == "rope":
        inputs, call = (s.q, s.k, s.v), lambda: swa.TiledSwaRope2D.apply(s.q, s.k, s.v, *s.rope, *s.win)
    elif s.train:
        inputs, call = (s.q, s.k, s.v), lambda: swa.TiledSwa.apply(s.q, s.k, s.v, *s.win)
    else:
        return (swa.tiled_swa_fwd(s.q, s.k, s.v, *s.win),)
    if not s.train:
        with torch.no_grad():
            return (call(),)
    o = call()
    return (o.detach(), *torch.autograd.grad(o, inputs, s.do))

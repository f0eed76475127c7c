"""The roles of the strip kernels at the ends of what they hand each other: streams of blocks shorter and longer than the
batch the masking warp works out, the record rings and the rings of keys and values."""
import ctypes as C

import pytest
import torch
from test_gpu_strips import DEV
from test_gpu_strips import test_strips_against_simt as against_simt

import dl_templates_b200 as swa
from dl_templates_b200 import _lib
from oracle import swa_oracle as orc

pytestmark = pytest.mark.gpu


# (test_strip_handover.py looks that these plans have what can differ: rings of keys and values, score buffers, resident buffers)
STREAMS = [
    (1, 8, 1, 0, 0, 64, 64, 0, 1), (2, 8, 1, 1, 1, 64, 64, 16, 1), (5, 9, 1, 1, 1, 64, 64, 16, 149), (32, 8, 1, 0, 1, 64, 64, 8, 1),
    (33, 8, 1, 3, 3, 64, 64, 16, 2), (257, 8, 1, 2, 2, 64, 64, 16, 1), (4, 8, 1, 1, 1, 128, 128, 32, 1), (17, 24, 1, 9, 15, 128, 128, 32, 3),
    (70, 20, 1, 12, 12, 128, 128, 16, 60), (19, 31, 1, 7, 7, 128, 64, 16, 9), (40, 17, 1, 15, 15, 96, 96, 8, 40), (8, 8, 16, 1, 1, 32, 32, 0, 2)]


@pytest.mark.parametrize("th,tw,b,wr,wc,dqk,dv,R,BH", STREAMS)
def test_streams_of_any_length(th, tw, b, wr, wc, dqk, dv, R, BH):
    against_simt(th, tw, b, wr, wc, dqk, dv, R, BH)


@pytest.mark.parametrize("dtype,bound", [(torch.bfloat16, 1e-2), (torch.float16, 1.25e-3)])   # P and o rounded: 2^-9, 2^-12 of a value each
@pytest.mark.parametrize("th,tw,b,wr,wc,BH", [(5, 24, 1, 2, 0, 700), (7, 24, 1, 0, 0, 900), (6, 24, 1, 1, 0, 600), (13, 24, 1, 2, 5, 500), (9, 12, 4, 2, 1, 300),
                                              (81, 65, 1, 1, 0, 150), (9, 93, 1, 7, 0, 120), (63, 33, 1, 1, 1, 150)])
def test_quarters_that_one_group_does_alone(th, tw, b, wr, wc, BH, dtype, bound):
    """Windows at which one of the two softmax groups has no part in some quarters, many items per CTA: every row against the
    CUDA-core kernels, and the same bits every time."""
    N, win = th * tw * b, (b, th, tw, wr, wc)
    g = torch.Generator(device=DEV).manual_seed(th * 1000 + tw)
    q, k, v = (torch.randn(1, BH, N, 64, device=DEV, generator=g).to(dtype) for _ in range(3))
    o, lse = swa.swa_forward(q, k, v, None, *win, 0.125, impl="tc")
    o1, l1 = swa.swa_forward(q, k, v, None, *win, 0.125, impl="simt")
    swa.check_status()
    assert (lse - l1).abs().max().item() < 1e-3
    row = (o.float() - o1.float()).norm(dim=-1) / (o1.float().norm(dim=-1) + 0.3 * 8 * o1.float().pow(2).mean().sqrt())
    assert row.max().item() < 6 * bound, f"row {int(row.argmax())} off by {row.max().item():.2e}"
    assert ((o.float() - o1.float()).norm() / o1.float().norm()).item() < bound
    for _ in range(3):
        again, l2 = swa.swa_forward(q, k, v, None, *win, 0.125, impl="tc")
        assert torch.equal(again, o) and torch.equal(l2, lse)


@pytest.mark.parametrize("th,tw,b,wr,wc,dqk,dv,R,BH", [(70, 33, 1, 28, 15, 128, 128, 32, 3), (64, 21, 1, 31, 0, 96, 96, 16, 4), (61, 3, 16, 29, 2, 96, 96, 0, 2)])
def test_tall_windows_of_wide_heads(th, tw, b, wr, wc, dqk, dv, R, BH):
    """Largest blocks beside the softmax statistics of the resident rows: not a byte of shared memory to spare."""
    against_simt(th, tw, b, wr, wc, dqk, dv, R, BH)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("th,tw,wr,wc,dv", [(24, 24, 6, 6, 64), (19, 35, 6, 5, 64), (40, 9, 5, 6, 64), (27, 18, 7, 7, 128)])
def test_rows_whose_maximum_comes_late(th, tw, wr, wc, dv, dtype):
    """Keys far down the grid are large, the others small: a row's maximum grows by far more than 2^8 after the first block of either
    softmax group, its accumulator is rescaled and, where only later blocks show it, the block is done again.  The result is close to
    single rows of v, |v| < 4.8; P and the output, rounded to 8 (11) bits, are off by 2^-9 (2^-12) of it each."""
    q, k, v, do = orc.seeded_inputs(1, 2, th * tw, 64, dv, dtype, th + tw)
    row = torch.arange(th * tw) // tw
    plan = (C.c_int32 * 12)()
    g = _lib.make_geom(dtype, 1, 2, 1, th, tw, wr, wc, 64, dv, 0.125)
    assert _lib.lib.swa_describe_plan(C.byref(g), None, 0, plan) == 0
    R4, KR = 32 // plan[1], plan[2]
    for sel in (row >= th // 2, row % 9 >= 5, row == th - 1):
        ks = torch.where(sel[:, None], k.float() * 40., k.float() * 0.05).to(dtype)
        # rows for which that is certain: the keys of the two first blocks against the others, in powers of two
        s = (q[0, 0].double() @ ks[0, 0].double().T) * 0.125 * 1.4427
        seen = ((row[:, None] - row).abs() <= wr) & ((torch.arange(th * tw) % tw)[:, None] - torch.arange(th * tw) % tw).abs().le(wc)
        early = row[None] < ((row // R4 * R4 - wr).clamp(min=0) + 2 * KR)[:, None]
        first, rest = (s.masked_fill(~(seen & m), -1e30).amax(1) for m in (early, ~early))
        assert ((first > -1e30) & (rest > first + 16)).sum() >= tw // 2
        want = orc.fused_ref(q.float(), ks.float(), v.float(), do.float(), None, None, None, 1, th, tw, wr, wc, 0.125)[0]
        o, lse = swa.swa_forward(q.to(DEV), ks.to(DEV), v.to(DEV), None, 1, th, tw, wr, wc, 0.125, impl="tc")
        swa.check_status()
        assert torch.isfinite(lse).all()
        assert orc.max_abs(o.float().cpu(), want) < (2e-2 if dtype == torch.bfloat16 else 5e-3)

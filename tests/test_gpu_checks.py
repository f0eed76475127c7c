"""Calls whose tensors do not fit each other are refused by name before anything is launched: a short index, a table or a
tensor on the wrong device, saved tensors of another shape or type.  (A kernel would read past their ends, or a host
address.)"""
import pytest
import torch

from oracle import swa_oracle as orc

import dl_templates_b200 as swa
from dl_templates_b200 import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TH, TW, D = 6, 7, 64
N = TH * TW
WIN = (1, TH, TW, 2, 2)


def case(dtype=torch.bfloat16):
    q, k, v, do = (t.to(DEV) for t in orc.seeded_inputs(1, 2, N, D, D, dtype, 3))
    rope = tuple(t.to(DEV) for t in (orc.encode_idx(TH, TW), orc.make_cs_table(8, TH), orc.make_cs_table(8, TW)))
    return q, k, v, do, rope


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_refused_before_any_launch(dtype):
    q, k, v, do, rope = case(dtype)
    idx, row, col = rope
    short, cpu = (idx[:-1].contiguous(), row, col), (idx.cpu(), row, col)
    qkv = torch.stack([t.permute(0, 2, 1, 3) for t in (q, k, v)], 2).contiguous()
    o, lse = swa.swa_forward(q, k, v, None, *WIN, 0.125)
    back = lambda **kw: swa.swa_backward(*{**dict(q=q, k=k, v=v, o=o, lse=lse, do=do), **kw}.values(), None, *WIN, 0.125)
    noalloc = lambda rope=None, dq=None, **kw: swa.swa_backward_noalloc(*{**dict(q=q, k=k, v=v, o=o, lse=lse, do=do), **kw}.values(), rope, *WIN,
                                                                       0.125, torch.empty_like(q) if dq is None else dq, torch.empty_like(k),
                                                                       torch.empty_like(v))
    bad = [(AssertionError, f) for f in (
        lambda: swa.TiledSwaRope2D.apply(q, k, v, *short, *WIN, 0.125),
        lambda: swa.TiledSwaPackedQKV.apply(qkv, *short, *WIN, 0.125),
        lambda: swa.swa_forward(q, k, v, short, *WIN, 0.125),
        lambda: swa.swa_forward_rot(q, k, v, short, *WIN, 0.125),
        lambda: swa.swa_backward(q, k, v, o, lse, do, short, *WIN, 0.125),
        lambda: swa.swa_backward_rot(q, k, v, o, lse, do, short, *WIN, 0.125),
        lambda: noalloc(short),
        lambda: swa.swa_backward(q, k, v, o, lse, do, None, 1, TH + 1, TW, 2, 2, 0.125))]
    bad += [(RuntimeError, f) for r in (cpu, (idx, row.cpu(), col), (idx, row, col.cpu())) for f in (
        lambda r=r: swa.TiledSwaRope2D.apply(q, k, v, *r, *WIN, 0.125),
        lambda r=r: swa.TiledSwaPackedQKV.apply(qkv, *r, *WIN, 0.125),
        lambda r=r: swa.swa_forward(q, k, v, r, *WIN, 0.125),
        lambda r=r: swa.swa_backward_rot(q, k, v, o, lse, do, r, *WIN, 0.125),
        lambda r=r: swa.rope2d_apply_(q[0], *r),
        lambda r=r: swa.rope2d_apply_to(q[0], *r))]
    bad += [(RuntimeError, f) for f in (lambda: back(o=o.cpu()), lambda: back(lse=lse.cpu()), lambda: back(do=do.cpu()), lambda: back(k=k.cpu()),
                                        lambda: noalloc(lse=lse.cpu()), lambda: swa.tiled_swa_fwd(q, k.cpu(), v, *WIN))]
    bad += [(TypeError, f) for f in (lambda: back(do=do.double()), lambda: back(o=o.double()), lambda: back(lse=lse.double()))]
    bad += [(ValueError, f) for f in (lambda: back(do=do[:, :, 1:]), lambda: back(o=o[..., :32]), lambda: back(lse=lse[:, :1]),
                                      lambda: noalloc(dq=torch.empty_like(q)[:, :, 1:]), lambda: noalloc(lse=lse.transpose(1, 2).contiguous().transpose(1, 2)))]
    torch.cuda.synchronize()
    before = _lib.launch_count()
    for i, (kind, f) in enumerate(bad):
        with pytest.raises(kind):
            f()
            pytest.fail(f"call {i} was accepted")
    assert _lib.launch_count() == before
    # ... and what fits is still taken: a longer index, a softmax statistic that is a view
    want = swa.swa_backward(q, k, v, o, lse, do, None, *WIN, 0.125)
    got = back(lse=lse.transpose(1, 2).contiguous().transpose(1, 2))
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    longer = (torch.cat([idx, idx]), row, col)
    assert torch.equal(swa.swa_forward(q, k, v, longer, *WIN, 0.125)[0], swa.swa_forward(q, k, v, rope, *WIN, 0.125)[0])


@pytest.mark.parametrize("mode", ["handoff", "fused"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_tables_that_start_off_a_16_byte_boundary(dtype, mode):
    q, k, v, do, rope = case(dtype)
    off = [rope[0]]
    for t in rope[1:]:
        buf = torch.empty(t.numel() + 1, device=DEV)
        buf[1:] = t.flatten()
        off.append(buf[1:].view(t.shape))
        assert off[-1].data_ptr() % 16 and off[-1].is_contiguous()
    prev = swa.set_rope_mode(mode)
    try:
        res = []
        for r in (rope, off):
            t = [x.clone().requires_grad_(True) for x in (q, k, v)]
            out = swa.TiledSwaRope2D.apply(*t, *r, *WIN, 0.125)
            res.append((out.detach(), *torch.autograd.grad(out, t, do)))
    finally:
        swa.set_rope_mode(prev)
    assert all(torch.equal(a, b) for a, b in zip(*res))

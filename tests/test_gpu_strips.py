"""Strip kernels (no streamed rotation) at the sizes where their walk can go wrong: quarters of a strip that meet a
single block, grids lower than a quarter or a block, heights and widths that leave remainders, strips cut into chunks,
windows at which quarters just slide or just do not, several column blocks per band, many items per CTA."""
import pytest
import torch

from oracle import swa_oracle as orc

import dl_templates_b200 as swa

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("th,tw,b,wr,wc,dqk,dv,R,BH", [
    (64, 64, 1, 0, 0, 64, 64, 0, 40), (63, 33, 1, 1, 1, 64, 64, 16, 64), (130, 9, 1, 1, 2, 32, 32, 8, 300),
    (1, 200, 1, 0, 3, 64, 64, 16, 7), (3, 17, 1, 2, 2, 64, 64, 8, 5), (300, 7, 1, 2, 1, 64, 64, 16, 9),
    (41, 24, 1, 5, 5, 64, 64, 16, 30), (41, 24, 1, 6, 6, 64, 64, 16, 30), (41, 24, 1, 7, 7, 64, 64, 8, 30),
    (200, 16, 1, 3, 3, 64, 64, 16, 160), (37, 19, 1, 4, 2, 128, 128, 32, 20), (26, 40, 1, 12, 3, 96, 64, 16, 6),
    (9, 6, 16, 1, 3, 32, 64, 0, 12), (12, 10, 2, 1, 2, 64, 128, 0, 33)])
def test_strips_against_simt(th, tw, b, wr, wc, dqk, dv, R, BH):
    N = th * tw * b
    g = torch.Generator(device=DEV).manual_seed(th * 1000 + tw)
    q, k = (torch.randn(1, BH, N, dqk, device=DEV, generator=g).to(torch.bfloat16) for _ in range(2))
    v, do = (torch.randn(1, BH, N, dv, device=DEV, generator=g).to(torch.bfloat16) for _ in range(2))
    win, sc = (b, th, tw, wr, wc), dqk ** -0.5
    if R:
        rope = tuple(t.to(DEV) for t in (orc.encode_idx(th, tw * b), orc.make_cs_table(R, max(th, 2)), orc.make_cs_table(R, max(tw * b, 2))))
        o, lse, qr, kr = swa.swa_forward_rot(q, k, v, rope, *win, sc, impl="tc")
        got = (o, *swa.swa_backward_rot(qr, kr, v, o, lse, do, rope, *win, sc, impl="tc"))
        o1, l1, qs, ks = swa.swa_forward_rot(q, k, v, rope, *win, sc, impl="simt")
        want = (o1, *swa.swa_backward_rot(qs, ks, v, o1, l1, do, rope, *win, sc, impl="simt"))
    else:
        o, lse = swa.swa_forward(q, k, v, None, *win, sc, impl="tc")
        got = (o, *swa.swa_backward(q, k, v, o, lse, do, None, *win, sc, impl="tc"))
        o1, l1 = swa.swa_forward(q, k, v, None, *win, sc, impl="simt")
        want = (o1, *swa.swa_backward(q, k, v, o1, l1, do, None, *win, sc, impl="simt"))
    swa.check_status()
    assert (lse - l1).abs().max().item() < 1e-3
    for a, c, n in zip(got, want, ("o", "dq", "dk", "dv")):
        assert torch.isfinite(a.float()).all(), n
        err = (a.float() - c.float()).norm() / max(c.float().norm(), 0.1 * c.numel() ** 0.5)     # (a 1 x 1 window has dq = dk = 0)
        assert err < 1e-2, f"{n}: relative error {float(err):.2e}"
        # ... and row by row: one bad quarter, corner or last row is nothing to the norm of the whole.  Both sides round P, dS and the
        # result to bf16 (2^-9 of a value each, sums of up to 325 pairs); rows up to 1.9e-2 apart are seen, a wrong one is near 1
        row = (a.float() - c.float()).norm(dim=-1) / (c.float().norm(dim=-1) + 0.3 * dv ** 0.5 * max(c.float().pow(2).mean().sqrt().item(), 0.1))
        assert row.max().item() < 6e-2, f"{n}: row {int(row.argmax())} off by {row.max().item():.2e}"


@pytest.mark.parametrize("th,tw,b,wr,wc,dqk,dv,R,BH", [
    (16, 16, 1, 3, 3, 32, 32, 8, 2), (9, 13, 1, 0, 0, 64, 64, 0, 3), (1, 5, 1, 2, 2, 4, 8, 1, 2), (33, 17, 1, 4, 6, 64, 64, 16, 5), (7, 10, 1, 2, 2, 100, 36, 8, 1),
    (20, 9, 2, 2, 1, 80, 48, 16, 3), (6, 5, 16, 1, 2, 96, 128, 8, 2), (40, 21, 1, 12, 12, 128, 128, 32, 2), (11, 30, 1, 1, 14, 128, 64, 0, 2)])
def test_fp32_tiles_against_oracle(th, tw, b, wr, wc, dqk, dv, R, BH):
    """fp32 (tiled CUDA-core kernels): tiles cut at the grid's edge, halos in one and several bands, head dims that leave
    lanes idle, both rotation paths' common kernels."""
    N = th * tw * b
    q, k, v, do = orc.seeded_inputs(1, BH, N, dqk, dv, torch.float32, th)
    rope_cpu = (orc.encode_idx(th, tw * b), orc.make_cs_table(R, max(th, 2)), orc.make_cs_table(R, max(tw * b, 2))) if R else (None,) * 3
    win, sc = (b, th, tw, wr, wc), dqk ** -0.5
    want = orc.fused_ref(q.double(), k.double(), v.double(), do.double(), *(t if t is None or t.dtype == torch.int32 else t.double() for t in rope_cpu),
                         *win, sc)
    qd, kd, vd = (t.to(DEV).requires_grad_(True) for t in (q, k, v))
    o = swa.TiledSwaRope2D.apply(qd, kd, vd, *(t if t is None else t.to(DEV) for t in rope_cpu), *win, sc)
    got = (o.detach(), *torch.autograd.grad(o, (qd, kd, vd), do.to(DEV)))
    for a, c, n in zip(got, want, ("o", "dq", "dk", "dv")):
        err = (a.cpu().double() - c).norm() / max(c.norm(), 0.1 * c.numel() ** 0.5)
        assert err < 2e-6, f"{n}: relative error {float(err):.2e}"


@pytest.mark.parametrize("dqk,dv,R", [(80, 80, 16), (48, 48, 8), (8, 24, 0), (72, 104, 8), (120, 40, 16), (32, 32, 8), (96, 96, 16)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_head_dims_of_any_multiple_of_8_as_they_are(dqk, dv, R, dtype):
    """The autograd surface hands such head dims to the tensor-core kernels without padded copies: no launch but its own,
    results against the oracle."""
    th, tw, win, sc = 21, 26, (1, 21, 26, 3, 2), dqk ** -0.5
    q, k, v, do = orc.seeded_inputs(1, 2, th * tw, dqk, dv, dtype, dqk)
    rope = (orc.encode_idx(th, tw), orc.make_cs_table(R, th), orc.make_cs_table(R, tw)) if R else (None,) * 3
    want = orc.fused_ref(q.float(), k.float(), v.float(), do.float(), *rope, *win, sc)
    qd, kd, vd = (t.to(DEV).requires_grad_(True) for t in (q, k, v))
    rd = tuple(None if t is None else t.to(DEV) for t in rope)
    before = swa._lib.launch_count()
    o = swa.TiledSwaRope2D.apply(qd, kd, vd, *rd, *win, sc)
    got = (o.detach(), *torch.autograd.grad(o, (qd, kd, vd), do.to(DEV)))
    swa.check_status()
    assert swa._lib.launch_count() - before <= (6 if R else 4)
    assert swa.tiled_swa._mode_for(qd, vd, rd if R else None, (*win, sc)) == ("handoff" if R else "none")
    for a, c, n in zip(got, want, ("o", "dq", "dk", "dv")):
        assert orc.max_abs(a.float().cpu(), c) < 2e-2 and orc.mean_rel(a.float().cpu(), c) < 5e-3, n


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("wr,wc", [(2 ** 31 - 1, 2 ** 31 - 1), (3, 2 ** 27), (2 ** 30, 2 ** 27 + 3), (2 ** 30 - 1, 1)])
def test_windows_of_any_size_beyond_the_grid(wr, wc, dtype):
    """A half-size that reaches past the grid is the whole grid, also where (2 wc + 1) * b or r + wr does not fit 32 bits."""
    b, th, tw = 16, 6, 5
    q, k, v, do = (t.to(DEV) for t in orc.seeded_inputs(1, 2, th * tw * b, 64, 64, dtype, 5))
    got, want = [], []
    for res, win in ((got, (b, th, tw, wr, wc)), (want, (b, th, tw, min(wr, th), min(wc, tw)))):
        t = [x.clone().requires_grad_(True) for x in (q, k, v)]
        o = swa.TiledSwa.apply(*t, *win, 0.125)
        res += [o.detach(), *torch.autograd.grad(o, t, do)]
    swa.check_status()
    for a, c in zip(got, want):
        assert orc.max_abs(a.float(), c.float()) < (2e-6 if dtype == torch.float32 else 2e-2)


@pytest.mark.parametrize("what", ["q", "k", "v", "do"])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("th,tw,b,wr,wc,dqk,dv,R", [(9, 11, 1, 2, 1, 64, 64, 8), (6, 5, 4, 1, 1, 32, 96, 0), (14, 30, 1, 3, 3, 100, 36, 16)])
def test_fp32_rows_are_not_touched_by_what_they_do_not_see(th, tw, b, wr, wc, dqk, dv, R, bad, what):
    """One token with an infinity or a NaN: the tiled kernels spoil exactly the rows that the one-warp-per-token kernels, which look at
    nothing but a row's own window, spoil; all others keep their values.  (A last stride of 2 takes those kernels.)"""
    N = th * tw * b
    q, k, v, do = (t.to(DEV) for t in orc.seeded_inputs(1, 2, N, dqk, dv, torch.float32, th))
    {"q": q, "k": k, "v": v, "do": do}[what][0, 1, (th // 2 * tw + tw // 2) * b, 5] = bad
    rope = tuple(t.to(DEV) for t in (orc.encode_idx(th, tw * b), orc.make_cs_table(R, th), orc.make_cs_table(R, tw * b))) if R else None
    win, sc = (b, th, tw, wr, wc), dqk ** -0.5
    wide = lambda t: torch.empty(*t.shape[:3], 2 * t.shape[3], device=DEV)[..., ::2].copy_(t)
    res = []
    for f in (lambda t: t, wide):
        if R:
            o, lse, qr, kr = swa.swa_forward_rot(f(q), k, f(v), rope, *win, sc)
            res.append((o, lse, *swa.swa_backward_rot(f(qr), kr, f(v), o, lse, do, rope, *win, sc)))
        else:
            o, lse = swa.swa_forward(f(q), k, f(v), None, *win, sc)
            res.append((o, lse, *swa.swa_backward(f(q), k, f(v), o, lse, do, None, *win, sc)))
    spoiled = 0
    for a, c, n in zip(*res, ("o", "lse", "dq", "dk", "dv")):
        ok, ref = torch.isfinite(a), torch.isfinite(c)
        # (a score of -inf has weight 0 here; where it is the first of a window, the running maximum of the one-warp kernels is -inf too
        # and makes the row a NaN: they may then spoil more)
        assert torch.equal(ok | ref, ok) if bad == float("inf") and what in "qk" else torch.equal(ok, ref), n
        spoiled += int((~ok).any(-1).sum())
        ok = ok & ref
        assert (a[ok] - c[ok]).abs().max().item() < 1e-5, n
    assert spoiled > 0

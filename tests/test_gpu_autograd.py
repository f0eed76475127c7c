"""The call surface as torch's autograd sees it: autograd.Functions whose plain calls run natively.  What only the general
path can answer -- forward-mode tangents, functorch's transforms, tracing -- is refused or handled as for any other such
function, never answered without it."""
import pytest
import torch
import torch.autograd.forward_ad as fwAD

from oracle import swa_oracle as orc

import dl_templates_b200 as swa

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
TH, TW, D = 6, 7, 64
N = TH * TW
WIN = (1, TH, TW, 2, 2, 0.125)


def case(dtype=torch.bfloat16, seed=3):
    q, k, v, do = (t.to(DEV) for t in orc.seeded_inputs(1, 2, N, D, D, dtype, seed))
    rope = tuple(t.to(DEV) for t in (orc.encode_idx(TH, TW), orc.make_cs_table(8, TH), orc.make_cs_table(8, TW)))
    return q, k, v, do, rope


def calls(rope):
    packed = lambda q, k, v: torch.stack([t.permute(0, 2, 1, 3) for t in (q, k, v)], 2)
    module = swa.FusedInplaceRotaryPositionEncoding2D(16, TH, TW).to(DEV)
    return {"plain": lambda q, k, v: swa.TiledSwa.apply(q, k, v, *WIN),
            "rope": lambda q, k, v: swa.TiledSwaRope2D.apply(q, k, v, *rope, *WIN),
            "packed": lambda q, k, v: swa.TiledSwaPackedQKV.apply(packed(q, k, v), *rope, *WIN),
            "module": lambda q, k, v: module(q.clone(), rope[0])}


@pytest.mark.parametrize("entry", ["plain", "rope", "packed", "module"])
def test_forward_mode_tangents_are_refused(entry):
    q, k, v, do, rope = case()
    f = calls(rope)[entry]
    for grad_mode in (True, False):
        with torch.set_grad_enabled(grad_mode), fwAD.dual_level():
            dual = fwAD.make_dual(q, torch.ones_like(q))
            with pytest.raises((RuntimeError, NotImplementedError)):
                f(dual, k, v)
    with pytest.raises((RuntimeError, NotImplementedError)):
        torch.func.jvp(lambda x: f(x, k, v), (q,), (torch.ones_like(q),))
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda x: f(x, k, v).float().sum())(q)
    with pytest.raises(RuntimeError):
        torch.vmap(lambda x: f(x, k, v))(torch.stack([q, q]))


@pytest.mark.parametrize("entry", ["plain", "rope", "packed"])
def test_general_path_gives_what_the_native_one_gives(entry, monkeypatch):
    """The autograd.Function bodies against the native nodes, in every rotation mode: the same launches, so the same bits."""
    q, k, v, do, rope = case()
    f = calls(rope)[entry]
    cls = {"plain": swa.TiledSwa, "rope": swa.TiledSwaRope2D, "packed": swa.TiledSwaPackedQKV}[entry]
    assert issubclass(cls, torch.autograd.Function)

    def step():
        t = [x.clone().requires_grad_(True) for x in (q, k, v)]
        o = f(*t)
        return (o.detach(), *torch.autograd.grad(o, t, do if entry != "packed" else do.permute(0, 2, 1, 3).reshape(1, N, -1)))

    for mode in ("handoff", "fused", "prerotate"):
        prev = swa.set_rope_mode(mode)
        try:
            want = step()
            with monkeypatch.context() as m:
                m.setattr(cls, "apply", super(cls, cls).apply)
                got = step()
        finally:
            swa.set_rope_mode(prev)
        assert all(torch.equal(a, b) for a, b in zip(got, want)), mode


@pytest.mark.parametrize("entry", ["plain", "rope", "packed"])
def test_a_trace_holds_the_call_and_not_its_result(entry):
    q, k, v, do, rope = case()
    f = calls(rope)[entry]
    with torch.no_grad():
        traced = torch.jit.trace(lambda q, k, v: f(q, k, v), (q, k, v), check_trace=False)
        q2, k2, v2, _, _ = case(seed=4)
        assert torch.equal(traced(q2, k2, v2), f(q2, k2, v2))


@pytest.mark.parametrize("entry", ["plain", "rope", "packed"])
def test_saved_tensor_hooks_and_checkpointing(entry):
    """Saved tensors go through the hooks of the forward pass; recomputation gives the same gradients."""
    from torch.utils.checkpoint import checkpoint
    q, k, v, do, rope = case()
    f = calls(rope)[entry]
    res = []
    for wrap in (lambda *t: f(*t), lambda *t: checkpoint(f, *t, use_reentrant=False), lambda *t: checkpoint(f, *t, use_reentrant=True)):
        t = [x.clone().requires_grad_(True) for x in (q, k, v)]
        o = wrap(*t)
        o.float().square().sum().backward()
        res.append([o.detach(), *(x.grad for x in t)])
    packs = []
    with torch.autograd.graph.saved_tensors_hooks(lambda x: (packs.append(1), x.cpu())[1], lambda x: x.to(DEV)):
        t = [x.clone().requires_grad_(True) for x in (q, k, v)]
        o = f(*t)
    o.float().square().sum().backward()
    res.append([o.detach(), *(x.grad for x in t)])
    assert len(packs) >= 4
    for r in res[1:]:
        assert all(torch.equal(a, b) for a, b in zip(r, res[0]))

"""Tiled 2D sliding-window attention: the call surface of the reference's
``src/tiled_swa.py`` on top of the sm_100a C-ABI library.

Same names and argument order as the reference:

  ``TiledSwa.apply(q, k, v, b_size, t_height, t_width, row_size, col_size, sm_scale)``   (src/tiled_swa.py:604)
  ``tiled_swa_fwd(q, k, v, b_size, t_height, t_width, row_size, col_size, sm_scale=1.0)`` (src/tiled_swa.py:564)

plus the composed entry the reference does not have (RoPE-2D and attention as one
autograd function; q and k stay untouched, their gradients come back un-rotated):

  ``TiledSwaRope2D.apply(q, k, v, idx, row_cs_buffer, col_cs_buffer, b_size, t_height,
  t_width, row_size, col_size, sm_scale)``

Layout: ``q, k [B,H,N,d_qk]``, ``v, o [B,H,N,d_v]``, ``N = t_height*t_width*b_size``,
token ``n = (tile_row*t_width + tile_col)*b_size + s``; a query attends every token
of every tile within ``row_size`` rows and ``col_size`` columns of its own tile,
truncated at the grid border (src/tiled_swa.py:76-79,212-214,704-710).

Departures from reference quirks (none changes the mathematics): outputs take the
dtype and device of ``q`` (the reference hard-codes fp16 on the default device,
src/tiled_swa.py:608-609); ``dq`` comes back in ``q.dtype`` (reference: fp32,
src/tiled_swa.py:656); backward works for every ``b_size`` (reference raises
below 16, src/tiled_swa.py:660-661); the saved softmax statistic is fp32.
"""
from __future__ import annotations

import ctypes as C
import os

import torch

from . import _lib
from ._lib import native as _native
from .fused_rope2d import rope2d_apply_, rope2d_apply_to


def _status(device: torch.device) -> torch.Tensor:
    """Per-device int32 words (pinned host memory, mapped into the device) the tensor-core kernels write to when one
    of their bounded waits gives up; zero in normal operation.  Every call looks at them first, so a timed-out kernel
    does not go unnoticed by callers that never synchronise on it."""
    return _native.status_words(torch.cuda.current_device() if device.index is None else device.index)


def check_status(device=None) -> None:
    """Synchronise and raise if any kernel reported a timed-out wait."""
    _native.check_status()


def _geom(q, v, b_size, t_height, t_width, row_size, col_size, sm_scale, impl):
    B, H, N, d_qk = q.shape
    return _lib.make_geom(q.dtype, B, H, b_size, t_height, t_width, row_size, col_size, d_qk, v.shape[-1], sm_scale,
                          impl)


def _ref(x):
    return C.byref(x) if x is not None else None


def padded_head_dims(q, v, rope, b_size, t_height, t_width, row_size, col_size, sm_scale=1.0, impl="auto"):
    """``(d_qk', d_v')`` if zero-padding the head dims to 64 or 128 moves this problem from the SIMT kernels to
    the tensor-core kernels, else ``None``.  Padding q and k with zero columns leaves every score unchanged,
    padding v adds zero columns to O.  Without ``rope`` the tensor-core kernels take any multiple of 8 as it is; with it the
    answer is that of the kernels that rotate what they stream (``set_rope_mode("fused")``), which take 64 and 128."""
    return _native.padded_dims(q, v.shape[-1], *(rope or _NO_ROPE), b_size, t_height, t_width, row_size, col_size,
                               sm_scale, _lib.impl_code(impl))


_NO_ROPE = (None, None, None)


def swa_forward(q, k, v, rope, b_size, t_height, t_width, row_size, col_size, sm_scale, impl="auto", out=None):
    """Launch the forward kernel; returns ``(o, lse)`` with ``lse`` fp32 ``[B,H,N]`` in
    the base-2 domain.  ``rope`` is ``None`` or ``(idx, row_cs, col_cs)``.  ``out``: an
    optional ``[B,H,N,d_v]`` tensor or strided view the kernel writes O into (e.g. a view
    of a ``[B,N,H*d_v]`` buffer for the output projection)."""
    return _native.forward(q, k, v, *(rope or _NO_ROPE), b_size, t_height, t_width, row_size, col_size, sm_scale,
                           _lib.impl_code(impl), out)


def swa_backward(q, k, v, o, lse, do, rope, b_size, t_height, t_width, row_size, col_size, sm_scale, impl="auto",
                 out=None):
    """Launch delta, dQ and dK/dV kernels; returns ``(dq, dk, dv)`` in the input dtype
    (gradients of the un-rotated q and k when ``rope`` is given).  ``out``: optional
    ``(dq, dk, dv)`` tensors or strided views to write into (e.g. the three slices of one
    packed ``[B,N,3,H,d]`` gradient buffer)."""
    return _native.backward(q, k, v, o, lse, do, *(rope or _NO_ROPE), b_size, t_height, t_width, row_size, col_size,
                            sm_scale, _lib.impl_code(impl), 0, *(out or _NO_ROPE))


def swa_forward_rot(q, k, v, rope, b_size, t_height, t_width, row_size, col_size, sm_scale, impl="auto", out=None):
    """Forward with the rotation handed on (``swa_fwd_rot``): returns ``(o, lse, q_rot, k_rot)``.

    Every query and key row is rotated once by a streaming pass into ``q_rot`` / ``k_rot``; ``q`` and ``k`` stay
    untouched.  ``q_rot`` and ``k_rot`` are what ``swa_backward_rot`` takes in place of ``q`` and ``k`` -- the tensors
    the reference keeps for backward as well, since its RoPE rotates q and k in place (src/fused_rope2d.py:143-145).
    ``rope`` = ``(idx, row_cs, col_cs)`` is required; ``out`` as in ``swa_forward``."""
    return _native.forward_rot(q, k, v, *rope, b_size, t_height, t_width, row_size, col_size, sm_scale,
                               _lib.impl_code(impl), out)


def swa_backward_rot(q_rot, k_rot, v, o, lse, do, rope, b_size, t_height, t_width, row_size, col_size, sm_scale,
                     impl="auto", out=None):
    """Backward pass on the rotated copies ``swa_forward_rot`` left behind: delta, ``swa_bwd_dq_rot``,
    ``swa_bwd_dkdv_rot``.  Returns ``(dq, dk, dv)``, gradients of the UN-rotated q and k (the kernels rotate dq and
    dk back in their epilogues).  ``out`` as in ``swa_backward``."""
    return _native.backward(q_rot, k_rot, v, o, lse, do, *rope, b_size, t_height, t_width, row_size, col_size, sm_scale,
                            _lib.impl_code(impl), 1, *(out or _NO_ROPE))


def swa_backward_noalloc(q, k, v, o, lse, do, rope, b_size, t_height, t_width, row_size, col_size, sm_scale, dq, dk,
                         dv, impl="auto"):
    """Backward pass into caller-provided ``dq, dk, dv`` through ``swa_bwd_noalloc``: the library
    neither allocates nor frees anything, the softmax-delta scratch lives in a fixed array
    inside the library (limit: ``B*H*N <= _lib.NOALLOC_MAX_ROWS``).  Meant for callers that own
    no allocator (everything, outputs included, comes from memory they reserved up front).
    Calls on one device share that array, so do not let two of them overlap on the GPU; the
    first call on a device does a one-time address lookup and should come before any stream
    capture.  Returns ``(dq, dk, dv)``."""
    _native.check_backward(q, k, v, o, lse, do, *(rope or _NO_ROPE), b_size, t_height, t_width, row_size, col_size, sm_scale)
    if not lse.is_contiguous():
        raise ValueError("lse must be contiguous")
    for t, like, what in ((dq, q, "dq"), (dk, k, "dk"), (dv, v, "dv")):
        if t.shape != like.shape or t.dtype != like.dtype or t.device != like.device:
            raise ValueError(f"{what}: expected shape {tuple(like.shape)}, dtype {like.dtype} on {like.device}")
    g = _geom(q, v, b_size, t_height, t_width, row_size, col_size, sm_scale, impl)
    r = _lib.make_rope(*rope) if rope is not None else None
    tq, tk, tv, to, tdo, tdq, tdk, tdv = (_lib.tensor4(t) for t in (q, k, v, o, do, dq, dk, dv))
    with torch.cuda.device(q.device):
        code = _lib.lib.swa_bwd_noalloc(C.byref(g), _ref(r), C.byref(tq), C.byref(tk), C.byref(tv), C.byref(to),
                                        C.byref(tdo), lse.data_ptr(), C.byref(tdq), C.byref(tdk), C.byref(tdv),
                                        _status(q.device).data_ptr(), _lib.stream_ptr(q.device))
    _lib.check(code, "swa_bwd_noalloc")
    return dq, dk, dv


def selected_impl(q, v, rope, b_size, t_height, t_width, row_size, col_size, sm_scale=1.0, which=0, impl="auto"):
    """'tc' or 'simt': the kernel family ``swa_forward`` / ``swa_backward`` (``which``: 0 forward, 1 dQ, 2 dK/dV) run for these
    shapes as they are; where that is 'simt', ``padded_head_dims`` says whether the call is padded instead."""
    g = _geom(q, v, b_size, t_height, t_width, row_size, col_size, sm_scale, impl)
    r = _lib.make_rope(*rope) if rope is not None else None
    code = (_lib.lib.swa_step_select_impl if r is None else _lib.lib.swa_select_impl)(C.byref(g), _ref(r), which)
    if code < 0:
        _lib.check(code, "swa_select_impl")
    return {_lib.IMPL_SIMT: "simt", _lib.IMPL_TC: "tc"}[code]


def tiled_swa_fwd(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, b_size: int, t_height: int, t_width: int,
                  row_size: int, col_size: int, sm_scale: float = 1.0) -> torch.Tensor:
    """Forward only, no autograd graph (src/tiled_swa.py:564-600)."""
    return swa_forward(q, k, v, None, b_size, t_height, t_width, row_size, col_size, sm_scale)[0]


class TiledSwa(torch.autograd.Function):
    """``TiledSwa.apply(q, k, v, b_size, t_height, t_width, row_size, col_size, sm_scale)``
    -- src/tiled_swa.py:602-689.

    ``apply`` runs natively, here and in the two functions below (argument checks, launches and the autograd node in C++).
    ``forward`` and ``backward`` are the general path: what carries forward-mode tangents, runs under functorch's transforms,
    is being traced or has a Python dispatch of its own, which the native entry hands to ``Function.apply``."""

    apply = staticmethod(_native.tiled_swa)

    @staticmethod
    def forward(ctx, q, k, v, *win):
        o, lse = swa_forward(q, k, v, None, *win)
        ctx.save_for_backward(q, k, v, lse, o)
        ctx.win = win
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, lse, o = ctx.saved_tensors
        return (*swa_backward(q, k, v, o, lse, do, None, *ctx.win), *(None,) * 6)


_rope_mode = "handoff"
_ROPE_MODES = ("none", "handoff", "fused", "prerotate")      # index = code of the native layer


def set_rope_mode(mode: str) -> str:
    """How ``TiledSwaRope2D`` and ``TiledSwaPackedQKV`` apply the rotation; returns the previous mode.

    ``"handoff"`` (default): every q and k row is rotated exactly once, by a streaming pass that writes rotated
    copies (``swa_forward_rot``); all three attention kernels read the copies, which replace q and k among the
    tensors saved for backward (the reference keeps the same thing: its RoPE rotates q and k in place,
    src/fused_rope2d.py:143-145), and the backward kernels rotate dq and dk back in their epilogues
    (``swa_backward_rot``).  ``"fused"``: every kernel rotates the rows it streams in shared memory (no temporaries,
    but a row is rotated once per tile whose window holds it: 4.4x at a 13 x 13 window).  ``"prerotate"``: the
    reference's own composition (src/fused_rope2d.py:126-168 around src/tiled_swa.py:604) -- rotated copies,
    attention without RoPE, separate in-place inverse rotation of dq and dk.  A module-level switch like the
    reference's ``use_fused_na()`` / ``use_autotuner()`` toggles."""
    global _rope_mode
    if mode == "auto":
        mode = "handoff"
    if mode not in _ROPE_MODES[1:]:
        raise ValueError(f"rope mode must be one of {_ROPE_MODES[1:]}")
    prev, _rope_mode = _rope_mode, mode
    _native.set_rope_mode(_ROPE_MODES.index(mode))
    return prev


set_rope_mode(os.environ.get("SWA_ROPE_MODE", "handoff"))


def _mode_for(q, v, rope, win) -> str:
    """The mode a call runs in: 'none' without RoPE; head dims that only reach the tensor-core kernels through
    zero padding take the fused path (the padding lives there)."""
    return _ROPE_MODES[_native.rope_mode(q, v.shape[-1], *(rope or _NO_ROPE), *win)]


class TiledSwaRope2D(torch.autograd.Function):
    """RoPE-2D and the attention as one differentiable function:
    ``TiledSwaRope2D.apply(q, k, v, idx, row_cs_buffer, col_cs_buffer, b_size, t_height, t_width, row_size, col_size,
    sm_scale)``.

    Equivalent to ``TiledSwa.apply(rope(q, idx), rope(k, idx), v, ...)`` with
    ``rope`` = ``RotaryPE2D`` (src/fused_rope2d.py:124-168), but q and k are left
    unmodified and ``dq``/``dk`` are gradients of the un-rotated tensors (rotated back
    inside the backward kernels).  How the rotation itself is done: ``set_rope_mode``.
    ``idx`` may be ``None`` (no rotation).
    """

    apply = staticmethod(_native.tiled_swa_rope2d)

    @staticmethod
    def forward(ctx, q, k, v, idx, row_cs_buffer, col_cs_buffer, *win):
        rope = None if idx is None else (idx, row_cs_buffer, col_cs_buffer)
        if rope is not None:
            assert idx.shape[0] == q.shape[2] and row_cs_buffer.shape[1] == col_cs_buffer.shape[1]
        ctx.mode, ctx.win = _mode_for(q, v, rope, win), win
        if ctx.mode == "handoff":            # q, k are the rotated copies from here on: they are what backward needs
            o, lse, q, k = swa_forward_rot(q, k, v, rope, *win)
        elif ctx.mode == "prerotate":
            q, k = (rope2d_apply_to(t.reshape(-1, *t.shape[2:]), *rope).view(t.shape) for t in (q, k))
            o, lse = swa_forward(q, k, v, None, *win)
        else:
            o, lse = swa_forward(q, k, v, rope, *win)
        ctx.save_for_backward(q, k, v, lse, o, *(rope or ()))
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, lse, o, *rope = ctx.saved_tensors
        if ctx.mode == "handoff":
            grads = swa_backward_rot(q, k, v, o, lse, do, rope, *ctx.win)
        elif ctx.mode == "prerotate":
            dq, dk, dv = swa_backward(q, k, v, o, lse, do, None, *ctx.win)
            dq, dk = dq.contiguous(), dk.contiguous()
            for t in (dq, dk):
                rope2d_apply_(t.view(-1, *t.shape[2:]), *rope, inverse=True)
            grads = dq, dk, dv
        else:
            grads = swa_backward(q, k, v, o, lse, do, tuple(rope) or None, *ctx.win)
        return (*grads, *(None,) * 9)


class TiledSwaPackedQKV(torch.autograd.Function):
    """The op between a packed QKV projection and the output projection, without the
    permute / contiguous copies either side of it.

    ``TiledSwaPackedQKV.apply(qkv, idx, row_cs_buffer, col_cs_buffer, b_size, t_height,
    t_width, row_size, col_size, sm_scale)`` takes ``qkv [B, N, 3, H, d]`` -- the output of
    one ``Linear(C, 3*H*d)`` viewed, the layout the reference's RoPE self-test slices its
    strided q and k from (src/fused_rope2d.py:259-262) -- and returns ``o [B, N, H*d]``,
    the layout the output projection consumes.  The kernels read q, k, v through strided
    tensor maps and write O, and in backward the three slices of one packed
    ``[B, N, 3, H, d]`` gradient, in place; ``idx`` may be ``None`` (no rotation).
    Same mathematics as ``TiledSwaRope2D`` on the permuted views.
    """

    apply = staticmethod(_native.tiled_swa_packed)

    @staticmethod
    def forward(ctx, qkv, idx, row_cs_buffer, col_cs_buffer, *win):
        if qkv.dim() != 5 or qkv.shape[2] != 3:
            raise ValueError("expected qkv [B, N, 3, H, d]")
        B, N, _, H, d = qkv.shape
        q, k, v = (qkv[:, :, i].permute(0, 2, 1, 3) for i in range(3))
        rope = None if idx is None else (idx, row_cs_buffer, col_cs_buffer)
        ctx.handoff, ctx.win = _mode_for(q, v, rope, win) == "handoff", win
        o = torch.empty((B, N, H, d), dtype=qkv.dtype, device=qkv.device)
        _, lse, *rotated = (swa_forward_rot if ctx.handoff else swa_forward)(q, k, v, rope, *win, out=o.permute(0, 2, 1, 3))
        ctx.save_for_backward(qkv, lse, o, *(rope or ()), *rotated)      # (v is read from the packed tensor again)
        return o.view(B, N, H * d)

    @staticmethod
    def backward(ctx, do):
        qkv, lse, o, *rest = ctx.saved_tensors
        B, N, _, H, d = qkv.shape
        if do.stride(-1) != 1 or do.stride(1) % 8 or do.stride(0) % 8 or do.data_ptr() % 16:
            do = do.contiguous()
        q, k, v = (qkv[:, :, i].permute(0, 2, 1, 3) for i in range(3))
        dqkv = torch.empty((B, N, 3, H, d), dtype=qkv.dtype, device=qkv.device)
        outs = tuple(dqkv[:, :, i].permute(0, 2, 1, 3) for i in range(3))
        saved = (o.permute(0, 2, 1, 3), lse, do.view(B, N, H, d).permute(0, 2, 1, 3))
        if ctx.handoff:
            swa_backward_rot(*rest[3:], v, *saved, rest[:3], *ctx.win, out=outs)
        else:
            swa_backward(q, k, v, *saved, tuple(rest) or None, *ctx.win, out=outs)
        return (dqkv, *(None,) * 9)


_native.set_general(*(super(cls, cls).apply for cls in (TiledSwa, TiledSwaRope2D, TiledSwaPackedQKV)))

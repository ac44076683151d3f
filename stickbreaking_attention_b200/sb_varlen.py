"""``sb_attn_varlen``: stick-breaking attention over a packed variable-length batch.

Drop-in for ``stickbreaking_attention.sb_varlen.sb_attn_varlen`` (``sb_varlen/__init__.py:24-82``):
same argument order and meaning, same ``(o, rem)`` outputs, gradients for q, k, v from upstream
gradients of both outputs.
"""
from __future__ import annotations

import math

import torch

from . import ops


def _require_ends(cu_seqlens):
    """(Without them the native call takes a batch for a fixed-length one.)"""
    ops._require(cu_seqlens is not None, "a packed batch needs cu_seqlens")


class StickBreakingAttention:
    """The reference's name for the differentiable operator (``sb_varlen/__init__.py:24-68``); the autograd node itself is
    native (``csrc/sb_torch.cpp``)."""

    @staticmethod
    def apply(q, k, v, cu_seqlens, max_seqlens, inv_temp, attend_current, leading_zero):
        return sb_attn_varlen_(q, k, v, inv_temp, cu_seqlens, max_seqlens, attend_current, leading_zero)


def sb_attn_varlen(q, k, v, cu_seqlens, max_seqlens=None, inv_temp=None, zero_start=True,
                   attend_current=False):
    """q, k, v: ``(heads, total_tokens, head_dim)``; ``cu_seqlens``: cumulative sequence ends on the
    device, with a leading 0 iff ``zero_start``.  Returns ``o`` like q and ``rem (heads, total_tokens)``.

    ``max_seqlens`` is optional here (the reference requires it): it is only an upper bound that keeps
    the backward's scratch memory small; leaving it out costs memory, never a host synchronisation.
    The leading zero is verified on the device (see ``ops.check_status``) rather than with the
    reference's host-side ``assert cu_seqlens[0] == 0`` (``sb_varlen/__init__.py:72-74``).
    """
    _require_ends(cu_seqlens)
    if inv_temp is None:
        inv_temp = 1 / math.sqrt(q.size(-1))
    if torch.compiler.is_compiling():   # one traceable operator with its own autograd formula
        o, rem, _ = ops.functional_fwd(q, k, v, cu_seqlens, max_seqlens, inv_temp, attend_current, bool(zero_start))
        return o, rem
    return sb_attn_varlen_(q, k, v, inv_temp, cu_seqlens, max_seqlens, attend_current, bool(zero_start))


def sb_attn_varlen_(q, k, v, inv_temp, cu_seqlens, max_seqlens, attend_current, leading_zero=False):
    _require_ends(cu_seqlens)
    o, rem = ops.attention(q, k, v, cu_seqlens, max_seqlens, inv_temp, attend_current, leading_zero)
    return o, rem


class StickBreakingAttentionFused:
    """The fused form's operator by the same interface."""

    @staticmethod
    def apply(q, k, v, cu_seqlens, max_seqlens, inv_temp, attend_current, leading_zero):
        _require_ends(cu_seqlens)
        return ops.attention(q, k, v, cu_seqlens, max_seqlens, inv_temp, attend_current, leading_zero, fused=True)[0]


def sb_attn_varlen_fused(q, k, v, cu_seqlens, max_seqlens=None, inv_temp=None, zero_start=True,
                         attend_current=False):
    """Same arguments as ``sb_attn_varlen``; returns the single tensor ``o + rem[..., None] * v`` that the reference's
    callers compute from its two outputs (``tests/test_varlen.py:101``), without the extra passes over o and v."""
    _require_ends(cu_seqlens)
    if inv_temp is None:
        inv_temp = 1 / math.sqrt(q.size(-1))
    if torch.compiler.is_compiling():
        return ops.functional_fwd(q, k, v, cu_seqlens, max_seqlens, inv_temp, attend_current, bool(zero_start),
                                  fuse_rem_v=True)[0]
    return ops.attention(q, k, v, cu_seqlens, max_seqlens, inv_temp, attend_current, bool(zero_start), fused=True)[0]

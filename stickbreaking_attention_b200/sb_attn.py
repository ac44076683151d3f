"""``sb_attn``: stick-breaking attention over a fixed-length ``(batch, heads, tokens, head_dim)`` batch.

Drop-in for ``stickbreaking_attention.sb_attn.sb_attn`` (``sb_attn/__init__.py:16-64``).
"""
from __future__ import annotations

import math

import torch

from . import ops


class StickBreakingAttention:
    """The reference's name for the differentiable operator (``sb_attn/__init__.py:16-54``); the autograd node itself is
    native (``csrc/sb_torch.cpp``)."""

    @staticmethod
    def apply(q, k, v, inv_temp, attend_current=False):
        return sb_attn_(q, k, v, inv_temp, attend_current)


def sb_attn(q, k, v, inv_temp=None, zero_start=True, attend_current=False):
    """``zero_start`` is accepted and ignored, as in the reference (``sb_attn/__init__.py:57``)."""
    if inv_temp is None:
        inv_temp = 1 / math.sqrt(q.size(-1))
    if torch.compiler.is_compiling():   # one traceable operator with its own autograd formula
        o, rem, _ = ops.functional_fwd(q, k, v, None, None, inv_temp, attend_current)
        return o, rem
    return sb_attn_(q, k, v, inv_temp, attend_current=attend_current)


def sb_attn_(q, k, v, inv_temp, attend_current):
    o, rem = ops.attention(q, k, v, None, None, inv_temp, attend_current, False)
    return o, rem


class StickBreakingAttentionFused:
    """The fused form's operator by the same interface."""

    @staticmethod
    def apply(q, k, v, inv_temp, attend_current=False):
        return ops.attention(q, k, v, None, None, inv_temp, attend_current, False, fused=True)[0]


def sb_attn_fused(q, k, v, inv_temp=None, zero_start=True, attend_current=False):
    """Same arguments as ``sb_attn``; returns ``o + rem[..., None] * v`` (``tests/test_attn.py:64`` of the reference)."""
    if inv_temp is None:
        inv_temp = 1 / math.sqrt(q.size(-1))
    if torch.compiler.is_compiling():
        return ops.functional_fwd(q, k, v, None, None, inv_temp, attend_current, fuse_rem_v=True)[0]
    return ops.attention(q, k, v, None, None, inv_temp, attend_current, False, fused=True)[0]

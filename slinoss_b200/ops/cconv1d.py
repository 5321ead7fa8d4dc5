"""Depthwise causal conv1d on B200 (channel-last, stride-aware).

``cconv1d_b200(x, weight, bias, conv_state)`` is the mixer-facing form
(slinoss/layers/mixer.py:456 ``_apply_cconv_cuda``): ``x (b,T,C)`` -- possibly a
column slice of the input projection -- and ``conv_state (b,C,W-1)`` give
``(y (b,T,C), next_state (b,C,W-1))``.  ``activation="silu"`` fuses the
activation the mixer applies next (mixer.py:562).
"""

from __future__ import annotations

from typing import Optional, Tuple

import torch

from .. import _lib
from . import _trace


def _check(x, weight, conv_state, rank: str, ndim: int) -> None:
    """Raises for arguments the kernels cannot take; the native path has found something unusual."""
    if x.device.type != "cuda":
        raise ValueError("slinoss_b200 cconv1d requires CUDA tensors.")
    if x.ndim != ndim:
        raise ValueError(f"x must be {rank}. Got {tuple(x.shape)}.")
    C = int(x.shape[-1])
    if weight.ndim != 2 or int(weight.shape[0]) != C:
        raise ValueError(f"weight must be ({C}, width). Got {tuple(weight.shape)}.")
    W = int(weight.shape[1])
    if W not in (2, 3, 4):
        raise ValueError(f"conv width must be 2, 3 or 4. Got {W}.")
    want = (int(x.shape[0]), C, W - 1)
    if conv_state is not None and tuple(conv_state.shape) != want:
        raise ValueError(f"conv_state must be {want}. Got {tuple(conv_state.shape)}.")
    _lib.dtype_code(x.dtype)


@torch.compiler.disable
def cconv1d_b200(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None,
                 conv_state: Optional[torch.Tensor] = None, *,
                 activation: Optional[str] = None) -> Tuple[torch.Tensor, torch.Tensor]:
    if activation not in (None, "silu", "swish"):
        raise NotImplementedError("activation must be None, silu, or swish")
    if _trace.tracing():
        return _trace.recorded(lambda *a: cconv1d_b200(*a, activation=activation), x, weight, bias, conv_state)
    out = _lib.host().cconv1d(x, weight, bias, conv_state, activation is not None)
    if out is not None:
        return out
    _check(x, weight, conv_state, "(batch, T, channels)", 3)
    b, T, C = map(int, x.shape)
    if T == 0:
        W = int(weight.shape[1])
        nxt = (torch.zeros((b, C, W - 1), device=x.device, dtype=x.dtype) if conv_state is None
               else conv_state.to(x.dtype))
        return x.new_empty((b, 0, C)), nxt
    _lib.same_device(x, weight, bias, conv_state)
    raise ValueError(f"cconv1d: batch, channels and bias must fit x {tuple(x.shape)}.")


def cconv1d_update_b200(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None,
                        conv_state: Optional[torch.Tensor] = None, *, activation: Optional[str] = None,
                        inplace: bool = False) -> Tuple[torch.Tensor, torch.Tensor]:
    """One decode token of the depthwise causal conv: the contract of the reference's
    ``causal_conv1d_update`` as ``SLinOSSMixer._apply_causal_depthwise_conv_step`` uses it
    (slinoss/layers/mixer.py:614-676).  ``x (b, C)`` -- possibly a column slice of the input
    projection's one-token output -- and the rolling ``conv_state (b, C, W-1)`` give
    ``(y (b, C), next_state (b, C, W-1))`` with ``y = act(bias + w . [state, x])`` and
    ``next_state = [state[..., 1:], x]``.  ``inplace=True`` rolls ``conv_state`` in place and returns
    it (it must then be contiguous and of ``x``'s dtype).  Inference only (no autograd)."""
    if activation not in (None, "silu", "swish"):
        raise NotImplementedError("activation must be None, silu, or swish")
    out = _lib.host().cconv1d_update(x, weight, bias, conv_state, activation is not None, inplace)
    if out is not None:
        return out
    _check(x, weight, conv_state, "(batch, channels)", 2)
    _lib.same_device(x, weight, bias, conv_state)
    if inplace:
        raise ValueError("inplace=True needs a contiguous conv_state of x's dtype.")
    raise ValueError(f"cconv1d: batch, channels and bias must fit x {tuple(x.shape)}.")


__all__ = ["cconv1d_b200", "cconv1d_update_b200"]

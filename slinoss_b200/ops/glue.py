"""Mixer glue on B200: skip connection, ``(b,H,T,P) -> (b,T,H*P)`` re-layout and SiLU gate in one
pass each way (``SLinOSSMixer._apply_gate_skip``, slinoss/layers/mixer.py:585-599, which runs five
elementwise passes and a transposing copy in eager mode)."""

from __future__ import annotations

import torch

from .. import _lib
from . import _trace


@torch.compiler.disable
def gate_skip_b200(scan_y: torch.Tensor, scan_u: torch.Tensor, gate: torch.Tensor, skip: torch.Tensor) -> torch.Tensor:
    """``(scan_y + scan_u * skip)`` re-laid from ``(b,H,T,P)`` to ``(b,T,H*P)`` and multiplied by
    ``silu(gate)``; ``gate (b,T,H*P)`` may be a column slice of the input projection's output,
    ``skip (H*P,)``.  Differentiable in all four."""
    if _trace.tracing():
        return _trace.recorded(lambda *a: (gate_skip_b200(*a),), scan_y, scan_u, gate, skip)[0]
    out = _lib.host().gate_skip(scan_y, scan_u, gate, skip)
    if out is not None:
        return out
    if scan_y.device.type != "cuda":
        raise ValueError("slinoss_b200 gate_skip requires CUDA tensors.")
    if scan_y.ndim != 4 or tuple(scan_u.shape) != tuple(scan_y.shape):
        raise ValueError(f"scan_y and scan_u must be (batch,heads,T,P) and equal. Got {tuple(scan_y.shape)}, "
                         f"{tuple(scan_u.shape)}.")
    b, H, T, P = map(int, scan_y.shape)
    if tuple(gate.shape) != (b, T, H * P):
        raise ValueError(f"gate must be {(b, T, H * P)}. Got {tuple(gate.shape)}.")
    if skip.numel() != H * P:
        raise ValueError(f"skip must have {H * P} entries. Got {tuple(skip.shape)}.")
    if P % 8 != 0:
        raise ValueError(f"head dim must be a multiple of 8. Got {P}.")
    _lib.same_device(scan_y, scan_u, gate, skip)
    if T == 0:
        return scan_y.new_empty((b, 0, H * P))
    _lib.dtype_code(scan_y.dtype)
    raise ValueError(f"gate_skip: sizes must be positive. Got {tuple(scan_y.shape)}.")


__all__ = ["gate_skip_b200"]

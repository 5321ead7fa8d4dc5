"""SLinOSSScanPrep on B200: ``(value, params, bc) -> (U, M, K, B, C)``.

``scanprep_b200`` has the argument list of the reference's ``scanprep_cute``
(slinoss/ops/scanprep/cute/api.py:10) and the results of
``SLinOSSScanPrep._prepare_inputs_reference`` (slinoss/layers/scanprep.py:351).
Inputs may be column slices of the mixer's input projection (only the last
dimension has to be dense); nothing is copied on the host side.
"""

from __future__ import annotations

from typing import Optional

import torch

from .. import _lib
from ..types import ScanInputs
from . import _trace

PARAM_DIM = 13


@torch.compiler.disable
def scanprep_b200(value, params, bc, *, n_heads: int, d_state: int, d_head: int,
                  normalize_bc: bool = True, dt_min: float, dt_max: float, r_min: float,
                  r_max: float, theta_bound: float, k_max: float, eps: float, dt_bias, gamma_bias,
                  omega_bias, mix_r_bias, mix_theta_bias, mix_k_prev_bias, mix_k_curr_bias,
                  b_scale: Optional[torch.Tensor] = None,
                  c_scale: Optional[torch.Tensor] = None) -> ScanInputs:
    """Same keyword list as ``scanprep_cute`` (scanprep.py:359-384 shows the call)."""
    if normalize_bc and (b_scale is None or c_scale is None):
        raise ValueError("b_scale and c_scale are required when normalize_bc is set.")
    pars = (dt_bias, gamma_bias, omega_bias, mix_r_bias, mix_theta_bias, mix_k_prev_bias, mix_k_curr_bias)
    if normalize_bc:
        pars += (b_scale, c_scale)
    hyper = (dt_min, dt_max, r_min, r_max, theta_bound, k_max, eps)
    if _trace.tracing():
        def call(value, params, bc, *pars):
            names = ("dt_bias", "gamma_bias", "omega_bias", "mix_r_bias", "mix_theta_bias", "mix_k_prev_bias",
                     "mix_k_curr_bias", "b_scale", "c_scale")
            o = scanprep_b200(value, params, bc, n_heads=n_heads, d_state=d_state, d_head=d_head,
                              normalize_bc=normalize_bc, dt_min=dt_min, dt_max=dt_max, r_min=r_min, r_max=r_max,
                              theta_bound=theta_bound, k_max=k_max, eps=eps, **dict(zip(names, pars)))
            return o.U, o.M, o.K, o.B, o.C
        return ScanInputs(*_trace.recorded(call, value, params, bc, *pars))
    out = _lib.host().scanprep(value, params, bc, n_heads, d_state, d_head, normalize_bc, hyper, pars)
    if out is not None:
        return ScanInputs(*out)
    for name, t in (("value", value), ("params", params), ("bc", bc)):
        if t.device.type != "cuda":
            raise ValueError(f"slinoss_b200 scanprep requires CUDA tensors ({name} is on {t.device}).")
    if value.ndim != 3 or value.shape[-1] != n_heads * d_head:
        raise ValueError(f"value must be (batch, T, {n_heads * d_head}). Got {tuple(value.shape)}.")
    b, T = int(value.shape[0]), int(value.shape[1])
    if params.ndim != 3 or tuple(params.shape) != (b, T, n_heads * PARAM_DIM):
        raise ValueError(f"params must be (batch, T, {n_heads * PARAM_DIM}). Got {tuple(params.shape)}.")
    if bc.ndim != 5 or tuple(bc.shape) != (b, T, n_heads, 4, d_state):
        raise ValueError(f"bc must be (batch, T, heads, 4, d_state). Got {tuple(bc.shape)}.")
    if not (value.dtype == params.dtype == bc.dtype):
        raise TypeError("value, params and bc must share one dtype.")
    if T == 0:
        dev, dt = value.device, value.dtype
        return ScanInputs(U=torch.empty((b, n_heads, 0, d_head), device=dev, dtype=dt),
                          M=torch.empty((b, n_heads, 0, 2), device=dev, dtype=torch.float32),
                          K=torch.empty((b, n_heads, 0, 2, 2), device=dev, dtype=torch.float32),
                          B=torch.empty((b, n_heads, 0, 2 * d_state), device=dev, dtype=dt),
                          C=torch.empty((b, n_heads, 0, 2 * d_state), device=dev, dtype=dt))
    _lib.dtype_code(value.dtype)
    pars = tuple(p.to(device=value.device, dtype=torch.float32) for p in pars)
    pars = tuple(p.expand(n_heads) for p in pars[:7]) + pars[7:]
    out = _lib.host().scanprep(value, params, bc, n_heads, d_state, d_head, normalize_bc, hyper, pars)
    if out is not None:
        return ScanInputs(*out)
    raise ValueError("scanprep: the biases must be (heads,), the scales (heads, 2, d_state), and every size positive.")


__all__ = ["scanprep_b200"]

"""One-token mixer decode step on B200 (inference only).

``mixer_decode_step_b200`` follows the keyword list and return values of the reference's
``mixer_decode_step_cute`` (slinoss/ops/v2x2ssd/cute/decode.py:117-149) without its shape
limits (P = 64, N = 64, batch in {1,2,4,8,16}); the arithmetic is
``SLinOSSMixer._decode_step_reference`` (slinoss/layers/mixer.py:714-748).  The carried
state is kept in fp32; passing ``final_state_out=initial_states`` (and likewise
``b_last_out`` / ``u_last_out``) updates a ``ScanState`` in place.
"""

from __future__ import annotations

from typing import Optional, Tuple

import torch

from .. import _lib

_DTYPES = (torch.float32, torch.bfloat16, torch.float16)


def _like(name: str, t: torch.Tensor, shape, dtype, device) -> torch.Tensor:
    if tuple(t.shape) != tuple(shape):
        raise ValueError(f"{name} must be {tuple(shape)}. Got {tuple(t.shape)}.")
    if t.device != device:
        raise ValueError(f"{name} must be on {device}.")
    if dtype is not None and t.dtype != dtype:
        raise TypeError(f"{name} must be {dtype}. Got {t.dtype}.")
    if not t.is_contiguous():
        raise ValueError(f"{name} must be contiguous; got strides {t.stride()}.")
    return t


@torch.compiler.disable
def mixer_decode_step_b200(value, params, bc, gate, skip, *, initial_states=None, B_prev=None,
                           U_prev=None, dt_min: float, dt_max: float, r_min: float, r_max: float,
                           theta_bound: float, k_max: float, eps: float, dt_bias, gamma_bias,
                           omega_bias, mix_r_bias, mix_theta_bias, mix_k_prev_bias, mix_k_curr_bias,
                           b_scale: Optional[torch.Tensor] = None,
                           c_scale: Optional[torch.Tensor] = None, normalize_bc: bool = True,
                           output_dtype: Optional[torch.dtype] = None,
                           final_state_out: Optional[torch.Tensor] = None,
                           b_last_out: Optional[torch.Tensor] = None,
                           u_last_out: Optional[torch.Tensor] = None
                           ) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor, torch.Tensor]:
    """``value, gate (b,H,P)``, ``params (b,H,13)``, ``bc (b,H,4,N)``, ``skip (H,P)`` ->
    ``(gated (b, H*P), final_state (b,H,P,2N) fp32, b_last (b,H,2N), u_last (b,H,P))``."""
    if normalize_bc and (b_scale is None or c_scale is None):
        if value.device.type != "cuda":
            raise ValueError("slinoss_b200 decode step requires CUDA tensors.")
        raise ValueError("b_scale and c_scale are required when normalize_bc is set.")
    hyper = (dt_min, dt_max, r_min, r_max, theta_bound, k_max, eps)
    pars = (dt_bias, gamma_bias, omega_bias, mix_r_bias, mix_theta_bias, mix_k_prev_bias, mix_k_curr_bias)
    if normalize_bc:
        pars += (b_scale, c_scale)
    if (output_dtype is None or output_dtype is value.dtype) and value.is_contiguous() and params.is_contiguous() \
            and bc.is_contiguous() and gate.is_contiguous():
        out = _lib.host().decode_step(value, params, bc, gate, skip, initial_states, B_prev, U_prev, normalize_bc, hyper,
                                      pars, final_state_out, b_last_out, u_last_out)
        if out is not None:
            return out
    return _decode_general(value, params, bc, gate, skip, initial_states, B_prev, U_prev, normalize_bc, hyper, pars,
                           output_dtype, final_state_out, b_last_out, u_last_out)


@torch.no_grad()
def _decode_general(value, params, bc, gate, skip, initial_states, B_prev, U_prev, normalize_bc, hyper, pars,
                    output_dtype, final_state_out, b_last_out, u_last_out):
    """Arguments the native path does not take as they are: raises what is wrong with them, or converts the carried
    tensors and the skip weights to the dtypes the kernel reads."""
    if value.device.type != "cuda":
        raise ValueError("slinoss_b200 decode step requires CUDA tensors.")
    if value.ndim != 3:
        raise ValueError(f"value must be (batch, heads, P). Got {tuple(value.shape)}.")
    dev, dt = value.device, value.dtype
    if dt not in _DTYPES:
        raise TypeError(f"value must be float32, bfloat16 or float16. Got {dt}.")
    if output_dtype is not None and output_dtype != dt:
        raise TypeError("the decode step writes its output in the dtype of value.")
    b, H, P = map(int, value.shape)
    if bc.ndim != 4 or tuple(bc.shape[:3]) != (b, H, 4):
        raise ValueError(f"bc must be (batch, heads, 4, N). Got {tuple(bc.shape)}.")
    N = int(bc.shape[-1])
    value = _like("value", value, (b, H, P), dt, dev)
    params = _like("params", params, (b, H, 13), dt, dev)
    bc = _like("bc", bc, (b, H, 4, N), dt, dev)
    gate = _like("gate", gate, (b, H, P), dt, dev)
    skip = skip.reshape(H, P).to(device=dev, dtype=dt).contiguous()
    if (B_prev is None) != (U_prev is None):
        raise ValueError("B_prev and U_prev must be passed together (or both omitted).")
    if initial_states is not None:
        initial_states = _like("initial_states", initial_states, (b, H, P, 2 * N), None, dev).to(torch.float32)
    if B_prev is not None:
        B_prev = _like("B_prev", B_prev, (b, H, 2 * N), None, dev).to(dt)
        U_prev = _like("U_prev", U_prev, (b, H, P), None, dev).to(dt)
    if final_state_out is not None:
        _like("final_state_out", final_state_out, (b, H, P, 2 * N), torch.float32, dev)
    if b_last_out is not None:
        _like("b_last_out", b_last_out, (b, H, 2 * N), dt, dev)
    if u_last_out is not None:
        _like("u_last_out", u_last_out, (b, H, P), dt, dev)
    pars = tuple(p.to(device=dev, dtype=torch.float32) for p in pars)
    pars = tuple(p.expand(H) for p in pars[:7]) + pars[7:]
    out = _lib.host().decode_step(value, params, bc, gate, skip, initial_states, B_prev, U_prev, normalize_bc, hyper,
                                  pars, final_state_out, b_last_out, u_last_out)
    if out is None:
        raise ValueError("decode step: the biases must be (heads,) and the scales (heads, 2, N), and every size positive.")
    return out


__all__ = ["mixer_decode_step_b200"]

"""Sizes at which the kernels' tilings and the dispatch between them change, against the float64 oracle."""

from __future__ import annotations

import types

import numpy as np
import pytest
import torch

import test_decode_gpu as decode_cases
import test_prep_conv_gpu as prep_cases
from gpu_util import SCAN_GRADS, make_scan_inputs, oracle_fwd_bwd, run_b200_fwd_bwd, to_np
from util import rel_err

pytestmark = pytest.mark.gpu

F32, BF16, F16 = torch.float32, torch.bfloat16, torch.float16


def _scan_errors(inp, run):
    Y, fin, grads = run()
    Yo, fino, go = oracle_fwd_bwd(inp)
    errs = {"Y": rel_err(to_np(Y), Yo), "final": rel_err(to_np(fin), fino)}
    errs.update({k: rel_err(to_np(grads[k]), go[k]) for k in SCAN_GRADS if grads[k] is not None})
    return errs


@pytest.mark.parametrize("L,T,N,P,dtype", [
    (16, 47, 2, 1, F32), (16, 48, 17, 33, F32),      # one row per thread; head tiles of 32 and 64, one slab and two
    (32, 33, 16, 32, F32), (32, 95, 40, 64, F16),
    (64, 64, 15, 31, F32), (64, 129, 33, 64, F32),   # last chunk full, last chunk of one token
    (128, 127, 16, 32, F32), (128, 130, 20, 48, BF16),
])
def test_cuda_core_chunks_as_requested(L, T, N, P, dtype, monkeypatch):
    import slinoss_b200 as sb

    op = sb.v2x2ssd_b200
    monkeypatch.setattr(sb, "v2x2ssd_b200", lambda *a, **kw: op(*a, retile=False, **kw))
    inp = make_scan_inputs(1, 2, T, N, P, dtype, seed=L + T, streaming=True, with_init=True)
    errs = _scan_errors(inp, lambda: run_b200_fwd_bwd(inp, L))
    assert max(errs.values()) < (1e-5 if dtype == F32 else 2e-2), errs


@pytest.mark.parametrize("b,h,T", [(1, 1, 40), (2, 80, 65)])   # tiled in 32 tokens; in 64
def test_cuda_core_tiling_follows_the_work(b, h, T):
    inp = make_scan_inputs(b, h, T, 4, 8, F32, seed=h, streaming=True, with_init=True)
    errs = _scan_errors(inp, lambda: run_b200_fwd_bwd(inp, 128))
    assert max(errs.values()) < 1e-5, errs


@pytest.mark.parametrize("dtype,N,T", [(BF16, 64, 129), (F16, 128, 256)])
def test_states_and_rows_in_the_activation_dtype(dtype, N, T):
    """Carried state, its gradient and the streaming rows are read and written in their own dtype."""
    inp = make_scan_inputs(1, 2, T, N, 64, dtype, seed=T, streaming=True, with_init=True)
    inp["initial_states"] = inp["initial_states"].to(dtype)
    errs = _scan_errors(inp, lambda: run_b200_fwd_bwd(inp, 128))
    assert max(errs.values()) < 2e-2, errs


@pytest.mark.parametrize("dtype,N,P,H,b,T", [
    (BF16, 16, 32, 4, 1, 37),      # four lanes per row
    (F16, 32, 64, 4, 2, 65),       # eight; rows aligned to 8 bytes only
    (BF16, 128, 64, 8, 1, 100),    # sixteen
    (F32, 128, 64, 4, 1, 50),      # thirty-two
    (F32, 8, 16, 4, 1, 19),
])
def test_prep_lane_groups(dtype, N, P, H, b, T):
    prep_cases.test_prep_seeded_vs_oracle(dtype, N, P, H, b, T)


@pytest.mark.parametrize("dtype", [BF16, F32])
def test_prep_parameters_in_half_precision(dtype):
    """bf16 parameters give what their values in fp32 give; gradients are rounded once."""
    H, N, P, b, T = 4, 32, 64, 2, 70
    gen = torch.Generator().manual_seed(3)
    r = lambda *s: torch.randn(*s, generator=gen)
    value, params, bc = r(b, T, H * P).to(dtype).cuda(), r(b, T, H * 13).to(dtype).cuda(), r(b, T, H, 4, N).to(dtype).cuda()
    pars = {n: (0.5 * r(H)).to(BF16).cuda() for n in prep_cases.BIAS_NAMES}
    pars.update({n: (1 + 0.3 * r(H, 2, N)).to(BF16).cuda() for n in ("b_scale", "c_scale")})
    hp = dict(dt_min=1e-4, dt_max=1e-1, r_min=0.9, r_max=1.0, theta_bound=float(np.pi), k_max=0.5, eps=1e-8)
    shapes = [(b, H, T, P), (b, H, T, 2), (b, H, T, 2, 2), (b, H, T, 2 * N), (b, H, T, 2 * N)]
    gouts = [r(*s).to(d).cuda() for s, d in zip(shapes, (dtype, F32, F32, dtype, dtype))]
    run = lambda p: prep_cases._run_prep(value.clone(), params.clone(), bc.clone(), p, hp, H, N, P, gouts)
    outs, grads = run(pars)
    outs32, grads32 = run({k: v.detach().float() for k, v in pars.items()})
    assert all(torch.equal(x, y) for x, y in zip(outs, outs32))
    for x, y in zip(grads, grads32):
        assert torch.equal(x, y.to(x.dtype))


@pytest.mark.parametrize("b,H,P,N,dtype", [
    (1000, 16, 8, 4, F32),       # more than 32 heads per CTA: the coefficients are made in groups
    (1, 1, 1, 2, F32),
    (2, 3, 33, 66, BF16),        # rows and items one past a step
    (37, 16, 64, 130, F16),      # several steps per row, more heads than CTAs
])
def test_decode_walk_over_heads(b, H, P, N, dtype):
    tol = {F32: 1e-5, BF16: 2e-2, F16: 5e-3}[dtype]
    decode_cases.test_decode_vs_oracle_and_in_place(b, H, P, N, dtype, tol)


def test_decode_half_parameters_and_strided_rows():
    import slinoss_b200 as sb

    b, H, P, N = 3, 4, 64, 32
    case, biases, cfg = decode_cases._random_case(b, H, P, N, BF16, seed=1)
    dev = {k: v.cuda() for k, v in case.items()}
    for k in ("b_scale", "c_scale"):
        dev[k] = dev[k].to(BF16)
    bias = {k: v.to(BF16).cuda() for k, v in biases.items()}
    hp = {k: getattr(cfg, k) for k in decode_cases.HP}

    def run(wide, conv):
        prep = types.SimpleNamespace(**hp, **{k: conv(v) for k, v in bias.items()}, b_scale=conv(dev["b_scale"]),
                                     c_scale=conv(dev["c_scale"]), normalize_bc=True)
        owner = types.SimpleNamespace(scanprep=prep, d_state=N, d_head=P, output_norm=None)
        row = {}
        for k in ("value", "params", "bc", "gate"):   # rows that are slices of a wider projection, or whole
            t = dev[k].reshape(b, -1)
            row[k] = (torch.cat([t, t], 1)[:, :t.shape[1]] if wide else t).view(dev[k].shape)
        state = sb.ScanState(state=dev["state"].clone(), b_prev=dev["b_prev"].clone(), u_prev=dev["u_prev"].clone())
        y, nxt = sb.B200MixerDecodeBackend()(owner, types.SimpleNamespace(skip=dev["skip"], **row), state)
        return y, nxt.state, nxt.b_prev, nxt.u_prev

    want = run(False, lambda t: t.float())
    for got in (run(True, lambda t: t), run(False, lambda t: t), run(True, lambda t: t.float())):
        assert all(torch.equal(x, y) for x, y in zip(got, want))


@pytest.mark.parametrize("dtype,skip_dtype,tol", [(F32, F32, 2e-5), (BF16, BF16, 1e-2), (F16, F32, 4e-3)])
@pytest.mark.parametrize("b,H,T,P", [(1, 2, 1, 64), (2, 3, 5, 32), (1, 8, 67, 64), (3, 4, 130, 24)])
def test_gate_tile_remainders(dtype, skip_dtype, tol, b, H, T, P):
    import slinoss_b200 as sb

    gen = torch.Generator().manual_seed(T)
    r = lambda *s: torch.randn(*s, generator=gen)
    y, u = (r(b, H, T, P).to(dtype).cuda().requires_grad_(True) for _ in range(2))
    wide = r(b, T, 2 * H * P + 8).to(dtype).cuda().requires_grad_(True)
    skip = r(H, P).to(skip_dtype).cuda().requires_grad_(True)
    out = sb.gate_skip_b200(y, u, wide[..., 8:8 + H * P], skip)
    d = r(*out.shape).to(dtype).cuda()
    got = (out,) + torch.autograd.grad(out, [y, u, wide, skip], d)
    y64, u64, w64, s64 = (t.detach().double().requires_grad_(True) for t in (y, u, wide, skip))
    s_row = s64.to(dtype).double() if dtype != skip_dtype else s64
    ref = (y64 + s_row[None, :, None] * u64).permute(0, 2, 1, 3).reshape(b, T, H * P)
    ref = ref * torch.nn.functional.silu(w64[..., 8:8 + H * P])
    want = (ref,) + torch.autograd.grad(ref, [y64, u64, w64, s64], d.double().view(ref.shape))
    for name, x, w in zip(("out", "dy", "du", "dgate", "dskip"), got, want):
        assert rel_err(to_np(x).reshape(-1), to_np(w).reshape(-1)) < tol, name

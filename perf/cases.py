"""Performance cases of the framework: what its users have it do, through its public entry points.

Three kinds of work, in the sizes of this repository's configurations and tests:

* ``scan``    the chunked scan by itself (``v2x2ssd_b200``), training (forward + all gradients) or inference;
* ``mixer``   the core of one mixer layer between its two projections: causal conv + SiLU, scan preparation, scan,
              skip / gate.  Inputs are the column slices of one input projection's output, as the layer hands them over;
              training (forward + all gradients) or prefill (states in and out);
* ``decode``  one token of the same core: rolling conv update, then the decode step on the carried state.

``listed()`` names twelve of them, ``draw(rng)`` gives more of the same ranges.
"""

from __future__ import annotations

import math
import types

import torch

import slinoss_b200 as sb

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
BIASES = ("dt_bias", "gamma_bias", "omega_bias", "mix_r_bias", "mix_theta_bias", "mix_k_prev_bias", "mix_k_curr_bias")
HYPER = dict(dt_min=1e-4, dt_max=1e-1, r_min=0.9, r_max=1.0, theta_bound=math.pi, k_max=0.5, eps=1e-8)


def _scan(name, dtype, b, h, T, N, *, P=64, chunk=64, train=True, state=False):
    return dict(name=name, kind="scan", dtype=dtype, b=b, h=h, T=T, P=P, N=N, chunk=chunk, train=train, state=state)


def _mixer(name, dtype, b, h, T, N, *, P=64, chunk=64, conv=4, train=True):
    return dict(name=name, kind="mixer", dtype=dtype, b=b, h=h, T=T, P=P, N=N, chunk=chunk, conv=conv, train=train)


def _decode(name, dtype, b, h, N, *, P=64, conv=4):
    return dict(name=name, kind="decode", dtype=dtype, b=b, h=h, P=P, N=N, conv=conv)


def listed():
    return [
        # the headline workload of the benchmark, at the chunk size the reference defaults to
        _scan("scan_train_headline", "bf16", 4, 32, 8192, 128),
        # one long document: few sequences, many chunks (half of the longest configured context)
        _scan("scan_train_long", "bf16", 1, 32, 131072, 128, chunk=128),
        # a training segment that carries state in and out, ragged length
        _scan("scan_train_segment", "fp16", 3, 12, 1537, 64, state=True),
        # the smallest configured shape, in fp32: a small model on a small batch
        _scan("scan_train_smallest_fp32", "fp32", 2, 4, 256, 16, P=32),
        # full-precision training of an ordinary model
        _scan("scan_train_fp32", "fp32", 2, 8, 2048, 64),
        # inference over the next segment of a stream, odd length
        _scan("scan_infer_stream", "bf16", 1, 16, 4093, 128, state=True, train=False),
        # the single-layer configuration: d_model 768, 12 heads, d_state 64
        _mixer("mixer_train_layer", "bf16", 8, 12, 2048, 64),
        # one layer of the language-model training configuration: d_model 1024, 16 heads, d_state 128
        _mixer("mixer_train_lm", "bf16", 16, 16, 4096, 128),
        # a small fp32 layer on short ragged sequences
        _mixer("mixer_train_short_fp32", "fp32", 2, 4, 77, 16, chunk=32),
        # serving: prompt of two requests through a small model
        _mixer("mixer_prefill", "fp16", 2, 8, 1000, 64, train=False),
        # one token of one request through a small model
        _decode("decode_single", "fp16", 1, 8, 64),
        # one token of a full serving batch
        _decode("decode_batch", "bf16", 256, 32, 128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["scan", "scan", "mixer", "mixer", "decode"])
    dtype = rng.choice(["bf16", "bf16", "fp16", "fp32"])
    h = rng.choice([2, 4, 8, 12, 16, 24, 32])
    N = rng.choice([16, 32, 64, 64, 128, 128])
    if kind == "decode":
        c = _decode("", dtype, _log_int(rng, 1, 256), h, N, conv=rng.choice([2, 3, 4, 4]))
    else:
        # head-tokens of one call: up to the headline's for half types, up to an eighth of it for fp32 and for the
        # narrow state the tensor-core kernels do not take
        most = (1 << 20) if dtype != "fp32" and N > 16 else (1 << 17)
        T = _log_int(rng, 48, min(most // h, 32768))
        b = _log_int(rng, 1, max(1, min(16, most // (h * T))))
        train = rng.random() < 0.65
        if kind == "scan":
            P = 32 if dtype == "fp32" and rng.random() < 0.3 else 64
            c = _scan("", dtype, b, h, T, N, P=P, chunk=rng.choice([32, 64, 64, 128]), train=train,
                      state=rng.random() < 0.4)
        else:
            c = _mixer("", dtype, b, h, T, N, chunk=rng.choice([32, 64, 64]), conv=rng.choice([3, 4, 4]), train=train)
    del c["name"]
    return c


# ---- inputs ------------------------------------------------------------------------------------------------------


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) + 1)

    def randn(*shape, dtype=torch.float32, scale=1.0):
        return torch.randn(shape, generator=g, device="cuda", dtype=dtype).mul_(scale)

    return randn


def _scan_state(case, randn, dt):
    b, h, T, P, N = (case[k] for k in ("b", "h", "T", "P", "N"))
    radius = torch.sigmoid(2.0 + randn(b, h, T))
    angle = torch.tanh(randn(b, h, T)) * (math.pi / 4)
    M = torch.view_as_real(torch.polar(radius, angle)).contiguous()
    s = dict(case=case, U=randn(b, h, T, P, dtype=dt), M=M, K=randn(b, h, T, 2, 2, scale=0.1),
             B=randn(b, h, T, 2 * N, dtype=dt, scale=N ** -0.5), C=randn(b, h, T, 2 * N, dtype=dt, scale=N ** -0.5))
    leaves = ["U", "M", "K", "B", "C"]
    if case["state"]:
        s.update(init=randn(b, h, P, 2 * N), B_prev=randn(b, h, 2 * N, dtype=dt, scale=N ** -0.5),
                 U_prev=randn(b, h, P, dtype=dt))
        leaves += ["init", "B_prev", "U_prev"]
    if case["train"]:
        s["dY"] = randn(b, h, T, P, dtype=dt)
        s["d_final"] = randn(b, h, P, 2 * N, dtype=dt, scale=0.1)
        for k in leaves:
            s[k].requires_grad_(True)
    s["leaves"] = [s[k] for k in leaves]
    return s


def _owner(case, randn, dt):
    """The parameters of one mixer layer, under the attribute names the backends read."""
    h, P, N, W = (case[k] for k in ("h", "P", "N", "conv"))
    prep = types.SimpleNamespace(
        n_heads=h, d_state=N, d_head=P, normalize_bc=True, **HYPER,
        **{k: randn(h, dtype=dt, scale=0.3) for k in BIASES},
        b_scale=1 + randn(h, 2, N, dtype=dt, scale=0.1), c_scale=1 + randn(h, 2, N, dtype=dt, scale=0.1))
    return types.SimpleNamespace(
        scanprep=prep, d_conv=W, d_state=N, output_norm=None,
        dw_weight=randn(h * P, W, dtype=dt, scale=W ** -0.5), dw_bias=randn(h * P, dtype=dt, scale=0.1),
        skip=1 + randn(h * P, dtype=dt, scale=0.1))


def _projection(case, randn, dt, rows):
    """Column slices (gate, value, params, bc) of one input projection's output.  A half-precision row is padded to
    a multiple of 8 values, as the framework's aligned projection leaves it."""
    h, P, N = (case[k] for k in ("h", "P", "N"))
    widths = [h * P, h * P, h * 13, h * 4 * N]
    total = sum(widths)
    pad = (-total) % 8 if dt != torch.float32 else 0
    proj = randn(*rows, total + pad, dtype=dt)
    return [t.detach() for t in torch.split(proj[..., :total], widths, dim=-1)]


def _mixer_state(case, randn, dt):
    b, h, T, P, N, W = (case[k] for k in ("b", "h", "T", "P", "N", "conv"))
    owner = _owner(case, randn, dt)
    gate, value, params, bc = _projection(case, randn, dt, (b, T))
    s = dict(case=case, owner=owner, gate=gate, value=value, params=params, bc=bc)
    if case["train"]:
        s["d_out"] = randn(b, T, h * P, dtype=dt)
        p = owner.scanprep
        s["leaves"] = [gate, value, params, bc, owner.dw_weight, owner.dw_bias, owner.skip,
                       *(getattr(p, k) for k in BIASES), p.b_scale, p.c_scale]
        for t in s["leaves"]:
            t.requires_grad_(True)
    else:
        s["conv"] = randn(b, h * P, W - 1, dtype=dt)
        s["scan"] = sb.ScanState(state=randn(b, h, P, 2 * N), b_prev=randn(b, h, 2 * N, dtype=dt),
                                 u_prev=randn(b, h, P, dtype=dt))
    s["prep_backend"], s["scan_backend"] = sb.B200ScanPrepBackend(), sb.B200ScanBackend()
    return s


def _decode_state(case, randn, dt):
    b, h, P, N, W = (case[k] for k in ("b", "h", "P", "N", "conv"))
    owner = _owner(case, randn, dt)
    gate, value, params, bc = _projection(case, randn, dt, (b,))
    return dict(case=case, owner=owner, gate=gate, value=value, params=params, bc=bc,
                conv=randn(b, h * P, W - 1, dtype=dt),
                scan=sb.ScanState(state=randn(b, h, P, 2 * N), b_prev=randn(b, h, 2 * N, dtype=dt),
                                  u_prev=randn(b, h, P, dtype=dt)),
                backend=sb.B200MixerDecodeBackend())


def prepare(case, seed):
    make = {"scan": _scan_state, "mixer": _mixer_state, "decode": _decode_state}[case["kind"]]
    return make(case, _generator(seed), DTYPES[case["dtype"]])


# ---- one pass ----------------------------------------------------------------------------------------------------


def _run_scan(s):
    case = s["case"]
    kw = dict(chunk_size=case["chunk"], return_state=case["state"])
    if case["state"]:
        kw.update(initial_states=s["init"], B_prev=s["B_prev"], U_prev=s["U_prev"])
    if not case["train"]:
        with torch.no_grad():
            return sb.v2x2ssd_b200(s["U"], s["M"], s["K"], s["B"], s["C"], **kw)
    out = sb.v2x2ssd_b200(s["U"], s["M"], s["K"], s["B"], s["C"], **kw)
    if not case["state"]:
        return [out.detach(), *torch.autograd.grad(out, s["leaves"], s["dY"])]
    grads = torch.autograd.grad(out[:2], s["leaves"], [s["dY"], s["d_final"]])
    return [*(t.detach() for t in out), *grads]


def _mixer_core(s, conv_state, scan_state, return_state):
    owner, case = s["owner"], s["case"]
    value, conv_next = sb.cconv1d_b200(s["value"], owner.dw_weight, owner.dw_bias, conv_state, activation="silu")
    bc = s["bc"].view(case["b"], case["T"], case["h"], 4, case["N"])
    inputs = s["prep_backend"](owner.scanprep, sb.ScanPrepInputs(value=value, params=s["params"], bc=bc))
    y = s["scan_backend"](inputs, chunk_size=case["chunk"], state=scan_state, return_state=return_state)
    y, scan_next = y if return_state else (y, None)
    return sb.gate_skip_b200(y, inputs.U, s["gate"], owner.skip), conv_next, scan_next


def _run_mixer(s):
    if s["case"]["train"]:
        out, _, _ = _mixer_core(s, None, None, False)
        return [out.detach(), *torch.autograd.grad(out, s["leaves"], s["d_out"])]
    with torch.no_grad():
        out, conv_next, st = _mixer_core(s, s["conv"], s["scan"], True)
        return [out, conv_next, st.state, st.b_prev, st.u_prev]


def _run_decode(s):
    owner, case = s["owner"], s["case"]
    b, h, P, N = (case[k] for k in ("b", "h", "P", "N"))
    with torch.no_grad():
        value, s["conv"] = sb.cconv1d_update_b200(s["value"], owner.dw_weight, owner.dw_bias, s["conv"],
                                                  activation="silu")
        inputs = types.SimpleNamespace(value=value.view(b, h, P), params=s["params"].view(b, h, 13),
                                       bc=s["bc"].view(b, h, 4, N), gate=s["gate"].view(b, h, P),
                                       skip=owner.skip.view(h, P))
        out, s["scan"] = s["backend"](owner, inputs, s["scan"])
        return [out, s["conv"], s["scan"].state, s["scan"].b_prev, s["scan"].u_prev]


def run(state):
    return {"scan": _run_scan, "mixer": _run_mixer, "decode": _run_decode}[state["case"]["kind"]](state)


# ---- what a pass cannot do without, and how close results have to be ------------------------------------------------


def _scan_flops(case, train):
    """Multiply-adds of the causal triangle in 64-token chunks plus the state terms, counted twice each."""
    P, D, L = case["P"], 2 * case["N"], 64
    per = (12 * P * D + (L + 1) * (8 * D + 6 * P)) if train else (4 * P * D + (L + 1) * (2 * D + 2 * P))
    return per * case["b"] * case["h"] * case["T"]


def work(case):
    b, h, P, N = (case[k] for k in ("b", "h", "P", "N"))
    D, es = 2 * N, torch.empty((), dtype=DTYPES[case["dtype"]]).element_size()
    state = b * h * P * D
    if case["kind"] == "decode":
        W = case["conv"]
        rows = es * b * h * (2 * P + 13 + 2 * D + P + 2 * P * (W - 1) + 2 * D + 2 * P)
        params = es * h * (P * (W + 2) + 7 + 2 * D)
        return dict(bytes=8 * state + rows + params, flops=b * h * P * (8 * D + 2 * D + 2 * W))
    ht = b * h * case["T"]
    train = case["train"]
    if case["kind"] == "scan":
        nbytes = ht * (es * (2 * P + 2 * D) + 24)
        if train:
            nbytes += ht * (es * (2 * P + 2 * D) + 24)
        if case["state"]:
            nbytes += (4 if train else 3) * state * 2 + 2 * es * b * h * (D + P)
        return dict(bytes=nbytes, flops=_scan_flops(case, train))
    row = es * (2 * P + 13 + 2 * D)  # one head's share of a projection row
    nbytes = ht * (row + es * P)
    if train:
        nbytes += ht * (row + es * P)
    else:
        nbytes += 4 * state + es * state + 2 * es * b * h * (P * (case["conv"] - 1) + D + P)
    return dict(bytes=nbytes, flops=_scan_flops(case, train) + ht * P * 2 * case["conv"] * (3 if train else 1))


def tolerance(case):
    if case["dtype"] == "fp32":
        # 32-bit sums; the layer's parameter gradients go through the tap formulas and long sums on top
        return {"rel": 2e-5 if case["kind"] == "mixer" else 1e-5}
    if case["dtype"] == "fp16":
        return {"rel": 3e-3}
    # bf16: the gradient of M divides sums of rounded operands by M itself; the repository's own exact and
    # tensor-core kernels differ by 1.2e-2 there (4e-3 on every other output)
    return {"rel": 1.5e-2 if case.get("train") else 1e-2}

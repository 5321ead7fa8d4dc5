"""Forms of arguments that the ops take besides the plain one: addresses, strides, storage types."""

from __future__ import annotations

import contextlib
import ctypes

import pytest
import torch

from gpu_util import make_scan_inputs, run_b200_fwd_bwd

F32, BF16, F16 = torch.float32, torch.bfloat16, torch.float16


def _at_odd_offset(t):
    """The same values, contiguous, one element past a 16-byte boundary."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    buf[1:].copy_(t.reshape(-1))
    return buf[1:].view(t.shape)


@pytest.mark.parametrize("which", ["B_prev", "U_prev"])
@pytest.mark.parametrize("dtype", [BF16, F32])
def test_entry_points_refuse_misaligned_streaming_rows(which, dtype):
    """No GPU needed: the addresses are looked at before anything is launched."""
    from slinoss_b200 import _lib

    s = _lib.scan_shape(2, 128, 64, 32, 128, dtype)
    a = 0x100000
    args = {"B_prev": a, "U_prev": a, which: a + 2}
    rows, lib = (args["B_prev"], args["U_prev"]), _lib.lib()
    by, code = ctypes.byref(s), _lib.dtype_code(dtype)

    class Ends(ctypes.Structure):  # slx_scan_ends and slx_scan_grad_ends: six pointers, then the dtypes
        _fields_ = [("p", ctypes.c_void_p * 6), ("codes", ctypes.c_int32 * 4)]

    fwd, bwd = Ends(), Ends()
    fwd.p[1], fwd.p[2], fwd.codes[1] = *rows, code
    bwd.p[0], bwd.p[1], bwd.codes[0] = *rows, code
    nbytes = lib.slx_v2x2ssd_bwd_workspace_bytes(by)
    calls = [lambda: lib.slx_v2x2ssd_fwd_stream(by, a, a, a, a, a, ctypes.byref(fwd), a, a, a, a, a, None),
             lambda: lib.slx_v2x2ssd_bwd_stream(by, a, a, a, a, a, ctypes.byref(bwd), *([a] * 9), a, nbytes, None)]
    if dtype == F32:
        calls += [lambda: lib.slx_chunk_increment_fwd(by, a, a, a, a, *rows, a, _lib.SLX_F32, a, None),
                  lambda: lib.slx_chunk_scan_fwd(by, a, a, a, a, a, a, *rows, a, None),
                  lambda: lib.slx_chunk_scan_bwd(by, a, a, a, a, a, *rows, *([a] * 11), None)]
    for call in calls:
        assert call() == -3 and b"aligned" in lib.slx_last_error_string()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,N,T", [(BF16, 64, 130), (F16, 32, 40), (F32, 17, 70)])
def test_streaming_rows_at_any_address(dtype, N, T):
    inp = make_scan_inputs(1, 2, T, N, 64, dtype, seed=T, streaming=True, with_init=True)
    Y, fin, g = run_b200_fwd_bwd(inp, 128)
    import slinoss_b200 as sb

    rows = {k: _at_odd_offset(inp[k]).requires_grad_(True) for k in ("B_prev", "U_prev")}
    assert all(t.data_ptr() % 16 for t in rows.values())
    leaves = [inp[k].detach().requires_grad_(True) for k in ("U", "M", "K", "B", "C", "initial_states")]
    out = sb.v2x2ssd_b200(*leaves[:5], chunk_size=128, initial_states=leaves[5], return_state=True, **rows)
    grads = torch.autograd.grad(out[:2], [*leaves, *rows.values()], [inp["dY"], inp["d_final"].to(out[1].dtype)])
    assert torch.equal(out[0], Y) and torch.equal(out[1], fin)
    names = ("dU", "dM", "dK", "dB", "dC", "d_initial", "dB_prev", "dU_prev")
    assert all(torch.equal(a, g[k]) for k, a in zip(names, grads))


def _one_token_forms(t):
    """(b, 1, ...) tensors with the values of ``t`` and other strides: the size-one axis leading in storage, trailing."""
    lead = t.transpose(0, 1).contiguous().transpose(0, 1)
    trail = torch.empty((*t.shape[:1], *t.shape[2:], 1), dtype=t.dtype, device=t.device).movedim(-1, 1).copy_(t)
    wide = torch.empty((t.shape[0], 3, *t.shape[2:]), dtype=t.dtype, device=t.device)[:, 1:2].copy_(t)
    return lead, trail, wide


def test_row_stride_of_one_token():
    """The distance of the rows that the scan preparation is given (no GPU needed)."""
    from slinoss_b200 import _lib

    rs = _lib.host().row_stride
    x = torch.zeros(4, 1, 24)
    assert [rs(t) for t in (x, *_one_token_forms(x))] == [24, 24, 24, 72]
    assert rs(x.view(4, 1, 3, 2, 4).transpose(0, 1).contiguous().transpose(0, 1)) == 24
    assert rs(torch.zeros(1, 1, 24)) == 24 and rs(torch.zeros(1, 24, 1).transpose(1, 2)) == 24
    assert rs(torch.zeros(2, 5, 30)[..., 3:27]) == 30 and rs(torch.zeros(2, 5, 24)[:, :4]) == 0
    assert rs(torch.zeros(1, 5, 24)[:, :4]) == 24 and rs(torch.zeros(5, 2, 24).transpose(0, 1)) == 0
    assert rs(torch.zeros(1, 1, 24).expand(3, 1, 24)) == 0 and rs(torch.zeros(2, 24, 5).transpose(1, 2)) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [BF16, F32])
@pytest.mark.parametrize("form", range(3))
def test_scanprep_and_gate_of_one_token(dtype, form):
    import slinoss_b200 as sb

    b, H, P, N = 3, 2, 16, 8
    g = torch.Generator().manual_seed(form)
    r = lambda *s: torch.randn(*s, generator=g).to(dtype).cuda()
    hp = dict(n_heads=H, d_state=N, d_head=P, normalize_bc=True, dt_min=1e-4, dt_max=1e-1, r_min=0.9, r_max=1.0,
              theta_bound=3.0, k_max=0.5, eps=1e-8, b_scale=r(H, 2, N), c_scale=r(H, 2, N),
              **{k: r(H) for k in ("dt_bias", "gamma_bias", "omega_bias", "mix_r_bias", "mix_theta_bias",
                                   "mix_k_prev_bias", "mix_k_curr_bias")})
    args = [r(b, 1, H * P), r(b, 1, H * 13), r(b, 1, H, 4, N)]
    gate, skip, y, u = r(b, 1, H * P), r(H * P), r(b, H, 1, P), r(b, H, 1, P)

    def both(value, params, bc, gate):
        leaves = [t.detach().requires_grad_(True) for t in (value, params, bc, gate)]
        o = sb.scanprep_b200(*leaves[:3], **hp)
        outs = [o.U, o.M, o.K, o.B, o.C, sb.gate_skip_b200(y, u, leaves[3], skip)]
        return outs + list(torch.autograd.grad([t.float().square().sum() for t in outs], leaves))

    want = both(*args, gate)
    for k, t in enumerate([*args, gate]):
        mixed = [*args, gate]
        mixed[k] = _one_token_forms(t)[form]
        assert all(torch.equal(a, w) for a, w in zip(both(*mixed), want)), k


@pytest.mark.gpu
@pytest.mark.parametrize("before,after", [(1, 0), (0, 1), (2, 0), (1, 2)])
def test_kernel_family_chosen_between_forward_and_backward(before, after):
    """Chunk starts are held in the dtype of the family that wrote them: the backward runs on the family chosen by then."""
    import slinoss_b200 as sb
    from slinoss_b200 import _lib

    inp = make_scan_inputs(1, 2, 300, 32, 64, BF16, seed=1, with_init=True)
    names = ("U", "M", "K", "B", "C", "initial_states")

    def grads(forward, backward):
        old = _lib.set_tensor_path(forward)
        try:
            leaves = [inp[k].detach().requires_grad_(True) for k in names]
            Y = sb.v2x2ssd_b200(*leaves[:5], chunk_size=128, initial_states=leaves[5])
            _lib.set_tensor_path(backward)
            return torch.autograd.grad(Y, leaves, inp["dY"])
        finally:
            _lib.set_tensor_path(old)

    for k, a, b in zip(names, grads(before, after), grads(after, after)):
        # the families' chunk starts differ by their storage, half against fp32: 2^-9 of a value
        assert (a.float() - b.float()).norm() < 4e-3 * b.float().norm(), k


@pytest.mark.gpu
def test_other_threads_run_while_a_launch_waits():
    """The interpreter lock is free while an op waits for room in the launch queue."""
    import threading
    import time

    import slinoss_b200 as sb

    x, w = torch.zeros(1, 8, device="cuda"), torch.zeros(8, 4, device="cuda")
    state = torch.zeros(1, 8, 3, device="cuda")
    sb.cconv1d_update_b200(x, w, None, state, inplace=True)
    torch.cuda.synchronize()
    gaps, done = [], threading.Event()

    def tick():
        last = time.perf_counter()
        while not done.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    torch.cuda._sleep(int(1.5e9))  # the GPU is busy for most of a second
    thread = threading.Thread(target=tick)
    thread.start()
    start = time.perf_counter()
    for _ in range(4000):  # more than the queue holds
        sb.cconv1d_update_b200(x, w, None, state, inplace=True)
    waited = time.perf_counter() - start
    done.set()
    thread.join()
    torch.cuda.synchronize()
    if waited < 0.4:
        pytest.skip("the launches did not have to wait")
    assert max(gaps) < 0.5 * waited, (max(gaps), waited)


@pytest.mark.gpu
@pytest.mark.parametrize("residual", ["keep", "recompute"])
def test_carried_tensors_may_be_overwritten_before_the_backward(residual):
    """A stream that keeps its carried tensors in place: the backward needs the rows and states that the forward read."""
    import slinoss_b200 as sb

    inp = make_scan_inputs(1, 2, 140, 32, 64, BF16, seed=2, streaming=True, with_init=True)
    inp["initial_states"] = inp["initial_states"].to(BF16)
    names = ("U", "M", "K", "B", "C")

    def grads(overwrite):
        leaves = [inp[k].detach().requires_grad_(True) for k in names]
        carried = {k: inp[k].clone() for k in ("initial_states", "B_prev", "U_prev")}
        Y, *nxt = sb.v2x2ssd_b200(*leaves, chunk_size=128, return_state=True, residual=residual, **carried)
        if overwrite:
            for t, n in zip(carried.values(), nxt):
                t.copy_(n.detach())
        return torch.autograd.grad(Y, leaves, inp["dY"])

    assert all(torch.equal(a, b) for a, b in zip(grads(True), grads(False)))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [BF16, F32])
def test_parameters_may_be_updated_before_the_backward(dtype):
    import slinoss_b200 as sb

    b, T, H, P, N = 2, 9, 2, 16, 8
    g = torch.Generator().manual_seed(5)
    r = lambda *s, dt=BF16: torch.randn(*s, generator=g).to(dt).cuda()
    value, params, bc = r(b, T, H * P), r(b, T, H * 13), r(b, T, H, 4, N)
    gate, y = r(b, T, H * P), r(b, H, T, P)
    names = ("dt_bias", "gamma_bias", "omega_bias", "mix_r_bias", "mix_theta_bias", "mix_k_prev_bias",
             "mix_k_curr_bias")
    pars = {k: r(H, dt=dtype) for k in names}
    pars.update(b_scale=r(H, 2, N, dt=dtype), c_scale=r(H, 2, N, dt=dtype))
    skip, w = r(H * P), r(H * P, 4, dt=F32)  # (fp32 skip weights and taps of x's own dtype are kept by reference)

    def grads(update):
        leaves = [t.clone().requires_grad_(True) for t in (value, params, bc, gate)]
        ps = {k: t.clone().requires_grad_(True) for k, t in pars.items()}
        ws = [t.clone().requires_grad_(True) for t in (skip, w)]
        x, _ = sb.cconv1d_b200(leaves[0], ws[1], None, activation="silu")
        o = sb.scanprep_b200(x, leaves[1], leaves[2], n_heads=H, d_state=N, d_head=P, normalize_bc=True, dt_min=1e-4,
                             dt_max=1e-1, r_min=0.9, r_max=1.0, theta_bound=3.0, k_max=0.5, eps=1e-8, **ps)
        outs = [o.U, o.M, o.K, o.B, o.C, sb.gate_skip_b200(y, o.U, leaves[3], ws[0])]
        if update:
            with torch.no_grad():
                for t in (*ps.values(), *ws):
                    t.mul_(0.5)
        return torch.autograd.grad([t.float().square().sum() for t in outs], [*leaves, *ps.values(), *ws])

    assert all(torch.equal(a, b) for a, b in zip(grads(True), grads(False)))


def _one_input_calls():
    """name -> (op as a function of its main input, shape of that input)"""
    import slinoss_b200 as sb

    g = torch.Generator().manual_seed(8)
    r = lambda *s: torch.randn(*s, generator=g).cuda()
    b, T, H, P, N = 1, 20, 2, 16, 8
    hp = dict(n_heads=H, d_state=N, d_head=P, normalize_bc=True, dt_min=1e-4, dt_max=1e-1, r_min=0.9, r_max=1.0,
              theta_bound=3.0, k_max=0.5, eps=1e-8, b_scale=r(H, 2, N), c_scale=r(H, 2, N),
              **{k: r(H) for k in ("dt_bias", "gamma_bias", "omega_bias", "mix_r_bias", "mix_theta_bias",
                                   "mix_k_prev_bias", "mix_k_curr_bias")})
    w, params, bc, gate, skip = r(H * P, 4), r(b, T, H * 13), r(b, T, H, 4, N), r(b, T, H * P), r(H * P)
    M = torch.view_as_real(torch.polar(0.5 + 0.5 * torch.rand(b, H, T, generator=g), torch.randn(b, H, T, generator=g)))
    scan = [M.contiguous().cuda(), r(b, H, T, 2, 2), r(b, H, T, 2 * N), r(b, H, T, 2 * N)]
    return {
        "conv": (lambda x: sb.cconv1d_b200(x, w, None, activation="silu")[0], (b, T, H * P)),
        "prep": (lambda x: sb.scanprep_b200(gate, params, x, **hp).B, (b, T, H, 4, N)),
        "gate": (lambda x: sb.gate_skip_b200(x, x, gate, skip), (b, H, T, P)),
        "scan": (lambda x: sb.v2x2ssd_b200(x, *scan, chunk_size=16, return_state=True)[1], (b, H, T, P)),
    }


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["conv", "prep", "gate", "scan"])
@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.filterwarnings("ignore")
def test_traced_calls_run_again(name, grad):
    fn, shape = _one_input_calls()[name]
    x, y = torch.randn(2, *shape, device="cuda").requires_grad_(grad)
    traced = torch.jit.trace(fn, x.detach().requires_grad_(grad), check_trace=False)
    leaf = y.detach().requires_grad_(grad)
    outs = traced(leaf), fn(leaf)
    assert torch.equal(*outs)
    if grad:
        assert torch.equal(*(torch.autograd.grad(o.square().sum(), leaf)[0] for o in outs))


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["conv", "prep", "gate", "scan"])
@pytest.mark.parametrize("grad", [False, True])
def test_tangents_are_refused(name, grad):
    """Forward-mode derivatives are not implemented: an error, not an output without its tangent."""
    import torch.autograd.forward_ad as forward_ad

    fn, shape = _one_input_calls()[name]
    x, t = torch.randn(2, *shape, device="cuda")
    with forward_ad.dual_level(), pytest.raises(NotImplementedError):
        fn(forward_ad.make_dual(x.requires_grad_(grad), t))


def _kernels(fn):
    """(name, grid) of the kernels that ``fn`` launches, in order."""
    import json
    import tempfile

    fn()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        fn()
        torch.cuda.synchronize()
    with tempfile.NamedTemporaryFile(suffix=".json") as f:
        prof.export_chrome_trace(f.name)
        events = json.load(open(f.name))["traceEvents"]
    found = sorted((e["ts"], e["name"], e["args"]["grid"]) for e in events if e.get("cat") == "kernel")
    if not found:
        pytest.skip("the profiler shows no kernels here")
    return [(n, g) for _, n, g in found]


@pytest.mark.gpu
def test_decode_grid_follows_the_state_width():
    """Wide states leave fewer CTAs per SM; the narrow ones before and after keep three."""
    import slinoss_b200 as sb

    def grid(N):
        b, H, P = 1024, 1, 64
        z = lambda *s: torch.zeros(*s, device="cuda")
        bias = {k: z(H) for k in ("dt_bias", "gamma_bias", "omega_bias", "mix_r_bias", "mix_theta_bias",
                                  "mix_k_prev_bias", "mix_k_curr_bias")}
        kern = _kernels(lambda: sb.mixer_decode_step_b200(
            z(b, H, P), z(b, H, 13), z(b, H, 4, N), z(b, H, P), z(H, P), initial_states=z(b, H, P, 2 * N),
            B_prev=z(b, H, 2 * N), U_prev=z(b, H, P), dt_min=1e-4, dt_max=0.1, r_min=0.9, r_max=1.0, theta_bound=3.0,
            k_max=0.5, eps=1e-8, b_scale=z(H, 2, N), c_scale=z(H, 2, N), **bias))
        return [g[0] for n, g in kern if "decode_step" in n][-1]

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert [grid(N) for N in (64, 1024, 64)] == [3 * sms, grid(1024), 3 * sms]
    assert grid(1024) in (sms, 2 * sms)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,N,P,vec", [(F16, 36, 12, 4), (BF16, 512, 64, 4), (F32, 6, 2, 2)])
def test_scanprep_rows_on_8_byte_boundaries(dtype, N, P, vec):
    """Rows wider than a warp's slices, or of half a slice's multiple: the forward reads 8 bytes at a time."""
    import slinoss_b200 as sb

    b, T, H = 2, 37, 4
    g = torch.Generator().manual_seed(N)
    r = lambda *s: torch.randn(*s, generator=g).to(dtype).cuda()
    hp = dict(n_heads=H, d_state=N, d_head=P, normalize_bc=True, dt_min=1e-4, dt_max=1e-1, r_min=0.9, r_max=1.0,
              theta_bound=3.0, k_max=0.5, eps=1e-8, b_scale=r(H, 2, N), c_scale=r(H, 2, N),
              **{k: r(H) for k in ("dt_bias", "gamma_bias", "omega_bias", "mix_r_bias", "mix_theta_bias",
                                   "mix_k_prev_bias", "mix_k_curr_bias")})
    per = 16 // (2 if dtype != F32 else 4)  # values of 16 bytes
    value, bc = r(b, T, H * P + per // 2)[..., :H * P], r(b, T, H * 4 * N + per // 2)[..., :H * 4 * N].view(b, T, H, 4, N)
    params = r(b, T, H * 13)
    call = lambda: sb.scanprep_b200(value, params, bc, **hp)
    names = [n for n, _ in _kernels(call) if "scanprep_fwd" in n]
    assert len(names) == 1 and f", {vec}, 16>" in names[0], names
    got = call()
    x = bc.double()
    x = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-5)
    want = x * torch.cat([hp["b_scale"], hp["c_scale"]], 1).double()[None, None]
    want = want.view(b, T, H, 2, 2, N).permute(3, 0, 2, 1, 5, 4).reshape(2, b, H, T, 2 * N)
    assert torch.equal(got.U, value.view(b, T, H, P).transpose(1, 2))
    for a, w in zip((got.B, got.C), want):  # one rounding of the result; fp32: of each of its few operations
        assert (a.double() - w).norm() < (1e-6 if dtype == F32 else 2.0 ** -8) * w.norm()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [BF16, F32])
def test_scanprep_gradient_of_huge_rows(dtype):
    """RMS norm does not see the scale of its row: the gradient is that of the scaled-down row, scaled down."""
    import slinoss_b200 as sb

    b, T, H, P, N = 1, 8, 2, 16, 16
    g = torch.Generator().manual_seed(4)
    r = lambda *s: torch.randn(*s, generator=g).to(dtype).cuda()
    hp = dict(n_heads=H, d_state=N, d_head=P, normalize_bc=True, dt_min=1e-4, dt_max=1e-1, r_min=0.9, r_max=1.0,
              theta_bound=3.0, k_max=0.5, eps=1e-8, b_scale=r(H, 2, N), c_scale=r(H, 2, N),
              **{k: r(H) for k in ("dt_bias", "gamma_bias", "omega_bias", "mix_r_bias", "mix_theta_bias",
                                   "mix_k_prev_bias", "mix_k_curr_bias")})
    value, params, bc, dB = r(b, T, H * P), r(b, T, H * 13), r(b, T, H, 4, N), r(b, H, T, 2 * N)

    def grad(scale):
        x = (bc * scale).requires_grad_(True)
        return torch.autograd.grad(sb.scanprep_b200(value, params, x, **hp).B, x, dB)[0].double() * scale

    # powers of two: the two differ by the norm's eps (1e-5 of x^2 = 1) and by the rounding of the result
    a, w = grad(2.0 ** 56), grad(2.0 ** 10)
    assert (a - w).norm() < (1e-6 if dtype == F32 else 2.0 ** -8) * w.norm()


@pytest.mark.gpu
def test_scanprep_refuses_parameters_of_other_shapes():
    import slinoss_b200 as sb

    b, T, H, P, N = 1, 3, 3, 16, 8
    r = lambda *s: torch.randn(*s, device="cuda")
    names = ("dt_bias", "gamma_bias", "omega_bias", "mix_r_bias", "mix_theta_bias", "mix_k_prev_bias",
             "mix_k_curr_bias")
    pars = dict({k: r(H) for k in names}, b_scale=r(H, 2, N), c_scale=r(H, 2, N))
    call = lambda **kw: sb.scanprep_b200(
        r(b, T, H * P), r(b, T, H * 13), r(b, T, H, 4, N), n_heads=H, d_state=N, d_head=P, dt_min=1e-4, dt_max=1e-1,
        r_min=0.9, r_max=1.0, theta_bound=3.0, k_max=0.5, eps=1e-8, **{**pars, **kw})
    for kw in (dict(dt_bias=r(1)), dict(mix_r_bias=r(())), dict(omega_bias=r(1, H)), dict(b_scale=r(H, 2 * N))):
        call(**kw)
    for kw in (dict(dt_bias=r(H, 1)), dict(b_scale=r(2 * H * N)), dict(c_scale=r(2, H, N)), dict(c_scale=r(H, 2, N + 1))):
        with pytest.raises((ValueError, RuntimeError)):
            call(**kw)


@pytest.mark.gpu
def test_saved_tensors_may_come_back_with_other_strides():
    """Column slices that a saved-tensor hook moves away come back dense: the backward takes the distances it gets."""
    import slinoss_b200 as sb

    b, T, H, P, N = 2, 7, 2, 16, 8
    g = torch.Generator().manual_seed(6)
    r = lambda *s: torch.randn(*s, generator=g).to(BF16).cuda()
    names = ("dt_bias", "gamma_bias", "omega_bias", "mix_r_bias", "mix_theta_bias", "mix_k_prev_bias",
             "mix_k_curr_bias")
    pars = dict({k: r(H) for k in names}, b_scale=r(H, 2, N), c_scale=r(H, 2, N))
    value, params, gate = r(b, T, 48)[..., 8:40], r(b, T, 40)[..., 8:34], r(b, T, 48)[..., 16:]
    bc, w, skip = r(b, T, 80)[..., 8:72].view(b, T, H, 4, N), r(H * P, 4), r(H * P)

    def grads(hooks):
        leaves = [t.detach().requires_grad_(True) for t in (value, params, bc, gate)]
        with hooks:
            x, _ = sb.cconv1d_b200(leaves[0], w, None, activation="silu")
            o = sb.scanprep_b200(x, leaves[1], leaves[2], n_heads=H, d_state=N, d_head=P, normalize_bc=True, dt_min=1e-4,
                                 dt_max=1e-1, r_min=0.9, r_max=1.0, theta_bound=3.0, k_max=0.5, eps=1e-8, **pars)
            y = sb.v2x2ssd_b200(o.U, o.M, o.K, o.B, o.C, chunk_size=16)
            out = sb.gate_skip_b200(y, o.U, leaves[3], skip)
        return torch.autograd.grad(out, leaves, torch.ones_like(out))

    moved = grads(torch.autograd.graph.saved_tensors_hooks(lambda t: t.contiguous().cpu(), lambda t: t.cuda()))
    assert all(torch.equal(x, y) for x, y in zip(moved, grads(contextlib.nullcontext())))

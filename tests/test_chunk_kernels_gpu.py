"""Chunk kernels of the scan at the points where their own geometry changes."""

from __future__ import annotations

from ctypes import byref

import pytest
import torch

from gpu_util import make_scan_inputs, oracle_fwd_bwd, run_b200_fwd_bwd, to_np
from util import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,T,BH", [(32, 128, 2), (96, 300, 2), (128, 129, 2), (32, 128, 150), (96, 300, 50), (128, 129, 76)])
def test_gradient_rows_off_a_32_byte_boundary(dtype, N, T, BH):
    """dB and dC leave as whole 32-byte sectors where their base allows it, else as two 16-byte stores: same bits."""
    import slinoss_b200 as sb
    from slinoss_b200 import _lib

    inp = make_scan_inputs(1, BH, T, N, 64, dtype, seed=N, dist="cfg2", with_init=True)
    U, M, K, B, C, dY = (inp[k] for k in ("U", "M", "K", "B", "C", "dY"))
    s = _lib.scan_shape(BH, T, 64, N, 128, dtype, _lib.starts_dtype(_lib.scan_shape(BH, T, 64, N, 128, dtype)))
    NC = (T + 127) // 128
    inc, mch = sb.chunk_increment_b200(U, M, K, B, chunk_size=128)
    starts, _ = sb.state_passing_b200(inc, mch, initial_states=inp["initial_states"])
    starts = starts.to(dtype).contiguous()
    d_inc = torch.randn_like(starts)
    zdot = torch.randn(BH, NC, 2, device="cuda")
    outs = []
    for off in (0, 8):
        flat = [torch.zeros(BH * T * 2 * N + 16, device="cuda", dtype=dtype) for _ in range(2)]
        dB, dC = (f[off:off + BH * T * 2 * N] for f in flat)
        assert dB.data_ptr() % 32 == 2 * off and dC.data_ptr() % 32 == 2 * off
        dU, dM, dK = torch.empty_like(U), torch.empty_like(M), torch.empty_like(K)
        cB, cU = torch.empty(BH, NC, 2 * N, device="cuda"), torch.empty(BH, NC, 64, device="cuda")
        rc = _lib.lib().slx_chunk_scan_bwd(
            byref(s), U.data_ptr(), M.data_ptr(), K.data_ptr(), B.data_ptr(), C.data_ptr(), None, None,
            starts.data_ptr(), d_inc.data_ptr(), zdot.data_ptr(), dY.data_ptr(), dU.data_ptr(), dM.data_ptr(),
            dK.data_ptr(), dB.data_ptr(), dC.data_ptr(), cB.data_ptr(), cU.data_ptr(), _lib.stream_ptr(U.device))
        _lib.check(rc, "chunk_scan_bwd")
        for f in flat:  # nothing outside the rows
            assert not f[:off].any() and not f[off + BH * T * 2 * N:].any()
        outs.append([dU, dM, dK, dB.clone(), dC.clone(), cB, cU])
    for x, y in zip(*outs):
        assert torch.equal(x, y)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,T", [(32, 77), (64, 300), (96, 128), (128, 257)])
@pytest.mark.parametrize("prev", ["none", "half", "fp32"])
def test_backward_on_either_side_of_one_cta_per_sm(dtype, N, T, prev):
    """Launches of up to 148 chunks run CTAs of 512 threads over 64-column slabs, larger ones CTAs of 256 over 32: the same
    operands and products, fp32 sums in another order.  Outputs in half precision may round to the other neighbour (half a
    step at most differs from one step by the sums' 1e-5); both sides are as far from the oracle as the operands' rounding."""
    heads = 150 // ((T + 127) // 128) + 1
    inp = make_scan_inputs(1, heads, T, N, 64, dtype, seed=N, dist="cfg2", with_init=True, streaming=prev != "none")
    if prev == "fp32":
        inp["B_prev"], inp["U_prev"] = inp["B_prev"].float() * 1.001, inp["U_prev"].float() * 1.001
    few = {k: None if v is None else v[:, :3].contiguous() for k, v in inp.items()}
    large, small = run_b200_fwd_bwd(inp, 128)[2], run_b200_fwd_bwd(few, 128)[2]
    exact = oracle_fwd_bwd(few)[2]
    tol = 2e-2 if dtype == torch.bfloat16 else 3e-3
    for k, x in small.items():
        if x is None:
            continue
        y = large[k][:, :3]
        assert rel_err(to_np(x), exact[k]) < tol, k
        assert rel_err(to_np(y), exact[k]) < tol, k
        assert rel_err(to_np(x), to_np(y)) < (2.0 ** -9 if x.dtype == dtype == torch.bfloat16 else
                                              2.0 ** -12 if x.dtype == dtype else 1e-4), k


@pytest.mark.parametrize("dtype,u", [(torch.bfloat16, 2.0 ** -8), (torch.float16, 2.0 ** -11), (torch.float32, 0.0)])
@pytest.mark.parametrize("BH,NC", [(222, 5), (223, 6), (2, 9)])
def test_reverse_state_pass_on_either_side_of_three_ctas_per_sm(dtype, u, BH, NC):
    """Half states of 64 x 64 are two CTAs per head; the kernel changes above 444.  d_inc is rounded to its dtype once (u:
    the largest relative error of that, 8 and 11 significant bits), the recurrence and the dots are fp32."""
    from slinoss_b200 import _lib

    g = torch.Generator().manual_seed(BH)
    P, N, code = 64, 32, _lib.dtype_code(dtype)
    dz, st = (torch.randn((BH, NC, P, 2 * N), generator=g).to(dtype) for _ in range(2))
    m = torch.view_as_real(torch.polar(0.5 + 0.5 * torch.rand((BH, NC), generator=g), torch.randn((BH, NC), generator=g)))
    fin, dfin = (torch.randn((BH, P, 2 * N), generator=g) for _ in range(2))
    z = lambda t: torch.view_as_complex(t.double().reshape(*t.shape[:-1], -1, 2))
    grad, want_inc, want_dot = z(dfin), [None] * NC, [None] * NC
    for c in reversed(range(NC)):
        want_inc[c] = torch.view_as_real(grad).flatten(-2)
        want_dot[c] = ((z(fin) if c + 1 == NC else z(st[:, c + 1])).conj() * grad).sum((1, 2))
        grad = z(dz[:, c]) + z(m)[:, c].reshape(-1, 1, 1).conj() * grad
    dev = [t.cuda() for t in (dz, m, st, fin, dfin)]
    inc, init, dot = torch.empty_like(dev[0]), torch.empty_like(dev[3]), torch.empty((BH, NC, 2), device="cuda")
    part = torch.empty(_lib.lib().slx_state_passing_bwd_partials_bytes(BH, NC, P, N) // 4, device="cuda")
    rc = _lib.lib().slx_state_passing_bwd(
        BH, NC, P, N, dev[0].data_ptr(), code, dev[1].data_ptr(), dev[2].data_ptr(), code, dev[3].data_ptr(),
        dev[4].data_ptr(), inc.data_ptr(), init.data_ptr(), dot.data_ptr(), part.data_ptr(), _lib.stream_ptr(inc.device))
    _lib.check(rc, "state_passing_bwd")
    want = torch.stack(want_inc, 1)
    err = (inc.double().cpu() - want).abs()
    assert (err <= u * want.abs() + 1e-5).all()
    assert (init.double().cpu() - torch.view_as_real(grad).flatten(-2)).abs().max() < 1e-5
    want = torch.view_as_real(torch.stack(want_dot, 1))
    assert (dot.double().cpu() - want).norm() < 1e-5 * want.norm()


@pytest.mark.parametrize("N,dtype", [(32, torch.bfloat16), (64, torch.bfloat16), (128, torch.float16)])
def test_rows_through_l2_leave_the_outputs_alone(N, dtype):
    """Forwards of more than 2664 chunks fetch whole rows into L2 (N > 32), the ragged last chunk's among them: same bits as
    the same heads in launches of half the size, which do not."""
    import slinoss_b200 as sb

    inp = make_scan_inputs(1, 1340, 128 + 71, N, 64, dtype, seed=N, dist="cfg2", with_init=True, streaming=True)
    names = ("U", "M", "K", "B", "C")
    carried = ("initial_states", "B_prev", "U_prev")

    def run(h):
        with torch.no_grad():
            return sb.v2x2ssd_b200(*(inp[k][:, h] for k in names), chunk_size=128, return_state=True,
                                   **{k: inp[k][:, h] for k in carried})

    whole, halves = run(slice(None)), [run(slice(i, i + 670)) for i in (0, 670)]
    for w, *h in zip(whole, *halves):
        assert torch.equal(w, torch.cat(h, 1))

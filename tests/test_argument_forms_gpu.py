"""Forms of arguments that the ops take besides the plain one: addresses, strides, storage types."""

from __future__ import annotations

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

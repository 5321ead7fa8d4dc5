"""Chunk kernels of the scan at the points where their own geometry changes."""

from __future__ import annotations

from ctypes import byref

import pytest
import torch

from gpu_util import make_scan_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,T", [(32, 128), (96, 300), (128, 129)])
def test_gradient_rows_off_a_32_byte_boundary(dtype, N, T):
    """dB and dC leave as whole 32-byte sectors where their base allows it, else as two 16-byte stores: same bits."""
    import slinoss_b200 as sb
    from slinoss_b200 import _lib

    inp = make_scan_inputs(1, 2, T, N, 64, dtype, seed=N, dist="cfg2", with_init=True)
    U, M, K, B, C, dY = (inp[k] for k in ("U", "M", "K", "B", "C", "dY"))
    s = _lib.scan_shape(2, T, 64, N, 128, dtype, _lib.starts_dtype(_lib.scan_shape(2, T, 64, N, 128, dtype)))
    NC = (T + 127) // 128
    inc, mch = sb.chunk_increment_b200(U, M, K, B, chunk_size=128)
    starts, _ = sb.state_passing_b200(inc, mch, initial_states=inp["initial_states"])
    starts = starts.to(dtype).contiguous()
    d_inc = torch.randn_like(starts)
    zdot = torch.randn(2, NC, 2, device="cuda")
    outs = []
    for off in (0, 8):
        flat = [torch.zeros(2 * T * 2 * N + 16, device="cuda", dtype=dtype) for _ in range(2)]
        dB, dC = (f[off:off + 2 * T * 2 * N] for f in flat)
        assert dB.data_ptr() % 32 == 2 * off and dC.data_ptr() % 32 == 2 * off
        dU, dM, dK = torch.empty_like(U), torch.empty_like(M), torch.empty_like(K)
        cB, cU = torch.empty(2, NC, 2 * N, device="cuda"), torch.empty(2, NC, 64, device="cuda")
        rc = _lib.lib().slx_chunk_scan_bwd(
            byref(s), U.data_ptr(), M.data_ptr(), K.data_ptr(), B.data_ptr(), C.data_ptr(), None, None,
            starts.data_ptr(), d_inc.data_ptr(), zdot.data_ptr(), dY.data_ptr(), dU.data_ptr(), dM.data_ptr(),
            dK.data_ptr(), dB.data_ptr(), dC.data_ptr(), cB.data_ptr(), cU.data_ptr(), _lib.stream_ptr(U.device))
        _lib.check(rc, "chunk_scan_bwd")
        for f in flat:  # nothing outside the rows
            assert not f[:off].any() and not f[off + 2 * T * 2 * N:].any()
        outs.append([dU, dM, dK, dB.clone(), dC.clone(), cB, cU])
    for x, y in zip(*outs):
        assert torch.equal(x, y)

"""More than 2^27 lines of an axis: every one is factorised."""
import ctypes

import numpy as np
import pytest

from heatsim2_gb300 import _native

pytestmark = pytest.mark.gpu


def test_last_lines_of_a_large_plane(cuda_ok):
    """One layer of 11600 x 11600 voxels (134.6 million z lines of one row).  A problem and a field that are symmetric in y
    stay so to rounding, 1e-13 of the field; the last rows hold the lines past the 2^27th."""
    import torch
    ny = nx = 11600
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("needs 60 GB of device memory")
    Gz, Gy, Gx = np.zeros((2, ny, nx)), np.full((1, ny + 1, nx), 2e6), np.full((1, ny, nx + 1), 3e6)
    Gy[:, [0, -1]] = 0.0
    Gx[:, :, [0, -1]] = 0.0
    M, fixed = np.full((1, ny, nx), 4e6), np.zeros((1, ny, nx), dtype=np.uint8)
    p = _native.DenseProblem(1, ny, nx, Gz.ctypes.data, Gy.ctypes.data, Gx.ctypes.data, M.ctypes.data, fixed.ctypes.data,
                             None)
    L, h = _native.load(), ctypes.c_void_p()
    _native.check(L.hs2g_create_dense(ctypes.byref(p), 0, ctypes.byref(h)))
    try:
        T = 293.0 + torch.rand(ny, nx, dtype=torch.float64, device="cuda")
        T = 0.5 * (T + T.flip(0))
        out = torch.empty_like(T)
        torch.cuda.synchronize()
        _native.check(L.hs2g_step(h, T.data_ptr(), out.data_ptr(), None, None, None, _native.DEVICE | _native.SYNC))
        assert torch.isfinite(out).all()
        assert (out - out.flip(0)).abs().max().item() <= 1e-13 * out.abs().max().item()
        assert (out - T).abs().max().item() > 0.01
    finally:
        L.hs2g_destroy(h)
        del T, out
        torch.cuda.empty_cache()

"""Steps and runs on host buffers through the C ABI: their waits are their own stream's."""
import numpy as np
import pytest

import heatsim2_gb300 as hs
from heatsim2_gb300 import _native
from heatsim2_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _panel(shape):
    nz, ny, nx = shape
    return W.composite_panel(seed=4, nz=nz - 1, ny=ny, nx=nx, top_layers=4, width_range=(5, min(ny, nx) // 4),
                             depth_range=(2, nz // 2), nsteps=3)


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("shape", [(9, 30, 41), (64, 256, 65)])
def test_host_steps_do_not_wait_for_other_streams(cuda_ok, shape, pinned):
    """A handle with a stream of its own: a step and a run on host buffers end while the default stream is still busy."""
    import torch
    spec = _panel(shape)
    P, S = hs.setup(*W.setup_args(hs, spec))
    T = torch.from_numpy(W.initial_temperature(spec))
    T, out = (T.pin_memory(), torch.empty_like(T).pin_memory()) if pinned else (T, torch.empty_like(T))
    L = _native.load()
    for f in (lambda: L.hs2g_step(P.handle.ptr, T.data_ptr(), out.data_ptr(), None, None, None, 0),
              lambda: L.hs2g_run(P.handle.ptr, 3, T.data_ptr(), out.data_ptr(), None, 0, None, 0)):
        for _ in range(2):                       # staging buffers, modules and graphs exist from here on
            _native.check(f())
        done = torch.cuda.Event()
        torch.cuda._sleep(1_000_000_000)         # about half a second
        done.record()
        _native.check(f())
        assert not done.query()
        torch.cuda.synchronize()


@pytest.mark.parametrize("shape", [(64, 256, 72), (64, 256, 65), (16, 256, 256), (17, 250, 247)])
def test_overlapped_steps_of_page_locked_buffers_equal_device_path(cuda_ok, shape):
    """Page-locked host buffers of 2^20 voxels or more go up in slabs of planes and come back in blocks of rows while the
    sweeps run; at 64 planes the first slab's x lines take two kernels, the last slab's one, and the device path's two.
    The same bits, with and without a source, class sources and a field beside them, and into the input buffer."""
    import torch
    from heatsim2_gb300.alternatingdirection import _ClassSources, source_table
    spec = _panel(shape)
    assert W.voxels(spec) >= 1 << 20
    L = _native.load()
    sources = _ClassSources(W.volumetric_tuple(hs, spec))
    P, S = hs.setup(*W.setup_args(hs, spec))
    D, _ = hs.setup(*W.setup_args(hs, spec))
    rng = np.random.default_rng(3)
    T = torch.from_numpy(293.0 + rng.random(shape)).pin_memory()
    field = torch.from_numpy(1e6 * rng.random(shape)).pin_memory()
    out, dev, dfield = torch.empty_like(T).pin_memory(), T.cuda(), field.cuda()
    dout = torch.empty_like(dev)
    for n in range(4):
        q, _ = source_table(sources, n * spec["dt"], spec["dt"], D.volume_array)
        _native.check(L.hs2g_step(P.handle.ptr, T.data_ptr(), out.data_ptr(), q.ctypes.data,
                                  field.data_ptr() if n == 1 else None, None, 0))
        torch.cuda.synchronize()
        _native.check(L.hs2g_step(D.handle.ptr, dev.data_ptr(), dout.data_ptr(), q.ctypes.data,
                                  dfield.data_ptr() if n == 1 else None, None, _native.DEVICE | _native.SYNC))
        np.testing.assert_array_equal(out.numpy(), dout.cpu().numpy())
        T, out = (out, out) if n == 2 else (out, T)      # the last step in place
        dev, dout = dout, dev

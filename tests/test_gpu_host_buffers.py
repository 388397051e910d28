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

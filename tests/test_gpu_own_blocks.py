"""Problems whose stencil blocks do not repeat: eight values per voxel, the weights as integers, or as doubles where no
integers stand for them.  Device memory, and steps through both forms of the x sweep."""
import ctypes

import numpy as np
import pytest

from conftest import rel_err
import oracle
from oracle_shim import HS
import heatsim2_gb300 as hs
from heatsim2_gb300 import _native
from heatsim2_gb300 import workloads as W
from heatsim2_gb300.batch import Batch

pytestmark = pytest.mark.gpu


def _random_faces(shape, conductances):
    spec = W.line_grid(shape, dt=0.01)
    spec["boundaries"] = [["conducting"], ["insulating"]] + [["thininsulatinglayer", float(h)] for h in conductances]
    spec["volumetric"] = [["none"]]
    a = spec["arrays"]
    a["volumetric"][:] = 0
    rng = np.random.default_rng(11)
    n = len(spec["boundaries"])
    for key, cut in (("boundary_z", np.s_[1:-1]), ("boundary_y", np.s_[:, 1:-1]), ("boundary_x", np.s_[:, :, 1:-1])):
        a[key][cut] = rng.integers(0, n, size=a[key][cut].shape).astype(np.uint8)
    return spec


def test_device_memory_of_blocks_that_do_not_repeat(cuda_ok):
    """Per voxel: three face conductances, capacity, mask, source class, two stage arrays, six line coefficients and
    eight stencil coefficients.  Line tables would only take less; a few words and allocations beside them."""
    shape = nz, ny, nx = (32, 64, 96)
    spec = _random_faces(shape, 50.0 + 37.0 * np.arange(40))
    P, S = hs.setup(*W.setup_args(hs, spec))
    faces = (nz + 1) * ny * nx + nz * (ny + 1) * nx + nz * ny * (nx + 1)
    most = 8 * faces + nz * ny * nx * (8 + 1 + 1 + 2 * 8 + 6 * 8 + 8 * 8) + 4096
    assert _native.load().hs2g_device_bytes(P.handle.ptr) <= most


@pytest.mark.parametrize("kind", ["kelvin", "rise", "mixed"])
@pytest.mark.parametrize("shape", [(9, 20, 70), (5, 130, 37), (40, 7, 1), (3, 4, 33)])
def test_steps_vs_oracle(cuda_ok, shape, kind):
    """Face conductances over twelve decades beside insulating ones: weights far below their voxel's largest, and none at
    all.  Single problem and batch (beside an instance whose blocks repeat): the same bits, within the parity bar."""
    spec = _random_faces(shape, 10.0 ** np.linspace(-6, 6, 40))
    rng = np.random.default_rng(4)
    T0 = 293.0 + rng.random(shape)
    if kind == "rise":
        T0 = 4.0 * rng.random(shape) ** 4
    elif kind == "mixed":
        T0 = np.where(rng.random(shape) < 0.5, T0 - 293.5, rng.choice([0.0, -0.0, 250.0, 1e-300, -7.0], size=shape))
    P, S = hs.setup(*W.setup_args(hs, spec))
    Po, _ = oracle.setup(*W.setup_args(HS, spec))
    vol = W.volumetric_tuple(hs, spec)
    T = ref = T0
    for t in (0.0, 0.01):
        T = hs.run_adi_steps(P, S, t, spec["dt"], T, spec["arrays"]["volumetric"], vol)
        ref = oracle.run_adi_steps(Po, None, t, spec["dt"], ref, spec["arrays"]["volumetric"], vol)
    assert rel_err(T, ref) <= 1e-12
    other = W.steel_slab(seed=2, nz=12, ny=20, nx=40, flaw=4, depth_range=(2, 9))
    b = Batch([W.setup_args(hs, spec), W.setup_args(hs, other)], precision=64)
    b.set_temperature([T0, W.initial_temperature(other)])
    b.run(2)
    np.testing.assert_array_equal(b.get_temperature()[0], T)


@pytest.mark.parametrize("negative", [False, True])
@pytest.mark.parametrize("nx", [1, 2, 33, 64, 400])
def test_few_equal_lines_with_blocks_of_their_own(cuda_ok, nx, negative):
    """x lines of one class in the one-kernel form of the x sweep, their blocks all different: line L has 2^L times the
    capacity and conductances of the first (the same line coefficients, another source weight).  Some negative
    conductances: weights that stay doubles.  Against dense solves."""
    nz, ny = 4, 4
    rng = np.random.default_rng(nx)
    g = rng.uniform(0.1, 1e6, nx + 1)
    if negative:
        g[1::3] *= -0.3
    g[0] = g[-1] = 0.0
    m = rng.uniform(1e6, 4e6, nx)
    scale = 2.0 ** np.arange(nz * ny).reshape(nz, ny, 1)
    Gx, M = np.ascontiguousarray(scale * g), np.ascontiguousarray(scale * m)
    Gz, Gy, fixed = np.zeros((nz + 1, ny, nx)), np.zeros((nz, ny + 1, nx)), np.zeros((nz, ny, nx), dtype=np.uint8)
    dense = _native.DenseProblem(nz, ny, nx, Gz.ctypes.data, Gy.ctypes.data, Gx.ctypes.data, M.ctypes.data,
                                 fixed.ctypes.data, None)
    L, h = _native.load(), ctypes.c_void_p()
    _native.check(L.hs2g_create_dense(ctypes.byref(dense), 0, ctypes.byref(h)))
    try:
        T = 293.0 + rng.random((nz, ny, nx))
        out, q = np.empty_like(T), 1e6 * scale * rng.random((nz, ny, nx))
        _native.check(L.hs2g_step(h, T.ctypes.data, out.ctypes.data, None, q.ctypes.data, None, 0))
    finally:
        L.hs2g_destroy(h)
    lap = np.diag(g[1:-1], 1) + np.diag(g[1:-1], -1) - np.diag(g[:-1] + g[1:])
    for k in range(nz):
        for j in range(ny):
            rhs = lap @ (T[k, j] - 293.0) + q[k, j] / scale[k, j]
            ref = T[k, j] + np.linalg.solve(np.diag(m) - lap / 2, rhs)
            assert rel_err(out[k, j], ref) <= 1e-12


@pytest.mark.parametrize("shape", [(1, 2050, 2112), (64, 256, 256)])
def test_setup_where_the_search_has_no_room(cuda_ok, shape):
    """200 bytes per voxel left on the device: what a handle keeps (162 and the planes' extra faces) and the factors' two
    arrays, but not the search for equal lines and blocks beside them.  The same step, bit for bit."""
    import torch
    L = _native.load()
    spec = _random_faces(shape, 50.0 + 37.0 * np.arange(40))
    args = W.setup_args(hs, spec)
    T = 293.0 + torch.rand(shape, dtype=torch.float64, device="cuda")
    out = [torch.empty_like(T), torch.empty_like(T)]
    hold = None
    try:
        for o in out:
            P, _ = hs.setup(*args)
            _native.check(L.hs2g_step(P.handle.ptr, T.data_ptr(), o.data_ptr(), None, None, None,
                                      _native.DEVICE | _native.SYNC))
            del P
            if hold is None:
                torch.cuda.empty_cache()
                hold = torch.empty(torch.cuda.mem_get_info()[0] - 200 * T.numel(), dtype=torch.uint8, device="cuda")
    finally:
        del hold
        torch.cuda.empty_cache()
    assert torch.equal(*out)


def test_batch_where_the_search_has_no_room(cuda_ok):
    """The same for a batch of one: 260 bytes per voxel left, which state, coefficients and blocks (137) and the
    compilation's own arrays (99) need without the scratch of the search."""
    import torch
    shape = (1, 2050, 2112)
    spec = _random_faces(shape, 50.0 + 37.0 * np.arange(40))
    args = W.setup_args(hs, spec)
    T = 293.0 + np.random.default_rng(1).random(shape)
    out, hold = [], None
    try:
        for _ in range(2):
            b = Batch([args], precision=64)
            b.set_temperature([T])
            b.run(2)
            out.append(b.get_temperature()[0])
            del b
            if hold is None:
                torch.cuda.empty_cache()
                hold = torch.empty(torch.cuda.mem_get_info()[0] - 260 * T.size, dtype=torch.uint8, device="cuda")
    finally:
        del hold
        torch.cuda.empty_cache()
    np.testing.assert_array_equal(*out)

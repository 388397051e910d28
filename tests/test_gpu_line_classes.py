"""The search for equal lines at its edges: lines of 16, 17, 1023 and 1024 rows (where the shares of a line change), counts
of lines around the 8 and 32 that a block takes, one line and one class, and classes of which a few lines differ in their
first, last or a middle row alone.  Against the oracle, and the same bits in a batch."""
import numpy as np
import pytest

from conftest import rel_err
import oracle
from oracle_shim import HS
import heatsim2_gb300 as hs
from heatsim2_gb300 import workloads as W
from heatsim2_gb300.batch import Batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 16), (3, 3, 17), (3, 11, 16), (9, 7, 15), (1100, 3, 9), (3, 1100, 5), (1023, 2, 33),
                                   (2, 1024, 31), (2, 3, 1030), (33, 8, 64), (8, 33, 65)])
def test_tables_of_lines_that_differ_in_one_row(cuda_ok, shape):
    nz, ny, nx = shape
    spec = W.line_grid(shape, dt=0.01)
    spec["boundaries"] = spec["boundaries"][:2] + [["thininsulatinglayer", 100.0], ["thininsulatinglayer", 300.0]]
    spec["volumetric"] = [["none"]]
    a = spec["arrays"]
    a["volumetric"][:] = 0
    for key, n, axis in (("boundary_z", nz, 0), ("boundary_y", ny, 1), ("boundary_x", nx, 2)):
        faces = np.moveaxis(a[key], axis, 0)
        for line, row in ((0, 1), (-1, n - 1), (1, n // 2)):
            if 0 < row < n:
                view = faces[row]
                view[np.unravel_index(line % view.size, view.shape)] = 3
    T = ref = 293.0 + np.random.default_rng(1).random(shape)
    P, S = hs.setup(*W.setup_args(hs, spec))
    Po, _ = oracle.setup(*W.setup_args(HS, spec))
    vol = W.volumetric_tuple(hs, spec)
    b = Batch([W.setup_args(hs, spec)] * 2, precision=64)
    b.set_temperature([T, T])
    b.run(2)
    for n in range(2):
        T = hs.run_adi_steps(P, S, n * spec["dt"], spec["dt"], T, a["volumetric"], vol)
        ref = oracle.run_adi_steps(Po, None, n * spec["dt"], spec["dt"], ref, a["volumetric"], vol)
    assert rel_err(T, ref) <= 1e-12
    np.testing.assert_array_equal(b.get_temperature()[1], T)

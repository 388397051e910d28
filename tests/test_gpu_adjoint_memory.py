"""Device memory of an adjoint: what its fields need, and one pad column per row of an odd nx."""
import numpy as np
import pytest

from heatsim2_gb300.adjoint import Adjoint

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(8, 9, 32), (8, 9, 33), (8, 9, 34), (7, 5, 3), (40, 50, 97)])
def test_fields_and_stores_hold_one_pad_column_at_most(cuda_ok, shape):
    nz, ny, nx = shape
    n, steps, ckpt = nz * ny * (nx + nx % 2), 6, 2
    a = Adjoint([(shape, (1e-3,) * 3)], 0.01)
    assert a.device_bytes <= 30 * 8 * n
    a.set_parameters(np.full(shape, 54.0), np.full(shape, 3.7e6), np.zeros(shape))
    a.forward(np.random.default_rng(1).random(shape), np.zeros((steps, ny, nx)), np.ones(steps), ckpt)
    a.backward()
    stores = (steps // ckpt + 2 * 4 * ckpt) * n + steps * ny * nx + 2 * 32 * steps
    assert a.device_bytes <= 8 * (30 * n + stores)

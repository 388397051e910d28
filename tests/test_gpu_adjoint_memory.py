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


def test_instances_after_one_of_an_odd_count_of_pairs(cuda_ok):
    """Instances start on whole sectors, a pair of voxels after the one before where that has an odd count of pairs: each
    one's loss and gradients are those it has alone, bit for bit."""
    shapes = [(3, 3, 2), (5, 3, 17), (1, 1, 1), (3, 3, 34), (2, 7, 5), (3, 1, 50)]
    rng = np.random.default_rng(3)
    k = [54.0 * np.exp(0.2 * rng.standard_normal(s)) for s in shapes]
    C, q = [3.6e6 * (1.0 + rng.random(s)) for s in shapes], [1e8 * rng.random(s) for s in shapes]
    T0, obs = [293.0 + rng.random(s) for s in shapes], [293.0 + rng.random((4,) + s[1:]) for s in shapes]
    schedule = [1.0, 0.0, 0.5, 0.0]

    def evaluate(sel):
        a = Adjoint([(shapes[i], (1e-3,) * 3) for i in sel], 0.01)
        out = []
        for _ in range(2):                       # the second forward pass keeps states in the stores
            a.set_parameters([k[i] for i in sel], [C[i] for i in sel], [q[i] for i in sel])
            loss = a.forward([T0[i] for i in sel], [obs[i] for i in sel], schedule, 2)
            out.append((loss, a.backward()))
        return out
    for n, (loss, grads) in enumerate(evaluate(range(len(shapes)))):
        for i in range(len(shapes)):
            alone, ga = evaluate([i])[n]
            assert loss[i] == alone[0]
            for x, y in zip(grads, ga):
                np.testing.assert_array_equal(x[i], y)

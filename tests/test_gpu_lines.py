"""The sweeps' line solves at the sizes where they can go wrong: line lengths around the blocks of eight rows of a half
line (1 to 3 rows, 15 to 18, 33), row widths around the warps' 16 lines with odd ones among them, coefficients from
tables per line class (a layered problem) and in voxel order (faces drawn at random, so that no two lines are alike),
forward values kept in shared memory and, for long lines, sent through global memory; double and float.  Against the
oracle, 2 steps: FP64 within the parity bar of 1e-12 of max|T|, FP32 within the 1e-7 of its stated error."""
import numpy as np
import pytest

from conftest import rel_err
import oracle
from oracle_shim import HS
import heatsim2_gb300 as hs
from heatsim2_gb300 import workloads as W
from heatsim2_gb300.batch import Batch

pytestmark = pytest.mark.gpu

SMALL = [(1, 2, 16), (2, 1, 15), (3, 3, 17), (15, 18, 33), (16, 17, 1), (17, 16, 31), (33, 15, 16), (18, 33, 47)]
LONG = [(2, 700, 80), (700, 2, 40), (8, 300, 1700), (300, 8, 1700)]


def _spec(shape, random_faces):
    nz, ny, nx = shape
    spec = W.line_grid(shape, dt=0.01)
    spec["boundaries"] = [["conducting"], ["insulating"]] + [["thininsulatinglayer", 50.0 + 37.0 * c] for c in range(40)]
    spec["volumetric"] = [["none"], ["stepped", 0.0, 1.0, 2e8]]
    a = spec["arrays"]
    a["volumetric"][:] = 0
    a["volumetric"][0] = 1
    if random_faces:
        rng = np.random.default_rng(sum(shape))
        for key, cut in (("boundary_z", np.s_[1:-1]), ("boundary_y", np.s_[:, 1:-1]), ("boundary_x", np.s_[:, :, 1:-1])):
            a[key][cut] = rng.choice([0] + list(range(2, 42)), size=a[key][cut].shape)
    return spec


def _field(shape, kind="kelvin"):
    T = 293.0 + np.random.default_rng(4).random(shape)
    if kind == "mixed":       # signs, binary exponents and zeros side by side: the stencil's FP64 chain, voxel by voxel
        rng = np.random.default_rng(5)
        T = np.where(rng.random(shape) < 0.5, T - 293.5, rng.choice([0.0, -0.0, 250.0, 260.0, 1e-300, -7.0], size=shape))
    elif kind == "negative":  # one sign and exponent
        T = -T
    return T


@pytest.mark.parametrize("kind", ["kelvin", "mixed", "negative"])
@pytest.mark.parametrize("shape", [(9, 20, 70), (5, 130, 37)])
def test_stencil_of_any_temperatures_vs_oracle(cuda_ok, shape, kind):
    """The stencil in integers and in FP64, for all voxels and for some of a warp's, and through the two layouts of the
    x sweep (the batch takes it in two kernels, the small problem in one): the same bits, within the parity bar."""
    spec = _spec(shape, False)
    vol = W.volumetric_tuple(hs, spec)
    P, S = hs.setup(*W.setup_args(hs, spec))
    Po, _ = oracle.setup(*W.setup_args(HS, spec))
    T0 = _field(shape, kind)
    T = hs.run_adi_steps(P, S, 0.0, spec["dt"], T0, spec["arrays"]["volumetric"], vol)
    assert rel_err(T, oracle.run_adi_steps(Po, None, 0.0, spec["dt"], T0, spec["arrays"]["volumetric"], vol)) <= 1e-12
    b = Batch([W.setup_args(hs, spec)], precision=64)
    b.set_temperature([T0])
    b.set_sources([0.0], spec["dt"])
    b.run(1)
    np.testing.assert_array_equal(b.get_temperature()[0], T)


@pytest.mark.parametrize("random_faces", [False, True])
@pytest.mark.parametrize("shape", SMALL + LONG)
def test_line_solves_vs_oracle(cuda_ok, shape, random_faces):
    spec = _spec(shape, random_faces)
    vol = W.volumetric_tuple(hs, spec)
    P, S = hs.setup(*W.setup_args(hs, spec))
    Po, _ = oracle.setup(*W.setup_args(HS, spec))
    T = ref = _field(shape)
    for t in (0.0, 0.01):
        T = hs.run_adi_steps(P, S, t, spec["dt"], T, spec["arrays"]["volumetric"], vol)
        ref = oracle.run_adi_steps(Po, None, t, spec["dt"], ref, spec["arrays"]["volumetric"], vol)
    assert rel_err(T, ref) <= 1e-12
    for precision, tol in ((64, 0.0), (32, 1e-7)):      # the batched form: the same bits in double
        b = Batch([W.setup_args(hs, spec)], precision=precision)
        b.set_temperature([_field(shape)])
        b.set_sources([0.0, 0.01], spec["dt"])
        b.run(2)
        got = b.get_temperature()[0]
        assert rel_err(got, T) <= tol, precision


def test_problems_of_several_sizes_side_by_side(cuda_ok):
    """What a problem's setup allows its kernels (shared memory) never takes from an earlier, larger problem."""
    made = []
    for shape in [(3, 3, 1000), (3, 700, 40), (3, 3, 400), (3, 300, 40)]:
        spec = _spec(shape, False)
        P, S = hs.setup(*W.setup_args(hs, spec))
        made.append((P, S, spec, shape))

    def step(P, S, spec, shape):
        return hs.run_adi_steps(P, S, 0.0, spec["dt"], _field(shape), spec["arrays"]["volumetric"],
                                W.volumetric_tuple(hs, spec))
    for P, S, spec, shape in made:
        alone, _ = oracle.setup(*W.setup_args(HS, spec))
        ref = oracle.run_adi_steps(alone, None, 0.0, spec["dt"], _field(shape), spec["arrays"]["volumetric"],
                                   W.volumetric_tuple(hs, spec))
        assert rel_err(step(P, S, spec, shape), ref) <= 1e-12

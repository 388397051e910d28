"""Fields at the ends of the number range, with infinities and NaN, and the two places a sweep keeps its forward values."""
import numpy as np
import pytest

from conftest import rel_err
import oracle
from oracle_shim import HS
import heatsim2_gb300 as hs
from heatsim2_gb300 import workloads as W
from heatsim2_gb300.batch import Batch

pytestmark = pytest.mark.gpu


def _spec(shape, random_faces):
    spec = W.line_grid(shape, dt=0.01)
    spec["boundaries"] = [["conducting"], ["insulating"]] + [["thininsulatinglayer", 50.0 + 37.0 * c] for c in range(40)]
    spec["volumetric"] = [["none"]]
    a = spec["arrays"]
    a["volumetric"][:] = 0
    if random_faces:
        rng = np.random.default_rng(sum(shape))
        for key, cut in (("boundary_z", np.s_[1:-1]), ("boundary_y", np.s_[:, 1:-1]), ("boundary_x", np.s_[:, :, 1:-1])):
            a[key][cut] = rng.integers(2, 42, size=a[key][cut].shape).astype(np.uint8)
    return spec


def _step(spec, T0, steps=1):
    """The single problem's field and the oracle's; the batch's is checked to be the same bits."""
    vol = W.volumetric_tuple(hs, spec)
    P, S = hs.setup(*W.setup_args(hs, spec))
    Po, _ = oracle.setup(*W.setup_args(HS, spec))
    T = ref = T0
    with np.errstate(all="ignore"):
        for n in range(steps):
            T = hs.run_adi_steps(P, S, n * spec["dt"], spec["dt"], T, spec["arrays"]["volumetric"], vol)
            ref = oracle.run_adi_steps(Po, None, n * spec["dt"], spec["dt"], ref, spec["arrays"]["volumetric"], vol)
    b = Batch([W.setup_args(hs, spec)], precision=64)
    b.set_temperature([T0])
    b.run(steps)
    np.testing.assert_array_equal(b.get_temperature()[0], T)
    return T, ref


@pytest.mark.parametrize("random_faces", [False, True])
@pytest.mark.parametrize("scale", [1e290, 1e-280, -1e290])
def test_fields_near_the_ends_of_the_range(cuda_ok, scale, random_faces):
    shape = (9, 20, 70)
    T, ref = _step(_spec(shape, random_faces), scale * (1.0 + 0.2 * np.random.default_rng(1).random(shape)), 2)
    assert rel_err(T / scale, ref / scale) <= 1e-12


@pytest.mark.parametrize("random_faces", [False, True])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_infinities_and_nan_reach_what_they_reach_in_the_oracle(cuda_ok, value, random_faces):
    """One such value among ordinary ones, in a corner, on a warp's and a block's edge and inside."""
    shape = (5, 20, 70)
    spec = _spec(shape, random_faces)
    for at in ((0, 0, 0), (2, 15, 31), (4, 16, 32), (3, 7, 50)):
        T0 = 293.0 + np.random.default_rng(2).random(shape)
        T0[at] = value
        T, ref = _step(spec, T0)
        np.testing.assert_array_equal(np.isfinite(T), np.isfinite(ref))


@pytest.mark.parametrize("random_faces", [False, True])
@pytest.mark.parametrize("value", [np.finfo(np.float64).max, np.finfo(np.float64).min])
def test_largest_and_lowest_value_among_ordinary_ones(cuda_ok, value, random_faces):
    """The step forms no product beyond the range (the oracle's M T overflows here): the oracle's step of the field scaled
    down, scaled up."""
    shape = (5, 20, 70)
    spec = _spec(shape, random_faces)
    Po, _ = oracle.setup(*W.setup_args(HS, spec))
    for at in ((0, 0, 0), (2, 15, 31), (4, 16, 32), (3, 7, 50)):
        T0 = 293.0 + np.random.default_rng(2).random(shape)
        T0[at] = value
        P, S = hs.setup(*W.setup_args(hs, spec))
        vol = W.volumetric_tuple(hs, spec)
        T = hs.run_adi_steps(P, S, 0.0, spec["dt"], T0, spec["arrays"]["volumetric"], vol)
        ref = oracle.run_adi_steps(Po, None, 0.0, spec["dt"], T0 / value, spec["arrays"]["volumetric"], vol)
        assert rel_err(T / value, ref) <= 1e-12


@pytest.mark.parametrize("random_faces", [False, True])
@pytest.mark.parametrize("shape", [(4, 700, 160), (700, 4, 160), (4, 100, 1000)])
def test_forward_values_in_shared_and_in_global_memory(cuda_ok, shape, random_faces):
    """Long lines of one problem keep them in shared memory; twelve such problems side by side are more warps than that
    leaves room for.  The same bits, with coefficients from tables and in voxel order."""
    spec = _spec(shape, random_faces)
    fields = [293.0 + np.random.default_rng(i).random(shape) for i in range(12)]
    b = Batch([W.setup_args(hs, spec)] * 12, precision=64)
    b.set_temperature(fields)
    b.run(2)
    got = b.get_temperature()
    P, S = hs.setup(*W.setup_args(hs, spec))
    for i in (0, 11):
        T = fields[i]
        for n in range(2):
            T = hs.run_adi_steps(P, S, n * spec["dt"], spec["dt"], T, spec["arrays"]["volumetric"],
                                 W.volumetric_tuple(hs, spec))
        np.testing.assert_array_equal(got[i], T)

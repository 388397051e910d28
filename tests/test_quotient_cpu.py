"""The quotient of adj_factor_kernel (heatsim2_gb300/csrc/hs2g_adjoint.cu), in / piv from the rounded reciprocal of piv and
one correction step, in exact arithmetic rounded where the kernel rounds: against ordinary division, for rows of ordinary
voxels and for rows beside fixed ones, whose capacity is 1e300."""
from fractions import Fraction

import numpy as np
import pytest


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def _quotient(num, piv):
    inv = 1.0 / piv
    q = num * inv
    return _fma(_fma(-q, piv, num), inv, q)


@pytest.mark.parametrize("kind", ["ordinary", "fixed", "beside_fixed"])
def test_corrected_quotient_is_the_quotient(kind):
    rng = np.random.default_rng(1)
    num = 10.0 ** rng.uniform(-3, 12, 4000)
    if kind == "fixed":                  # the fixed voxel's own row
        piv = 1e300 + num
    elif kind == "beside_fixed":         # a row whose neighbour's half conductance is its pivot's largest part
        piv = num * (1.0 + 10.0 ** rng.uniform(-15, 0, num.size))
    else:
        piv = num * 10.0 ** rng.uniform(0, 8, num.size) + 10.0 ** rng.uniform(3, 10, num.size)
    for a, b in zip(num.tolist(), piv.tolist()):
        assert _quotient(a, b) == a / b

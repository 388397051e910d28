"""Rounding of the adjoint's single operations, where a gradient shows them by themselves."""
import numpy as np
import pytest

from heatsim2_gb300.adjoint import Adjoint

pytestmark = pytest.mark.gpu


def _solve(lo, d, hi, b):
    """Tridiagonal solve in extended precision."""
    n, d, b = len(d), d.copy(), b.copy()
    for i in range(1, n):
        f = lo[i] / d[i - 1]
        d[i] -= f * hi[i - 1]
        b[i] -= f * b[i - 1]
    b[-1] /= d[-1]
    for i in range(n - 2, -1, -1):
        b[i] = (b[i] - hi[i] * b[i + 1]) / d[i]
    return b


@pytest.mark.parametrize("nx", [37, 600])
def test_face_gradient_keeps_the_digits_of_small_increments(cuda_ok, nx):
    """One step of a line whose halves are at +1000 and -1000 K and warm by some 1e-5 K: the increments' differences make
    the gradient of k away from the jump.  Two neighbours' shares are within 1e-11 of the larger one: the residual rounds
    lambda T = 1e-3 K (lambda = G / M = 1e-6) to 1e-19, 1e-14 of an increment, and a difference of two values of the
    misfit's gradient loses at most two digits; rounding an increment to the last place of T would leave 1e-8."""
    d, dt, k, C = 1e-3, 1e-4, 0.04, 4e6
    G, M = np.longdouble(k) / np.longdouble(d) ** 2, np.longdouble(C) / np.longdouble(dt)
    rng = np.random.default_rng(nx)
    T0 = np.where(np.arange(nx) < nx // 2, 1000.0, -1000.0)
    q = 1e-5 * C / dt * (1.0 + np.arange(nx) % 3)
    obs = rng.uniform(-3000.0, 3000.0, nx)
    a = Adjoint([((1, 1, nx), (d, d, d))], dt)
    a.set_parameters(np.full((1, 1, nx), k), np.full((1, 1, nx), C), q.reshape(1, 1, nx))
    shift = T0.mean()
    a.forward(T0.reshape(1, 1, nx), obs.reshape(1, 1, nx), [1.0], 1)
    got = a.backward()[0].reshape(-1).astype(np.longdouble)
    T, ob = (T0 - shift).astype(np.longdouble), (obs - shift).astype(np.longdouble)
    lo, hi = np.full(nx, -G / 2), np.full(nx, -G / 2)
    lo[0] = hi[-1] = 0
    dg = M - lo - hi
    r = q.astype(np.longdouble)
    r[1:] += G * (T[:-1] - T[1:])
    r[:-1] += G * (T[1:] - T[:-1])
    y = _solve(lo, dg, hi, r)
    mu = _solve(lo, dg, hi, 2 * (T + y - ob))
    face = np.zeros(nx + 1, dtype=np.longdouble)
    face[1:-1] = -np.diff(mu) * (np.diff(T) + np.diff(y) / 2)
    half = face / (2 * np.longdouble(d) ** 2)
    err = np.abs(got - (half[:-1] + half[1:])) / np.maximum(np.abs(half[:-1]), np.abs(half[1:]))
    assert err.max() <= 1e-11

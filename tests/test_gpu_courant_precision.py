"""The Courant step of the float64 SPH is as exact as its last operations allow: its mean error against
extended precision stays below one rounding, 2^-53, on neighbourhoods of a search (a cloud, a flat
disk with a wide range of densities, a core in a cloud)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(kind, n, rng):
    x = rng.normal(size=(n, 3))
    if kind == "disk":
        x *= np.array([3.0, 3.0, 0.3]) * rng.exponential(size=(n, 1))
    elif kind == "core":
        x[::2] *= 0.05
    return x


def _step(x, v, nb, h, u, alpha, beta):
    long = np.longdouble
    if np.finfo(long).eps >= np.finfo(np.float64).eps:
        pytest.skip("no extended precision in this NumPy")
    x, v, h, u = (a.astype(long) for a in (x, v, h, u))
    gamma = long(5.0 / 3.0)
    d = x[:, None, :] - x[nb]
    vr = ((v[:, None, :] - v[nb]) * d).sum(2)
    hb = (h[:, None] + h[nb]) / 2
    mu = np.where(vr < 0, hb * vr / ((d * d).sum(2) + long("0.01") * hb * hb), long(0))
    c = np.sqrt(gamma * (gamma - 1) * u)
    return long("0.3") * h / (c + long("1.2") * (alpha * c + beta * (-mu).max(1)) + long("1e-30"))


@pytest.mark.parametrize("kind", ["cloud", "disk", "core"])
@pytest.mark.parametrize("n", [6000, 20000])
def test_mean_error_of_the_courant_step(gpulib, kind, n):
    from galaxy_formation_gb300 import sph

    rng = np.random.default_rng(n)
    x = _points(kind, n, rng)
    v, m, u = rng.normal(size=(n, 3)), rng.uniform(0.5, 1.5, n) / n, rng.uniform(0.1, 10.0, n)
    dist, nb = sph.knn(x, 32)
    h = 0.5 * dist[:, -1]
    rho, acc, dudt, dt = np.empty(n), np.empty((n, 3)), np.empty(n), np.empty(n)
    sph.sph_forces(x, v, m, nb, h, u, 5.0 / 3.0, 1.0, 2.0, rho, acc, dudt, dt)
    want = _step(x, v, nb, h, u, 1, 2)
    assert float(np.mean(np.abs((dt - want) / want))) < 2.0**-53

"""The direct sum split over a cluster's blocks: particle counts at the edges of the source tiles and
parts (fewer tiles than parts, a partial last tile), target lists, and distances outside the range
of the fast power (which take the division), against NumPy in float64. A pair term takes fewer
than 30 rounded operations and a component sums n <= 1000 of them, so it is within (n + 30) 2^-53 <
1.2e-13 of the sum of the terms' absolute values (x_j - x_i is the same rounded number on both
sides)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(x, m, eps, rows):
    d = x[None, :, :] - x[rows][:, None, :]
    r2 = (d * d).sum(2) + eps * eps
    with np.errstate(divide="ignore", invalid="ignore"):
        t = (m[None, :] / (r2 * np.sqrt(r2)))[..., None] * d
    return t.sum(1), np.abs(t).sum(1)


@pytest.mark.parametrize("scale", [1.0, 1e95, 1e-95])
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 511, 512, 513, 1000])
def test_direct_sum(gpulib, n, scale):
    from galaxy_formation_gb300.engine import Engine

    rng = np.random.default_rng(n)
    x, m, eps = rng.normal(size=(n, 3)) * scale, rng.uniform(0.5, 1.5, n), 0.05 * scale
    ref, size = _reference(x, m, eps, np.arange(n))
    acc = Engine().gravity_direct(x, m, eps)
    assert np.all(np.abs(acc - ref) <= 1.2e-13 * size)
    rows = rng.integers(0, n, size=min(n, 70))
    at = Engine().gravity_direct_targets(x, m, rows, eps)
    assert np.array_equal(at, acc[rows])


def test_direct_sum_without_softening(gpulib):
    from galaxy_formation_gb300.engine import Engine

    rng = np.random.default_rng(1)
    x, m = rng.normal(size=(100, 3)), rng.uniform(0.5, 1.5, 100)
    assert np.isnan(Engine().gravity_direct(x, m, 0.0)).all()  # the pair with itself is 0 / 0, as in the reference

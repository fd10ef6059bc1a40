"""Opening angles at the ends of the range: a node's opening radius is 2 half / theta plus the distance
of its centre of mass, whatever theta is."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("theta", [np.inf, -np.inf, 1e39, 1e30, 0.7, 1e-30, -0.7])
@pytest.mark.parametrize("n", [50, 3000, 40000])
def test_opening_radii(gpulib, n, theta):
    from galaxy_formation_gb300.engine import Engine

    rng = np.random.default_rng(n)
    x, m = rng.normal(size=(n, 3)), rng.uniform(0.5, 1.5, n)
    t = Engine().build_tree(x, m, theta)
    half = t["half"].astype(float)
    com = np.stack([t["cx"], t["cy"], t["cz"]], 1).astype(float)
    centre = np.stack([t["gx"], t["gy"], t["gz"]], 1).astype(float)
    with np.errstate(over="ignore"):
        want = 2 * half / np.float64(np.float32(theta)) + np.linalg.norm(com - centre, axis=1)
    # float32 records: each of their 2^-24 roundings counts with the values that it rounds
    size = np.abs(want) + half + np.abs(centre).max(axis=1)
    finite = np.abs(want) < 1e37
    got = t["open_r"].astype(float)
    assert np.all(np.abs(got - want)[finite] <= 8 * 2.0**-24 * size[finite])
    assert np.all(np.abs(got[~finite]) > 1e36)

"""A particle with no neighbour but itself is not heated (sph.py:72-106 adds nothing up), also where
its pressure over density squared is no number: without mass, with an internal energy or a smoothing
length that is no number. With each number of lanes per particle, and rows of one entry or several."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ODD = 100


@pytest.mark.parametrize("n", [600, 20000, 200000, 300000])
@pytest.mark.parametrize("k", [1, 7])
@pytest.mark.parametrize("field,value", [("mass", 0.0), ("u", np.nan), ("u", np.inf), ("h", np.nan), ("h", 0.0)])
def test_no_heating_without_neighbours(gpulib, n, k, field, value):
    from galaxy_formation_gb300 import sph

    rng = np.random.default_rng(n)
    d = {"mass": rng.uniform(0.5, 1.5, n) / n, "h": rng.uniform(0.3, 3.0, n), "u": rng.uniform(0.1, 10.0, n)}
    nb = np.ascontiguousarray((np.arange(n)[:, None] + np.arange(k)[None, :]) % n, np.int64)
    nb[ODD] = ODD
    d[field][ODD] = value
    rho, acc, dudt, dt = np.empty(n), np.empty((n, 3)), np.full(n, 7.0), np.empty(n)
    sph.sph_forces(rng.normal(size=(n, 3)), rng.normal(size=(n, 3)), d["mass"], nb, d["h"], d["u"], 5.0 / 3.0, 1.0, 2.0,
                   rho, acc, dudt, dt)
    assert dudt[ODD] == 0.0
    assert np.all(acc[ODD] == 0.0)
    if k == 1:
        assert np.all(dudt == 0.0)

"""A full search that starts from a previous h far too large (the particles have collapsed since, or are
another set altogether) still finds every particle's neighbours: the same ones and the same h as a
search without a previous h (in a row, distances equal to float32 rounding may come in either order). The sets have points on all scales down to 1e-6 of their size, so that a sphere
of the first radius meets far more points at its rim than near its centre."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fractal(n, rng):
    return rng.normal(size=(n, 3)) * 10 ** rng.uniform(-6, 0, (n, 1))


def _clump_in_field(n, rng):
    x = rng.uniform(size=(n, 3))
    x[::2] *= 1e-5
    return x


@pytest.mark.parametrize("make", [_fractal, _clump_in_field])
@pytest.mark.parametrize("n,size", [(60000, 3.0), (60000, 300.0), (7000, 300.0), (100000, 3e5)])
def test_search_from_a_stale_h(gpulib, make, n, size):
    from galaxy_formation_gb300 import _lib

    lib = gpulib
    rng = np.random.default_rng(1)
    x = np.ascontiguousarray(make(n, rng))
    before = np.random.default_rng(5).uniform(size=(n, 3)) * size
    v, m, kind, u = np.zeros((n, 3)), np.full(n, 1.0 / n), np.zeros(n, np.int8), np.ones(n)

    def evaluate(pos):
        acc, dt = np.empty((n, 3)), np.empty(n)
        _lib.check(lib.gf_accelerations(n, pos, v, m, kind, u, 0.7, 1e-12, 5 / 3, 1.0, 2.0, None, 1, 1, 1, acc, dt))
        return _lib.read_gas(lib)

    for key in (_lib.OPT_SPH_FLOAT32, _lib.OPT_GRAVITY_QUAD, _lib.OPT_GRAVITY_REL, _lib.OPT_WALK_MERGE,
                _lib.OPT_HGUESS):
        lib.gf_set_option(key, 0)
    lib.gf_set_option(_lib.OPT_FORGET_H, 1)
    first = evaluate(x)
    evaluate(before)
    then = evaluate(x)
    assert np.array_equal(np.sort(then["nb"]), np.sort(first["nb"]))
    assert np.array_equal(then["h"], first["h"])

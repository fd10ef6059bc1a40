"""The direct sum with masses at the ends of the range: infinite and no numbers (each term's kind as
NumPy's), subnormal and huge ones (within 2^-53 of the terms' sum per rounded operation, as
test_gpu_direct_parts derives it; a subnormal term has the spacing of subnormals beside)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("odd", [np.inf, -np.inf, np.nan, 1e-310, 1e-300, 1e290, -1.0, 0.0])
@pytest.mark.parametrize("n", [3, 300])
def test_one_odd_mass(gpulib, n, odd):
    from galaxy_formation_gb300.engine import Engine
    from test_gpu_direct_parts import _reference

    rng = np.random.default_rng(n)
    x, m, eps = rng.normal(size=(n, 3)), rng.uniform(0.5, 1.5, n), 0.05
    if abs(odd) < 1e-290:
        m[:] = odd  # all of them, or nothing of it shows
    m[2] = odd
    with np.errstate(all="ignore"):
        want, size = _reference(x, m, eps, np.arange(n))
    got = Engine().gravity_direct(x, m, eps)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[np.isinf(want)], want[np.isinf(want)])
    ok = np.isfinite(want)
    assert np.all(np.abs(got[ok] - want[ok]) <= 1.2e-13 * size[ok] + n * 5e-324)

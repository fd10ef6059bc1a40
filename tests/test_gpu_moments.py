"""The bottom-up moments passes leave their arrival counters ready for the next pass: several
refits in a row give the bits of one refit of the same tree to the last positions, in the plain
form (float64 sums) and in the mixed form (quadrupoles), with leaves of coincident points (larger
than a leaf's register tile) in the tree."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 9, 3000])
@pytest.mark.parametrize("quad", [0, 1])
def test_refits_in_a_row(gpulib, n, quad):
    from galaxy_formation_gb300 import _lib

    lib = gpulib
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, 3))
    if n > 100:
        x[100:140] = x[100]
    v, m = rng.normal(size=(n, 3)) * 1e-3, rng.uniform(0.5, 1.5, n)
    kind, u = np.full(n, 2, np.int8), np.zeros(n)

    def evaluate(pos, rebuild):
        acc, dt = np.empty((n, 3)), np.empty(n)
        _lib.check(lib.gf_accelerations(n, np.ascontiguousarray(pos), v, m, kind, u, 0.7, 0.05, 5 / 3, 1.0, 2.0,
                                        None, rebuild, 0, 0, acc, dt))
        return acc

    for key in (_lib.OPT_GRAVITY_REL, _lib.OPT_WALK_MERGE):
        lib.gf_set_option(key, 0)
    lib.gf_set_option(_lib.OPT_GRAVITY_QUAD, quad)
    try:
        evaluate(x, 1)
        for t in (1, 2, 3):
            several = evaluate(x + t * v, 0)
        evaluate(x, 1)
        once = evaluate(x + 3 * v, 0)
    finally:
        lib.gf_set_option(_lib.OPT_GRAVITY_QUAD, 0)
    assert np.array_equal(several, once)
    assert np.isfinite(several).all()

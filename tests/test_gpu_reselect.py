"""The reselection of the 32 nearest among the cached candidates ranks them by buckets of their
distance: smoothing lengths and neighbour sets of both forms against NumPy on the candidates of the
first positions, after drifts that leave the order, shuffle it, or pile distances up (coincident
points), and with candidates that are no gas any more.

Tolerance: h is half the 32nd distance, three squares of float64 differences on both sides (at most
6 roundings of 2^-53 each): 1e-14 relative. The mixed form measures that distance in float64 as well.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _d2(x, rows):
    d = x[:, None, :] - x[rows]
    return (d[..., 0] ** 2 + d[..., 1] ** 2) + d[..., 2] ** 2


@pytest.mark.parametrize("float32", [0, 1])
@pytest.mark.parametrize("n", [48, 65, 300, 2501])
@pytest.mark.parametrize("change", ["drift", "shuffle", "groups", "stars"])
def test_reselection(gpulib, n, float32, change):
    from galaxy_formation_gb300 import _lib, params

    lib = gpulib
    for key in (_lib.OPT_GRAVITY_QUAD, _lib.OPT_GRAVITY_REL, _lib.OPT_WALK_MERGE, _lib.OPT_HGUESS):
        lib.gf_set_option(key, 0)
    lib.gf_set_option(_lib.OPT_SPH_FLOAT32, float32)
    lib.gf_set_option(_lib.OPT_FORGET_H, 1)
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, 3))
    kind = np.zeros(n, np.int8)
    acc, dt = np.empty((n, 3)), np.empty(n)

    def evaluate(fresh):
        _lib.check(lib.gf_accelerations(n, x, np.zeros((n, 3)), np.full(n, 1.0 / n), kind, np.ones(n), params.THETA,
                                        params.EPS, params.GAMMA, 1.0, 2.0, None, 1, 1, fresh, acc, dt))
        return _lib.read_gas(lib)

    try:
        evaluate(1)
        cand = np.argsort(_d2(x, np.broadcast_to(np.arange(n), (n, n))), axis=1, kind="stable")[:, :48]
        if change == "groups":  # six points on each place: equal distances, and h of the softening
            x = np.ascontiguousarray(x[np.arange(n) // 6 * 6])
        else:
            x = x + {"drift": 1e-3, "shuffle": 0.3, "stars": 1e-3}[change] * rng.normal(size=(n, 3))
        if change == "stars":
            kind[rng.permutation(n)[: n // 12]] = 2
        g = evaluate(0)
    finally:
        lib.gf_set_option(_lib.OPT_SPH_FLOAT32, 0)
    gas = kind == 0
    assert np.array_equal(g["gidx"], np.flatnonzero(gas))
    d2 = np.where(gas[cand], _d2(x, cand), np.inf)[gas]
    assert np.all(np.isfinite(d2).sum(axis=1) >= 32)
    near = np.sqrt(np.sort(d2, axis=1)[:, :32])
    h = np.maximum(0.5 * near[:, 31], 0.5 * params.EPS)
    assert np.all(np.abs(g["h"] - h) <= 1e-14 * h)
    rows = g["gidx"][g["nb"]]
    own = np.sort(np.sqrt(((x[gas][:, None, :] - x[rows]) ** 2).sum(axis=2)), axis=1)
    assert np.all(np.abs(own - near) <= 1e-14 * near[:, 31:])
    assert all(len(set(r)) == 32 for r in rows.tolist())

"""The neighbour search without a previous h starts from the distances to the points next to the
query in the tree's order: the result must not depend on the start.

* gf_knn against NumPy's brute force (the same float64 operations per pair, none contracted, so
  the distances are equal to the bit) at the edges of the window (fewer points than the
  window's 128, exactly 128, one more), for the smallest and largest k, on sets where the window
  misleads: a sparse cloud around a dense core (first spheres with far more points than a search
  keeps), tight groups of coincident points, a plane.
* The fused evaluation's first search from this start against the cell-density start: the same
  neighbour rows and h.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _set(kind, n, seed=11):
    rng = np.random.default_rng(seed)
    x = rng.normal(size=(n, 3))
    if kind == "core":  # half of the points in a core 1e4 times denser in each dimension
        x[::2] *= 1e-4
    elif kind == "groups":  # groups of 5 coincident points
        x = x[rng.integers(0, max(1, n // 5), n)]
    elif kind == "plane":
        x[:, 2] *= 1e-9
    return np.ascontiguousarray(x)


@pytest.mark.parametrize("kind", ["normal", "core", "groups", "plane"])
@pytest.mark.parametrize("n,k", [(1, 1), (2, 2), (64, 64), (127, 48), (128, 48), (129, 33), (700, 1), (3001, 48),
                                 (3001, 64)])
def test_knn_start(gpulib, kind, n, k):
    from galaxy_formation_gb300 import sph

    x = _set(kind, n)
    dist, nb = sph.knn(x, k)
    dx, dy, dz = (x[:, None, c] - x[None, :, c] for c in range(3))
    d2 = (dx * dx + dy * dy) + dz * dz
    rnb = np.argsort(d2, axis=1, kind="stable")[:, :k]
    rd = np.sqrt(np.take_along_axis(d2, rnb, axis=1))
    assert np.array_equal(dist, rd)
    if kind != "groups":  # coincident points: any of them may come first
        assert np.array_equal(nb, rnb)


def test_first_search_does_not_depend_on_its_start(gpulib):
    from galaxy_formation_gb300 import _lib, params, synthetic

    lib = gpulib
    for key in (_lib.OPT_SPH_FLOAT32, _lib.OPT_GRAVITY_QUAD, _lib.OPT_GRAVITY_REL, _lib.OPT_WALK_MERGE):
        lib.gf_set_option(key, 0)
    d = synthetic.disk_halo(n_gas=20011, n_dm=5000, n_clumps=20)
    n = len(d["mass"])
    acc, dt = np.empty((n, 3)), np.empty(n)
    rows, iters = {}, {}
    for mode in (0, 1):
        lib.gf_set_option(_lib.OPT_HGUESS, mode)
        lib.gf_set_option(_lib.OPT_FORGET_H, 1)
        _lib.check(lib.gf_accelerations(n, d["pos"], d["vel"], d["mass"], d["kind"], d["u"], params.THETA,
                                        params.EPS, params.GAMMA, 1.0, 2.0, None, 1, 1, 1, acc, dt))
        rows[mode] = _lib.read_gas(lib)
        st = np.zeros(9)
        lib.gf_force_stats(st, 9)
        iters[mode] = st[3] / st[0]
    lib.gf_set_option(_lib.OPT_HGUESS, 0)
    assert np.array_equal(rows[0]["nb"], rows[1]["nb"])
    assert np.array_equal(rows[0]["h"], rows[1]["h"])
    assert iters[0] < iters[1], iters

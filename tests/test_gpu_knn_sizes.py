"""The neighbour search serves one, two or three queries per warp by their number and sorts a
query's points by buckets of their distance.

* gf_knn against a float64 search in a k-d tree: the distances of the k nearest, on both sides of
  the sizes where the number of queries per warp changes, with every remainder of three.
  Tolerance: both sum three squares of differences in float64, contracted or not: each rounding
  is 2^-53 relative and there are at most 6 on a side, so 1e-14 relative bounds the difference.
* Distances that pile up in few buckets (points on a sphere around a query, coincident points),
  against the same sums in NumPy. A search settles at most 64 points within float32 rounding (2e-5
  of the squared distance) of its last one in float64, so the query in the sphere's centre, with
  more of them, has its distances within that band; with more than 128 of them no radius encloses
  k to 128 points, which is an error.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8192, 8193, 65536, 65537, 65538, 65539])
def test_knn_sizes(gpulib, n):
    from scipy.spatial import cKDTree

    from galaxy_formation_gb300 import sph

    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, 3))
    x[::3] *= 0.05  # dense core: several radius steps for some queries of a warp
    dist, nb = sph.knn(x, 48)
    ref, _ = cKDTree(x).query(x, 48)
    assert np.all(np.abs(dist - ref) <= 1e-14 * ref)
    d = x[nb] - x[:, None, :]
    own = np.sqrt((d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1]) + d[..., 2] * d[..., 2])
    assert np.all(np.abs(own - dist) <= 1e-14 * ref)
    assert np.all(np.sort(nb, axis=1)[:, 1:] != np.sort(nb, axis=1)[:, :-1])


@pytest.mark.parametrize("n,k", [(66, 48), (100, 64), (126, 32), (500, 48)])
def test_knn_piled_distances(gpulib, n, k):
    from galaxy_formation_gb300 import _lib, sph

    rng = np.random.default_rng(n)
    v = rng.normal(size=(n, 3))
    shell = v / np.linalg.norm(v, axis=1)[:, None]
    shell[0] = 0.0  # the centre: all its distances within rounding of 1
    shell[1 : n // 3] = shell[1]
    x = np.ascontiguousarray(shell)
    if n > 128:
        with pytest.raises(_lib.GpuError):
            sph.knn(x, k)
        return
    dist, _ = sph.knn(x, k)
    dx, dy, dz = (x[:, None, c] - x[None, :, c] for c in range(3))
    d2 = np.sort((dx * dx + dy * dy) + dz * dz, axis=1)[:, :k]
    assert np.array_equal(dist[1:], np.sqrt(d2[1:]))
    assert np.all(np.abs(dist[0] - np.sqrt(d2[0])) <= 1e-5)

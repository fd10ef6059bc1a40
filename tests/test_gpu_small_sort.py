"""The one-launch bounding box, keys and sort of small sets: the tree equals the oracle's node for
node (structure, particle order) at the edges of the split over the cluster's blocks (fewer
particles than blocks, empty last blocks, uneven shares) and of the launch rules (28,672 particles
and one more; 147,456 and one more for the keys per thread of the larger sorts), with coincident
points, points on cell walls and cells deeper than a key; and sets whose keys share their top
40 bits in runs just short enough for the insertion sort of the one launch, one longer, and in one
run over several blocks."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 17, 63, 1023, 8191, 8193, 10000, 28671, 28672, 28673,
                               32768, 32769, 144 * 1024, 144 * 1024 + 1])
@pytest.mark.parametrize("kind", ["normal", "grid", "deep"])
def test_small_sort_builds_the_same_tree(gpulib, oracle, n, kind):
    from galaxy_formation_gb300.engine import Engine

    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, 3))
    if kind == "grid":  # many ties and coordinates on cell walls
        x = np.round(x * 4) / 4
    elif kind == "deep":  # groups that only separate below level 21, and coincident ones
        x = x[rng.integers(0, max(1, n // 12), n)]
        x[::2] *= 1 + 1e-9 * rng.integers(0, 4, size=(len(x[::2]), 1))
    x = np.ascontiguousarray(x)
    m = rng.uniform(0.5, 1.5, n)
    a, b = Engine().build_tree(x, m, 0.7), oracle.build_tree(x, m, 0.7)
    for f in ("start", "count", "next", "leaf", "order", "groups"):
        assert np.array_equal(a[f], b[f]), f


@pytest.mark.parametrize("n", [16384, 16385, 524288, 524289])
def test_scan_tiles_build_the_same_tree(gpulib, oracle, n):
    """The most entries that the scans take in one launch and one per thread, and one more."""
    test_small_sort_builds_the_same_tree(gpulib, oracle, n, "normal")


@pytest.mark.parametrize("n", [31, 4097, 28672])
@pytest.mark.parametrize("run", [2, 15, 16, 17, 5000])
def test_keys_that_share_their_top_bits(gpulib, oracle, n, run):
    from galaxy_formation_gb300.engine import Engine

    rng = np.random.default_rng(n + run)
    # places half way between the walls of the 2^13 grid, `run` points within 1e-5 of the box on each
    # (a 13th of that grid's cell): the same top bits, different keys
    places = (rng.choice(8192, size=(n // run + 1, 3)) + 0.5) / 8192
    x = np.repeat(places, run, axis=0)[:n] + 1e-5 * rng.uniform(-1, 1, (n, 3))
    x = np.ascontiguousarray(x[rng.permutation(n)])
    x[:2] = [[0.0, 0.0, 0.0], [1.0, 1.0, 1.0]]  # the box
    m = rng.uniform(0.5, 1.5, n)
    a, b = Engine().build_tree(x, m, 0.7), oracle.build_tree(x, m, 0.7)
    for f in ("start", "count", "next", "leaf", "order", "groups"):
        assert np.array_equal(a[f], b[f]), f

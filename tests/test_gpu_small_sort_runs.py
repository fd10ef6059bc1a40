"""Runs of keys that share their top 40 bits side by side: each is sorted by the thread of its first
key, next to the runs of other threads that are moving theirs. Places are consecutive cells of the
2^13 grid in the curve's order, so no key lies between two runs; every length from 1 to the longest
that is sorted in place occurs (the 40th bit halves a cell: a quarter of it is used), within and across the shares of the cluster's blocks. The tree
equals the oracle's node for node."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [tuple(range(1, 17)), (2,), (16,), (16, 1), (1, 2, 3)])
@pytest.mark.parametrize("n", [18, 4097, 28672])
def test_adjacent_runs(gpulib, oracle, n, lengths):
    from galaxy_formation_gb300.engine import Engine

    rng = np.random.default_rng(n + len(lengths))
    cell = np.repeat(np.arange(n), np.resize(lengths, n))[:n]
    grid = np.zeros((n, 3), np.int64)
    for bit in range(5):
        for axis in range(3):
            grid[:, axis] |= (cell >> (3 * bit + axis) & 1) << bit
    x = (4096 + grid + 0.25) / 8192 + 1e-5 * rng.uniform(-1, 1, (n, 3))
    x = np.ascontiguousarray(x[rng.permutation(n)])
    x[:2] = [[0.0, 0.0, 0.0], [1.0, 1.0, 1.0]]  # the box
    m = rng.uniform(0.5, 1.5, n)
    a, b = Engine().build_tree(x, m, 0.7), oracle.build_tree(x, m, 0.7)
    for f in ("start", "count", "next", "leaf", "order", "groups"):
        assert np.array_equal(a[f], b[f]), f

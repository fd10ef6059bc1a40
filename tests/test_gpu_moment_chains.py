"""Chains of cells with one child each, above coincident or tightly grouped particles: the moments
pass of the plain form climbs a warp's chains side by side, and each record of a chain is that of its
child, measured against its own cell."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STAGE_MOMENTS = 12


def _groups(count, each, spread, seed=3):
    rng = np.random.default_rng(seed)
    x = np.repeat(rng.uniform(-1, 1, size=(count, 3)), each, axis=0)
    return np.ascontiguousarray(x + spread * rng.normal(size=x.shape)), rng.uniform(0.5, 1.5, len(x))


def _compare(got, want):
    """The structure to the bit, the float32 records to two roundings (float64 sums in another order
    can move one). An opening radius also holds the distance of a float64 centre of mass from its cell's
    centre, coordinates below 1 of a few roundings of 2^-53 each: 1e-15."""
    for f in ("start", "count", "next", "leaf", "order", "groups"):
        assert np.array_equal(got[f], want[f]), f
    for f in ("cx", "cy", "cz", "m", "open_r", "gx", "gy", "gz", "half"):
        a, b = got[f].astype(np.float64), want[f].astype(np.float64)
        tol = 2.0 * np.spacing(np.abs(want[f])) + (1e-15 if f == "open_r" else 0.0)
        assert np.all(np.abs(a - b) <= tol), f


SETS = [(1, 9, 0.0), (5, 20, 0.0), (100, 20, 0.0), (200, 9, 1e-7), (40, 30, 1e-10)]


@pytest.mark.parametrize("count,each,spread", SETS)
@pytest.mark.parametrize("theta", [0.5, 0.7])
def test_records_of_chains(gpulib, oracle, count, each, spread, theta):
    from galaxy_formation_gb300.engine import Engine

    x, m = _groups(count, each, spread)
    _compare(Engine().build_tree(x, m, theta), oracle.build_tree(x, m, theta))


@pytest.mark.parametrize("count,each,spread", SETS)
def test_records_of_chains_after_a_refit(gpulib, oracle, count, each, spread):
    from galaxy_formation_gb300.engine import Engine

    x, m = _groups(count, each, spread)
    eng = Engine()
    eng.build_tree(x, m, 0.7)
    oracle.build_tree(x, m, 0.7)
    x1 = np.ascontiguousarray(x + 1e-3 * np.random.default_rng(4).normal(size=x.shape))
    nobody, acc = np.zeros(len(m), np.uint8), np.zeros_like(x)
    eng.gravity(x1, m, acc, 0.7, 0.1, nobody, False)
    oracle.accel_active(x1, m, acc.copy(), 0.7, 0.1, nobody, False)
    _compare(eng.tree(), oracle.tree_export())


def test_many_chains_take_no_longer_than_a_few(gpulib):
    """48 levels up from 96 groups of coincident particles as from 4 (eight times the chains per
    warp, side by side; one after another they took eight times as long)."""
    from galaxy_formation_gb300.engine import Engine

    lib, eng = gpulib, Engine()

    def moments_ms(count):
        x, m = _groups(count, 20, 0.0)
        eng.build_tree(x, m, 0.7)
        best = np.inf
        for _ in range(10):
            ms, launches = ctypes.c_double(), ctypes.c_int()
            lib.gf_profile(1)
            try:
                eng.build_tree(x, m, 0.7)
                assert lib.gf_profile_stage(STAGE_MOMENTS, ctypes.byref(ms), ctypes.byref(launches)) == 0
            finally:
                lib.gf_profile(0)
            assert launches.value == 1
            best = min(best, ms.value)
        return best

    few, many = moments_ms(4), moments_ms(96)
    assert many < 3.0 * few, (few, many)

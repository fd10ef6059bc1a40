"""The float64 SPH passes on values outside the ordinary range, with each number of lanes per particle
(eight, four, two, one by the particle count): what one such particle does to the others' results.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COUNTS = (600, 20000, 200000, 300000)
ODD = 100  # the particle that is out of the ordinary


def _set(n, k=7):
    rng = np.random.default_rng(n)
    nb = np.ascontiguousarray((np.arange(n)[:, None] + np.arange(k)[None, :]) % n, np.int64)
    return {"pos": rng.normal(size=(n, 3)), "vel": rng.normal(size=(n, 3)), "mass": rng.uniform(0.5, 1.5, n) / n,
            "nb": nb, "h": rng.uniform(0.3, 3.0, n), "u": rng.uniform(0.1, 10.0, n)}


def _forces(d):
    from galaxy_formation_gb300 import sph

    n = len(d["mass"])
    rho, acc, dudt, dt = np.empty(n), np.empty((n, 3)), np.empty(n), np.empty(n)
    sph.sph_forces(d["pos"], d["vel"], d["mass"], d["nb"], d["h"], d["u"], 5.0 / 3.0, 1.0, 2.0, rho, acc, dudt, dt)
    return {"rho": rho, "acc": acc, "dudt": dudt, "dt": dt}


def _with(d, **changes):
    out = {key: val.copy() for key, val in d.items()}
    for key, val in changes.items():
        out[key][ODD] = val
    return out


@pytest.mark.parametrize("n", COUNTS)
@pytest.mark.parametrize("distance", [1e150, 1e160, 1e200])
def test_a_neighbour_whose_squared_distance_overflows(gpulib, n, distance):
    """Outside both supports and receding, it adds zero to every sum, like one far enough for that at an
    ordinary distance: the same bits."""
    d = _set(n)
    near = _forces(_with(d, pos=[1e6, 0, 0], vel=[1e3, 0, 0]))
    far = _forces(_with(d, pos=[distance, 0, 0], vel=[1e3, 0, 0]))
    for key in near:
        assert np.isfinite(near[key]).all()
        assert np.array_equal(far[key], near[key]), key


@pytest.mark.parametrize("n", COUNTS)
@pytest.mark.parametrize("h", [-2.9, -40.0])
def test_the_courant_step_ignores_receding_and_odd_pairs(gpulib, n, h):
    """Only a negative mu counts: with a negative smoothing length the approaching pairs have a positive
    one, whatever the number of lanes. Each rounding of the step is within 2^-53, fewer than 50 of them."""
    d = _with(_set(n), h=h)
    dt = _forces(d)["dt"][ODD]
    gamma, j = 5.0 / 3.0, d["nb"][ODD, 1:]
    dx = d["pos"][ODD] - d["pos"][j]
    vr = ((d["vel"][ODD] - d["vel"][j]) * dx).sum(1)
    hb = 0.5 * (h + d["h"][j])
    mu = np.where(vr < 0, hb * vr / ((dx * dx).sum(1) + 0.01 * hb * hb), 0.0)
    c = np.sqrt(gamma * (gamma - 1) * d["u"][ODD])
    want = 0.3 * h / (2.2 * c + 1.2 * 2.0 * max(0.0, (-mu).max()))
    assert abs(dt - want) <= 1e-14 * abs(want)


def _rows_of(d):
    """The rows that hold ODD, and no other particle's: those whose results it can change."""
    return np.flatnonzero((d["nb"] == ODD).any(axis=1))


def _close_to_numpy(d, got, rows):
    """Within 1e-13 of the terms' scales of NumPy's restatement (test_gpu_sph_lanes derives both)."""
    from test_gpu_sph_lanes import _reference

    with np.errstate(all="ignore"):
        rho, acc, s_acc, dudt, s_dudt, dt = _reference(*(d[key] for key in ("pos", "vel", "mass", "nb", "h", "u")))
    for key, want, size in (("rho", rho, np.abs(rho)), ("acc", acc, np.abs(s_acc)), ("dudt", dudt, np.abs(s_dudt)),
                            ("dt", dt, np.abs(dt))):
        assert np.all(np.abs(got[key] - want)[rows] <= 1e-13 * size[rows]), key


@pytest.mark.parametrize("n", COUNTS)
@pytest.mark.parametrize("h", [-0.7, -2.9, -40.0])
def test_a_negative_smoothing_length(gpulib, n, h):
    """The kernels of sph.py:31-54 take the branch of q < 1 for it; so do the passes here."""
    d = _with(_set(n), h=h)
    _close_to_numpy(d, _forces(d), _rows_of(d))


@pytest.mark.parametrize("n", COUNTS)
@pytest.mark.parametrize("nan", [np.nan, -np.nan])
def test_a_smoothing_length_that_is_no_number(gpulib, n, nan):
    """Its own density is 0 (no pair is inside its support); the others' densities stay."""
    d = _set(n)
    got, plain = _forces(_with(d, h=nan)), _forces(d)
    assert got["rho"][ODD] == 0.0
    others = np.arange(n) != ODD
    assert np.array_equal(got["rho"][others], plain["rho"][others])


@pytest.mark.parametrize("n", COUNTS)
@pytest.mark.parametrize("h", [1e-70, 1e-76, 1e-77, 1e-80])
def test_a_smoothing_length_whose_fourth_power_underflows(gpulib, n, h):
    """The normalisation of its gradient is beyond float64; its neighbours lie outside its support."""
    d = _with(_set(n), h=h)
    _close_to_numpy(d, _forces(d), _rows_of(d))


@pytest.mark.parametrize("n", COUNTS)
def test_a_smoothing_length_of_zero(gpulib, n):
    """Its density is zero; the heating of the others does not see its pressure and stays a number."""
    d = _with(_set(n), h=0.0)
    got = _forces(d)
    assert got["rho"][ODD] == 0.0
    assert np.isfinite(got["dudt"][np.arange(n) != ODD]).all()


@pytest.mark.parametrize("n", COUNTS)
@pytest.mark.parametrize("h", [1e-309, 1e-310, 5e-324])
def test_a_subnormal_smoothing_length(gpulib, n, h):
    """W(0, h) of sph.py:31-40 is then infinite, and with it the particle's own density."""
    d = _set(n)
    got, plain = _forces(_with(d, h=h)), _forces(d)
    assert got["rho"][ODD] == np.inf
    others = np.arange(n) != ODD
    assert np.array_equal(got["rho"][others], plain["rho"][others])


@pytest.mark.parametrize("n", COUNTS)
@pytest.mark.parametrize("x", [np.nan, -np.nan, np.inf, -np.inf])
def test_a_position_that_is_no_number(gpulib, n, x):
    """Its distances are no numbers either, that to itself included: density zero. The others' densities
    are as if it were far away."""
    d = _set(n)
    got, far = _forces(_with(d, pos=[x, 0, 0])), _forces(_with(d, pos=[1e6, 0, 0]))
    assert got["rho"][ODD] == 0.0
    others = np.arange(n) != ODD
    assert np.array_equal(got["rho"][others], far["rho"][others])

"""The float64 SPH passes at the edges of their launch rule and of their pair arithmetic.

Particle counts on both sides of the switches between eight, four, two and one lanes per particle, rows
of 1 to 33 neighbours (not a multiple of the lanes), coincident particles, pairs outside both
supports, and sets scaled so far that the squared distances leave the range of the fast inverse
root. Against NumPy's float64 restatement of sph.py:57-106. A pair term takes fewer than 60
rounded operations and a row has at most 33 terms, so each sum is within 100 x 2^-53 = 1.2e-14 of
the sum of its terms' scales; 1e-13 is allowed (the libraries' own roots and divisions). A term's
scale is its absolute value where its factors are products and quotients; a factor that is a
difference counts with the values it came from: the kernel gradient with its change for a relative
change of q (it vanishes at the support's edge), v.d with the sum of its three products' absolute
values.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _reference(x, v, m, nb, h, u, gamma=5.0 / 3.0, alpha=1.0, beta=2.0):
    d = x[:, None, :] - x[nb]
    r2 = (d * d).sum(2)
    r = np.sqrt(r2)

    def shape(q):
        return np.where(q < 1, 1 - 1.5 * q**2 + 0.75 * q**3, np.where(q < 2, 0.25 * (2 - q) ** 3, 0.0))

    def grad(q):
        return np.where(q < 1, -3 * q + 2.25 * q**2, np.where(q < 2, -0.75 * (2 - q) ** 2, 0.0))

    hi, hj = h[:, None], h[nb]
    rho = (m[nb] * shape(r / hi)).sum(1) / (np.pi * h**3)
    cs = np.sqrt(gamma * (gamma - 1) * u)
    pr2 = (gamma - 1) * u / rho
    other = nb != np.arange(len(x))[:, None]
    inv_r = 1 / np.maximum(r, 1e-30)
    gi = grad(r / hi) / (np.pi * hi**4) * inv_r
    gj = grad(r / hj) / (np.pi * hj**4) * inv_r
    vr = ((v[:, None, :] - v[nb]) * d).sum(2)
    hb = 0.5 * (hi + hj)
    mu = np.where((vr < 0) & other, hb * vr / (r2 + 0.01 * hb * hb), 0.0)
    visc = (-alpha * 0.5 * (cs[:, None] + cs[nb]) * mu + beta * mu * mu) / (0.5 * (rho[:, None] + rho[nb]))
    gb = 0.5 * (gi + gj)
    mj = np.where(other, m[nb], 0.0)
    pair = -(mj * (pr2[:, None] * gi + pr2[nb] * gj + visc * gb))[..., None] * d
    heat = mj * (pr2[:, None] * gi + 0.5 * visc * gb) * vr

    def slope(q):  # |q d(gradient)/dq|
        return q * np.where(q < 1, np.abs(-3 + 4.5 * q), np.where(q < 2, 1.5 * (2 - q), 0.0))

    si = np.abs(gi) + slope(r / hi) / (np.pi * hi**4) * inv_r
    sj = np.abs(gj) + slope(r / hj) / (np.pi * hj**4) * inv_r
    sv = np.abs((v[:, None, :] - v[nb]) * d).sum(2)
    smu = hb * sv / (r2 + 0.01 * hb * hb)
    svisc = (alpha * 0.5 * (cs[:, None] + cs[nb]) * smu + beta * smu * smu) / (0.5 * (rho[:, None] + rho[nb]))
    s_pair = (mj * (pr2[:, None] * si + pr2[nb] * sj + 0.5 * svisc * (si + sj)))[..., None] * np.abs(d)
    s_heat = mj * (pr2[:, None] * si + 0.25 * svisc * (si + sj)) * sv
    dt = 0.3 * h / (cs + 1.2 * (alpha * cs + beta * (-mu).max(1, initial=0.0)) + 1e-30)
    return rho, pair.sum(1), s_pair.sum(1), heat.sum(1), s_heat.sum(1), dt


@pytest.mark.parametrize("n,k,scale", [(3, 1, 1.0), (257, 5, 1.0), (4001, 33, 1.0), (4001, 32, 1e-38),
                                       (4001, 32, 1e30), (8 * 1024, 19, 1.0),
                                       (8 * 1024 + 1, 21, 1.0), (128 * 1024, 8, 1.0), (128 * 1024 + 1, 7, 1.0),
                                       (256 * 1024, 6, 1.0), (256 * 1024 + 1, 5, 1.0)])
def test_sph_forces_lanes(gpulib, n, k, scale):
    from galaxy_formation_gb300 import sph

    rng = np.random.default_rng(n + k)
    x = rng.normal(size=(n, 3))
    if n > 10:
        x[1::7] = x[::7][: len(x[1::7])]  # coincident pairs
    nb = (np.arange(n)[:, None] + np.arange(k)[None, :]) % n  # self first, then the next ones
    nb = np.ascontiguousarray(nb, np.int64)
    h = rng.uniform(0.3, 3.0, n)  # q below 1, in 1..2 and beyond
    v = rng.normal(size=(n, 3))
    m = rng.uniform(0.5, 1.5, n) / n
    u = rng.uniform(0.1, 10.0, n)
    x, h = x * scale, h * scale
    rho, acc, dudt, dt = np.empty(n), np.empty((n, 3)), np.empty(n), np.empty(n)
    sph.sph_forces(x, v, m, nb, h, u, 5.0 / 3.0, 1.0, 2.0, rho, acc, dudt, dt)
    with np.errstate(over="ignore", under="ignore"):
        r_rho, r_acc, s_acc, r_du, s_du, r_dt = _reference(x, v, m, nb, h, u)
    assert np.all(np.abs(rho - r_rho) <= 1e-13 * r_rho)
    assert np.all(np.abs(dt - r_dt) <= 1e-13 * r_dt)
    assert np.all(np.abs(acc - r_acc) <= 1e-13 * s_acc)
    assert np.all(np.abs(dudt - r_du) <= 1e-13 * s_du)

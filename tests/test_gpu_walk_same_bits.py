"""Walks of the same work list by different kernels: the same bits where every particle's sum keeps its
order, the same list interactions to the last one where it does not.

Reference form: items shared by two warps or not, two particles per lane by packed instructions or not,
against the walk that also sums potentials, whose kernel does neither; with the particle counts on both sides
of the switch between the kernels, and with more and fewer items than are shared. Mixed form: 2 or 8 nodes per
lane and every launch shape. The library's own steps are called one by one: the work list of the tree walked
last is prepared again and walked again.
"""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 0.05


class Walker:
    """prepare_walk and walk of the last walked tree."""

    def __init__(self, lib):
        self.lib = lib
        last = lib["_ZN2gf11last_walkedEv"]
        last.restype = ctypes.c_void_p
        self.tree = ctypes.c_void_p(ctypes.cast(last(), ctypes.POINTER(ctypes.c_void_p))[0])
        self.prepare = lib["_ZN2gf6Octree12prepare_walkEPKhP11CUstream_stiPKdff"]
        self.prepare.restype, self.prepare.argtypes = None, [ctypes.c_void_p] * 3 + [
            ctypes.c_int, ctypes.c_void_p, ctypes.c_float, ctypes.c_float]
        self.walk = lib["_ZN2gf6Octree4walkEdPdP11CUstream_stS1_ii"]
        self.walk.restype, self.walk.argtypes = None, [
            ctypes.c_void_p, ctypes.c_double, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.c_int]

    def __call__(self, acc, active=None, pot=None, npl=2, shape=0, chunk=0, aold=None, alpha=0.0, alpha_q=0.0):
        import torch

        torch.cuda.synchronize()
        stream, ptr = self.lib.gf_stream(), lambda t: None if t is None else t.data_ptr()
        self.prepare(self.tree, ptr(active), stream, chunk, ptr(aold), alpha, alpha_q)
        self.walk(self.tree, EPS, acc.data_ptr(), stream, ptr(pot), npl, shape)
        torch.cuda.synchronize()
        assert self.lib.gf_last_status() == 0
        return self.lib.gf_walk_pairs(), self.lib.gf_walk_quad_pairs()


def _clusters(sizes, seed=5):
    rng = np.random.default_rng(seed)
    return np.concatenate([rng.normal(size=(m, 3)) * 0.01 + rng.normal(size=3) * 5 for m in sizes])


def _set(kind, n):
    if kind == "clusters":
        return _clusters((1, 2, 8, 9, 16, 17, 31, 32, 33, 48, 63, 64, 65, 130) * 4)
    if kind == "coincident":
        return np.concatenate([_clusters((20, 40, 64)), np.repeat([[1.0, 2.0, 3.0]], n, axis=0)])
    rng = np.random.default_rng(n)
    return rng.normal(size=(n, 3)) * rng.random((n, 1))


@pytest.mark.parametrize("kind,n", [("clusters", 0), ("coincident", 150), ("cloud", 1000), ("cloud", 10000),
                                    ("cloud", 400000), ("cloud", 400001)])
@pytest.mark.parametrize("which", ["all", "every other", "every 7th", "a half"])
def test_reference_form(gpulib, kind, n, which):
    import torch
    from galaxy_formation_gb300.engine import Engine

    x = torch.from_numpy(np.ascontiguousarray(_set(kind, n))).cuda()
    n = len(x)
    m = torch.rand(n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1)) + 0.5
    index = torch.arange(n, device="cuda")
    active = {"all": None, "every other": index % 2 == 0, "every 7th": index % 7 == 0, "a half": x[:, 0] > 0}[which]
    active = None if active is None else active.to(torch.uint8)
    acc, again, pot = (torch.full((n, 3), 7.0, dtype=torch.float64, device="cuda") for _ in range(3))
    Engine().gravity(x, m, acc, 0.7, EPS, active)
    pairs = gpulib.gf_walk_pairs()
    assert Walker(gpulib)(again, active, pot)[0] == pairs > 0
    assert torch.equal(acc, again)
    assert torch.isfinite(acc).all()


@pytest.mark.parametrize("alpha,alpha_q", [(0.0, 0.0), (4e-3, 0.0), (4e-3, 1.5e-4)])
@pytest.mark.parametrize("every,chunk", [(400, 4), (400, 8), (37, 0), (37, 72), (1, 0)])
def test_mixed_form(gpulib, alpha, alpha_q, every, chunk):
    """Each row of the acceleration: two sums of the same terms in another order, over tiles of up to 256 entries
    at a time: 2 x 272 x 2^-24 of the terms' scales, of which the monopoles' are at most m / (d^2 + eps^2) and the
    quadrupoles' at most half of that."""
    import torch
    from galaxy_formation_gb300 import _lib, params, synthetic

    lib = gpulib
    d = synthetic.make_config(1)
    n = len(d["mass"])
    assert n >= 200000
    acc0, dt = np.empty((n, 3)), np.empty(n)
    lib.gf_set_option(_lib.OPT_GRAVITY_REL, 0)
    lib.gf_set_option(_lib.OPT_WALK_MERGE, 0)
    lib.gf_set_option(_lib.OPT_GRAVITY_QUAD, 1)
    try:
        _lib.check(lib.gf_accelerations(n, d["pos"], d["vel"], d["mass"], np.full(n, params.DM, np.int8), d["u"], 0.55, EPS,
                                        params.GAMMA, 1.0, 2.0, None, 1, 0, 0, acc0, dt))
    finally:
        lib.gf_set_option(_lib.OPT_GRAVITY_QUAD, 0)
    walk = Walker(lib)
    x, m, aold = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (d["pos"], d["mass"], acc0))
    rows = torch.arange(0, n, every, device="cuda")
    active = None
    if every > 1:
        active = torch.zeros(n, dtype=torch.uint8, device="cuda")
        active[rows] = 1
    results = []
    for npl, shape in ((2, 0), (2, 1), (2, 2), (2, 3), (8, 0)):
        acc = torch.full((n, 3), 7.0, dtype=torch.float64, device="cuda")
        counts = walk(acc, active, None, npl, shape, chunk, aold if alpha else None, alpha, alpha_q)
        results.append((counts, acc))
    assert len({c for c, _ in results}) == 1 and results[0][0][1] > 0, [c for c, _ in results]
    some = rows[:: max(1, len(rows) // 2000)]
    scale = torch.cat([(m / (((x[None] - x[part, None]) ** 2).sum(2) + EPS * EPS)).sum(1) for part in some.split(50)])
    for _, acc in results[1:]:
        diff = (acc[some] - results[0][1][some]).abs().amax(1)
        assert torch.all(diff <= 1.5 * 2 * 272 * 2.0**-24 * scale)
        if every > 1:
            others = torch.ones(n, dtype=torch.bool, device="cuda")
            others[rows] = False
            assert torch.all(acc[others] == 7.0)

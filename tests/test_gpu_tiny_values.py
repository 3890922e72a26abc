"""FP64 values near and below the smallest normal number -- the far front of a
disturbance or of a tracer reaches them after some 150 updates -- and infinite
densities: the GPU's bits are the CPU oracle's.
"""

import numpy as np
import pytest

from scenarios import two_spheres

pytestmark = pytest.mark.gpu


def tracer(L, scale, big=False):
    lb = L.newlb(10, 11, 12, "null")
    lb.tau = 0.8
    if L.has("lbpull"):
        L.lbpull(lb)
    rng = np.random.default_rng(11)
    a = lb.array("a")
    a[:] = (rng.random(a.shape) - 0.3) * 8.0  # values of order one, so that an ulp of p / rho shows
    if big:
        a[300] = 1.5e308  # an infinite density of finite populations
    if L.has("lbpush"):
        L.lbpush(lb)
    mp = L.newmp(lb, "null")
    mp.alpha = 0.3
    L.mpinit(mp)
    L.mprhoinit(mp)
    if L.has("mppull"):
        L.mppull(mp)
    f = mp.field()
    f[:] = (rng.random(f.shape) - 0.2) * scale
    f[::17] = 0.0
    f[::19] = -0.0
    if L.has("mppush"):
        L.mppush(mp)
    L.mpstep(mp)
    if L.has("mppull"):
        L.mppull(mp)
    return mp.field().copy()


@pytest.mark.parametrize("scale", [1.0, 1e-270, 1e-292, 1e-303, 1e-306, 1e-308, 1e-315])
def test_tiny_tracer_equals_oracle(gpu, orc, scale):
    got, want = tracer(gpu, scale), tracer(orc, scale)
    assert np.array_equal(got, want), int((got != want).sum())


def test_infinite_density_equals_oracle(gpu, orc):
    got, want = tracer(gpu, 1.0, big=True), tracer(orc, 1.0, big=True)
    assert np.isfinite(want).all()  # p over an infinite density is 0
    assert np.array_equal(got, want), int((got != want).sum())


def populations(L, scale, stokes, dims):
    """Four updates of random populations around two spheres."""
    lb = two_spheres(L, dims=dims, steps=0, measure=False, bf=(0.0, 0.0, 0.0), stokes=stokes)
    if L.has("lbpull"):
        L.lbpull(lb)
    a = lb.array("a")
    a[:] = (np.random.default_rng(5).random(a.shape) - 0.5) * scale
    a[::7] = 0.0
    if L.has("lbpush"):
        L.lbpush(lb)
    for _ in range(4):
        L.lbstep(lb)
    return lb.pops()


@pytest.mark.parametrize("scale", [1e-250, 1e-270, 1e-290, 1e-300, 1e-306, 1e-308, 1e-312, 1e-318])
@pytest.mark.parametrize("stokes", [1, 0])
@pytest.mark.parametrize("dims", [(9, 10, 11), (5, 6, 32)])  # a plane as one run of nodes, rows of whole warps
def test_tiny_populations_equal_oracle(gpu, orc, scale, stokes, dims):
    got, want = populations(gpu, scale, stokes, dims), populations(orc, scale, stokes, dims)
    assert np.array_equal(got, want), int((got != want).sum())

"""Object forces and torques from the pieces of the boundary list: many small
objects (a thread each), one object of several pieces (a warp each), both in one
lattice, and an object without boundary nodes, against the oracle.  The sums
differ by their order: at most N 2^-53 of the sum of magnitudes for N nodes, torques
by the box's length times that.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def build(L, kind):
    if kind == "many":
        lb = L.newlb(60, 60, 60, "null")
        spheres = [(1.5 + 0.1 * (x % 3), 6 + 12 * x, 6 + 12 * y, 6 + 12 * z) for x in range(5) for y in range(5) for z in range(5)]
    elif kind == "one":
        lb = L.newlb(72, 70, 71, "null")
        spheres = [(31.0, 36, 35, 35)]
    elif kind == "both":
        lb = L.newlb(72, 70, 110, "null")
        spheres = [(31.0, 36, 35, 36)] + [(2.0, 10 + 17 * x, 10 + 16 * y, 88 + 6 * z) for x in range(4) for y in range(4) for z in range(3)]
    else:  # and an object without nodes
        lb = L.newlb(20, 20, 20, "null")
        spheres = [(6.0, 10, 10, 10)]
    lb.tau = 0.8
    objs = [L.insertsph(lb, *s) for s in spheres]
    L.addbf(lb, 1e-4, 3e-5, -2e-5)
    if kind == "empty":
        objs.append(L.addobj(lb))
    L.lbstep(lb)
    L.lbstep(lb)
    L.measure(lb)
    return lb, np.array([[o.frcx, o.frcy, o.frcz, o.trqx, o.trqy, o.trqz] for o in objs])


@pytest.mark.parametrize("kind", ["many", "one", "both", "empty"])
def test_object_sums(gpu, orc, kind):
    lb, got = build(gpu, kind)
    _, want = build(orc, kind)
    gpu.lbpull(lb)
    f = [np.abs(lb.array(c)) for c in ("fx", "fy", "fz")]
    n = int((f[0] > 0).sum())
    scale = n * 2.0 ** -53 * max(v.sum() for v in f)
    assert n > 0 and np.abs(want[:, :3]).max() > 0
    assert (np.abs(got - want)[:, :3] <= scale).all()
    assert (np.abs(got - want)[:, 3:] <= 2 * 110 * scale).all()

"""FP64 update on rows along k that fill whole warps (one row per block row)
and on rows that do not (a plane as one run of nodes): both against the CPU
oracle, bit for bit, with both update kinds, spheres across the periodic
faces, moving walls, inertia and a per-node body force.
"""

import numpy as np
import pytest

from scenarios import two_spheres

pytestmark = pytest.mark.gpu

CASES = [  # rows of 30 (31/32 full), 32, 33, 64, 70, 97 nodes; thin planes
    dict(dims=(7, 6, 30)),
    dict(dims=(6, 5, 32), moving=1),
    dict(dims=(5, 7, 33), stokes=0, tau=0.7),
    dict(dims=(4, 9, 64), stokes=0, moving=1),
    dict(dims=(3, 1, 70)),
    dict(dims=(1, 4, 97), skip=1),
    dict(dims=(9, 8, 97), stokes=0, moving=1, skip=1),
]


@pytest.mark.parametrize("cfg", CASES, ids=lambda c: "x".join(map(str, c["dims"])))
@pytest.mark.parametrize("steps", [7, 12])
def test_rows_and_runs_equal_oracle(gpu, orc, cfg, steps):
    pops = []
    for L in (gpu, orc):
        lb = two_spheres(L, steps=0, measure=False, **cfg)
        lb.array("bx")[: lb.nnodes // 3] *= 3.0  # per-node body force
        if L is gpu:
            L.lbpush(lb)
        for _ in range(steps):
            L.lbstep(lb)
        pops.append(lb.pops())
    assert np.array_equal(pops[0], pops[1])


@pytest.mark.parametrize("axis", ["x", "y", "z"])
@pytest.mark.parametrize("precision", [0, 1])
def test_wall_fills_and_injected_total(gpu, orc, axis, precision):
    """Plane fills along every axis (and a slab, a sphere, all nodes), several
    blocks each, counted by the block that finishes last: field and injected
    total equal the oracle's (FP64 field bit for bit; totals to the rounding
    of at most 1e5 FP64 additions of O(1) terms, 1e-11)."""
    out = []
    for L in (gpu, orc):
        lb = two_spheres(L, dims=(40, 50, 60), steps=3, measure=False, precision=precision if L is gpu else 0)
        mp = L.newmp(lb, "null")
        if L is gpu:
            mp.precision = precision
        mp.alpha = 0.3
        L.mpinit(mp)
        L.mpall(mp, 0.25)
        L.mpwall(mp, axis, 3, 1.5)
        L.mpslab(mp, 2.0, 9.0, 1.0, 20.0, 5.0, 44.0, 0.5)
        L.mpsph(mp, 9.5, 20.0, 25.0, 30.0, 0.75)
        L.mpwall(mp, axis, 0, 0.0)
        if L is gpu:
            L.mppull(mp)
        out.append((mp.field().copy(), L.mptotal(mp, "injected")))
    assert np.array_equal(out[0][0], out[1][0])  # the values are exact in FP32 too
    assert abs(out[0][1] - out[1][1]) <= 1e-11 * max(1.0, abs(out[1][1]))

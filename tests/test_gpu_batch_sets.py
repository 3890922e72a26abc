"""Batches larger than the L2, whose lattices go through all steps set by set:
the same bits as one lattice at a time, with moving and fixed walls, a uniform
and a per-node body force and members at both parities spread over the sets,
and for step counts below and above a graph's.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def members(L, precision, side, count):
    out = []
    for d in range(count):
        n = side + d % 3
        lb = L.newlb(n, side, side + d % 2, "null")
        lb.precision = precision
        lb.tau = 0.8 + 0.02 * d
        lb.stokes_flow = d % 2
        lb.objects_moving = (d // 2) % 2
        o = L.insertsph(lb, 0.2 * side + d, 0.5 * n, 0.45 * side, 0.4 * side)
        if lb.objects_moving:
            o.velx, o.angz = 1e-3, 1e-4
            L.vspread(lb)
        L.addbf(lb, 1e-5, 0.0, 2e-6)
        if d % 3 == 0:
            lb.array("bx")[: lb.nnodes // 2] *= 2.0
            L.lbpush(lb)
        L.lbsteps(lb, 1 + d % 2)
        out.append(lb)
    return out


@pytest.mark.parametrize("precision, side, count", [(1, 70, 8), (0, 64, 6)])  # 175 MB and 195 MB of state
@pytest.mark.parametrize("steps", [5, 104])
def test_sets_equal_one_at_a_time(gpu, precision, side, count, steps):
    batch, alone = members(gpu, precision, side, count), members(gpu, precision, side, count)
    b = gpu.newbatch()
    for lb in batch:
        gpu.batchadd(b, lb)
    gpu.batchsteps(b, steps)
    for one, two in zip(batch, alone):
        gpu.lbsteps(two, steps)
        assert np.array_equal(one.pops(), two.pops())
    gpu.freebatch(b)
    for lb in batch + alone:
        gpu.freelb(lb)

"""Batches of one large member and many small ones, in every launch class: the
bits of one lattice at a time, wherever the large one stands, and no more
launches per step than the sets and classes need.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lattice(L, side, i, precision):
    lb = L.newlb(side, side + i % 3, side, "null")
    lb.precision = precision
    lb.tau = 0.8 + 0.01 * (i % 7)
    lb.objects_moving = (i // 2) % 2
    o = L.insertsph(lb, 0.22 * side, 0.5 * side, 0.45 * side, 0.4 * side)
    if lb.objects_moving:
        o.velx, o.angz = 1e-3, 1e-4
        L.vspread(lb)
    L.addbf(lb, 1e-5, 0.0, 2e-6)
    if i % 2:
        lb.array("bx")[: lb.nnodes // 2] *= 2.0
        L.lbpush(lb)
    L.lbsteps(lb, 1 + (i // 4) % 2)
    return lb


@pytest.mark.parametrize("precision, large, small, count", [(1, 130, 20, 80), (0, 104, 16, 80)])  # 136 MB and 135 MB: past the L2
@pytest.mark.parametrize("place", [0, 40])
@pytest.mark.parametrize("steps", [3, 102])
def test_large_among_small(gpu, precision, large, small, count, place, steps):
    sides = [small] * place + [large] + [small] * (count - place)
    batch = [lattice(gpu, s, i, precision) for i, s in enumerate(sides)]
    alone = [lattice(gpu, s, i, precision) for i, s in enumerate(sides)]
    b = gpu.newbatch()
    for lb in batch:
        gpu.batchadd(b, lb)
    before = gpu.lbkernelcount()
    gpu.batchsteps(b, steps)
    # the small members (41 and 48 MB) are at most one set besides the large one:
    # 8 classes and 1, and a conversion or swap of layout per member
    assert gpu.lbkernelcount() - before <= 9 * steps + 2 * len(batch)
    for one, two in zip(batch, alone):
        gpu.lbsteps(two, steps)
        assert np.array_equal(one.pops(), two.pops())
    gpu.freebatch(b)
    for lb in batch + alone:
        gpu.freelb(lb)

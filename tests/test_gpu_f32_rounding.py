"""Rounding of the FP32 collision: its distance from the FP64 collision of the
same populations (root mean square over 336 nodes and 15 populations of order
0.1), no larger than that of the reference's expressions contracted by the
compiler, 5.824e-9 (Stokes) and 5.838e-9 (Navier-Stokes); a form that rounds
the trace of the stress on its own gives 5.96e-9 and 5.95e-9.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def collided(gpu, precision, stokes):
    lb = gpu.newlb(6, 7, 8, "null")
    lb.precision = precision
    lb.tau = 0.8
    lb.stokes_flow = stokes
    gpu.lbpull(lb)
    a = lb.array("a")
    a[:] = ((np.random.default_rng(2).random(a.shape) - 0.4) * 0.3).astype(np.float32)
    gpu.lbpush(lb)
    gpu.bblforce(lb)
    gpu.propagate(lb)
    gpu.collide(lb)
    out = lb.pops()
    gpu.freelb(lb)
    return out


@pytest.mark.parametrize("stokes, rms", [(1, 5.824e-9), (0, 5.838e-9)])
def test_collision_rounding(gpu, stokes, rms):
    e = collided(gpu, 1, stokes) - collided(gpu, 0, stokes)
    assert np.sqrt((e ** 2).mean()) <= 1.001 * rms

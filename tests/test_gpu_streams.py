"""Lattices set up while the program's default stream is still busy.

A lattice works on a stream of its own that does not wait for the default
stream, so nothing of its set-up may be queued on the default stream: the
geometry, forces and populations of a lattice created behind a long kernel
there must be those of one created on an idle GPU.
"""

import numpy as np
import pytest

from scenarios import objects_ft, two_spheres

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1, 2])
def test_setup_behind_a_busy_default_stream(gpu, precision):
    torch = pytest.importorskip("torch")
    cfg = dict(dims=(20, 17, 34), precision=precision, steps=3)
    ref = two_spheres(gpu, **cfg)
    want_p, want_f = ref.pops(), objects_ft(ref)
    for _ in range(3):
        torch.cuda._sleep(20_000_000)  # about 10 ms on the default stream
        lb = two_spheres(gpu, **cfg)
        assert np.array_equal(objects_ft(lb), want_f)
        assert np.array_equal(lb.pops(), want_p)
        gpu.freelb(lb)
    gpu.freelb(ref)

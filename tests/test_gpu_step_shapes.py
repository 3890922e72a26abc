"""Launch shapes of the FP64 update (lbtuning / lbsettuning): rows along k or the
nodes of a plane as one run, whichever is asked for.

A lattice reports the shape it runs, takes either form where both apply, and
gives the oracle's bits in each; the run form is refused where it does not apply
and in blocks it has no form for.
"""

import ctypes as C

import numpy as np
import pytest

from scenarios import two_spheres

pytestmark = pytest.mark.gpu

RUN = -1


def shape_of(L, lb):
    cfg = (C.c_int * 4)()
    state = L.lbtuning(lb, C.addressof(cfg))
    return state, list(cfg)


@pytest.mark.parametrize("dims, even", [
    ((7, 6, 30), [RUN, 32]),   # 30 of 32 lanes: below 16/17
    ((5, 7, 33), [RUN, 32]),
    ((6, 5, 32), [1, 128]),
    ((4, 5, 62), [1, 128]),    # 62 of 64
    ((40, 64, 65), [RUN, 128]),  # 166,400 nodes: full blocks
])
def test_default_shape_is_the_one_that_runs(gpu, dims, even):
    lb = two_spheres(gpu, steps=1, measure=False, dims=dims)
    assert shape_of(gpu, lb) == (-1, even * 2)


@pytest.mark.parametrize("steps", [7, 12])
@pytest.mark.parametrize("shape", [(1, 64, 1, 64), (2, 128, 4, 32), (RUN, 32, RUN, 128), (RUN, 64, 1, 256), (1, 32, RUN, 64)],
                         ids=lambda s: ",".join(map(str, s)))
@pytest.mark.parametrize("dims", [(5, 7, 33), (6, 5, 32), (4, 3, 130)], ids=lambda d: "x".join(map(str, d)))
def test_either_form_equals_oracle(gpu, orc, dims, shape, steps):
    pops = []
    for L in (gpu, orc):
        lb = two_spheres(L, steps=0, measure=False, dims=dims, moving=1, stokes=0)
        if L is gpu:
            assert L.lbsettuning(lb, C.addressof((C.c_int * 4)(*shape))) == 0
        for _ in range(steps):
            L.lbstep(lb)
        if L is gpu:
            assert shape_of(L, lb) == (1, list(shape))
        pops.append(lb.pops())
    assert np.array_equal(pops[0], pops[1])


@pytest.mark.parametrize("shape", [(RUN, 256), (RUN, 16), (RUN, 0), (-2, 128), (-4, 128)])
def test_shapes_without_a_form_are_refused(gpu, shape):
    lb = two_spheres(gpu, dims=(5, 7, 33), steps=1, measure=False)
    before = shape_of(gpu, lb)
    assert gpu.lbsettuning(lb, C.addressof((C.c_int * 4)(*(shape * 2)))) != 0
    assert gpu.lbsettuning(lb, C.addressof((C.c_int * 4)(1, 64, *shape))) != 0
    assert shape_of(gpu, lb) == before


@pytest.mark.parametrize("precision", [1, 2])
def test_runs_are_fp64_only(gpu, precision):
    lb = two_spheres(gpu, dims=(6, 7, 33), steps=1, measure=False, precision=precision)
    assert gpu.lbsettuning(lb, C.addressof((C.c_int * 4)(RUN, 128, RUN, 128))) != 0

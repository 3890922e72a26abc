"""Velocity and density field (slbc_get_state_dev) at the edges of its range:
infinite populations and sums beyond FP32, any factor of a per-node body force,
and lattices whose rows along k are short or whose sides are long.

Against FP64 numpy of the same populations.  FP64 sums of 15 terms of order one
are exact to 1e-15 relative, the FP32 lattice's pairs to about 2^-44: a result
is the FP32 value nearest to numpy's, up to half an ulp and 2^-10 of one, where
rounding falls on the other side.
"""

import ctypes as C

import numpy as np
import pytest

from test_gpu_stream_order import ptr

pytestmark = pytest.mark.gpu

CX = np.array([0, 1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 1, -1, 1, -1.0])
CY = np.array([0, 0, 0, 1, -1, 0, 0, 1, 1, -1, -1, 1, 1, -1, -1.0])
CZ = np.array([0, 0, 0, 0, 0, 1, -1, 1, 1, 1, 1, -1, -1, -1, -1.0])


def field(gpu, dims, precision, pops, force=None, fac=0.0, steps=0):
    """(u, drho) of the GPU, FP32; with steps, of the state after that many
    updates on a lattice without objects, and the state."""
    torch = pytest.importorskip("torch")
    d, n = gpu.dll, int(np.prod(dims))
    h = C.c_void_p()
    assert d.slbc_create(C.byref(h), *dims, precision) == 0
    assert d.slbc_put_pops(h, ptr(pops)) == 0
    if force is not None:
        assert d.slbc_set_bodyforce(h, *(ptr(v) for v in force)) == 0
    if steps:
        assert d.slbc_step(h, steps, 0) == 0
    u = torch.full((3, n), 7.0, device="cuda")
    dr = torch.full((n,), 7.0, device="cuda")
    torch.cuda.synchronize()
    d.slbc_get_state_dev.argtypes = [C.c_void_p, C.c_double, C.c_void_p, C.c_void_p]
    assert d.slbc_get_state_dev(h, fac, u.data_ptr(), dr.data_ptr()) == 0
    assert d.slbc_synchronize(h) == 0
    state = np.empty((n, 15))
    assert d.slbc_get_pops(h, ptr(state)) == 0
    d.slbc_destroy(h)
    return u.cpu().numpy(), dr.cpu().numpy(), state


def plain(pops, force, fac):
    with np.errstate(all="ignore"):
        r = pops.sum(1)
        inv = 1.0 / (72.0 + r)
        u = [sum(c[q] * pops[:, q] for q in range(15)) for c in (CX, CY, CZ)]
        if force is not None:
            u = [m + fac * b for m, b in zip(u, force)]
        return np.array([m * inv for m in u]), r


def near(got, want):
    with np.errstate(all="ignore"):
        w32 = want.astype(np.float32)
        same = (got == w32) | (np.isnan(got) & np.isnan(w32))
        half = np.abs(got.astype(float) - want) <= (0.5 + 2.0 ** -10) * np.spacing(np.abs(w32))
    return same | (np.isfinite(want) & half)


@pytest.mark.parametrize("precision", [1, 0])
def test_infinite_and_large_sums(gpu, precision):
    a = np.zeros((210, 15))
    a[17, 3], a[40, 5], a[60, 0] = np.inf, -np.inf, np.inf
    a[61, [0, 1, 7]] = 1e38, 3e38, 3.3e38  # each in FP32, their sum not
    a[70, 0] = -72.0                       # density zero, no momentum
    a[71, [0, 1]] = -73.0, 1.0             # density zero, momentum along x
    a[72, 4] = np.nan
    a = a.astype(np.float32).astype(float)
    u, dr, _ = field(gpu, (5, 6, 7), precision, a)
    wu, wr = plain(a, None, 0.0)
    assert near(dr, wr).all()
    assert near(u, wu).all(), np.argwhere(~near(u, wu))
    assert np.isposinf(dr[17]) and np.isneginf(dr[40]) and np.isfinite(u[:, 61]).all() and np.isposinf(dr[61])


@pytest.mark.parametrize("precision", [1, 0])
@pytest.mark.parametrize("fac", [0.5, -0.5, 0.3, -1.7, 1e-3])
def test_any_factor_of_a_per_node_force(gpu, precision, fac):
    dims, rng = (7, 8, 9), np.random.default_rng(6)
    n = int(np.prod(dims))
    force = [rng.random(n).astype(np.float32).astype(float) for _ in range(3)]
    pops = ((rng.random((n, 15)) - 0.5) * 0.1).astype(np.float32).astype(float)
    u, dr, _ = field(gpu, dims, precision, pops, force, fac)
    wu, wr = plain(pops, force, fac)
    assert near(dr, wr).all()
    assert near(u, wu).all(), int((~near(u, wu)).sum())


SHAPES = [  # dims: rows of 1 to 260 nodes, a line, a side beyond 65,535
    (17, 19, 1), (700, 1, 1), (1, 700, 1), (9, 11, 3), (5, 7, 31), (6, 5, 32), (5, 6, 33), (4, 5, 48), (3, 5, 65), (3, 4, 97),
    (3, 3, 128), (2, 3, 130), (2, 2, 260), (2, 70000, 2), (70000, 2, 1),
]


@pytest.mark.parametrize("precision", [1, 0])
@pytest.mark.parametrize("dims", SHAPES, ids=lambda d: "x".join(map(str, d)))
def test_every_shape_and_layout(gpu, dims, precision):
    """The uploaded layout and those after one and two updates (sides beyond
    65,535 take no update: the uploaded one)."""
    n = int(np.prod(dims))
    pops = ((np.random.default_rng(8).random((n, 15)) - 0.5) * 0.1).astype(np.float32).astype(float)
    for steps in (0, 1, 2) if max(dims[:2]) <= 65535 else (0,):
        u, dr, state = field(gpu, dims, precision, pops, fac=0.5, steps=steps)
        wu, wr = plain(state, None, 0.0)
        assert near(dr, wr).all(), steps
        assert near(u, wu).all(), (steps, int((~near(u, wu)).sum()))

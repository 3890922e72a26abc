"""Uploads of lattices, batches and tracers go by the lattice's (or batch's) own
stream: with the default stream busy for a long time the set-up and the steps
finish before it does, and leave the same fields.

Everything runs once on an idle GPU first, so that no kernel or buffer is
created while the default stream is busy.
"""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = (12, 13, 40)
N = int(np.prod(DIMS))


def ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def geometry(objects):
    """Object map of two blocks and its boundary list, by object then node."""
    obj = np.full(DIMS, -1, np.int32)
    obj[2:6, 3:7, 5:20] = 0
    if objects > 1:
        obj[8:11, 8:12, 22:38] = 1
    solid = obj >= 0
    near = np.zeros(DIMS, bool)
    links = [(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 1), (1, 1, -1), (1, -1, 1), (1, -1, -1)]
    for c in links:
        for s in (1, -1):
            near |= ~np.roll(solid, [s * x for x in c], (0, 1, 2))
    node = [np.flatnonzero((obj == o).ravel() & near.ravel()) for o in range(objects)]
    return obj, np.concatenate(node).astype(np.int64), np.repeat(np.arange(objects, dtype=np.int32), [len(x) for x in node])


class Case:
    """Two lattices, a batch of them and, for FP64 and FP32 lattices, a tracer."""

    def __init__(self, d, precision, mode):
        self.d, self.precision = d, precision
        rng = np.random.default_rng(4)
        self.h, self.tracer, self.batch = [], [], C.c_void_p()
        for l in range(2):
            h = C.c_void_p()
            assert d.slbc_create(C.byref(h), *DIMS, precision) == 0
            self.h.append(h)
        self.pops = np.ascontiguousarray(rng.random((N, 15)) * 1e-2)
        self.vec = [rng.random(N) * 1e-4 for _ in range(6)]
        if precision != 2:
            arr = (C.c_void_p * 2)(*self.h)
            assert d.slbc_batch_create(C.byref(self.batch), arr, 2) == 0
            assert d.slbc_batch_set_mode(self.batch, mode) == 0

    def work(self):
        d = self.d
        for l, h in enumerate(self.h):
            obj, node, bobj = geometry(1 + l)
            assert d.slbc_set_geometry(h, ptr(obj), 1 + l, ptr(node), ptr(bobj), C.c_long(len(node))) == 0
            assert d.slbc_set_bodyforce(h, *(ptr(v) for v in self.vec[:3])) == 0
            if l:
                assert d.slbc_set_wallvel(h, *(ptr(v) for v in self.vec[3:])) == 0
            if self.precision != 2:
                assert d.slbc_put_pops(h, ptr(self.pops)) == 0
                t = C.c_void_p()
                assert d.slbc_mp_create(h, C.byref(t), 1 - self.precision) == 0
                geo = (C.c_double * 6)(0.0, 3.0)
                assert d.slbc_mp_fill(t, 2, geo, C.c_double(1.0)) == 0
                assert d.slbc_mp_step(t, 3, C.c_double(0.3), C.c_double(1.0), 0, None, 0) == 0
                self.tracer.append(t)
        if self.batch:
            assert d.slbc_batch_step(self.batch, 5) == 0
        for h in self.h:
            assert d.slbc_step(h, 3, 0) == 0
            assert d.slbc_synchronize(h) == 0

    def results(self):
        out = []
        for h in self.h:
            a = np.empty((N, 15))
            assert self.d.slbc_get_pops(h, ptr(a)) == 0
            out.append(a)
        for t in self.tracer:
            p = np.empty(N)
            assert self.d.slbc_mp_get(t, ptr(p)) == 0
            out.append(p)
        return out

    def free(self):
        for t in self.tracer:
            self.d.slbc_mp_destroy(t)
        if self.batch:
            self.d.slbc_batch_destroy(self.batch)
        for h in self.h:
            self.d.slbc_destroy(h)


@pytest.mark.parametrize("precision, mode", [(0, 0), (0, 1), (1, 0), (1, 1), (2, 0)])
def test_setup_does_not_wait_for_the_default_stream(gpu, precision, mode):
    torch = pytest.importorskip("torch")
    idle = Case(gpu.dll, precision, mode)
    idle.work()
    want = idle.results()
    busy = Case(gpu.dll, precision, mode)
    torch.cuda.synchronize()
    torch.cuda._sleep(1_000_000_000)  # about half a second on the default stream
    done = torch.cuda.Event()
    done.record()
    busy.work()
    assert not done.query()
    torch.cuda.synchronize()
    for a, b in zip(busy.results(), want):
        assert np.array_equal(a, b)
    idle.free()
    busy.free()

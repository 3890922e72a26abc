"""Tracer updates captured in a graph: the first update ever of a lattice, and
replays after other flows' density snapshots, equal the same updates called one
by one.
"""

import ctypes as C

import numpy as np
import pytest

from test_gpu_stream_order import ptr

pytestmark = pytest.mark.gpu

DIMS = (9, 10, 40)
N = int(np.prod(DIMS))


class Flow:
    def __init__(self, d, stream):
        rng = np.random.default_rng(2)
        self.d, self.h, self.t = d, C.c_void_p(), C.c_void_p()
        assert d.slbc_create(C.byref(self.h), *DIMS, 0) == 0
        if stream:
            d.slbc_set_stream.argtypes = [C.c_void_p, C.c_void_p]
            assert d.slbc_set_stream(self.h, stream) == 0
        assert d.slbc_put_pops(self.h, ptr(np.ascontiguousarray(rng.random((N, 15)) * 0.3))) == 0
        force = [rng.random(N) * 1e-3 for _ in range(3)]
        assert d.slbc_set_bodyforce(self.h, *(ptr(v) for v in force)) == 0
        assert d.slbc_step(self.h, 2, 0) == 0
        assert d.slbc_mp_create(self.h, C.byref(self.t), 1) == 0
        assert d.slbc_mp_put(self.t, ptr(rng.random(N))) == 0
        assert d.slbc_synchronize(self.h) == 0

    def update(self):
        self.d.slbc_mp_step.argtypes = [C.c_void_p, C.c_int, C.c_double, C.c_double, C.c_int, C.c_void_p, C.c_int]
        assert self.d.slbc_mp_step(self.t, 2, 0.3, 1.0, 0, None, 0) == 0

    def snapshot(self):
        assert self.d.slbc_step(self.h, 2, 0) == 0
        assert self.d.slbc_mp_rhoinit(self.h) == 0

    def field(self):
        p = np.empty(N)
        assert self.d.slbc_mp_get(self.t, ptr(p)) == 0
        return p

    def end(self):
        self.d.slbc_mp_destroy(self.t)
        self.d.slbc_destroy(self.h)


def test_replays_follow_the_snapshots(gpu):
    torch = pytest.importorskip("torch")
    first = Flow(gpu.dll, None)  # kernels loaded and set up outside the capture
    first.update()
    first.snapshot()
    first.end()
    eager, stream = Flow(gpu.dll, None), torch.cuda.Stream()
    replayed = Flow(gpu.dll, stream.cuda_stream)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        replayed.update()
    for turn in range(4):
        eager.update()
        with torch.cuda.stream(stream):
            graph.replay()
        torch.cuda.synchronize()
        want = eager.field()
        assert np.isfinite(want).all() and want.std() > 0
        assert np.array_equal(replayed.field(), want), turn
        eager.snapshot()
        replayed.snapshot()
    del graph
    torch.cuda.synchronize()
    eager.end()
    replayed.end()

"""Lists of tensors in one launch: more tensors than a launch takes, sizes
around a block's 2048 elements, against PyTorch.

Adam and the scaling round a few FP32 operations per element (2^-21 relative of
the terms); squares are summed in FP64; layouts are copies rounded to BF16, so
equal bits.
"""

import ctypes as C

import pytest

from sunlightlb_gb300.warmstart import Kernels, pointers

pytestmark = pytest.mark.gpu

SIZES = [1, 32, 2047, 2048, 2049, 70001] * 9  # 54 tensors: two launches


def test_adam_squares_and_scale(gpu):
    torch = pytest.importorskip("torch")
    k = Kernels(gpu.dll)
    st = torch.cuda.current_stream().cuda_stream
    gen = torch.Generator(device="cuda").manual_seed(5)
    make = lambda n: torch.randn(n, device="cuda", generator=gen)
    P, G, M = ([make(n) for n in SIZES] for _ in range(3))
    V = [make(n).abs() for n in SIZES]
    n = (C.c_longlong * len(SIZES))(*SIZES)
    ptr = lambda ts: pointers(t.data_ptr() for t in ts)
    lr, b1, b2, eps, t = 1e-2, 0.9, 0.999, 1e-8, 3
    want = []
    for p, g, m, v in zip(P, G, M, V):
        m2 = b1 * m.double() + (1 - b1) * g.double()
        v2 = b2 * v.double() + (1 - b2) * g.double() ** 2
        step = lr * (m2 / (1 - b1 ** t)) / ((v2 / (1 - b2 ** t)).sqrt() + eps)
        want.append((p.double() - step, m2, v2, step))
    state = torch.tensor([0.5, 2.0, 0.0], device="cuda", dtype=torch.float64)
    k.nn_sqsum_list(len(SIZES), ptr(G), n, state.data_ptr(), st)
    total = 0.5 + sum(float((g.double() ** 2).sum()) for g in G)
    assert abs(float(state[0]) - total) <= 1e-12 * total
    k.nn_adam_list(len(SIZES), ptr(P), ptr(G), ptr(M), ptr(V), n, lr, b1, b2, eps, t, st)
    for p, m, v, (wp, wm, wv, step) in zip(P, M, V, want):
        assert ((m - wm).abs() <= 2.0 ** -21 * (wm.abs() + 4)).all()
        assert ((v - wv).abs() <= 2.0 ** -21 * (wv.abs() + 4)).all()
        # b2 and 1 - b2^t in FP32 keep 2^-24 of 1, t 2^-24 / 0.003 < 2^-14 of the difference
        assert ((p - wp).abs() <= 2.0 ** -22 * wp.abs() + 2.0 ** -13 * step.abs()).all()
    before = [g.clone() for g in G]
    for scale in (0.25, 1.0, 0.0):
        state[2] = scale
        k.nn_scale_list(len(SIZES), ptr(G), n, state.data_ptr(), st)
        before = [b * scale for b in before]
        assert all(torch.equal(g, b) for g, b in zip(G, before))


def test_layouts(gpu):
    torch = pytest.importorskip("torch")
    k = Kernels(gpu.dll)
    st = torch.cuda.current_stream().cuda_stream
    jobs = [(32, 32, 0, 0), (32, 96, 0, 96), (48, 64, 0, 0), (64, 40, 8, 24), (256, 32, 0, 32)] * 10
    masters = [torch.randn(27, co, ci, device="cuda") for co, ci, _, _ in jobs]
    outs = [torch.zeros(27 * co * (nci or ci), device="cuda", dtype=torch.bfloat16) for co, ci, _, nci in jobs]
    ints = lambda j: (C.c_int * len(jobs))(*(job[j] for job in jobs))
    k.nn_layouts(len(jobs), pointers(m.data_ptr() for m in masters), ints(0), ints(1), ints(2), ints(3),
                 pointers(o.data_ptr() for o in outs), st)
    for m, o, (co, ci, c0, nci) in zip(masters, outs, jobs):
        if nci:
            w = m.flip(0)[:, :, c0:c0 + nci].reshape(27, co // 32, 32, nci).permute(0, 1, 3, 2)
        else:
            w = m.reshape(27, co, ci // 32, 32).permute(0, 2, 1, 3)
        assert torch.equal(o, w.reshape(-1).to(torch.bfloat16))

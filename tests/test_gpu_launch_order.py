"""Launches that overlap the end of their predecessor read what it wrote,
whatever it is: a library's kernel that runs long, a copy, a fill, an event of
another stream, another of these kernels, eagerly and inside a captured graph.

Pooling and upsampling of small integers are exact, so the results are equal
bits; a kernel that did not wait would read the poison that was there before.
"""

import pytest

from sunlightlb_gb300.warmstart import Kernels

pytestmark = pytest.mark.gpu

B, D, C = 2, 48, 32


def chain(torch, k, kind, value, src, mid, out, side):
    """src = value by way of `kind`, then pooled to mid and upsampled to out."""
    stream = torch.cuda.current_stream()
    if kind == "event":
        side.wait_stream(stream)
        with torch.cuda.stream(side):
            src.copy_(value)
        stream.wait_stream(side)
    elif kind == "fill":
        src.zero_()
    elif kind == "copy":
        src.view(torch.uint8).copy_(value.view(torch.uint8))
    else:  # a kernel that takes far longer than a launch
        src.copy_(torch.cumsum(value.view(-1).float() * 0, 0).view_as(value) + value)
    st = stream.cuda_stream
    for _ in range(3):
        k.nn_pool(src.data_ptr(), C, 0, mid.data_ptr(), C, 0, B, D, D, D, C, st)
        k.nn_up(mid.data_ptr(), C, 0, out.data_ptr(), C, 0, B, D, D, D, C, st)


@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("kind", ["kernel", "copy", "fill", "event"])
def test_results_of_the_predecessor(gpu, kind, captured):
    torch = pytest.importorskip("torch")
    k = Kernels(gpu.dll)
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    buf = lambda n: torch.full((B, n + 2, n + 2, n + 2, C), 7.0, device="cuda", dtype=torch.bfloat16)
    src, mid, out, value = buf(D), buf(D // 2), buf(D), buf(D)
    torch.cuda.synchronize()
    with torch.cuda.stream(main):
        chain(torch, k, kind, value, src, mid, out, side)
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=main):
                chain(torch, k, kind, value, src, mid, out, side)
    torch.cuda.synchronize()
    for turn in range(4):
        with torch.cuda.stream(main):
            fine = torch.randint(-4, 5, (B, D // 2, D // 2, D // 2, C), device="cuda").to(torch.bfloat16)
            fine = fine.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)
            value[:, 1:-1, 1:-1, 1:-1] = fine
            for t in (src, mid, out):
                t.fill_(7.0)
            if captured:
                graph.replay()
            else:
                chain(torch, k, kind, value, src, mid, out, side)
        torch.cuda.synchronize()
        want = torch.zeros_like(fine) if kind == "fill" else fine
        assert torch.equal(out[:, 1:-1, 1:-1, 1:-1], want)

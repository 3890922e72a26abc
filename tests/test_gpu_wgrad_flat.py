"""Weight gradients from flat channels-last copies (slbc_tc_flat,
slbc_tc_wgrad_flat) against the channel-major form with the same splits: the
same products in the same order, so equal bits; the copies against indexing.
Shapes: every output width, tap groups of nine, three, two and one, input
chunks, rows that touch (W + 2 a multiple of 8), tiles over sample ends, more
splits than K tiles.
"""

import pytest

from sunlightlb_gb300.warmstart import Kernels, flat_geometry

pytestmark = pytest.mark.gpu

CASES = [  # B, D, H, W, cin, cout, splits
    (1, 8, 8, 16, 32, 32, 5),
    (2, 3, 5, 6, 32, 64, 3),      # rows touch
    (1, 4, 4, 62, 96, 32, 7),     # rows touch, three taps per block
    (3, 4, 6, 10, 64, 64, 2),
    (2, 4, 4, 8, 128, 128, 4),
    (1, 2, 4, 16, 192, 64, 2),
    (1, 4, 4, 4, 384, 128, 1),    # input channels in two chunks
    (1, 2, 2, 2, 32, 32, 64),     # more splits than tiles
    (4, 16, 16, 16, 32, 128, 37),
]


@pytest.mark.parametrize("case", CASES)
def test_same_bits_as_channel_major(gpu, case):
    torch = pytest.importorskip("torch")
    k = Kernels(gpu.dll)
    B, D, H, W, cin, cout, splits = case
    Wp, ps = flat_geometry(D, H, W)
    g = torch.Generator(device="cuda").manual_seed(sum(case))
    st = torch.cuda.current_stream().cuda_stream
    make = lambda c: torch.randn(B, D + 2, H + 2, W + 2, c, device="cuda", generator=g).to(torch.bfloat16)
    dy, x = make(cout + 16), make(cin + 8)
    bf = lambda *shape: torch.full(shape, 7.0, device="cuda", dtype=torch.bfloat16)
    gt, xt, gf, xf = bf(B * ps // 64, 3, cout, 64), bf(cin, B * ps), bf(B * ps, cout), bf(B * ps, cin)
    k.tc_cmajor_shifts(dy.data_ptr(), B, D, H, W, cout + 16, 8, cout, Wp, ps, 1, gt.data_ptr(), st)
    k.tc_cmajor(x.data_ptr(), B, D, H, W, cin + 8, 8, cin, Wp, ps, 0, 1, xt.data_ptr(), st)
    k.tc_flat(dy.data_ptr(), B, D, H, W, cout + 16, 8, cout, Wp, ps, 0, gf.data_ptr(), st)
    k.tc_flat(x.data_ptr(), B, D, H, W, cin + 8, 8, cin, Wp, ps, 1, xf.data_ptr(), st)
    assert torch.equal(xf.T, xt)
    assert torch.equal(gf.view(-1, 64, cout).permute(0, 2, 1), gt[:, 1])
    n = 27 * cout * cin
    ws = torch.empty(splits * n, device="cuda")
    a, b = torch.zeros(n, device="cuda"), torch.ones(n, device="cuda")
    k.tc_wgrad_tiles(gt.data_ptr(), xt.data_ptr(), B, D, H, W, Wp, ps, cin, cout, ws.data_ptr(), splits * n, splits,
                     a.data_ptr(), st)
    k.tc_wgrad_flat(gf.data_ptr(), xf.data_ptr(), B, D, H, W, Wp, ps, cin, cout, ws.data_ptr(), splits * n, splits,
                    b.data_ptr(), st)
    assert gpu.dll.slbc_tc_status() == 0
    assert float(a.abs().max()) > 0
    assert torch.equal(a, b)

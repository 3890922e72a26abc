"""Channel-major copies (slbc_tc_cmajor, slbc_tc_cmajor_shifts) of long rows, of
row pitches beyond 16 bits and of samples of 2^31 positions, against indexing.
"""

import pytest

from sunlightlb_gb300.warmstart import Kernels, flat_geometry

pytestmark = pytest.mark.gpu


def expected(torch, src, coff, nch, Wp, shift):
    """[nch][B][(D + 2) * (H + 2) * Wp] of a padded channels-last buffer."""
    B, Dp, Hp, Wd, _ = src.shape
    out = torch.zeros(nch, B, Dp, Hp, Wp, device=src.device, dtype=src.dtype)
    lo, hi = max(0, shift), min(Wp, Wd + shift)
    out[..., lo:hi] = src[..., lo - shift:hi - shift, coff:coff + nch].permute(4, 0, 1, 2, 3)
    return out.reshape(nch, B, Dp * Hp * Wp)


@pytest.mark.parametrize("W, Wp", [(16381, None), (16384, None), (20000, None), (40000, None), (10, 32776), (10, 65536), (70000, None)])
def test_long_rows(gpu, W, Wp):
    torch = pytest.importorskip("torch")
    k = Kernels(gpu.dll)
    B, D, H, nch = 2, 1, 2, 40
    Wp = Wp or flat_geometry(D, H, W)[0]
    ps = ((D + 2) * (H + 2) * Wp + 63) // 64 * 64
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(W + Wp)
    src = torch.randn(B, D + 2, H + 2, W + 2, nch + 8, device="cuda", generator=g).to(torch.bfloat16)
    dst = torch.full((3, nch, B, ps), 7.0, device="cuda", dtype=torch.bfloat16)
    per = (D + 2) * (H + 2) * Wp
    k.tc_cmajor_shifts(src.data_ptr(), B, D, H, W, nch + 8, 8, nch, Wp, ps, 0, dst.data_ptr(), st)
    for i, shift in enumerate((-1, 0, 1)):
        assert torch.equal(dst[i, :, :, :per], expected(torch, src, 8, nch, Wp, shift)), shift
        assert not dst[i, :, :, per:].any()
    for shift in (-1, 0, 1):
        one = torch.full((nch, B, ps), 7.0, device="cuda", dtype=torch.bfloat16)
        k.tc_cmajor(src.data_ptr(), B, D, H, W, nch + 8, 8, nch, Wp, ps, shift, 0, one.data_ptr(), st)
        assert torch.equal(one, dst[shift + 1])


def test_samples_of_two_to_the_31_positions(gpu):
    torch = pytest.importorskip("torch")
    k = Kernels(gpu.dll)
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("not enough memory on the GPU")
    B, D, H, W, nch = 1, 3, 4, 6, 8
    Wp, ps = 8, 1 << 31
    st = torch.cuda.current_stream().cuda_stream
    src = torch.randn(B, D + 2, H + 2, W + 2, nch, device="cuda").to(torch.bfloat16)
    dst = torch.full((nch, ps), 7.0, device="cuda", dtype=torch.bfloat16)  # 34 GB
    k.tc_cmajor(src.data_ptr(), B, D, H, W, nch, 0, nch, Wp, ps, 0, 0, dst.data_ptr(), st)
    per = (D + 2) * (H + 2) * Wp
    assert torch.equal(dst[:, :per], expected(torch, src, 0, nch, Wp, 0)[:, 0])
    for c in range(nch):
        assert int(torch.count_nonzero(dst[c, per:])) == 0
    del dst
    torch.cuda.empty_cache()

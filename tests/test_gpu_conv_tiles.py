"""Persistent convolution tiles (32, 64 or 128 output channels) at the sizes
where they can go wrong: more tiles than blocks (several accumulator rounds
per block), two and four z slices, several channel chunks, one tile in all.

Against PyTorch in FP32 on BF16-rounded inputs; tolerance as in
test_gpu_tc.py: the result is off by its BF16 rounding (2^-9) and the FP32
accumulation.
"""

import pytest

from sunlightlb_gb300.warmstart import Kernels
from test_gpu_tc import conv_fns, gemm_weights, to_padded

pytestmark = pytest.mark.gpu


CONV = [  # B, D, H, W, cin, cout
    (1, 64, 64, 64, 32, 32),   # 512 tiles of four slices on 152 blocks
    (2, 8, 32, 64, 96, 32),
    (1, 2, 8, 16, 32, 32),     # one tile
    (1, 32, 64, 64, 64, 64),
    (3, 6, 16, 32, 32, 64),    # D a multiple of 2 only
    (1, 32, 64, 64, 32, 128),
]


@pytest.mark.parametrize("case", CONV)
def test_conv_tiles_match_torch(gpu, case):
    torch = pytest.importorskip("torch")
    F = torch.nn.functional
    conv, halo = conv_fns(gpu)
    B, D, H, W, cin, cout = case
    g = torch.Generator(device="cuda").manual_seed(sum(case))
    x = torch.randn(B, cin, D, H, W, device="cuda", generator=g).to(torch.bfloat16).float()
    wt = (torch.randn(cout, cin, 3, 3, 3, device="cuda", generator=g) / (27 * cin) ** 0.5).to(torch.bfloat16).float()
    bias = torch.randn(cout, device="cuda", generator=g) * 0.1
    st = torch.cuda.current_stream().cuda_stream
    xin = to_padded(torch, x, cin, 0)
    assert halo(xin.data_ptr(), B, D, H, W, cin, 0, cin, st) == 0
    w = gemm_weights(torch, wt)
    out = torch.zeros(B, D + 2, H + 2, W + 2, cout, device="cuda", dtype=torch.bfloat16)
    assert conv(xin.data_ptr(), B, D, H, W, cin, 0, cin, w.data_ptr(), bias.data_ptr(), cout, out.data_ptr(), cout, 0,
                1, None, st) == 0
    assert gpu.dll.slbc_tc_status() == 0
    ref = F.conv3d(F.pad(x, (1, 1, 1, 1, 1, 1), mode="circular"), wt, bias).clamp_min(0.0)
    got = out[:, 1:-1, 1:-1, 1:-1].float().permute(0, 4, 1, 2, 3)
    assert ((got - ref).abs() <= 4e-3 * ref.abs() + 2e-3 * ref.abs().max().item()).all()


SHIFTS = [  # B, D, H, W, ctot, coff, nch (multiples of 8)
    (1, 8, 8, 8, 32, 0, 32),       # rows of 10 voxels at a pitch of 16
    (2, 3, 5, 6, 48, 8, 40),       # W + 2 equal to the row pitch: rows touch
    (1, 4, 8, 62, 72, 0, 72),      # the same, with 64-position tiles across rows
    (2, 16, 16, 16, 256, 0, 256),
    (1, 2, 4, 130, 40, 16, 24),
]


@pytest.mark.parametrize("case", SHIFTS)
def test_channel_major_copies_match_definition(gpu, case):
    """slbc_tc_cmajor (every shift, with and without the halo),
    slbc_tc_cmajor_tiles and slbc_tc_cmajor_shifts against indexing; copies,
    so equal bits."""
    torch = pytest.importorskip("torch")
    k = Kernels(gpu.dll)
    B, D, H, W, ctot, coff, nch = case
    Wp = (W + 2 + 7) // 8 * 8
    ps = ((D + 2) * (H + 2) * Wp + 63) // 64 * 64
    g = torch.Generator(device="cuda").manual_seed(sum(case))
    src = torch.randn(B, D + 2, H + 2, W + 2, ctot, device="cuda", generator=g).to(torch.bfloat16)
    st = torch.cuda.current_stream().cuda_stream

    def expect(shift, zero_halo):
        v = src[..., coff:coff + nch].clone()
        if zero_halo:
            keep = torch.zeros(D + 2, H + 2, W + 2, 1, device="cuda", dtype=torch.bool)
            keep[1:-1, 1:-1, 1:-1] = True
            v = v * keep
        rows = torch.zeros(B, D + 2, H + 2, Wp, nch, device="cuda", dtype=torch.bfloat16)
        for x in range(Wp):
            if 0 <= x - shift <= W + 1:
                rows[..., x, :] = v[..., x - shift, :]
        flat = torch.zeros(B, ps, nch, device="cuda", dtype=torch.bfloat16)
        flat[:, :(D + 2) * (H + 2) * Wp] = rows.reshape(B, -1, nch)
        return flat.reshape(B * ps, nch).T.contiguous()

    args = (src.data_ptr(), B, D, H, W, ctot, coff, nch, Wp, ps)
    whole = torch.full((3, nch, B * ps), 7.0, device="cuda", dtype=torch.bfloat16)
    k.tc_cmajor_shifts(*args, 0, whole.data_ptr(), st)
    tiles = torch.full((B * ps // 64, 3, nch, 64), 7.0, device="cuda", dtype=torch.bfloat16)
    k.tc_cmajor_shifts(*args, 1, tiles.data_ptr(), st)
    one = torch.full((B * ps // 64, 3, nch, 64), 7.0, device="cuda", dtype=torch.bfloat16)
    for i, shift in enumerate((-1, 0, 1)):
        want = expect(shift, False)
        assert torch.equal(whole[i], want)
        assert torch.equal(tiles[:, i].permute(1, 0, 2).reshape(nch, -1), want)
        k.tc_cmajor_tiles(*args, shift, i, 3, one.data_ptr(), st)
        for zero in (0, 1):
            got = torch.full((nch, B * ps), 7.0, device="cuda", dtype=torch.bfloat16)
            k.tc_cmajor(*args, shift, zero, got.data_ptr(), st)
            assert torch.equal(got, expect(shift, bool(zero)))
    assert torch.equal(one, tiles)

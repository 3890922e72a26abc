"""Convolutions that stage each input voxel once (32 and 64 output channels, y a
multiple of 16): run lengths from one slice to the longest, uneven runs, rings
that wrap, several chunks, and the shapes next to the rule's edges (y of 8, x
of 8).

Against PyTorch in FP32 on BF16-rounded inputs; tolerance as in
test_gpu_tc.py: the result is off by its BF16 rounding (2^-9) and the FP32
accumulation.
"""

import pytest

from sunlightlb_gb300.warmstart import Kernels  # noqa: F401 (declares the entry points)
from test_gpu_tc import conv_fns, gemm_weights, to_padded

pytestmark = pytest.mark.gpu

CONV = [  # B, D, H, W, cin, cout
    (1, 1, 16, 8, 32, 32),       # one slice, one block
    (1, 16, 16, 8, 32, 64),      # 16 slices on one column
    (2, 64, 64, 64, 32, 32),     # 9 or 10 planes per item, several items per block
    (1, 64, 64, 64, 64, 64),     # 19 runs of 3 and 4 slices
    (3, 4, 16, 16, 96, 32),
    (1, 128, 32, 16, 128, 64),
    (1, 32, 8, 16, 64, 64),      # y of 8
    (2, 8, 16, 8, 64, 32),       # x of 8
    (1, 16, 16, 16, 32, 96),     # two slices per item
    (4, 7, 32, 16, 64, 128),     # an odd number of planes
]


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("case", CONV)
def test_conv_runs_match_torch(gpu, case, f32):
    torch = pytest.importorskip("torch")
    F = torch.nn.functional
    conv, halo = conv_fns(gpu)
    k = Kernels(gpu.dll)
    B, D, H, W, cin, cout = case
    g = torch.Generator(device="cuda").manual_seed(sum(case))
    x = torch.randn(B, cin, D, H, W, device="cuda", generator=g).to(torch.bfloat16).float()
    wt = (torch.randn(cout, cin, 3, 3, 3, device="cuda", generator=g) / (27 * cin) ** 0.5).to(torch.bfloat16).float()
    bias = torch.randn(cout, device="cuda", generator=g) * 0.1
    st = torch.cuda.current_stream().cuda_stream
    xin = to_padded(torch, x, cin, 0)
    assert halo(xin.data_ptr(), B, D, H, W, cin, 0, cin, st) == 0
    w = gemm_weights(torch, wt)
    out = torch.full((B, D + 2, H + 2, W + 2, cout + 8), 7.0, device="cuda", dtype=torch.float32 if f32 else torch.bfloat16)
    if f32:
        k.tc_conv3d_f32(xin.data_ptr(), B, D, H, W, cin, 0, cin, w.data_ptr(), bias.data_ptr(), cout, out.data_ptr(),
                        cout + 8, 8, st)
    else:
        assert conv(xin.data_ptr(), B, D, H, W, cin, 0, cin, w.data_ptr(), bias.data_ptr(), cout, out.data_ptr(),
                    cout + 8, 8, 0, None, st) == 0
    assert gpu.dll.slbc_tc_status() == 0
    ref = F.conv3d(F.pad(x, (1, 1, 1, 1, 1, 1), mode="circular"), wt, bias)
    got = out[:, 1:-1, 1:-1, 1:-1, 8:].float().permute(0, 4, 1, 2, 3)
    assert ((got - ref).abs() <= 4e-3 * ref.abs() + 2e-3 * ref.abs().max().item()).all()
    out[:, 1:-1, 1:-1, 1:-1, 8:] = 7.0
    assert (out == 7.0).all()   # nothing else was written

"""Glue kernels of the warm-start network on grids whose rows are shorter and
longer than a block's reach, against PyTorch on the same BF16 values.

Pooling, upsampling and the encoding's distances are exact (sums of eight BF16
values times 1/8 in FP32, rounded once; copies; integers), so equal bits; the
bias gradient sums in FP32 in another order than the FP64 reference: each of
its at most N terms adds at most 2^-24 of the partial sums, bounded by
N^(1/2) 2^-23 of the sum of magnitudes.
"""

import numpy as np
import pytest

from sunlightlb_gb300.warmstart import Kernels

pytestmark = pytest.mark.gpu

SHAPES = [  # B, D, H, W, C, channels of the buffer, offset
    (1, 2, 2, 2, 8, 8, 0),
    (2, 4, 6, 10, 24, 40, 8),
    (1, 4, 4, 130, 32, 32, 0),
    (3, 2, 4, 6, 256, 256, 0),
]


def padded(torch, x, ctot, coff):
    B, D, H, W, C = x.shape
    buf = torch.zeros(B, D + 2, H + 2, W + 2, ctot, device="cuda", dtype=torch.bfloat16)
    buf[:, 1:-1, 1:-1, 1:-1, coff:coff + C] = x
    return buf


@pytest.mark.parametrize("case", SHAPES)
def test_pool_up_and_bias(gpu, case):
    torch = pytest.importorskip("torch")
    k = Kernels(gpu.dll)
    B, D, H, W, C, ctot, coff = case
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(sum(case))
    fine = torch.randn(B, D, H, W, C, device="cuda", generator=g).to(torch.bfloat16)
    src = padded(torch, fine, ctot, coff)
    out = torch.zeros(B, D // 2 + 2, H // 2 + 2, W // 2 + 2, C, device="cuda", dtype=torch.bfloat16)
    k.nn_pool(src.data_ptr(), ctot, coff, out.data_ptr(), C, 0, B, D, H, W, C, st)
    acc = torch.zeros(B, D // 2, H // 2, W // 2, C, device="cuda")
    for c in range(8):
        acc += fine[:, c >> 2::2, (c >> 1) & 1::2, c & 1::2].float()
    assert torch.equal(out[:, 1:-1, 1:-1, 1:-1], (acc * 0.125).to(torch.bfloat16))

    coarse = torch.randn(B, D // 2, H // 2, W // 2, C, device="cuda", generator=g).to(torch.bfloat16)
    csrc = padded(torch, coarse, C, 0)
    up = padded(torch, fine, ctot, coff)
    k.nn_up(csrc.data_ptr(), C, 0, up.data_ptr(), ctot, coff, B, D, H, W, C, st)
    want = coarse.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)
    assert torch.equal(up[:, 1:-1, 1:-1, 1:-1, coff:coff + C], want)

    back = torch.zeros_like(csrc)
    k.nn_up_bwd(src.data_ptr(), ctot, coff, back.data_ptr(), C, 0, csrc.data_ptr(), C, 0, B, D, H, W, C, st)
    assert torch.equal(back[:, 1:-1, 1:-1, 1:-1], torch.where(coarse > 0, acc, torch.zeros_like(acc)).to(torch.bfloat16))

    gf = torch.zeros(B, D + 2, H + 2, W + 2, C, device="cuda", dtype=torch.bfloat16)
    k.nn_pool_bwd(csrc.data_ptr(), C, 0, gf.data_ptr(), C, 0, src.data_ptr(), ctot, coff, src.data_ptr(), ctot, coff, B,
                  D, H, W, C, st)
    v = want.float() * 0.125 + fine.float()
    assert torch.equal(gf[:, 1:-1, 1:-1, 1:-1], torch.where(fine > 0, v, torch.zeros_like(v)).to(torch.bfloat16))

    if 256 % (C // 8) == 0:
        db = torch.zeros(C, device="cuda")
        k.nn_bias_grad(src.data_ptr(), ctot, coff, B, D, H, W, C, db.data_ptr(), st)
        ref = fine.double().sum(dim=(0, 1, 2, 3))
        bound = (B * D * H * W) ** 0.5 * 2.0 ** -23 * fine.double().abs().sum(dim=(0, 1, 2, 3))
        assert ((db.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("shape", [(1, 3, 5, 7), (2, 16, 16, 20), (1, 4, 30, 300)])
@pytest.mark.parametrize("features", [1, 2])
def test_encoding_distances(gpu, shape, features):
    torch = pytest.importorskip("torch")
    k = Kernels(gpu.dll)
    B, D, H, W = shape
    R = 5 if features == 1 else 12
    rng = np.random.default_rng(sum(shape))
    solid = rng.random(shape) < 0.01
    solid[0, 0, 0, 0] = True
    d2 = np.full(shape, R * R)
    for dz in range(-R, R + 1):
        for dy in range(-R, R + 1):
            for dx in range(-R, R + 1):
                r = dx * dx + dy * dy + dz * dz
                if r < R * R:
                    d2 = np.where(np.roll(solid, (dz, dy, dx), (1, 2, 3)), np.minimum(d2, r), d2)
    out = torch.full((B, D + 2, H + 2, W + 2, 16), 7.0, device="cuda", dtype=torch.bfloat16)
    dev = torch.as_tensor(solid.astype(np.uint8), device="cuda")
    k.nn_encode(dev.data_ptr(), B, D, H, W, out.data_ptr(), 16, features, torch.cuda.current_stream().cuda_stream)
    got = out[:, 1:-1, 1:-1, 1:-1].float()
    s = torch.as_tensor(solid, device="cuda")
    dist = torch.sqrt(torch.as_tensor(d2, device="cuda").float())
    d = torch.where(s, torch.zeros_like(dist), dist * torch.tensor(1.0 / R, device="cuda"))
    assert torch.equal(got[..., 0], s.float())
    # the FP32 products before the BF16 rounding may differ in their last bit
    assert ((got[..., 1] - d).abs() <= 2.0 ** -8 * d).all()
    assert ((got[..., 2] - d * d).abs() <= 2.0 ** -8 * d * d).all()
    assert (got[..., 4:] == 0).all()
    # the squared distances themselves, recovered exactly: neighbouring squares are more than a BF16 step apart below 36
    near = (torch.as_tensor(d2, device="cuda") < 25) & ~s
    assert torch.equal(torch.round((got[..., 1][near] * R) ** 2), torch.as_tensor(d2, device="cuda").float()[near])

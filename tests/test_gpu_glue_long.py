"""Glue kernels of the warm-start network on grids of few long rows, which are cut
into pieces for the blocks: pooling, upsampling and distances as in
test_gpu_glue_rows.py, the loss and the decoded fields against PyTorch.

The loss is an FP64 sum of at most N terms in another order, 1e-12 of it; its BF16
gradient is the FP32 product 2 / count * d, rounded: one BF16 step, 2^-7.
"""

import pytest

import test_gpu_glue_rows
from sunlightlb_gb300.warmstart import Kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [(1, 2, 2, 3000, 64, 64, 0), (2, 2, 2, 20000, 8, 24, 8), (1, 4, 2, 1026, 256, 256, 0)])
def test_pool_and_up(gpu, case):
    test_gpu_glue_rows.test_pool_up_and_bias(gpu, case)


@pytest.mark.parametrize("features", [1, 2])
@pytest.mark.parametrize("shape", [(1, 2, 3, 4000), (1, 1, 1, 1537)])
def test_encoding(gpu, shape, features):
    test_gpu_glue_rows.test_encoding_distances(gpu, shape, features)


@pytest.mark.parametrize("shape", [(1, 1, 1, 70001), (2, 2, 3, 5000), (1, 40, 70, 600), (3, 5, 6, 7)])
def test_loss_and_decoded_fields(gpu, shape):
    torch = pytest.importorskip("torch")
    k = Kernels(gpu.dll)
    B, D, H, W = shape
    st = torch.cuda.current_stream().cuda_stream
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    pred = torch.randn(B, D + 2, H + 2, W + 2, 8, device="cuda", generator=g)
    label = torch.randn(B, D, H, W, 4, device="cuda", generator=g)
    weight = torch.rand(B, device="cuda", generator=g)
    grad = torch.full((B, D + 2, H + 2, W + 2, 16), 7.0, device="cuda", dtype=torch.bfloat16)
    loss = torch.zeros(1, device="cuda", dtype=torch.float64)
    k.nn_mse(pred.data_ptr(), 8, label.data_ptr(), 4, weight.data_ptr(), B, D, H, W, grad.data_ptr(), 16, loss.data_ptr(), st)
    d = pred[:, 1:-1, 1:-1, 1:-1, :4] - label
    count = 4.0 * B * D * H * W
    want = float((weight.double().view(-1, 1, 1, 1, 1) * d.double() * d.double()).sum() / count)
    assert abs(float(loss) - want) <= 1e-12 * want
    inner = grad[:, 1:-1, 1:-1, 1:-1]
    ref = 2.0 / count * weight.view(-1, 1, 1, 1, 1) * d
    assert ((inner[..., :4].float() - ref).abs() <= 2.0 ** -7 * ref.abs()).all()
    assert not inner[..., 4:].any()

    solid = (torch.rand(D, H, W, device="cuda", generator=g) < 0.3).to(torch.uint8)
    u = torch.full((3, D, H, W), 7.0, device="cuda")
    drho = torch.full((D, H, W), 7.0, device="cuda")
    k.nn_decode(pred.data_ptr(), 8, solid.data_ptr(), D, H, W, 0.5, 0.25, u.data_ptr(), 2.0, drho.data_ptr(), st)
    v = pred[0, 1:-1, 1:-1, 1:-1].permute(3, 0, 1, 2)
    fluid = solid == 0
    for c in range(3):
        assert torch.equal(u[c], torch.where(fluid, 0.5 * v[c] - (0.25 if c == 0 else 0.0), torch.zeros_like(v[c])))
    assert torch.equal(drho, torch.where(fluid, 2.0 * v[3], torch.zeros_like(v[3])))

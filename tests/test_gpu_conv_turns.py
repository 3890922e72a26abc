"""Convolutions on grids 8 high (y), whose tiles go two slices at a time: more
tiles than twice the SMs, so that a block uses its accumulator sets and its ring
of stages again and walks over several tiles; one tile more than one and two
turns; every width, several channel chunks, batches.

Against PyTorch in FP32 on BF16-rounded inputs; tolerance as in
test_gpu_tc.py: the result is off by its BF16 rounding (2^-9) and the FP32
accumulation.
"""

import pytest

import test_gpu_conv_runs

pytestmark = pytest.mark.gpu

CONV = [  # B, D, H, W, cin, cout; tiles of 16 x 8 x 2
    (1, 64, 8, 256, 32, 32),    # 512 tiles
    (1, 64, 8, 256, 64, 64),    # 512: up to four turns of a block
    (1, 64, 8, 256, 64, 128),
    (1, 64, 8, 256, 96, 32),    # three chunks
    (5, 32, 8, 64, 32, 64),     # 320 tiles over the samples of a batch
    (1, 38, 8, 128, 32, 128),   # 152: one turn
    (9, 34, 8, 16, 32, 32),     # 153: one tile more
    (1, 76, 8, 128, 64, 128),   # 304: two turns
    (5, 122, 8, 16, 64, 64),    # 305
    (1, 2, 8, 8192, 32, 64),    # 512 along x
]


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("case", CONV)
def test_tiles_eight_high_match_torch(gpu, case, f32):
    test_gpu_conv_runs.test_conv_runs_match_torch(gpu, case, f32)

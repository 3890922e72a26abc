"""Weight gradients of layers whose input channels (above 256) split evenly into
blocks of 16 but not at once of 32, as in a network whose coarsest level is much
wider than the next: the bits of the channel-major form, and the gradients of
such a network against the CPU oracle.
"""

import pytest

import test_gpu_warm
import test_gpu_wgrad_flat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [(1, 4, 4, 8, 288, 32, 3), (1, 2, 4, 6, 416, 64, 2), (2, 2, 2, 8, 288, 128, 2)])
def test_same_bits_as_channel_major(gpu, case):
    test_gpu_wgrad_flat.test_same_bits_as_channel_major(gpu, case)


def test_network_with_one_wide_level(gpu):
    test_gpu_warm.test_unet_gradients_match_cpu_oracle(gpu, 4, (32, 32, 32, 256), 1)

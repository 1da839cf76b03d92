"""Weight gradients whose CTAs take their tiles in several sums (accumulators that are added to dW, zeroed
and restarted, with the ring of stages going on), against FP64."""
import pytest

from test_conv_plans import SUMS, sums
from test_gpu_conv import _torch
from test_gpu_wgrad_tiles import test_wgrad_tile_edges as against_fp64

pytestmark = pytest.mark.gpu


# Layers of so many groups of pairs that fewer than 34 CTAs share the pixels, and at least 136 tiles of
# 32 x 4: 224 x 96 as the denoiser's training has it (256 tiles), and 256 x 128 with tiles that neither the
# CTAs nor the sums divide (3 x 3 x 17 = 153, of single rows and columns at the edges).
@pytest.mark.parametrize("B,H,W,cin,cout", SUMS)
@pytest.mark.parametrize("skip", [0, 1])
def test_several_sums(B, H, W, cin, cout, skip):
    """An FP32 sum of up to 2^15 products of unit variance is off by at most 2^-24 x 2^15 = 2e-3 of its rms
    in the worst order; the tiles' MMAs sum 16 products at a time, 2^11 steps: 1.3e-4, below the 1e-3."""
    assert sums(B, H, W, cin, cout, _torch().cuda.get_device_properties(0).multi_processor_count) >= 2
    against_fp64(B, H, W, cin, cout, skip)

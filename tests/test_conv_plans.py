"""Which kernel and how many partial sums the convolutions' plans choose, on the host: the shapes by which the
GPU tests reach the row tiles and the weight gradient's restarted sums."""
import pytest

from gknextengine_gb300 import native

# B, H, W, cin, cout, flags, n_store, extras: three chunks through the ring, pooled rows with the sums by chunk,
# FP32 in groups of 16 columns with a ragged store, two chunks that stay, 16-column groups with two chunks
ROWS = [(80, 31, 128, 96, 32, 1, 0, False), (48, 32, 255, 32, 32, 0, 0, True), (80, 31, 128, 32, 16, 2, 3, False),
        (48, 29, 250, 64, 64, 0, 0, False), (64, 33, 129, 64, 48, 1, 0, True), (80, 29, 127, 160, 16, 0, 0, False)]
SUMS = [(8, 64, 64, 224, 96), (3, 65, 65, 256, 128), (1, 541, 33, 256, 128)]


def row_tiles(B, H, W, cin, cout, extras, sms=152):
    return native.load().gkrt_internal_conv_row_tiles(B, H, W, cin, cout, int(extras), sms)


def sums(B, H, W, cin, cout, sms=152):
    return native.load().gkrt_internal_wgrad_sums(B, H, W, cin, cout, sms)


@pytest.mark.parametrize("B,H,W,cin,cout,flags,n_store,extras", ROWS)
def test_batches_take_row_tiles_and_single_images_do_not(gkrt_lib, B, H, W, cin, cout, flags, n_store, extras):
    assert row_tiles(B, H, W, cin, cout, extras) >= B * H // 3 * (W // 128)
    assert row_tiles(1, min(H, 60), W, cin, cout, extras) == 0


@pytest.mark.parametrize("shape", SUMS)
def test_several_sums(gkrt_lib, shape):
    assert sums(*shape) >= 2
    assert sums(1, 64, 64, *shape[3:]) == 1     # 32 tiles

"""Row-tile convolutions of further shapes against the 16 x 8- and 16 x 16-tile ones, and what a NaN
becomes; the plan's answer on this device says that the row tiles ran."""
import pytest

from test_conv_plans import ROWS, row_tiles
from test_gpu_conv import _torch
from test_gpu_conv_rows import run, test_rows_equal_tiles as rows_equal_tiles

pytestmark = pytest.mark.gpu


def sms():
    return _torch().cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("B,H,W,cin,cout,flags,n_store,extras", ROWS)
def test_rows(B, H, W, cin, cout, flags, n_store, extras):
    assert row_tiles(B, H, W, cin, cout, extras, sms()) > 0
    assert row_tiles(1, min(H, 60), W, cin, cout, extras, sms()) == 0
    rows_equal_tiles(B, H, W, cin, cout, flags, n_store, extras)


# row tiles (80 images), 16 x 16 tiles (layers whose weights do not fit beside a row tile) and 8 x 16 ones
@pytest.mark.parametrize("B,H,W,cin,cout", [(80, 29, 250, 64, 64), (2, 40, 45, 160, 64), (1, 9, 17, 32, 32)])
@pytest.mark.parametrize("extras", [False, True])
def test_relu_of_nan_is_zero(B, H, W, cin, cout, extras):
    """As max(x, 0) of every kernel: a pixel whose window holds a NaN is 0, in all channels; all others are as
    without it."""
    torch = _torch()
    H, W = H + H % 2, W + W % 2
    g = torch.Generator(device="cuda").manual_seed(B + cin)
    x = torch.randn((B, H, W, cin), device="cuda", generator=g).bfloat16()
    w = (torch.randn((cout, 3, 3, cin), device="cuda", generator=g) / (3 * cin ** 0.5)).bfloat16()
    bias = torch.randn(cout, device="cuda", generator=g) * 0.1
    clean = run(x, w, bias, 1, extras=extras)[0]
    y0, x0 = H // 2, W // 2
    x[B - 1, y0, x0, 5] = float("nan")
    out = run(x, w, bias, 1, extras=extras)
    window = (slice(y0 - 1, y0 + 2), slice(x0 - 1, x0 + 2))
    clean[B - 1][window][..., 16:16 + cout] = 0
    assert torch.equal(out[0], clean)
    if extras:   # averages and copies of the stored values
        inner = out[0][..., 16:16 + cout]
        up = inner.repeat_interleave(2, 1).repeat_interleave(2, 2)
        assert torch.equal(out[2][..., 8:8 + cout], up)
        f = inner.float()
        pool = (((f[:, 0::2, 0::2] + f[:, 0::2, 1::2]) + f[:, 1::2, 0::2]) + f[:, 1::2, 1::2]) * 0.25
        assert torch.equal(out[1][..., 16:16 + cout], pool.bfloat16())

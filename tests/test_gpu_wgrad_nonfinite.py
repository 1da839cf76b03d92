"""The weight gradient of infinite inputs: a tap's sum takes a pixel's products only where the tap and the
pixel both lie in the image, so one infinite value leaves the other taps finite. (TMA's zeros beside the
image are the horizontal padding: an infinity next to its left or right end is not covered.)"""
import ctypes as C

import pytest

from gknextengine_gb300 import abi, native
from test_gpu_conv import _torch

pytestmark = pytest.mark.gpu


def reference(x, dy):
    """Every tap's sum over the pixels that have it, in FP64."""
    torch = _torch()
    H, W = x.shape[1:3]
    x, dy = x.double(), dy.double()
    dw = torch.zeros((dy.shape[3], 3, 3, x.shape[3]), dtype=torch.float64, device=x.device)
    for ky in range(3):
        for kx in range(3):
            y0, y1, x0, x1 = max(0, 1 - ky), min(H, H + 1 - ky), max(0, 1 - kx), min(W, W + 1 - kx)
            if y0 >= y1 or x0 >= x1:
                continue
            p = dy[:, y0:y1, x0:x1].reshape(-1, dy.shape[3])
            q = x[:, y0 + ky - 1:y1 + ky - 1, x0 + kx - 1:x1 + kx - 1].reshape(-1, x.shape[3])
            dw[:, ky, kx] = (p[:, :, None] * q[:, None, :]).sum(0)
    return dw


# one row, one past and one short of a tile's four, two tiles; several images, channel groups and pairs
@pytest.mark.parametrize("B,H,W,cin,cout", [(1, 1, 32, 32, 32), (1, 2, 40, 32, 64), (2, 3, 33, 48, 40),
                                            (1, 4, 32, 96, 32), (2, 5, 64, 64, 64), (1, 8, 32, 16, 8)])
@pytest.mark.parametrize("last", [False, True])
@pytest.mark.parametrize("where", ["x", "dy"])
def test_infinite_value_in_an_outer_row(B, H, W, cin, cout, last, where):
    torch = _torch()
    g = torch.Generator(device="cuda").manual_seed(H + cin)
    x = torch.randn((B, H, W, cin), device="cuda", generator=g).bfloat16()
    dy = torch.randn((B, H, W, cout), device="cuda", generator=g).bfloat16()
    (x if where == "x" else dy)[B - 1, H - 1 if last else 0, 5, 3] = float("inf")
    dw = torch.zeros((cout, 3, 3, cin), device="cuda")
    rc = native.load().gkrt_conv3x3_wgrad_bf16(C.c_void_p(dy.data_ptr()), C.c_void_p(x.data_ptr()), B, H, W, cin, cout,
                                               C.c_void_p(dw.data_ptr()), None)
    assert rc == abi.GKRT_OK
    torch.cuda.synchronize()
    ref = reference(x, dy)
    finite = torch.isfinite(ref)
    assert torch.equal(dw[~finite].double(), ref[~finite])
    # FP32 sums of at most 640 products of unit variance: off by at most 2^-24 x 640 of their rms
    torch.testing.assert_close(dw[finite].double(), ref[finite], rtol=1e-4, atol=1e-4 * float(ref[finite].abs().max()))

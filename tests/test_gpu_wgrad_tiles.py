"""The weight gradient at the edges of its tiles, boxes and blocks, against FP64."""
import ctypes as C

import pytest

from gknextengine_gb300 import abi, native
from test_gpu_conv import _torch

pytestmark = pytest.mark.gpu


# tiles of 32 pixels x 4 rows, boxes of 32 channels, blocks of four boxes: single pixels, one past and
# one short of a tile, channels that end inside a box, the smallest and the widest layers
@pytest.mark.parametrize("B,H,W", [(1, 1, 1), (1, 4, 32), (2, 5, 33), (1, 3, 31), (1, 131, 97)])
@pytest.mark.parametrize("cin,cout", [(16, 8), (32, 32), (48, 40), (64, 64), (96, 32), (256, 128)])
@pytest.mark.parametrize("skip", [0, 1])   # 16-byte additions to dw, or single ones
def test_wgrad_tile_edges(B, H, W, cin, cout, skip):
    """As test_wgrad_matches_torch, against the FP64 gradient; dw is added to. An FP32 sum of up to
    12,707 products of unit variance is off by at most 2^-24 x 12,707 of its rms, well below 1e-3."""
    torch = _torch()
    g = torch.Generator(device="cuda").manual_seed(cin + H)
    x = torch.randn((B, H, W, cin), device="cuda", generator=g).bfloat16()
    dy = torch.randn((B, H, W, cout), device="cuda", generator=g).bfloat16()
    dw = torch.ones(skip + cout * 9 * cin, device="cuda")[skip:].view(cout, 3, 3, cin)
    rc = native.load().gkrt_conv3x3_wgrad_bf16(C.c_void_p(dy.data_ptr()), C.c_void_p(x.data_ptr()), B, H, W, cin, cout,
                                               C.c_void_p(dw.data_ptr()), None)
    assert rc == abi.GKRT_OK
    torch.cuda.synchronize()
    ref = 1.0 + torch.nn.grad.conv2d_weight(x.double().permute(0, 3, 1, 2), (cout, cin, 3, 3),
                                            dy.double().permute(0, 3, 1, 2), padding=1).permute(0, 2, 3, 1)
    torch.testing.assert_close(dw.double(), ref, rtol=1e-3, atol=1e-3 * float(ref.abs().max()))

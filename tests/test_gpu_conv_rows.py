"""Row-tile convolutions against the 16 x 8-tile ones: both take an output's FP32 sums in the same order,
so a batch large enough for row tiles equals its images one at a time, bit for bit."""
import ctypes as C

import pytest

from gknextengine_gb300 import abi, native
from gknextengine_gb300.denoiser import Unet
from gknextengine_gb300.renderer import PathTracingRenderer
import test_gpu_conv as base
from test_gpu_conv import _torch

pytestmark = pytest.mark.gpu


def run(x, w, bias, flags, n_store=0, extras=False):
    torch = _torch()
    B, H, W, cin = x.shape
    cout = w.shape[0]
    f32 = bool(flags & 2)
    out = torch.full((B, H, W, n_store if f32 else cout + 32), 3.0, device="cuda",
                     dtype=torch.float32 if f32 else torch.bfloat16)
    res = [out]
    L = native.load()
    p = lambda t: C.c_void_p(t.data_ptr() if t is not None else 0)
    if extras:
        pool = torch.full((B, H // 2, W // 2, cout + 24), 5.0, device="cuda").bfloat16()
        up = torch.full((B, 2 * H, 2 * W, cout + 8), 6.0, device="cuda").bfloat16()
        rc = L.gkrt_conv3x3_bf16_fused(p(x), B, H, W, cin, p(w), p(bias), cout, p(out), cout + 32, 16, flags, p(pool),
                                       cout + 24, 16, p(up), cout + 8, 8, None)
        res += [pool, up]
    else:
        rc = L.gkrt_conv3x3_bf16(p(x), B, H, W, cin, p(w), p(bias), cout, p(out), out.shape[3], 0 if f32 else 16,
                                 n_store, flags, None)
    assert rc == abi.GKRT_OK, rc
    return res


# tiles of 128 x 2 or 3 pixels: one pixel short of, at and past an edge; rows that end inside a tile; one,
# two and three chunks; split output channels; every epilogue
@pytest.mark.parametrize("B,H,W,cin,cout,flags,n_store,extras", [
    (40, 31, 128, 32, 32, 1, 0, False), (24, 32, 255, 32, 32, 0, 0, True), (33, 35, 127, 32, 64, 1, 0, False),
    (24, 30, 257, 64, 64, 1, 0, True), (24, 29, 250, 64, 128, 0, 0, False), (40, 33, 125, 32, 128, 1, 0, True),
    (40, 31, 128, 96, 32, 1, 0, False), (24, 37, 256, 32, 96, 1, 0, True), (33, 31, 128, 32, 16, 2, 3, False),
    (40, 32, 127, 32, 48, 1, 0, False), (40, 35, 128, 64, 32, 3, 32, False), (2, 539, 120, 64, 64, 1, 0, True)])
def test_rows_equal_tiles(B, H, W, cin, cout, flags, n_store, extras):
    torch = _torch()
    g = torch.Generator(device="cuda").manual_seed(B + W + cin + cout)
    x = torch.randn((B, H, W, cin), device="cuda", generator=g).bfloat16()
    w = (torch.randn((cout, 3, 3, cin), device="cuda", generator=g) / (3 * cin ** 0.5)).bfloat16()
    bias = torch.randn(cout, device="cuda", generator=g) * 0.1 if flags & 1 else None
    batch = run(x, w, bias, flags, n_store, extras)
    for i in range(0, B, 7):
        # 60 rows at a time: few enough for the tiles, of which the inner ones see all their taps
        for y0 in range(0, H, 56):
            a, b = max(0, y0 - 2), min(H, y0 + 58)
            one = run(x[i:i + 1, a:b].contiguous(), w, bias, flags, n_store, extras)
            lo, hi = y0 - a, min(H, y0 + 56) - a
            for full, part, num, den in zip(batch, one, (1, 1, 2), (1, 2, 1)):
                s = slice(lo * num // den, hi * num // den)
                got = full[i, y0 * num // den:y0 * num // den + (s.stop - s.start)]
                assert torch.equal(got, part[0, s])


def test_unet_batch_equals_single_images():
    """The whole forward (the sub-pixel addend, the 16-channel input, FP32 outputs included)."""
    torch = _torch()
    B, H, W = 8, 136, 248
    with PathTracingRenderer(0) as r:
        net = Unet(r, seed=5)
        g = torch.Generator(device="cuda").manual_seed(6)
        x = torch.rand((B, H, W, 10), device="cuda", generator=g)
        raw = torch.zeros((B, H, W, 4), device="cuda")
        net.forward(x, out_raw=raw)
        for i in (0, B - 1):
            one = torch.zeros((1, H, W, 4), device="cuda")
            net.forward(x[i:i + 1].contiguous(), out_raw=one)
            assert torch.equal(raw[i], one[0])


# 16 x 16 tiles: one pixel short of, at and past an edge and a half; channels that end in half a stage;
# groups of 32 and of 16 output channels; two and three stages
@pytest.mark.parametrize("B,H,W,cin,cout", [(2, 15, 17, 96, 96), (1, 33, 31, 160, 64), (1, 9, 16, 224, 96),
                                            (3, 24, 48, 128, 128), (1, 17, 15, 160, 48), (1, 8, 8, 320, 80),
                                            (1, 1, 1, 96, 128), (2, 200, 130, 192, 64)])
def test_tiles_match_torch(B, H, W, cin, cout):
    """As the other convolutions' tests, with their tolerances."""
    base.test_conv_matches_torch(B, H, W, cin, cout, True)
    if H > 1:
        base.test_conv_fused_pool_and_upsample(B, H, W, cin, cout)


def test_chain_in_a_graph():
    """Kernels that start while their predecessors end, captured: a chain on one stream, replayed on new
    inputs, equals the same calls outside."""
    torch = _torch()
    L = native.load()
    g = torch.Generator(device="cuda").manual_seed(9)
    x = torch.randn((4, 100, 256, 64), device="cuda", generator=g).bfloat16()
    w = (torch.randn((64, 3, 3, 64), device="cuda", generator=g) / 24.0).bfloat16()
    w2 = (torch.randn((96, 3, 3, 64), device="cuda", generator=g) / 24.0).bfloat16()
    y, z, dw = torch.zeros_like(x), torch.zeros((4, 100, 256, 96), device="cuda").bfloat16(), torch.zeros((64, 3, 3, 64),
                                                                                                          device="cuda")

    def chain(stream):
        p = lambda t: C.c_void_p(t.data_ptr())
        st = C.c_void_p(stream.cuda_stream)
        for src, dst, k in ((x, y, w), (y, z, w2)):
            assert L.gkrt_conv3x3_bf16(p(src), 4, 100, 256, 64, p(k), None, dst.shape[3], p(dst), dst.shape[3], 0, 0, 1,
                                       st) == abi.GKRT_OK
        assert L.gkrt_conv3x3_wgrad_bf16(p(y), p(x), 4, 100, 256, 64, 64, p(dw), st) == abi.GKRT_OK

    chain(torch.cuda.current_stream())
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain(torch.cuda.current_stream())
    for _ in range(3):
        x.copy_(torch.randn(x.shape, device="cuda", generator=g))
        dw.zero_()
        graph.replay()
        torch.cuda.synchronize()
        got, got_dw = z.clone(), dw.clone()
        dw.zero_()
        chain(torch.cuda.current_stream())
        torch.cuda.synchronize()
        assert torch.equal(got, z)
        # FP32 sums over 102,400 pixels, added in any order
        torch.testing.assert_close(got_dw, dw, rtol=1e-3, atol=1e-3 * float(dw.abs().max()))

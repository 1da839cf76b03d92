"""Calls with scratch of their own, captured into a graph by a context's first such call, and replayed."""
import numpy as np
import pytest

from gknextengine_gb300 import abi, camera, scenes
from gknextengine_gb300.renderer import PathTracingRenderer
from test_gpu_parity import _torch

pytestmark = pytest.mark.gpu


def capture(torch, calls):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        calls(torch.cuda.current_stream())
    return graph


@pytest.mark.parametrize("W,H", [(96, 64), (700, 500)])   # pools of one warp's worth of paths, and larger ones
def test_adjoint(W, H):
    torch = _torch()
    sc, cam, st = scenes.cornell_materials(tiles=4)
    st.has_sky, st.sky_color = True, (0.4, 0.5, 0.6, 1.0)
    fc = camera.FrameBuilder(W, H, st).build(cam, 2)
    with PathTracingRenderer(0) as r:
        r.load_scene(sc)
        r.create_swap_chain(W, H)
        r.build_bvh()
        nm = r.material_count
        img = torch.zeros((H, W, 4), device="cuda")
        d = torch.randn((H, W, 4), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
        ga = torch.zeros((nm, 3), dtype=torch.float64, device="cuda")
        gr = torch.zeros((nm,), dtype=torch.float64, device="cuda")

        def calls(stream):
            r.adjoint_forward(fc, 2, img.data_ptr(), stream=stream)
            r.adjoint_backward(fc, 2, d.data_ptr(), ga.data_ptr(), gr.data_ptr(), stream=stream)

        r.synchronize()
        graph = capture(torch, calls)
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
        got = [t.clone() for t in (img, ga, gr)]
        img.zero_(), ga.zero_(), gr.zero_()
        calls(torch.cuda.current_stream())
        torch.cuda.synchronize()
        assert torch.equal(got[0], img)
        # the sums of three replays; FP64 additions in any order
        torch.testing.assert_close(got[1], 3.0 * ga, rtol=1e-9, atol=1e-9 * float(ga.abs().max()))
        torch.testing.assert_close(got[2], 3.0 * gr, rtol=1e-9, atol=1e-9 * float(gr.abs().max()))


def test_probe_bake():
    torch = _torch()
    sc, cam, st = scenes.cornell()
    st.has_sky, st.sky_color = True, (0.5, 0.7, 1.0, 1.0)
    fc = camera.FrameBuilder(64, 64, st).build(cam, 2)
    grids = []
    for captured in (True, False):
        with PathTracingRenderer(0) as r:
            r.load_scene(sc)
            r.create_swap_chain(64, 64)
            r.probe_voxelize()
            first = 1 * 192 * 192 + 64 * 192

            def calls(stream):
                r.probe_bake(fc, first, 64 * 192, stream=stream)

            r.synchronize()
            if captured:
                graph = capture(torch, calls)
            for _ in range(3):
                graph.replay() if captured else calls(torch.cuda.current_stream())
            torch.cuda.synchronize()
            grids.append(r.probe_download())
    assert grids[0][0].any()
    for a, b in zip(*grids):
        assert np.array_equal(a, b)

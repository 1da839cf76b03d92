"""The rt pass where one-warp pools end and where the larger pools' share of the pixels is rounded down,
against the oracle."""
import pytest

from gknextengine_gb300 import scenes
from gknextengine_gb300.renderer import PathTracingRenderer
from test_gpu_path_pools import _pass

pytestmark = pytest.mark.gpu


# on 152 SMs: 56 warps' worth of pixels per SM (272,384 = 532 x 512), one column more (a share of 112 pixels
# per warp, pools of 96), and the largest share below 128
@pytest.mark.parametrize("W,H", [(532, 512), (533, 512), (607, 512)])
def test_mid_frames(W, H):
    sc, cam, st = scenes.cornell()
    st.has_sun, st.sun_intensity, st.sun_direction = True, 2.0, (0.1, 0.5, 0.8)
    with PathTracingRenderer(0) as r:
        r.load_scene(sc)
        _pass(r, sc, cam, st, W, H)

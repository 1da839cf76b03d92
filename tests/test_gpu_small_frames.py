"""The rt pass on pools of one warp's worth of paths against the oracle: the largest frames that use them
and the smallest that do not, frames with fewer pixels than lanes, several samples per pixel."""
import pytest

from gknextengine_gb300 import abi, scenes
from gknextengine_gb300.renderer import PathTracingRenderer
from test_gpu_path_pools import _pass, test_adjoint_sizes as adjoint_sizes

pytestmark = pytest.mark.gpu


# 64 warps' worth of pixels per SM on 152 SMs: 311,296 pixels = 608 x 512
@pytest.mark.parametrize("W,H,samples,nee", [(608, 512, 1, abi.NEE_REFERENCE), (609, 512, 1, abi.NEE_REFERENCE),
                                             (130, 3, 8, abi.NEE_REFERENCE), (304, 128, 1, abi.NEE_REFERENCE),
                                             (305, 129, 1, abi.NEE_EMISSIVE), (255, 129, 4, abi.NEE_EMISSIVE),
                                             (456, 128, 2, abi.NEE_REFERENCE)])
def test_one_warp_pools(W, H, samples, nee):
    sc, cam, st = scenes.cornell()
    st.samples, st.nee_mode = samples, nee
    st.has_sun, st.sun_intensity, st.sun_direction = True, 2.0, (0.1, 0.5, 0.8)
    with PathTracingRenderer(0) as r:
        r.load_scene(sc)
        _pass(r, sc, cam, st, W, H)


# up to 16 warps' worth of pixels per SM, up to 48 and beyond (152 SMs: 77,824 and 233,472 pixels)
@pytest.mark.parametrize("W,H,spp,bounces", [(304, 255, 1, 2), (304, 257, 1, 2), (456, 513, 1, 2), (9, 31, 5, 4)])
def test_adjoint_one_warp_pools(W, H, spp, bounces):
    adjoint_sizes(W, H, spp, bounces, False)

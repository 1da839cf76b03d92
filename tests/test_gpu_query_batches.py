"""Ray queries at the batch sizes where the persistent kernel's shape changes (less than a warp's
lanes, one lane per warp, ragged last runs, several runs per warp), on buffers of any 4-byte
alignment and with the hits written over the rays: hits as the oracle's, exactly."""
import numpy as np
import pytest

from gknextengine_gb300 import abi, scenes
from gknextengine_gb300.renderer import PathTracingRenderer
from oracle import oracle as O
from test_gpu_parity import _torch, assert_hits_equal, random_rays

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    sc, _, _ = scenes.cornell()
    r = PathTracingRenderer(0)
    r.load_scene(sc)
    yield r, O.OracleScene(sc)
    r.close()


# 3040 warps: 1 lane each up to 3040 rays, 32 lanes from 97249, a second run from 97281
@pytest.mark.parametrize("n", [1, 5, 33, 3040, 3041, 20001, 97281, 200003])
@pytest.mark.parametrize("call", ["trace_rays_device", "trace_rays_noalloc_device"])
@pytest.mark.parametrize("shift,inplace", [(0, False), (4, False), (0, True)])
def test_batches(env, n, call, shift, inplace):
    torch = _torch()
    r, osc = env
    rays = random_rays(np.random.default_rng(n), n, (-0.6, -0.1, -0.6), (0.6, 1.1, 0.9))
    rays["tmin"] = np.where(np.arange(n) % 3 == 0, 0.2, 1e-3)
    rays["tmax"] = np.where(np.arange(n) % 5 == 0, 0.5, 1000.0)
    rb = torch.zeros(n * 32 + 16, dtype=torch.uint8, device="cuda")
    rb[shift:shift + 32 * n] = torch.from_numpy(rays.view(np.uint8).copy()).cuda()
    hb = rb if inplace else torch.full((n * 32 + 16,), 77, dtype=torch.uint8, device="cuda")
    getattr(r, call)(rb.data_ptr() + shift, hb.data_ptr() + shift, n, abi.TRACE_CLOSEST)
    r.synchronize()
    got = hb[shift:shift + 32 * n].cpu().numpy().view(abi.HIT_DTYPE)
    assert_hits_equal(got, osc.trace_rays(rays))
    assert not got["pad"].any()
    miss = got["inst"] == 0xFFFFFFFF
    assert (got["t"][miss] == -1).all() and (got["prim"][miss] == 0xFFFFFFFF).all()
    s = r.stats()
    assert s.rays_traced == n and s.device_error == 0 and s.hit_fetches == (~miss).sum()

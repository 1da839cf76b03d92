"""Rays whose direction is far from unit length (the caller's own units, or an instance scaled down by
many orders): hits as the oracle's, exactly, where products of FP32 values approach the largest one."""
import numpy as np
import pytest

from gknextengine_gb300 import abi, scenes
from gknextengine_gb300.renderer import PathTracingRenderer
from oracle import oracle as O
from test_gpu_parity import _torch, assert_hits_equal

pytestmark = pytest.mark.gpu


def triangles(z, e):
    """A triangle of size e at z, across the z axis, and a smaller one 1e13 behind it."""
    m = scenes.MeshBuilder()
    n = ((0, 0, -1),) * 3
    m.tri((-e, -e, z), (e, -e, z), (0, 2 * e, z), *n, 0)
    far = z + np.copysign(1e13, z)
    m.tri((-e / 64, -e / 64, far), (e / 64, -e / 64, far), (0, e / 32, far), *n, 0)
    pos, nrm, slot, idx, meshes = scenes._concat_meshes([m])
    return abi.SceneArrays(pos, nrm, slot, idx, meshes, np.array([scenes.lambertian((0.5, 0.5, 0.5))], abi.MATERIAL_DTYPE),
                           np.array([scenes.make_instance(0, scenes.trs(), [0], instance_id=0)], abi.INSTANCE_DTYPE))


# The determinant of the large triangle is 6 e^2 |d| (small one: / 4096): lengths |d| on both sides of
# where it passes 2^126 and the largest float.
@pytest.mark.parametrize("z,e,length", [(2e15, 1e10, 1e16), (2e15, 1e10, 1.3e17), (2e15, 1e10, 2e17), (2e15, 1e10, 4e17),
                                        (2e15, 1e10, 5e17), (2e15, 1e10, 2e18), (-2e15, 1e10, 2e17), (2e15, 1e9, 2e19)])
@pytest.mark.parametrize("call", ["trace_rays_device", "trace_rays_noalloc_device"])
def test_long_directions(z, e, length, call):
    torch = _torch()
    sc = triangles(z, e)
    n = 64
    rng = np.random.default_rng(5)
    rays = np.zeros(n, abi.RAY_DTYPE)
    rays["origin"][:, :2] = rng.uniform(-1.5 * e, 1.5 * e, (n, 2))
    rays["origin"][n // 2:, :2] /= 128.0
    rays["dir"][:, 2] = np.copysign(length, z)
    t = abs(z) / length
    rays["tmin"], rays["tmax"] = t / 1024, t * 1024
    rays["tmin"][::4] = t * (1.0 + 2e12 / abs(z))      # past the first triangle
    rb = torch.from_numpy(rays.view(np.uint8).copy()).cuda()
    hb = torch.empty(n * 32, dtype=torch.uint8, device="cuda")
    with PathTracingRenderer(0) as r:
        r.load_scene(sc)
        r.build_bvh()
        getattr(r, call)(rb.data_ptr(), hb.data_ptr(), n, abi.TRACE_CLOSEST)
        r.synchronize()
        assert r.stats().device_error == 0
    want = O.OracleScene(sc).trace_rays(rays)
    assert (want["inst"] == 0).sum() >= n // 2
    assert_hits_equal(hb.cpu().numpy().view(abi.HIT_DTYPE), want)

"""The rt pass's path pools against the oracle, at the frame sizes where a pool's shape changes: less
than a warp of pixels, ragged tiles, one warp's worth of paths per pool (32), two, and a full pool,
with closest-hit, sun and emitter rays mixed and several samples per pixel; and the four-child nodes
on single-leaf and two-leaf trees. Ids and radiance as in test_gpu_parity."""
import numpy as np
import pytest

from gknextengine_gb300 import abi, camera, scenes
from gknextengine_gb300.renderer import PathTracingRenderer
from oracle import oracle as O
from test_gpu_parity import _compare_trace_images

pytestmark = pytest.mark.gpu


def _pass(r, sc, cam, st, W, H):
    st.flags = abi.FRAME_PRIMARY_IDS
    r.create_swap_chain(W, H)
    fc = camera.FrameBuilder(W, H, st).build(cam, 3)
    r.trace_pass(fc)
    r.synchronize()
    oim = O.new_images(W, H)
    orays = O.OracleScene(sc).trace_pass(fc, W, H, oim)
    _compare_trace_images(r.images(), oim)
    assert r.stats().rays_traced == orays


# pixels per warp of the full grid (2432 or 3040 warps): < 1, 27, 34, 55, 105, 261
@pytest.mark.parametrize("W,H", [(1, 1), (7, 3), (33, 5), (129, 67), (257, 256), (383, 271), (512, 509), (1031, 771)])
@pytest.mark.parametrize("nee", [abi.NEE_REFERENCE, abi.NEE_EMISSIVE])
def test_frame_sizes(W, H, nee):
    sc, cam, st = scenes.cornell()
    st.samples = 3 if W < 200 else 1
    st.nee_mode = nee
    st.has_sky, st.sky_color = True, (0.4, 0.5, 0.6, 1.0)
    st.has_sun, st.sun_intensity, st.sun_direction = True, 2.0, (0.1, 0.5, 0.8)
    with PathTracingRenderer(0) as r:
        r.load_scene(sc)
        _pass(r, sc, cam, st, W, H)


@pytest.mark.parametrize("instances", [1, 2, 3])
@pytest.mark.parametrize("host", [False, True])
def test_shallow_trees(instances, host):
    """Meshes of one triangle (a root with one leaf) and of two, instance levels of one to three."""
    sc, cam, st = scenes.cornell()
    b = [scenes.MeshBuilder(), scenes.MeshBuilder()]
    b[0].tri((-0.5, 0, 0), (0.5, 0, 0), (0, 1, 0), (0, 0, 1), (0, 0, 1), (0, 0, 1), 0)
    b[1].quad((-0.5, 0, -0.2), (0.5, 0, -0.2), (0.5, 1, -0.3), (-0.5, 1, -0.3), (0, 0, 1), 0)
    pos, nrm, slot, idx, meshes = scenes._concat_meshes(b)
    inst = np.array([scenes.make_instance(k % 2, scenes.trs((0.3 * k - 0.3, 0.1 * k, 0.2 * k)), [k], k)
                     for k in range(instances)], dtype=abi.INSTANCE_DTYPE)
    sc = abi.SceneArrays(pos, nrm, slot, idx, meshes, sc.materials, inst, name="shallow")
    st.has_sky, st.sky_color = True, (0.4, 0.5, 0.6, 1.0)
    with PathTracingRenderer(0) as r:
        r.load_scene(sc)
        r.build_bvh(abi.BUILD_ALL | (abi.BUILD_ON_HOST if host else 0))
        _pass(r, sc, cam, st, 96, 64)


@pytest.mark.parametrize("offset,scale", [(0.0, 1.0), (1.0e3, 1.0), (0.0, 1e-3), (-2.0e4, 50.0)])
def test_far_and_scaled(offset, scale):
    """The four-child nodes' fused slabs and the edge-form triangle test far from the origin and at
    small and large scales (the camera moves along)."""
    sc, cam, st = scenes.cornell()
    inst = sc.instances.copy()
    for k in range(inst.shape[0]):
        w = np.eye(4)
        w[:3] = inst["world"][k].astype(np.float64).reshape(3, 4)
        m = np.diag([scale, scale, scale, 1.0])
        m[:3, 3] = offset
        w = (m @ w)[:3].reshape(-1).astype(np.float32)
        inst["world"][k] = w
        inst["world_inv"][k] = scenes.affine_inverse(w)
    sc = abi.SceneArrays(sc.positions, sc.normals, sc.material_slots, sc.indices, sc.meshes, sc.materials, inst,
                         lights=sc.lights, name="placed")
    cam = camera.Camera(eye=cam.eye * scale + offset, center=cam.center * scale + offset, fov_deg=cam.fov_deg)
    with PathTracingRenderer(0) as r:
        r.load_scene(sc)
        _pass(r, sc, cam, st, 160, 120)


# the adjoint's pools at the same edges; bounds of tests/test_gpu_adjoint.py
@pytest.mark.parametrize("W,H,spp,bounces", [(1, 1, 5, 16), (33, 5, 3, 16), (129, 67, 2, 1), (301, 203, 1, 4)])
@pytest.mark.parametrize("fast_gather", [False, True])
def test_adjoint_sizes(W, H, spp, bounces, fast_gather):
    import torch
    sc, cam, st = scenes.cornell_materials(tiles=4)
    st.bounces = st.max_bounces = bounces
    st.has_sky, st.sky_color, st.fast_gather = True, (0.4, 0.5, 0.6, 1.0), fast_gather
    fc = camera.FrameBuilder(W, H, st).build(cam, 2)
    dimg = np.zeros((H, W, 4), np.float32)
    dimg[..., :3] = np.random.default_rng(3).normal(size=(H, W, 3))
    with PathTracingRenderer(0) as r:
        r.load_scene(sc)
        r.create_swap_chain(W, H)
        nm = r.material_count
        streams = [torch.cuda.Stream() for _ in range(2)]
        img = [torch.empty((H, W, 4), device="cuda") for _ in streams]
        ga = [torch.zeros((nm, 3), dtype=torch.float64, device="cuda") for _ in streams]
        gr = [torch.zeros((nm,), dtype=torch.float64, device="cuda") for _ in streams]
        d = torch.as_tensor(dimg, device="cuda")
        torch.cuda.synchronize()
        for k, s in enumerate(streams):     # calls that may overlap
            r.adjoint_forward(fc, spp, img[k].data_ptr(), stream=s)
            r.adjoint_backward(fc, spp, d.data_ptr(), ga[k].data_ptr(), gr[k].data_ptr(), stream=s)
        torch.cuda.synchronize()
    o, oa, orr = O.OracleScene(sc).adjoint(fc, W, H, spp, dimage=dimg, window=(0, 0, W, H))
    for k in range(2):
        np.testing.assert_allclose(img[k].cpu().numpy(), o, rtol=1e-4, atol=1e-6)
        np.testing.assert_allclose(ga[k].cpu().numpy(), oa, rtol=1e-3, atol=1e-5 * max(np.abs(oa).max(), 1e-30))
        np.testing.assert_allclose(gr[k].cpu().numpy(), orr, rtol=1e-3, atol=1e-5 * max(np.abs(orr).max(), 1e-30))

"""One bake step at the batch sizes where the kernels' shapes change (a single probe, ragged groups,
one batch whose rays read the grid in place, one probe more than a batch, which reads a snapshot),
with and without the extra light and sun rays: the oracle's words, exactly."""
import numpy as np
import pytest

from gknextengine_gb300 import abi, camera
from gknextengine_gb300.renderer import PathTracingRenderer
from oracle import oracle as O
from test_gpu_probes import LAYER, XY, big_cornell

pytestmark = pytest.mark.gpu

FIRST = 3 * LAYER + 88 * XY + 77        # inside the room's rows, at an odd index


@pytest.mark.parametrize("light", [False, True])
@pytest.mark.parametrize("sun", [False, True])
def test_batch_sizes(light, sun):
    sc, cam, st = big_cornell()
    if not light:
        sc = abi.SceneArrays(sc.positions, sc.normals, sc.material_slots, sc.indices, sc.meshes, sc.materials,
                             sc.instances, name="no-light")
    st.has_sun = sun
    fc = camera.FrameBuilder(64, 64, st).build(cam, 0)
    osc = O.OracleScene(sc)
    with PathTracingRenderer(0) as r:
        r.load_scene(sc)
        r.probe_voxelize()
        for count in (1, 31, 257, 65536, 65537):
            prev, vox = r.probe_download()
            r.probe_bake(fc, FIRST, count)
            r.synchronize()
            cubes, vox2 = r.probe_download()
            o, ages = osc.probe_bake(fc, FIRST, count, prev, vox)
            assert np.array_equal(cubes[FIRST:FIRST + count], o), count
            assert np.array_equal(vox2[FIRST:FIRST + count, 1], ages)
            assert np.array_equal(cubes[:FIRST], prev[:FIRST])
            assert np.array_equal(cubes[FIRST + count:], prev[FIRST + count:])
        assert (cubes != 0).any() and r.stats().device_error == 0

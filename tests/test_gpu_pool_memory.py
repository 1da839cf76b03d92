"""Device memory that a renderer takes for its frame: the images, the a-trous passes' two, and the rt pass's
path pools for as many warps as can be resident."""
import pytest

from gknextengine_gb300 import abi
from gknextengine_gb300.renderer import PathTracingRenderer
from test_gpu_parity import _torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(1920, 1080), (3840, 2160), (512, 256)])
def test_frame_memory(W, H):
    torch = _torch()
    with PathTracingRenderer(0) as r:
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info(0)[0]
        r.create_swap_chain(W, H)
        torch.cuda.synchronize()
        used = before - torch.cuda.mem_get_info(0)[0]
        views = [r.image_view(i) for i in abi.IMAGE_FORMATS]
        images = sum(v.height * v.pitch_bytes for v in views) + 2 * W * H * 16
        # at most four blocks of four warps per SM: 256 paths of 15 16-byte fields and 8 for each lane's ray in
        # flight, or, for a frame of up to 56 warps' worth of pixels per SM, 32 paths; and 2 MiB pages
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        paths = 32 if W * H // sms <= 56 * 32 else 256
        pools = 16 * sms * (paths * 15 + (8 * 32 if paths > 32 else 0)) * 16
        assert images <= used <= images + pools + (len(views) + 3) * (2 << 20)

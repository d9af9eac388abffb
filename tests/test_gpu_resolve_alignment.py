"""The flat resolve, alone and with motion vectors, of a scene whose material
records lie at each address that their 4-byte fields allow: the same image."""
import numpy as np
import pytest
import torch

import gpu_util as U
from vk_gltf_viewer_gb300 import abi, scene
from vk_gltf_viewer_gb300.renderer import DeviceScene

pytestmark = pytest.mark.gpu

W, H = 173, 97


@pytest.mark.parametrize("views", [1, 3])
@pytest.mark.parametrize("flags", [abi.RESOLVE_FLAT, abi.RESOLVE_FLAT | abi.WRITE_MOTION, abi.WRITE_MOTION,
                                   abi.RESOLVE_TEXTURED | abi.WRITE_MOTION])
def test_materials_at_every_alignment(renderer, flags, views):
    host = U.small_grid()
    cam = scene.camera((4.0, 3.5, -3.0), (4.0, 1.0, 4.0), (0, 1, 0), 70.0, W / H)
    flags |= abi.CULL_FRUSTUM | abi.CULL_CONE | abi.WRITE_IDS

    def images(shift):
        dev = DeviceScene(host, "cuda")
        raw = dev.materials.reshape(-1).view(torch.uint8)
        buf = torch.zeros(raw.numel() + 32, dtype=torch.uint8, device="cuda")
        at = (shift - buf.data_ptr()) % 16
        buf[at:at + raw.numel()].copy_(raw)
        dev.scene.material_buffer = buf.data_ptr() + at
        vs = [U.ViewBuffers.allocate(W, H, cam, host.draw_count, motion=True) for _ in range(views)]
        renderer.frame(dev, vs, flags)
        torch.cuda.synchronize()
        return [t.cpu().numpy() for v in vs for t in (v.visbuffer, v.color, v.motion)]

    aligned = images(0)
    assert (aligned[0].view(np.uint32) != abi.VISBUFFER_CLEAR).any()
    if flags & abi.RESOLVE_FLAT:
        assert len(np.unique(aligned[1])) > 1
    for shift in (4, 8, 12):
        for a, b in zip(aligned, images(shift)):
            assert np.array_equal(a, b)

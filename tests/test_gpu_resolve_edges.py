"""The textured resolve where its loads and its texture addressing have two
forms: scene arrays at every alignment that the layout allows, and repeated
textures of odd sizes at coordinates inside, below and far outside [0, 1]."""
import numpy as np
import pytest
import torch

import gpu_util as U
from oracle import binding as ob
from vk_gltf_viewer_gb300 import abi, scene
from vk_gltf_viewer_gb300.renderer import DeviceScene

pytestmark = pytest.mark.gpu

W, H = 173, 97
FLAGS = (abi.CULL_FRUSTUM | abi.CULL_CONE | abi.RESOLVE_TEXTURED | abi.WRITE_IDS)
CAM = ((4.0, 3.5, -3.0), (4.0, 1.0, 4.0))


def _shifted(t: torch.Tensor, align: int, shift: int) -> torch.Tensor:
    """The tensor's bytes at an address of `shift` modulo `align`."""
    raw = t.reshape(-1).view(torch.uint8)
    buf = torch.zeros(raw.numel() + 2 * align, dtype=torch.uint8, device="cuda")
    at = (shift - buf.data_ptr()) % align
    out = buf[at:at + raw.numel()]
    out.copy_(raw)
    return out


def _frame(renderer, dev, host):
    cam = scene.camera(*CAM, (0, 1, 0), 70.0, W / H)
    v = U.ViewBuffers.allocate(W, H, cam, host.draw_count)
    renderer.frame(dev, [v], FLAGS)
    torch.cuda.synchronize()
    return U.u32(v.visbuffer), U.u32(v.color), np.sort(v.survivor_list())


def test_scene_arrays_at_their_least_alignment(renderer):
    host = U.small_grid()
    aligned = _frame(renderer, DeviceScene(host, "cuda"), host)
    dev = DeviceScene(host, "cuda")
    keep = []
    for name, shift in (("primitive_buffer", 8), ("material_buffer", 4), ("texture_table", 8)):
        src = {"primitive_buffer": dev.primitives, "material_buffer": dev.materials,
               "texture_table": dev.texture_table}[name]
        if name == "primitive_buffer":
            # the vertices and cones move too: 8-byte and 4-byte addresses
            p = src.cpu().numpy().view(np.uint64).reshape(-1, 8)
            for k in range(len(host.meshes)):
                raw = torch.from_numpy(host.meshes[k].vertices.view(np.uint8).reshape(-1).copy()).cuda()
                keep.append(_shifted(raw, 16, 8))
                p[k, 2] = keep[-1].data_ptr()
                raw = torch.from_numpy(host.meshes[k].cones.view(np.uint8).reshape(-1).copy()).cuda()
                keep.append(_shifted(raw, 16, 4))
                dev.cone_table.view(torch.int64)[k] = keep[-1].data_ptr()
            src = torch.from_numpy(p.reshape(-1).view(np.uint8).copy()).cuda()
        keep.append(_shifted(src, 16, shift))
        setattr(dev.scene, name, keep[-1].data_ptr())
    moved = _frame(renderer, dev, host)
    for a, b in zip(aligned, moved):
        assert np.array_equal(a, b)
    assert (aligned[0] != abi.VISBUFFER_CLEAR).any()


@pytest.mark.parametrize("size", [(1, 1), (3, 5), (8, 7), (1, 16)])
@pytest.mark.parametrize("offset,scale", [(0.0, 4.0), (-3.25, 2.5), (4000.0, -1.5), (1e9, 3.0), (-1e12, 1e8)])
def test_repeated_textures_match_oracle(renderer, size, offset, scale):
    host = U.small_grid()
    w, h = size
    rng = np.random.default_rng(w * 10 + h)
    host.textures = [scene.Texture(rng.integers(0, 256, size=(h, w, 4), dtype=np.uint8), abi.TEXTURE_RGBA8)]
    host.materials["uv_offset"][1] = (offset, 0.5 * offset)
    host.materials["uv_scale"][1] = (scale, 0.75 * scale)
    dev = DeviceScene(host, "cuda")
    ids, rgba, _ = _frame(renderer, dev, host)
    orc = ob.OracleScene(host)
    cam = scene.camera(*CAM, (0, 1, 0), 70.0, W / H)
    exp = ob.frame(orc, cam, W, H, U.oracle_flags(FLAGS))
    assert np.array_equal(ids, exp["ids"])
    close, off = U.rgba_close(rgba, exp["rgba"])
    assert close, f"{off} pixels differ"


@pytest.mark.parametrize("extra", [-1, 1])
def test_views_about_the_pixels_per_thread_line(renderer, extra):
    """A view just below and one just above the size from which a resolve
    thread takes four pixels."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    h = 1301
    w = 20 * 1024 * sms // h + extra
    assert (w * h >= 20 * 1024 * sms) == (extra > 0)
    host = U.small_grid()
    dev = DeviceScene(host, "cuda")
    cam = scene.camera(*CAM, (0, 1, 0), 70.0, w / h)
    v = U.ViewBuffers.allocate(w, h, cam, host.draw_count)
    renderer.frame(dev, [v], FLAGS)
    exp = ob.frame(ob.OracleScene(host), cam, w, h, U.oracle_flags(FLAGS))
    assert np.array_equal(U.u32(v.visbuffer), exp["ids"])
    close, off = U.rgba_close(U.u32(v.color), exp["rgba"])
    assert close, f"{off} pixels differ"

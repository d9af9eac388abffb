"""Triangles whose clip coordinates lie at the ends of the float range: w that
overflows to infinity, and w so small that its reciprocal does.  Such vertices
snap to no place and their triangles are not drawn, whichever way their meshlet
takes through the raster; the others have the oracle's bits."""
import numpy as np
import pytest
import torch

import gpu_util as U
from oracle import binding as ob
from vk_gltf_viewer_gb300 import scene

pytestmark = pytest.mark.gpu

W, H = 128, 96


@pytest.fixture(scope="module")
def triangles(built):
    """One triangle a meshlet, anywhere in the frustum at depths 0.3 to 8."""
    rng = np.random.default_rng(12)
    f = np.tan(np.radians(40.0))
    meshes = [scene.mesh_from_arrays(np.array([[0, 0, -2], [0.9, 0.2, -2], [-3.6, 3.5, -7]], np.float32),
                                     np.array([[0, 1, 2]]))]
    for _ in range(60):
        z = np.exp(rng.uniform(np.log(0.3), np.log(8.0), 3))
        p = np.stack([rng.uniform(-0.9, 0.9, 3) * f * W / H * z, rng.uniform(-0.9, 0.9, 3) * f * z, -z], 1)
        meshes.append(scene.mesh_from_arrays(p.astype(np.float32), np.array([[0, 1, 2]])))
    mats = np.concatenate([scene.make_material(double_sided=True), scene.default_material()])
    host = scene.HostScene(meshes=meshes, prim_materials=[int(k % 4 == 3) for k in range(len(meshes))], materials=mats,
                           transforms=np.stack([scene.to_column_major(scene.mat_scale(m.position_scale)) for m in meshes]),
                           node_meshes=[[k] for k in range(len(meshes))])
    return U.Pair(host)


@pytest.mark.parametrize("exponent", [127, 126, 125, 101, 100, 99, 0, -99, -100, -101, -126, -128, -129, -130, -140])
def test_view_projections_scaled_to_the_ends_of_the_range(renderer, triangles, exponent):
    cam = scene.camera((0.0, 0.0, 0.0), (0.0, 0.0, -1.0), (0.0, 1.0, 0.0), 80.0, W / H)
    with np.errstate(over="ignore"):
        vp = np.array(cam.view_projection, np.float32) * np.float32(2.0 ** exponent)
    cam.view_projection[:] = [float(x) for x in vp]
    every = np.arange(triangles.host.draw_count, dtype=np.uint32)
    exp = ob.raster(triangles.orc, cam, W, H, every)
    drawn = len(np.unique(exp.astype(np.uint32))) - 1
    if exponent in (127, 126, -128, -129):  # some have such a vertex, and some of the others are seen
        assert 5 < drawn < 45
    v = U.view(triangles, cam, W, H)
    renderer.clear(triangles.dev, v)
    lst = torch.from_numpy(every.view(np.int32)).cuda()
    cnt = torch.tensor([every.size], dtype=torch.int32, device="cuda")
    renderer.raster(triangles.dev, v, lst, cnt)
    got = U.u64(v.depth_id)
    assert np.array_equal(got, exp), f"{(got != exp).sum()} pixels differ"
    assert renderer.device_status() == (0, 0)

"""Triangles around the sizes at which their raster changes hands (drawn by
the meshlet's warp, queued as one rectangle, queued as several by the slow
instance), at every bin size, on and across the view's edges, and with a queue
that has room for one rectangle: the oracle's bits."""
import numpy as np
import pytest

import gpu_util as U
from oracle import binding as ob
from vk_gltf_viewer_gb300 import scene
from vk_gltf_viewer_gb300.renderer import Renderer

pytestmark = pytest.mark.gpu

W, H = 331, 257
SIZES = [3, 4, 7, 8, 9, 15, 16, 17, 31, 32, 33, 34, 62, 63, 64, 65, 66, 100]


@pytest.fixture(scope="module")
def patches(built):
    """Per size a fan of triangles about `size` pixels wide and of heights up
    to it, thin ones in both directions included, at sub-pixel offsets."""
    rng = np.random.default_rng(3)
    f = 1.0 / np.tan(np.radians(30.0))  # 60 degrees: at depth 1 a pixel is 2 / (f H)
    px = 2.0 / (f * H)
    meshes = []
    for size in SIZES:
        pos, idx = [], []
        for k in range(24):
            w, h = size + rng.uniform(-0.6, 0.6), (size, 1.2, size / 2)[k % 3] + rng.uniform(-0.6, 0.6)
            if k % 2:
                w, h = h, w
            x, y = rng.uniform(-0.52 * W, 0.52 * W), rng.uniform(-0.52 * H, 0.52 * H)
            z = rng.uniform(-0.05, 0.05)
            tri = [(x, y, z), (x + w, y + h * rng.uniform(0, 0.3), z), (x + w * rng.uniform(0, 1), y + h, z)]
            if k % 5 == 0:
                tri = tri[::-1]
            idx.append(len(pos) + np.arange(3))
            pos += [((a + 0.001 * c) * px, b * px, c) for a, b, c in tri]
        meshes.append(scene.mesh_from_arrays(np.array(pos, np.float32), np.array(idx)))
    mats = np.concatenate([scene.default_material(), scene.make_material(double_sided=True)])
    host = scene.HostScene(meshes=meshes, prim_materials=[k % 2 for k in range(len(meshes))], materials=mats,
                           transforms=np.stack([scene.to_column_major(scene.mat_scale(m.position_scale)) for m in meshes]),
                           node_meshes=[[k] for k in range(len(meshes))])
    return U.Pair(host)


@pytest.mark.parametrize("capacity", [0, 1, 40])
@pytest.mark.parametrize("bin_size", [8, 16, 32, 64])
def test_sizes_match_oracle(patches, bin_size, capacity):
    cam = scene.camera((0.0, 0.0, 1.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 60.0, W / H)
    r = Renderer(0, bin_size=bin_size, big_capacity=capacity)
    try:
        v = U.view(patches, cam, W, H)
        r.frame(patches.dev, [v], 0)
        exp = ob.frame(patches.orc, cam, W, H, 0)
        got = U.u64(v.depth_id)
        assert np.count_nonzero(exp["depth_id"]) > 20000
        assert np.array_equal(got, exp["depth_id"])
        code = r.device_status()[0]
        assert code == (2 if capacity else 0)  # a full queue draws in place and says so
    finally:
        r.close()

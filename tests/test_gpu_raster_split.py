"""The raster's split work list (the last meshlets of a launch are drawn one
32-triangle round a warp) and its test for meshlets inside the view volume:
list lengths around the split, meshlets of every number of rounds, views that
cut meshlets at the near plane, the guard band and the view edges, against the
oracle bit for bit."""
import numpy as np
import pytest
import torch

import gpu_util as U
from oracle import binding as ob
from vk_gltf_viewer_gb300 import scene

pytestmark = pytest.mark.gpu

W, H = 203, 117


def _strip(triangles):
    """A flat strip of `triangles` triangles: one meshlet (or a few past the
    limits) facing +z."""
    n = triangles + 2
    i = np.arange(n)
    pos = np.stack([0.02 * (i // 2), 0.05 * (i % 2), np.zeros(n)], 1).astype(np.float32)
    t = np.arange(triangles)
    idx = np.stack([t, np.where(t % 2, t + 2, t + 1), np.where(t % 2, t + 1, t + 2)], 1)
    return scene.mesh_from_arrays(pos, idx)


@pytest.fixture(scope="module")
def rounds(built):
    """Nodes of strips of 1 to 62 triangles, and grid patches up to 98
    triangles a meshlet, on a lattice."""
    meshes = [_strip(t) for t in (1, 31, 32, 33, 62)] + [scene.torus(seg_major=40, seg_minor=24)]
    nodes, xf = [], []
    for k in range(720):
        nodes.append([k % len(meshes)])
        s = meshes[k % len(meshes)].position_scale
        m = scene.mat_translate((1.3 * (k % 12) - 7.0, 1.1 * (k // 12 % 10) - 5.0, -0.4 * (k % 5) - 2.5 * (k // 120))) @ \
            scene.mat_rotate_y(0.2 * k) @ scene.mat_scale(s)
        xf.append(scene.to_column_major(m))
    mats = np.concatenate([scene.default_material(), scene.make_material(double_sided=True)])
    host = scene.HostScene(meshes=meshes, prim_materials=[1] * len(meshes), materials=mats, transforms=np.stack(xf),
                           node_meshes=nodes)
    return U.Pair(host)


# in front; among the nodes (near plane, view edges, guard band); close up
EYES = [(0.0, 0.0, 9.0), (-6.6, -4.9, 0.3), (0.3, 0.1, 0.55)]


@pytest.mark.parametrize("eye", EYES)
@pytest.mark.parametrize("count", [1, 7, 1063, 1064, 1065, 2700, None])
def test_split_lists_match_oracle(renderer, rounds, eye, count):
    draws = rounds.host.draw_count
    rng = np.random.default_rng(draws + (count or 0))
    lst = rng.permutation(draws).astype(np.uint32)[:count]
    cam = scene.camera(eye, (eye[0] + 0.2, eye[1] + 0.1, eye[2] - 3.0), (0.0, 1.0, 0.0), 70.0, W / H)
    v = U.view(rounds, cam, W, H)
    exp = ob.raster(rounds.orc, cam, W, H, lst)
    renderer.clear(rounds.dev, v)
    dev = torch.from_numpy(lst.view(np.int32).copy()).cuda()
    cnt = torch.tensor([lst.size], dtype=torch.int32, device="cuda")
    renderer.raster(rounds.dev, v, dev, cnt)
    torch.cuda.synchronize()
    assert np.array_equal(U.u64(v.depth_id), exp.reshape(-1))
    assert renderer.device_status() == (0, 0)


def test_list_covers_the_split(rounds):
    # longer than the split of any launch here, so both kinds of item occur
    assert rounds.host.draw_count > 2700
    counts = set(int(t) for m in rounds.host.meshes for t in m.meshlets["triangle_count"])
    assert {1, 31, 32, 33, 62} <= counts and max(counts) > 64

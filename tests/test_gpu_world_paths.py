"""Node transforms by one group of lanes per path and by one thread per node:
paths of 1 to 10 nodes, slot counts around a block's edge, nodes reached from
several roots, and trees large enough for the second form; every matrix has
the oracle's bits."""
import numpy as np
import pytest
import torch

from oracle import binding as ob
from vk_gltf_viewer_gb300 import abi
from vk_gltf_viewer_gb300.world import DeviceWorld, HostWorld, Sampler, make_nodes, quat_axis_angle

pytestmark = pytest.mark.gpu


def _forest(paths: int, depth: int, every: int, shared: bool) -> HostWorld:
    """`paths` chains of `depth` nodes, a mesh on each `every`-th node; with
    `shared` all chains end in one common last node."""
    n = paths * depth
    nodes = make_nodes(n)
    k = np.arange(n)
    inner = k % depth != depth - 1
    nodes["child_count"] = inner
    nodes["first_child"] = np.where(inner, k - k // depth, 0)
    children = (k[inner] + 1).astype(np.uint32)
    if shared and depth > 1:
        children[depth - 2:: depth - 1] = n - 1
    rng = np.random.default_rng(paths * 31 + depth)
    nodes["translation"] = rng.normal(size=(n, 3))
    q = rng.normal(size=(n, 4))
    nodes["rotation"] = q / np.linalg.norm(q, axis=1, keepdims=True)
    nodes["scale"] = rng.uniform(0.5, 1.5, (n, 3))
    nodes["mesh_index"] = np.where((k % depth) % every == every - 1, 0, abi.INVALID_HANDLE)
    samplers = [Sampler(np.array([0.0, 2.0], np.float32),
                        np.stack([quat_axis_angle((1, 0, 0), 0.1), quat_axis_angle((0, 1, 0), 1.5)]),
                        abi.INTERP_LINEAR),
                Sampler(np.array([0.0, 1.0], np.float32), np.array([[0, 0, 0], [1, 2, 3]], np.float32),
                        abi.INTERP_LINEAR)]
    moved = k[::3]
    channels = np.stack([moved % 2, moved, np.where(moved % 2, abi.PATH_TRANSLATION, abi.PATH_ROTATION),
                         np.zeros_like(moved)], 1)
    return HostWorld(nodes=nodes, children=children, roots=k[::depth].astype(np.uint32), mesh_primitives=[[0]],
                     primitive_meshlet_counts=np.array([1], np.uint32), samplers=samplers, channels=channels)


@pytest.mark.parametrize("paths,depth,every,shared",
                         [(1, 1, 1, False), (129, 1, 1, False), (64, 2, 2, False), (65, 2, 1, True), (31, 3, 1, False),
                          (33, 4, 2, True), (17, 5, 1, False), (16, 8, 1, False), (33, 8, 8, False), (3, 9, 1, False),
                          (40, 10, 3, True), (4097, 4, 1, False), (8193, 4, 1, True), (3000, 6, 1, False),
                          (70000, 2, 2, False), (70000, 2, 1, False)])
def test_transforms_by_path_length(renderer, paths, depth, every, shared):
    host = _forest(paths, depth, every, shared)
    dw = DeviceWorld(renderer, host)
    try:
        for time in (0.0, 0.7, 5.0):
            # room behind the last slot shows a store past it
            out = torch.full((dw.transform_count * 16 + 64,), float("nan"), device="cuda")
            dw.update_transforms(time, out)
            got = out.cpu().numpy()
            exp = ob.world_transforms(host, time)
            assert np.array_equal(got[:-64].view(np.uint32), exp.reshape(-1).view(np.uint32))
            assert np.isnan(got[-64:]).all()
        assert renderer.device_status() == (0, 0)
    finally:
        dw.close()

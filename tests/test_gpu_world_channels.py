"""Node trees whose shared nodes have many channels: one launch that samples a
path's channels again for every slot below them up to its line, a launch of one
thread per node past it, and the oracle's bits on both sides."""
import numpy as np
import pytest
import torch

from graph_util import captured_kernels
from oracle import binding as ob
from vk_gltf_viewer_gb300 import abi
from vk_gltf_viewer_gb300.world import DeviceWorld, HostWorld, Sampler, make_nodes

pytestmark = pytest.mark.gpu


def _star(leaves: int, root_channels: int, leaf_channels: int) -> HostWorld:
    """A root with `root_channels` channels over `leaves` meshes."""
    n = 1 + leaves
    rng = np.random.default_rng(leaves)
    nodes = make_nodes(n)
    nodes["translation"] = rng.normal(size=(n, 3))
    nodes["mesh_index"][1:] = 0
    nodes["child_count"][0] = leaves
    times = np.array([0.0, 0.5, 2.0], np.float32)
    q = rng.normal(size=(3, 4))
    samplers = [Sampler(times, (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32), abi.INTERP_LINEAR),
                Sampler(times, rng.normal(size=(3, 3)).astype(np.float32), abi.INTERP_LINEAR)]
    channels = [(k % 2, 0, abi.PATH_TRANSLATION if k % 2 else abi.PATH_ROTATION, 0) for k in range(root_channels)]
    channels += [(k % 2, 1 + i, abi.PATH_SCALE if k % 2 else abi.PATH_ROTATION, 0)
                 for i in range(leaves) for k in range(leaf_channels)]
    return HostWorld(nodes=nodes, children=np.arange(1, n, dtype=np.uint32), roots=np.array([0], np.uint32),
                     mesh_primitives=[[0]], primitive_meshlet_counts=np.array([1], np.uint32), samplers=samplers,
                     channels=np.asarray(channels, np.uint32))


# the root's channels are sampled again leaves - 1 times; its leaves' are not
@pytest.mark.parametrize("leaves,root,leaf,one", [(1025, 192, 0, True), (1026, 192, 0, False), (1025, 192, 5, True),
                                                  (2000, 500, 1, False), (1, 300, 2, True), (3, 70000, 0, True)])
def test_shared_channels(renderer, leaves, root, leaf, one):
    assert ((leaves - 1) * root <= 196608) == one
    host = _star(leaves, root, leaf)
    dw = DeviceWorld(renderer, host)
    try:
        out = torch.full((dw.transform_count * 16 + 64,), float("nan"), device="cuda")
        names = [k for k, _ in captured_kernels(lambda: dw.update_transforms(0.7, out))]
        assert len(names) == (1 if one else 2)
        assert ("k_world_slots" in names[0]) == one
        for time in (0.0, 0.7, 5.0):
            out.fill_(float("nan"))
            dw.update_transforms(time, out)
            got, exp = out.cpu().numpy(), ob.world_transforms(host, time)
            assert np.array_equal(got[:-64].view(np.uint32), exp.reshape(-1).view(np.uint32))
            assert np.isnan(got[-64:]).all()
        assert renderer.device_status() == (0, 0)
    finally:
        dw.close()

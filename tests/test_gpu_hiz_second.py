"""Pyramids on both sides of the sizes from which a reduce takes a second tiled
launch, alone and as views of one frame, at sizes whose level 4 does not halve
exactly: the oracle's bits."""
import numpy as np
import pytest
import torch

import gpu_util as U
from graph_util import frame_kernels
from oracle import binding as ob
from vk_gltf_viewer_gb300 import abi, scene

pytestmark = pytest.mark.gpu

# texels in level 5 about the two lines: 2,048 (several views) and 5,120 (one)
BELOW_MANY, ABOVE_MANY = (2853, 743), (2079, 1055)   # 89 x 23, 64 x 32
BELOW_ONE, ABOVE_ONE = (3819, 1399), (2575, 2063)    # 119 x 43, 80 x 64


@pytest.fixture(scope="module")
def mesh(built):
    return U.Pair(scene.scene_icosphere(1))


def _depth(w, h):
    rng = np.random.default_rng(w * 7 + h)
    d = rng.random(w * h, dtype=np.float32)
    d[rng.random(w * h) < 0.2] = 0.0
    return (d.view(np.uint32).astype(np.uint64) << np.uint64(32)) | np.uint64(3)


def _view(pair, w, h):
    return U.view(pair, scene.camera((0, 0, 3), (0, 0, 0), (0, 1, 0), 60, w / h), w, h)


def test_sizes_lie_about_the_lines():
    texels = [(w >> 5) * (h >> 5) for w, h in (BELOW_MANY, ABOVE_MANY, BELOW_ONE, ABOVE_ONE)]
    assert texels == [2047, 2048, 5117, 5120]


@pytest.mark.parametrize("size", [BELOW_MANY, ABOVE_MANY, BELOW_ONE, ABOVE_ONE, (3840, 2160), (3001, 1999), (3333, 2222),
                                  (8191, 1021), (797, 8191), (5119, 2881)])
def test_one_view(renderer, mesh, size):
    w, h = size
    depth = _depth(w, h)
    v = _view(mesh, w, h)
    v.depth_id.copy_(torch.from_numpy(depth.view(np.int64)).cuda())
    v.pyramid.fill_(-1.0)
    for _ in range(2):  # the second reduce finds the counters as the first left them
        renderer.hiz(mesh.dev, v)
        exp = ob.hiz(depth, w, h)
        assert np.array_equal(v.pyramid.cpu().numpy()[:exp.size], exp)
        v.pyramid.fill_(-1.0)
    assert renderer.device_status() == (0, 0)


@pytest.mark.parametrize("sizes", [[(640, 361), ABOVE_MANY, (1920, 1080), (3840, 2160), BELOW_MANY],
                                   [(3001, 1999), (97, 61)], [BELOW_MANY, (1, 700), (331, 5)], [ABOVE_ONE, ABOVE_MANY]])
def test_views_of_both_forms_in_one_frame(renderer, mesh, sizes):
    flags = abi.CULL_FRUSTUM | abi.BUILD_PYRAMID
    views = [_view(mesh, w, h) for w, h in sizes]
    for _ in range(2):
        for v in views:
            v.pyramid.fill_(-1.0)
        renderer.frame(mesh.dev, views, flags)
        torch.cuda.synchronize()
        for v, (w, h) in zip(views, sizes):
            depth = U.u64(v.depth_id)
            assert np.count_nonzero(depth) > 0 or min(w, h) < 8
            exp = ob.hiz(depth, w, h)
            assert np.array_equal(v.pyramid.cpu().numpy()[:exp.size], exp), (w, h)
    assert renderer.device_status() == (0, 0)


@pytest.mark.parametrize("sizes,launches", [([BELOW_ONE], 1), ([ABOVE_ONE], 2), ([(2560, 1440)], 1),
                                            ([BELOW_MANY, BELOW_MANY], 1), ([BELOW_MANY, ABOVE_MANY], 2)])
def test_launches_by_size_and_view_count(renderer, mesh, sizes, launches):
    graph = renderer.capture(mesh.dev, [_view(mesh, w, h) for w, h in sizes], abi.CULL_FRUSTUM | abi.BUILD_PYRAMID)
    try:
        assert sum("k_hiz" in name for name, _ in frame_kernels(graph)) == launches
    finally:
        graph.close()

"""The raster shapes that the autotuner tries hold both forms that an untuned
renderer chooses between: the fast and the slow kernel of its frame are those
of a renderer with one of the explicit shapes."""
import pytest

import gpu_util as U
from graph_util import frame_kernels
from vk_gltf_viewer_gb300 import abi, scene
from vk_gltf_viewer_gb300.renderer import Renderer

pytestmark = pytest.mark.gpu


def _raster_kernels(pair, views, meshlets_per_cta):
    r = Renderer(0, meshlets_per_cta=meshlets_per_cta)
    try:
        cam = scene.camera((4.0, 3.5, -3.0), (4.0, 1.0, 4.0), (0, 1, 0), 70.0, 1.5)
        graph = r.capture(pair.dev, [U.view(pair, cam, 96, 64) for _ in range(views)], abi.CULL_FRUSTUM)
        kernels = [(name.split("k_raster")[1], block) for name, block in frame_kernels(graph) if "k_rasterI" in name]
        graph.close()
        return kernels
    finally:
        r.close()


@pytest.mark.parametrize("views,shape", [(1, 4), (2, 1), (512, 1), (513, 4)])
def test_the_default_is_one_of_the_candidates(built, views, shape):
    pair = U.Pair(U.small_grid(tex=0))
    assert pair.host.draw_count == 13184  # one view below the line at 16,384 meshlets, two above
    default = _raster_kernels(pair, views, 0)
    assert len(default) == 2 and default[0][1] == 32 * shape
    assert default == _raster_kernels(pair, views, shape)

"""The raster's choice of one or four warps a CTA: launches of draws times
views on both sides of the line, and view counts up to and past the most that
one warp a CTA takes, against the oracle bit for bit."""
import numpy as np
import pytest

import gpu_util as U
from oracle import binding as ob
from vk_gltf_viewer_gb300 import scene

pytestmark = pytest.mark.gpu

W, H = 61, 47


@pytest.fixture(scope="module")
def grid(built):
    return U.Pair(U.small_grid())


@pytest.mark.parametrize("views", [1, 2, 512, 513])
def test_batches_match_oracle(renderer, grid, views):
    draws = grid.host.draw_count
    assert draws < 16384 <= 2 * draws
    cams = []
    for k in range(views):
        a = 2.0 * np.pi * k / views
        eye = (4.0 + 7.0 * np.cos(a), 3.0 + (k % 5), 4.0 + 7.0 * np.sin(a))
        cams.append(scene.camera(eye, (4.0, 1.0, 4.0), (0.0, 1.0, 0.0), 70.0, W / H))
    vs = [U.view(grid, c, W, H) for c in cams]
    renderer.frame(grid.dev, vs, 0)
    for k in sorted({0, 1 % views, views // 2, views - 1}):
        exp = ob.frame(grid.orc, cams[k], W, H, 0)
        assert np.count_nonzero(exp["depth_id"]) > 300
        assert np.array_equal(U.u64(vs[k].depth_id), exp["depth_id"]), k
    assert renderer.device_status() == (0, 0)

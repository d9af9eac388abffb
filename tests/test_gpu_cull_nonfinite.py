"""The occlusion tests on boxes that are not ordinary: nodes scaled to nothing,
by huge factors or mirrored, with infinite or NaN transforms, and boxes that
the camera plane cuts (corners with w <= 0), against the oracle's survivors
and rejects."""
import numpy as np
import pytest
import torch

import gpu_util as U
from oracle import binding as ob
from vk_gltf_viewer_gb300 import abi, scene

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def odd(built):
    host = scene.scene_torus_grid(texture_size=0, grid=(4, 4, 2))
    t = host.transforms.reshape(-1, 4, 4)  # column-major: t[n][column][row]
    t[1, :3, :3] = 0.0
    t[2, :3, :3] *= 1e30
    t[3, :3, :3] *= -1.0
    t[5, 0, 0] = np.inf
    t[6, 3, 1] = -np.inf
    t[7, 1, 2] = np.nan
    t[9] = np.nan
    t[10, :3, :3] *= 40.0
    t[12, :3, :3] *= 1e-30
    return U.Pair(host)


@pytest.mark.parametrize("size", [(512, 384), (640, 360), (257, 129)])
@pytest.mark.parametrize("fine", [False, True])
def test_odd_boxes_match_oracle(renderer, odd, size, fine):
    w, h = size
    flags = abi.CULL_FRUSTUM | abi.CULL_OCCLUSION | (abi.CULL_OCCLUSION_FINE if fine else 0)
    rng = np.random.default_rng(w)
    floats = ob.pyramid_floats(w, h)
    for kind in range(3):
        # empty, partly covered and full depth
        prev = np.zeros(floats, np.float32)
        if kind:
            prev[:] = rng.uniform(0, 0.05 * kind, floats)
        for eye in [(3.0, 1.2, 3.0), (-4.0, 2.0, -5.0), (0.1, 0.0, 0.2)]:
            cam = scene.camera(eye, (4.0, 1.0, 4.0), (0, 1, 0), 70.0, w / h)
            v = U.view(odd, cam, w, h, prev=prev)
            renderer.clear(odd.dev, v)
            renderer.cull(odd.dev, v, flags, 1)
            torch.cuda.synchronize()
            exp, _ = ob.cull(odd.orc, cam, w, h, U.oracle_flags(flags), 1, pyramid=prev)
            assert np.array_equal(np.sort(v.survivor_list()), np.sort(exp)), (kind, eye)

"""The loss of a captured step over many CTAs: how far launches of the same step
lie apart.  Each addition to the one float rounds by at most 2^-24 of the sum, in
an order that changes from launch to launch; with one addition a CTA (456 on
152 SMs) the spread is some sqrt(456 / 3) 2^-24 / sqrt(3) = 4e-7 of the sum at
most, with one a warp sqrt(8) times that."""
import numpy as np
import pytest
import torch

from vk_gltf_viewer_gb300 import diff, scene

pytestmark = pytest.mark.gpu


def test_spread_over_launches(renderer):
    rng = np.random.default_rng(5)
    mesh = scene.icosphere(5)
    nv = mesh.positions.shape[0]
    ds = diff.DiffScene.create(mesh, rng.random((nv, 3)).astype(np.float32),
                               rng.random((256, 256, 3)).astype(np.float32))
    eyes = rng.normal(size=(48, 3))
    eyes = 3.0 * eyes / np.linalg.norm(eyes, axis=1, keepdims=True)
    views = [diff.DiffViewBuffers.allocate(512, 512, scene.camera(tuple(e), (0, 0, 0), scene.safe_up(e, np.zeros(3)),
                                                                  60.0, 1.0)) for e in eyes]
    targets = [torch.rand(3 * 512 * 512, device="cuda") for _ in views]
    loss = torch.zeros(1, device="cuda")
    grad = torch.zeros_like(ds.positions)
    step = diff.capture_step(renderer, ds, views, targets=targets, grad_positions=grad,
                             rgb_out=[torch.empty_like(t) for t in targets], scale=1e-7, loss=loss)
    try:
        seen = []
        for _ in range(60):
            step.launch()
            seen.append(loss.item())
    finally:
        step.close()
    seen = np.array(seen, np.float64)
    assert seen.mean() > 0.0
    assert seen.std() / seen.mean() < 6e-7

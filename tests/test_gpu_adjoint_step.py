"""The captured forward + backward step, which is one pass unless an image
overlaps what the backward pass reads: against the two passes captured one
after the other, for images on their own, an image given as its own dL/drgb
or target, and an image that overlaps the next view's target."""
import numpy as np
import pytest
import torch

from vk_gltf_viewer_gb300 import abi, diff, scene

pytestmark = pytest.mark.gpu

SIZES = [(65, 40), (96, 96), (31, 17)]


def setup_views(rng):
    views = []
    for w, h in SIZES:
        v = rng.normal(size=3)
        eye = 3.0 * v / np.linalg.norm(v)
        views.append(diff.DiffViewBuffers.allocate(w, h, scene.camera(
            tuple(eye), (0, 0, 0), scene.safe_up(eye, (0, 0, 0)), 60.0, w / h)))
    return views


def images(alias):
    """(rgb, targets, grad_rgb) of the views, aliased as asked, filled alike."""
    n = [3 * w * h for w, h in SIZES]
    o = np.concatenate([[0], np.cumsum(n)])
    g = torch.Generator(device="cuda").manual_seed(4)
    a = torch.rand(int(o[-1]), generator=g, device="cuda")
    b = torch.rand(int(o[-1]), generator=g, device="cuda")
    cut = lambda t, d=0: [t[int(o[i]) + d:int(o[i]) + d + n[i]] for i in range(len(n))]  # noqa: E731
    if alias == "none":
        return cut(a), cut(b), None
    if alias == "upstream":
        return cut(a), None, cut(b)
    if alias == "rgb is grad":
        return cut(a), None, cut(a)
    if alias == "rgb is target":
        return cut(a), cut(a), None
    c = torch.rand(int(o[-1]) + 64, generator=g, device="cuda")
    return cut(c), cut(c, 64), None  # "shifted": each image's end is in the next target


@pytest.mark.parametrize("alias", ["none", "upstream", "rgb is grad", "rgb is target", "shifted"])
def test_one_pass_step_matches_two_passes(renderer, alias):
    rng = np.random.default_rng(21)
    mesh = scene.icosphere(3)
    sc = diff.DiffScene.create(mesh, rng.uniform(0, 1, (mesh.positions.shape[0], 3)),
                               rng.uniform(0, 1, (33, 47, 3)), uv_scale=(2.0, 1.5), uv_rotation=0.3)
    views = setup_views(rng)
    scale = 1.0 / (3 * sum(w * h for w, h in SIZES))
    got = []
    for split in (False, True):
        rgb, targets, upstream = images(alias)
        grads = [torch.full_like(t, 5.0) for t in (sc.positions, sc.colors, sc.texture)]
        loss = torch.full((1,), 5.0, device="cuda")
        kw = dict(rgb_out=rgb, targets=targets, grad_rgb=upstream, grad_positions=grads[0], grad_colors=grads[1],
                  grad_texture=grads[2], scale=scale, loss=loss)
        steps = ([abi.DIFF_ZERO_GRADS | abi.DIFF_FORWARD, abi.DIFF_BACKWARD] if split
                 else [abi.DIFF_ZERO_GRADS | abi.DIFF_FORWARD | abi.DIFF_BACKWARD])
        graphs = [diff.capture_step(renderer, sc, views, passes=p, **kw) for p in steps]
        for g in graphs:
            g.launch()
        torch.cuda.synchronize()
        got.append((rgb, grads, loss, [g.kernel_count() for g in graphs]))
        for g in graphs:
            g.close()
    (rgb1, grads1, loss1, k1), (rgb2, grads2, loss2, k2) = got
    # one pass where it may be, two where an image is read back
    assert (sum(k1) < sum(k2)) == (alias in ("none", "upstream"))
    for a, b in zip(rgb1, rgb2):
        assert torch.equal(a, b)
    assert any(bool((a != 0).any()) for a in rgb1)
    # the sums differ by the order of fp32 atomics only
    assert abs(float(loss1) - float(loss2)) <= 1e-5 * abs(float(loss2))
    for a, b in zip(grads1, grads2):
        assert torch.linalg.vector_norm(a - b) <= 1e-5 * torch.linalg.vector_norm(b)

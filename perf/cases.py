"""The work whose speed this repository is judged by, as its users run it.

Five kinds, each through the package's public classes:

  frame    one view per pass: the captured frame of a viewer or a headless
           renderer (Renderer.capture, Graph.launch), or an uncaptured one
           (Renderer.frame) of a small scene
  batch    many views of one scene in one captured frame
  adjoint  the differentiable resolve: zero + forward + backward in one
           captured step, or the separate calls an autograd function makes
  world    the node tree: animated transforms and the draw list
  decode   block-compressed base-colour textures into texels

listed() names the fixed cases, draw() gives more of the same ranges.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from vk_gltf_viewer_gb300 import abi, diff, scene, texture, world
from vk_gltf_viewer_gb300.renderer import DeviceScene, Renderer, ViewBuffers, pyramid_layout

DEVICE = "cuda:0"
CULL = abi.CULL_FRUSTUM | abi.CULL_CONE
OCCLUSION = abi.CULL_OCCLUSION | abi.CULL_OCCLUSION_FINE | abi.CULL_TWO_PASS | abi.BUILD_PYRAMID

# One 200 x 100 displaced torus: 40,000 triangles in 412 meshlets.
TORUS_MESHLETS, TORUS_VERTICES, TORUS_TRIANGLES = 412, 20000, 40000

FORMATS = {"bc1": abi.BC1, "bc2": abi.BC2, "bc3": abi.BC3, "bc4": abi.BC4, "bc5": abi.BC5, "bc7": abi.BC7,
           "bc6h_uf16": abi.BC6H_UF16, "bc6h_sf16": abi.BC6H_SF16}
NARROW = ("bc1", "bc4")  # 8-byte blocks; the others have 16

# How often encoders choose each BC7 mode (0-7) and BC6H mode field in colour
# and HDR images: mostly the one-subset modes, every mode present.
BC7_SHARE = (0.04, 0.24, 0.04, 0.10, 0.05, 0.10, 0.36, 0.07)
BC6H_MODES = (0x00, 0x01, 0x02, 0x06, 0x0A, 0x0E, 0x12, 0x16, 0x1A, 0x1E, 0x03, 0x07, 0x0B, 0x0F)
BC6H_SHARE = (0.09, 0.09, 0.04, 0.04, 0.04, 0.05, 0.04, 0.04, 0.04, 0.05, 0.16, 0.14, 0.11, 0.07)


# ------------------------------------------------------------------- cases

def _grid(kind, gx, gz, gy, tex, **kw):
    return dict(kind=kind, scene="grid", gx=gx, gz=gz, gy=gy, texture=tex, **kw)


def listed():
    return [
        # the per-frame host update of an animated scene: 2,048 animated tori
        # under 8 layers, and the draw list that a scene change rebuilds
        dict(name="world_2048_nodes", kind="world", gx=16, gz=16, gy=8),
        # a thumbnail or asset check: one small mesh, one uncaptured frame
        dict(name="frame_sphere_thumb", kind="frame", scene="sphere", level=4, width=256, height=256, shade="flat",
             occlusion=False, motion=False, moving=False, animated=False, captured=False),
        # one mesh, constant base colour, frustum and cone culling only
        dict(name="frame_sphere_720p", kind="frame", scene="sphere", level=6, width=1280, height=720, shade="flat",
             occlusion=False, motion=False, moving=False, animated=False, captured=True),
        # the viewer inside a dense instanced scene (82M triangles), two-pass
        # occlusion, textured resolve, steady state
        dict(_grid("frame", 16, 16, 8, 2048, inside=True, width=1920, height=1080, shade="textured", occlusion=True,
                   motion=False, moving=False, animated=False, captured=True), name="frame_grid_1080p"),
        # the viewer in motion at an odd window size: animated nodes, a moving
        # camera (the pyramid is last pose's), motion vectors for an upscaler
        dict(_grid("frame", 12, 12, 6, 1024, inside=True, width=1365, height=767, shade="textured", occlusion=True,
                   motion=True, moving=True, animated=True, captured=True), name="frame_grid_moving_odd"),
        # a 4K still of the whole scene from outside
        dict(_grid("frame", 16, 16, 8, 2048, inside=False, width=3840, height=2160, shade="textured", occlusion=True,
                   motion=False, moving=False, animated=False, captured=True), name="frame_grid_4k"),
        # many small observations of a small scene (simulation, dataset renders)
        dict(_grid("batch", 4, 4, 2, 512, views=256, width=128, height=128, shade="textured"), name="batch_small_views"),
        # 256 poses at mixed sizes of the dense scene in one launch
        dict(_grid("batch", 16, 16, 8, 2048, views=256, width=0, height=0, shade="textured"), name="batch_grid_256"),
        # inverse rendering: a 20,480-triangle sphere, 64 views
        dict(name="adjoint_sphere_64", kind="adjoint", level=5, displace=0.0, texture=1024, views=64, min_edge=512,
             max_edge=512, captured=True),
        # a 1.3M-triangle mesh, uneven views
        dict(name="adjoint_dense_128", kind="adjoint", level=8, displace=0.02, texture=2048, views=128, min_edge=256,
             max_edge=1024, captured=True),
        # texture loading: a 4096^2 colour map, and a ragged HDR map
        dict(name="decode_bc7_4096", kind="decode", format="bc7", width=4096, height=4096),
        dict(name="decode_bc6h_ragged", kind="decode", format="bc6h_uf16", width=2050, height=1023),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "batch", "batch", "adjoint", "adjoint", "world", "decode", "decode"])
    if kind == "world":
        return dict(kind="world", gx=rng.randint(1, 24), gz=rng.randint(1, 24), gy=rng.randint(1, 9))
    if kind == "decode":
        return dict(kind="decode", format=rng.choice(sorted(FORMATS)), width=_log(rng, 61, 8192),
                    height=_log(rng, 61, 8192))
    if kind == "adjoint":
        level = rng.randint(3, 8)
        lo = _log(rng, 64, 512)
        return dict(kind="adjoint", level=level, displace=rng.choice([0.0, 0.02]), texture=_log(rng, 200, 2048),
                    views=_log(rng, 1, 128), min_edge=lo, max_edge=min(1024, int(lo * rng.uniform(1, 2.5))),
                    captured=rng.random() < 0.7)
    if kind == "batch":
        g = rng.choice([(4, 4, 2), (8, 8, 4), (12, 12, 6)])
        w = _log(rng, 96, 1280)
        return _grid("batch", *g, _log(rng, 64, 2048), views=_log(rng, 2, 192), width=w,
                     height=max(64, int(w * rng.uniform(0.5, 1.0))), shade=rng.choice(["flat", "textured"]))
    w = _log(rng, 200, 3840)
    h = max(100, int(w * rng.uniform(0.45, 0.8)))
    common = dict(width=w, height=h, shade=rng.choice(["flat", "textured", "textured"]), motion=rng.random() < 0.4,
                  moving=rng.random() < 0.5, captured=rng.random() < 0.8)
    if rng.random() < 0.3:
        common["shade"] = "flat"  # the sphere scene has no texture
        return dict(kind="frame", scene="sphere", level=rng.randint(3, 7), occlusion=rng.random() < 0.5,
                    animated=False, **common)
    g = rng.choice([(4, 4, 2), (8, 8, 4), (12, 12, 6), (16, 16, 8)])
    return _grid("frame", *g, _log(rng, 64, 2048), inside=rng.random() < 0.6, occlusion=rng.random() < 0.8,
                 animated=rng.random() < 0.5, **common)


# ------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=4)
def _sphere_mesh(level, displace, seed):
    return scene.icosphere(level, displace=displace, seed=seed)


def _aim(eye, target, fovy, w, h, prev=None):
    return scene.camera(tuple(eye), tuple(target), scene.safe_up(eye, target), fovy, w / h, prev=prev)


def _centre(case):
    return np.array([(case["gx"] - 1), (case["gy"] - 1), (case["gz"] - 1)], np.float64) * scene.SPACING / 2


def _flags(case, occlusion, motion):
    shade = abi.RESOLVE_TEXTURED if case["shade"] == "textured" else abi.RESOLVE_FLAT
    return CULL | shade | abi.WRITE_IDS | (OCCLUSION if occlusion else 0) | (abi.WRITE_MOTION if motion else 0)


def _grid_scene(case, seed):
    return scene.scene_torus_grid(seed=seed, texture_size=case["texture"], grid=(case["gx"], case["gz"], case["gy"]),
                                  tex_seed=seed + 1)


def _poses(case, rng, n):
    """Eye points on a sphere around the grid, scaled with it (30 for the
    16 x 16 x 8 grid), aimed at its centre."""
    c = _centre(case)
    v = rng.normal(size=(n, 3))
    radius = 30.0 * max(case["gx"], case["gz"]) / 16 + 1.0
    return c, c + radius * v / np.linalg.norm(v, axis=1, keepdims=True)


def _prepare_frame(case, seed):
    rng = np.random.default_rng(seed)
    w, h = case["width"], case["height"]
    r = Renderer(0)
    dw = t_now = None
    if case["scene"] == "sphere":
        host = scene.scene_icosphere(case["level"], albedo=(*rng.uniform(0.2, 1.0, 3), 1.0))
        eye, target, fovy = np.array([0.0, 0.0, 3.0]) + rng.uniform(-0.1, 0.1, 3), np.zeros(3), 60.0
        step = np.array([0.03, 0.01, 0.02])
    else:
        host = _grid_scene(case, seed)
        if case["inside"]:
            c = _centre(case)
            eye = np.array([0.25 * scene.SPACING, c[1], c[2]]) + rng.uniform(-0.2, 0.2, 3)
            target = eye + np.array([10.0, 0.0, 0.0]) + rng.uniform(-0.3, 0.3, 3)
        else:
            target, eyes = _poses(case, rng, 1)
            eye = eyes[0]
        fovy, step = 75.0, np.array([0.08, 0.01, 0.03])
    dev = DeviceScene(host, DEVICE)
    if case["animated"]:
        mesh = host.meshes[0]
        dw = world.DeviceWorld(r, world.grid_world(mesh.meshlet_count, mesh.position_scale, seed=seed,
                                                   grid=(case["gx"], case["gz"], case["gy"])))
        t_now = float(rng.uniform(0.1, 3.9))
        dw.update_transforms(max(0.0, t_now - 1 / 60), dev.transforms)
    before = eye - step if case["moving"] else eye
    prev = _aim(before, target, fovy, w, h)
    v = ViewBuffers.allocate(w, h, prev, host.draw_count, device=DEVICE, pyramid=case["occlusion"],
                             prev_pyramid=case["occlusion"], motion=case["motion"])
    flags = _flags(case, case["occlusion"], case["motion"])
    # last frame, from the previous pose: its pyramid is this frame's input
    v.use_prev = False
    r.frame(dev, [v], flags)
    if case["occlusion"]:
        v.prev_pyramid.copy_(v.pyramid)
    v.use_prev = True
    if case["moving"]:
        v.set_camera(_aim(eye, target, fovy, w, h, prev=prev))
    graph = r.capture(dev, [v], flags) if case["captured"] else None
    torch.cuda.synchronize()
    return dict(case=case, renderer=r, scene=dev, view=v, flags=flags, graph=graph, world=dw, time=t_now)


def _run_frame(s):
    v = s["view"]
    if s["world"] is not None:
        s["world"].update_transforms(s["time"], s["scene"].transforms)
    if s["graph"] is not None:
        s["graph"].launch()
    else:
        s["renderer"].frame(s["scene"], [v], s["flags"])
    return dict(depth_id=v.depth_id, ids=v.visbuffer, color=v.color, pyramid=v.pyramid, motion=v.motion,
                survivors=v.survivor_count)


def _batch_sizes(case):
    rng = np.random.default_rng(case["views"])
    if case["width"]:
        return [(case["width"], case["height"])] * case["views"]
    return [scene.BATCH_SIZES[int(k)] for k in rng.integers(0, len(scene.BATCH_SIZES), case["views"])]


def _prepare_batch(case, seed):
    rng = np.random.default_rng(seed)
    n = case["views"]
    r = Renderer(0)
    host = _grid_scene(case, seed)
    dev = DeviceScene(host, DEVICE)
    sizes = _batch_sizes(case)
    target, eyes = _poses(case, rng, n)
    # the views' images are slices of one tensor of each kind, as a program
    # that hands the whole batch on keeps them (16-byte aligned starts)
    px = [(w * h + 3) // 4 * 4 for w, h in sizes]
    lay = [pyramid_layout(w, h) for w, h in sizes]
    fl = [(f + 3) // 4 * 4 for _, f in lay]
    po, fo = np.concatenate([[0], np.cumsum(px)]), np.concatenate([[0], np.cumsum(fl)])
    big = dict(depth_id=torch.zeros(int(po[-1]), dtype=torch.int64, device=DEVICE),
               ids=torch.zeros(int(po[-1]), dtype=torch.int32, device=DEVICE),
               color=torch.zeros(int(po[-1]), dtype=torch.int32, device=DEVICE),
               pyramid=torch.zeros(int(fo[-1]), dtype=torch.float32, device=DEVICE))
    last = torch.zeros_like(big["pyramid"])
    cams = [_aim(eyes[i], target, 75.0, w, h) for i, (w, h) in enumerate(sizes)]
    cam_bytes = torch.from_numpy(np.stack([scene.camera_bytes(c) for c in cams])).to(DEVICE)
    views = []
    for i, (w, h) in enumerate(sizes):
        a, b = int(po[i]), int(fo[i])
        views.append(ViewBuffers(width=w, height=h, camera=cam_bytes[i], depth_id=big["depth_id"][a:a + w * h],
                                 visbuffer=big["ids"][a:a + w * h], color=big["color"][a:a + w * h],
                                 pyramid=big["pyramid"][b:b + lay[i][1]], prev_pyramid=last[b:b + lay[i][1]],
                                 survivors=None, survivor_count=None, levels=lay[i][0], use_prev=False))
    flags = _flags(case, True, False)
    r.frame(dev, views, flags)
    last.copy_(big["pyramid"])
    for v in views:
        v.use_prev = True
    graph = r.capture(dev, views, flags)
    torch.cuda.synchronize()
    return dict(case=case, renderer=r, scene=dev, views=views, graph=graph, out=big, cams=cam_bytes, last=last)


def _run_batch(s):
    s["graph"].launch()
    return s["out"]


def _adjoint_sizes(case):
    rng = np.random.default_rng(case["views"])
    lo, hi = case["min_edge"], case["max_edge"]
    return [(int(a), int(b)) for a, b in rng.integers(lo, hi + 1, (case["views"], 2))]


def _adjoint_inputs(case, seed):
    rng = np.random.default_rng(seed)
    mesh = _sphere_mesh(case["level"], case["displace"], seed)
    t = case["texture"]
    eyes = rng.normal(size=(case["views"], 3))
    eyes = 3.0 * eyes / np.linalg.norm(eyes, axis=1, keepdims=True)
    sizes = _adjoint_sizes(case)
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    nv = mesh.positions.shape[0]
    p = torch.tensor(mesh.positions, device=DEVICE)

    def image():
        # a colour map with features of some 16 texels
        low = torch.rand(1, 3, t // 16 + 2, t // 16 + 2, generator=g, device=DEVICE)
        up = torch.nn.functional.interpolate(low, (t, t), mode="bicubic", align_corners=True)
        return up[0].clamp(0, 1).permute(1, 2, 0).contiguous()

    return dict(mesh=mesh, sizes=sizes, positions=p, colors=torch.rand(nv, 3, generator=g, device=DEVICE),
                texture=image(), texture_target=image(),
                positions_target=p + 0.01 * torch.randn(nv, 3, generator=g, device=DEVICE),
                cams=[_aim(e, np.zeros(3), 60.0, w, h) for e, (w, h) in zip(eyes, sizes)],
                scale=1.0 / (3 * sum(w * h for w, h in sizes)))


def _diff_scene(i, positions, tex):
    mesh = i["mesh"]

    def u8(a):
        return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()).to(DEVICE)

    return diff.DiffScene(mesh=mesh, meshlets=u8(mesh.meshlets), vertex_indices=u8(mesh.vertex_indices),
                          primitive_indices=u8(mesh.primitive_indices), positions=positions, colors=i["colors"],
                          uvs=torch.tensor(mesh.uvs, device=DEVICE), texture=tex)


def _adjoint_targets(case, seed, r):
    """The inputs, and the views' target images (a render of the perturbed
    mesh with another texture) and image buffers as slices of one tensor."""
    i = _adjoint_inputs(case, seed)
    px = [(w * h + 3) // 4 * 4 for w, h in i["sizes"]]
    o = np.concatenate([[0], np.cumsum(px)])
    images = {k: torch.zeros(3 * int(o[-1]), device=DEVICE) for k in ("target", "rgb")}
    cut = {k: [t[3 * int(o[j]):3 * (int(o[j]) + w * h)] for j, (w, h) in enumerate(i["sizes"])]
           for k, t in images.items()}
    views = [diff.DiffViewBuffers.allocate(w, h, c, device=DEVICE) for (w, h), c in zip(i["sizes"], i["cams"])]
    diff.forward(r, _diff_scene(i, i["positions_target"], i["texture_target"]), views, cut["target"])
    torch.cuda.synchronize()
    return i, o, images, cut, views


def _prepare_adjoint(case, seed):
    r = Renderer(0)
    i, _, images, cut, views = _adjoint_targets(case, seed, r)
    ds = _diff_scene(i, i["positions"], i["texture"])
    s = dict(case=case, renderer=r, scene=ds, views=views, cut=cut, images=images, scale=i["scale"], graph=None,
             grads=dict(positions=torch.zeros_like(ds.positions), colors=torch.zeros_like(ds.colors),
                        texture=torch.zeros_like(ds.texture)), loss=torch.zeros(1, device=DEVICE))
    if case["captured"]:
        s["graph"] = diff.capture_step(r, ds, views, rgb_out=cut["rgb"], targets=cut["target"],
                                       grad_positions=s["grads"]["positions"], grad_colors=s["grads"]["colors"],
                                       grad_texture=s["grads"]["texture"], scale=s["scale"], loss=s["loss"])
    else:
        s["upstream"] = torch.zeros_like(images["rgb"])
        off = [c.storage_offset() for c in cut["rgb"]]
        s["upstream_cut"] = [s["upstream"][a:a + c.numel()] for a, c in zip(off, cut["rgb"])]
    torch.cuda.synchronize()
    return s


def _run_adjoint(s):
    if s["graph"] is not None:
        s["graph"].launch()
    else:
        # what an autograd function's forward and backward do around a loss
        # of the program's own
        diff.forward(s["renderer"], s["scene"], s["views"], s["cut"]["rgb"])
        torch.sub(s["images"]["rgb"], s["images"]["target"], out=s["upstream"])
        s["loss"].copy_(s["scale"] * torch.linalg.vector_norm(s["upstream"]).square().reshape(1))
        s["upstream"].mul_(2.0 * s["scale"])
        for g in s["grads"].values():
            g.zero_()
        diff.backward(s["renderer"], s["scene"], s["views"], grad_positions=s["grads"]["positions"],
                      grad_colors=s["grads"]["colors"], grad_texture=s["grads"]["texture"],
                      grad_rgb=s["upstream_cut"])
    return dict(rgb=s["images"]["rgb"], loss=s["loss"], **s["grads"])


def _world_inputs(case, seed):
    tree = world.grid_world(TORUS_MESHLETS, 1.4, seed=seed, grid=(case["gx"], case["gz"], case["gy"]))
    return tree, float(np.float32(np.random.default_rng(seed).uniform(0.1, 3.9)))


def _prepare_world(case, seed):
    tree, t = _world_inputs(case, seed)
    r = Renderer(0)
    dw = world.DeviceWorld(r, tree)
    return dict(case=case, renderer=r, world=dw, time=t,
                transforms=torch.zeros(16 * dw.transform_count, device=DEVICE),
                draws=torch.zeros(3 * dw.draw_count, dtype=torch.int32, device=DEVICE))


def _run_world(s):
    s["world"].update_transforms(s["time"], s["transforms"])
    s["world"].build_draws(s["draws"])
    return dict(transforms=s["transforms"], draws=s["draws"])


def _block_bytes(case):
    n = ((case["width"] + 3) // 4) * ((case["height"] + 3) // 4)
    return n, n * (8 if case["format"] in NARROW else 16)


def _prepare_decode(case, seed):
    n, size = _block_bytes(case)
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    blocks = torch.randint(0, 256, (n, size // n), generator=g, device=DEVICE, dtype=torch.uint8)
    if case["format"] == "bc7":  # mode m: the lowest set bit of the first byte is bit m
        m = torch.multinomial(torch.tensor(BC7_SHARE, device=DEVICE), n, replacement=True, generator=g)
        first = blocks[:, 0].to(torch.int64)
        blocks[:, 0] = ((((first >> (m + 1)) << (m + 1)) | (1 << m)) & 255).to(torch.uint8)
    elif case["format"].startswith("bc6h"):  # a 2-bit (0, 1) or 5-bit mode field
        k = torch.multinomial(torch.tensor(BC6H_SHARE, device=DEVICE), n, replacement=True, generator=g)
        m = torch.tensor(BC6H_MODES, device=DEVICE)[k]
        keep = torch.where(m < 2, 0xFC, 0xE0)
        blocks[:, 0] = ((blocks[:, 0].to(torch.int64) & keep) | m).to(torch.uint8)
    return dict(case=case, renderer=Renderer(0), blocks=blocks.reshape(-1))


def _run_decode(s):
    c = s["case"]
    call = texture.decode_bc6h if c["format"].startswith("bc6h") else texture.decode_bc
    return call(s["renderer"], FORMATS[c["format"]], s["blocks"], c["width"], c["height"])


def prepare(case, seed):
    return {"frame": _prepare_frame, "batch": _prepare_batch, "adjoint": _prepare_adjoint, "world": _prepare_world,
            "decode": _prepare_decode}[case["kind"]](case, seed)


def run(state):
    return {"frame": _run_frame, "batch": _run_batch, "adjoint": _run_adjoint, "world": _run_world,
            "decode": _run_decode}[state["case"]["kind"]](state)


# -------------------------------------------------------------------- work

def work(case):
    """Bytes: each input once and each output once.  Flops: the box tests of
    every draw and view, and the per-pixel shading."""
    kind = case["kind"]
    if kind == "world":
        slots = case["gx"] * case["gz"] * case["gy"]
        return {"bytes": 40 * slots + 64 * slots + 12 * TORUS_MESHLETS * slots, "flops": 200 * slots}
    if kind == "decode":
        _, size = _block_bytes(case)
        px = case["width"] * case["height"]
        return {"bytes": size + px * (12 if case["format"].startswith("bc6h") else 4), "flops": 0}
    if kind == "adjoint":
        nv, px = 10 * 4 ** case["level"] + 2, sum(w * h for w, h in _adjoint_sizes(case))
        tris, tex = 20 * 4 ** case["level"], case["texture"] ** 2
        # visibility (8), target and image per pixel; parameters read,
        # gradients written; indices
        return {"bytes": px * (8 + 12 + 12) + nv * (12 + 12 + 8 + 24) + tex * 24 + 7 * tris, "flops": 300 * px}
    if case["scene"] == "sphere":
        tris, verts = 20 * 4 ** case["level"], 10 * 4 ** case["level"] + 2
        draws, nodes, tex = tris // 93 + 1, 1, 0
    else:
        tris, verts, nodes = TORUS_TRIANGLES, TORUS_VERTICES, case["gx"] * case["gz"] * case["gy"]
        draws, tex = TORUS_MESHLETS * nodes, case["texture"]
    sizes = [(case["width"], case["height"])] if kind == "frame" else _batch_sizes(case)
    px = sum(w * h for w, h in sizes)
    occlusion = kind == "batch" or case["occlusion"]
    motion = kind == "frame" and case["motion"]
    shaded = case["shade"] == "textured"
    per_px = 8 + 4 + 4 + (8 / 3 if occlusion else 0) + (4 if motion else 0)
    return {"bytes": 12 * draws + 64 * nodes + 28 * verts + 3 * tris + per_px * px + (4 * tex * tex if shaded else 0),
            "flops": 150 * draws * len(sizes) + (300 if shaded else 20) * px}


# ------------------------------------------------------------------- exact
# Visibility buffers, colours and draw lists are whole numbers.  The world
# transforms and the adjoint's image, loss and gradients are computed here in
# 64 bits with numpy and torch alone.

def _quat_mat(q):
    x, y, z, w = q
    return np.array([[1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y)],
                     [2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x)],
                     [2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]])


def _sample64(s, path, time):
    """A glTF animation sampler at `time` (looped), in 64 bits."""
    keys, out = np.asarray(s.input, np.float64), np.asarray(s.output, np.float64)
    t = math.fmod(time, keys[-1])
    i = int(np.searchsorted(keys, t, side="left"))
    cubic = s.interpolation == abi.INTERP_CUBICSPLINE
    if i == 0:
        return out[1 if cubic else 0]
    if i == len(keys):
        return out[-2 if cubic else -1]
    dt = keys[i] - keys[i - 1]
    u = (t - keys[i - 1]) / dt
    if s.interpolation == abi.INTERP_STEP:
        return out[i - 1]
    if cubic:
        p0, m0, p1, m1 = out[3 * i - 2], out[3 * i - 1], out[3 * i + 1], out[3 * i]
        v = ((2 * u ** 3 - 3 * u ** 2 + 1) * p0 + dt * (u ** 3 - 2 * u ** 2 + u) * m0
             + (-2 * u ** 3 + 3 * u ** 2) * p1 + dt * (u ** 3 - u ** 2) * m1)
        return v / np.linalg.norm(v) if path == abi.PATH_ROTATION else v
    a, b = out[i - 1], out[i]
    if path != abi.PATH_ROTATION:
        return (1 - u) * a + u * b
    if a @ b < 0:
        b = -b
    th = 2 * math.atan2(np.linalg.norm(a - b), np.linalg.norm(a + b))
    if th < 1e-6:
        return (1 - u) * a + u * b
    return (math.sin((1 - u) * th) * a + math.sin(u * th) * b) / math.sin(th)


def _exact_world(case, seed):
    tree, time = _world_inputs(case, seed)
    trs = [[n["translation"].astype(np.float64), n["rotation"].astype(np.float64), n["scale"].astype(np.float64)]
           for n in tree.nodes]
    for sampler, node, path, _ in tree.channels:
        if node != abi.INVALID_HANDLE and path != abi.PATH_WEIGHTS:
            at = {abi.PATH_TRANSLATION: 0, abi.PATH_ROTATION: 1, abi.PATH_SCALE: 2}[int(path)]
            trs[int(node)][at] = _sample64(tree.samplers[int(sampler)], int(path), time)
    out = []

    def walk(n, parent):
        t, q, s = trs[n]
        m = np.eye(4)
        m[:3, :3] = _quat_mat(q) * s[None, :]
        m[:3, 3] = t
        m = parent @ m
        node = tree.nodes[n]
        if node["mesh_index"] != abi.INVALID_HANDLE:
            out.append(m.T.reshape(16))
        first = int(node["first_child"])
        for c in tree.children[first:first + int(node["child_count"])]:
            walk(int(c), m)

    for root in tree.roots:
        walk(int(root), np.eye(4))
    return dict(transforms=np.concatenate(out), draws=None)


def _visible64(pos, tri, vp, w, h):
    """Index of the triangle at every pixel (-1: none): fp32 vertices snapped
    to 1/256 pixel, top-left rule, reverse-Z, back faces dropped.  The spheres
    here lie inside the near and far planes and the guard band."""
    m = torch.tensor(vp, device=DEVICE).reshape(4, 4)  # column-major: m[c][j]
    x, y, z = pos[:, 0], pos[:, 1], pos[:, 2]
    clip = [((m[0, j] * x + m[1, j] * y) + m[2, j] * z) + m[3, j] for j in range(4)]
    rw = 1.0 / clip[3]
    sx = torch.round(((clip[0] * rw) * (0.5 * w) + 0.5 * w) * 256).to(torch.int64)[tri]
    sy = torch.round(((clip[1] * rw) * (0.5 * h) + 0.5 * h) * 256).to(torch.int64)[tri]
    sz = (clip[2] * rw)[tri]
    (p0, q0, r0), (p1, q1, r1), (p2, q2, r2) = (clip[k][tri].unbind(1) for k in (0, 1, 3))
    det = (p0 * (q1 * r2 - r1 * q2) - q0 * (p1 * r2 - r1 * p2)) + r0 * (p1 * q2 - q1 * p2)
    area = (sx[:, 1] - sx[:, 0]) * (sy[:, 2] - sy[:, 0]) - (sy[:, 1] - sy[:, 0]) * (sx[:, 2] - sx[:, 0])
    x0 = ((sx.amin(1) + 127) >> 8).clamp(min=0)
    x1 = ((sx.amax(1) - 128) >> 8).clamp(max=w - 1)
    y0 = ((sy.amin(1) + 127) >> 8).clamp(min=0)
    y1 = ((sy.amax(1) - 128) >> 8).clamp(max=h - 1)
    keep = torch.nonzero((det <= 0) & (area != 0) & (x0 <= x1) & (y0 <= y1)).reshape(-1)
    sx, sy, sz, x0, y0, area = sx[keep], sy[keep], sz[keep], x0[keep], y0[keep], area[keep]
    bw = x1[keep] - x0 + 1
    n = bw * (y1[keep] - y0 + 1)
    k = torch.repeat_interleave(torch.arange(len(keep), device=DEVICE), n)
    local = torch.arange(len(k), device=DEVICE) - torch.repeat_interleave(torch.cumsum(n, 0) - n, n)
    px, py = x0[k] + local % bw[k], y0[k] + local // bw[k]
    order = torch.where((area < 0)[:, None], torch.tensor([0, 2, 1], device=DEVICE), torch.tensor([0, 1, 2], device=DEVICE))
    sx, sy, sz = (v.gather(1, order)[k] for v in (sx, sy, sz))
    qx, qy = px * 256 + 128, py * 256 + 128
    inside = torch.ones(len(k), dtype=torch.bool, device=DEVICE)
    for a, b in ((0, 1), (1, 2), (2, 0)):
        dx, dy = sx[:, b] - sx[:, a], sy[:, b] - sy[:, a]
        own = (dy < 0) | ((dy == 0) & (dx > 0))
        inside &= dx * (qy - sy[:, a]) - dy * (qx - sx[:, a]) >= torch.where(own, 0, 1)
    k, px, py, qx, qy, sx, sy, sz = (v[inside] for v in (k, px, py, qx, qy, sx, sy, sz))
    # the depth plane, in fp32 as the rasteriser pins it
    dx1, dy1, dx2, dy2 = (v.float() for v in (sx[:, 1] - sx[:, 0], sy[:, 1] - sy[:, 0], sx[:, 2] - sx[:, 0],
                                              sy[:, 2] - sy[:, 0]))
    ra = 1.0 / ((sx[:, 1] - sx[:, 0]) * (sy[:, 2] - sy[:, 0]) - (sy[:, 1] - sy[:, 0]) * (sx[:, 2] - sx[:, 0])).float()
    dz1, dz2 = sz[:, 1] - sz[:, 0], sz[:, 2] - sz[:, 0]
    pa, pb = (dz1 * dy2 - dz2 * dy1) * ra, (dz2 * dx1 - dz1 * dx2) * ra
    fma = lambda a, b, c: (a.double() * b.double() + c.double()).float()  # noqa: E731
    depth = fma(pa, (qx - sx[:, 0]).float(), fma(pb, (qy - sy[:, 0]).float(), sz[:, 0]))
    bits = depth.clamp(0, 1).view(torch.int32).to(torch.int64)
    best = torch.full((w * h,), -1, dtype=torch.int64, device=DEVICE)
    best.scatter_reduce_(0, py * w + px, (bits << 32) | keep[k], "amax")
    return torch.where(best < 0, best, best & 0xFFFFFFFF)


def _exact_adjoint(case, seed):
    sizes = _adjoint_sizes(case)
    # On displaced and very fine meshes the sums hang on a few edge-on
    # slivers whose barycentrics (far outside [0, 1] where the snapped
    # triangle covers a pixel centre that the exact one misses) have no digit
    # in common with 64 bits.
    if case["displace"] or case["level"] > 6:
        return None
    r = Renderer(0)
    i, o, images, cut, _ = _adjoint_targets(case, seed, r)  # the target images are inputs
    mesh, T = i["mesh"], case["texture"]
    tri = torch.tensor(np.asarray(mesh.indices, np.int64), device=DEVICE)
    P = i["positions"].double().requires_grad_()
    C = i["colors"].double().requires_grad_()
    X = i["texture"].double().reshape(-1, 3).requires_grad_()
    UV = torch.tensor(mesh.uvs, device=DEVICE).double()
    rgb = torch.zeros(3 * int(o[-1]), dtype=torch.float64, device=DEVICE)
    total = 0.0
    for j, (w, h) in enumerate(sizes):
        vp = np.frombuffer(scene.camera_bytes(i["cams"][j]).tobytes(), np.float32)[32:48].copy()
        vis = _visible64(i["positions"], tri, vp, w, h)
        at = torch.nonzero(vis >= 0).reshape(-1)
        t = tri[vis[at]]
        # the sample point is the fp32 NDC of the pixel centre
        nx = (((at % w).float() + 0.5) / w * 2 - 1).double()[:, None]
        ny = (((at // w).float() + 0.5) / h * 2 - 1).double()[:, None]
        m = torch.tensor(vp, device=DEVICE).double().reshape(4, 4)
        q = P[t]
        cx, cy, cw = (q @ m[:3, k] + m[3, k] for k in (0, 1, 3))
        a, b = cx - nx * cw, cy - ny * cw
        lam = torch.linalg.cross(a, b)
        s = lam.sum(1, keepdim=True)
        lam = lam / s
        col, uv = (lam[:, :, None] * C[t]).sum(1), (lam[:, :, None] * UV[t]).sum(1)
        xy = uv * T - 0.5
        f = torch.floor(xy.detach())
        ax, ay = (xy[:, 0] - f[:, 0])[:, None], (xy[:, 1] - f[:, 1])[:, None]
        x0, y0 = f[:, 0].to(torch.int64) % T, f[:, 1].to(torch.int64) % T
        x1, y1 = (x0 + 1) % T, (y0 + 1) % T
        tex = ((X[y0 * T + x0] * (1 - ax) + X[y0 * T + x1] * ax) * (1 - ay)
               + (X[y1 * T + x0] * (1 - ax) + X[y1 * T + x1] * ax) * ay)
        out = col * tex
        target = cut["target"][j].double().reshape(-1, 3)
        loss = i["scale"] * (out - target[at]).square().sum()
        loss.backward()
        img = rgb[3 * int(o[j]):3 * (int(o[j]) + w * h)].reshape(-1, 3)
        img[at] = out.detach()
        empty = vis < 0
        total += float(loss.detach()) + i["scale"] * float(target[empty].square().sum())
    torch.cuda.synchronize()
    return dict(rgb=rgb, loss=torch.tensor([total], dtype=torch.float64), positions=P.grad, colors=C.grad,
                texture=X.grad.reshape(T, T, 3))


def exact(case, seed):
    if case["kind"] == "world":
        return _exact_world(case, seed)
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed)
    return None

"""The work that programs have this library do, as cases that can be timed and compared.

`listed()` names twelve cases, `draw(rng)` gives further ones of the same ranges.  `prepare` makes
what a program holds before the call (scenes, rays, cameras, buffers, captured frames), `run` is one
pass through the package's public entry points, `work` the bytes and operations a pass cannot do
without, and `exact` the values of a pass's computed outputs in 64 bits where plain torch gives them.

Kinds of cases:
  query    host rays through CudaOctree.castRays: picking, line-of-sight and physics probes of a
           program that holds its rays in host memory; one to a few thousand rays
  cast     Scene.cast_rays_dev: primary rays of a camera (pixel rows or 8 x 4 tiles) or incoherent
           rays (ambient probes), with the colour payload, with or without a level-of-detail cone
  render   Scene.render_dev: ray generation, cast and shading of a frame into an RGBA8 image
  shadow   a camera's primary rays and the compacted shadow ray of every hit (city scenes)
  batch    Batch.cast: the rays of several scenes in one launch
  frame    Batch.capture_frame_compact / launch_frame: the primary rays of many scenes and two bounce
           rays per hit as one CUDA graph
  train    one step of fitting colours to images: forward views, gradient cleared, adjoint
  adjoint  the backward pass alone, from recorded hits (images of a closed surface)
  encode   the compressed payloads of a scene's bricks: normals, and material ids to DXT1 colours
  scene    a procedural scene from nothing to its first image: noise, octree, payloads, render

Scenes are the ones this repository measures itself on: value noise at 10 to 50 % fill and city
grids, 64 to 2048 voxels a side.  Hits come back as 32-bit words (t's bits among them), which are
whole numbers: they have no 64-bit counterpart, the traversal being defined in binary32.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    """The repository's package (its folder's name is not an identifier) and its workload builders."""
    if "vx_b200" not in sys.modules:
        folder = os.path.join(_ROOT, "vbvs--vixen_b200")
        spec = importlib.util.spec_from_file_location("vx_b200", os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        module = importlib.util.module_from_spec(spec)
        sys.modules["vx_b200"] = module
        spec.loader.exec_module(module)
    from vx_b200 import workloads
    return sys.modules["vx_b200"], workloads


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # a single pick against a small scene: latency of the whole host call
        {"name": "query_1", "kind": "query", "R": 256, "fill": 0.1, "rays": 1},
        # the small plain configuration: 256^3 with a box shell, RGBA8, 512 x 512 primary rays in pixel rows
        {"name": "cast_256_512sq", "kind": "cast", "R": 256, "fill": 0.1, "shell": True, "color": "rgba8",
         "rays": "camera", "width": 512, "height": 512, "fov": 60.0, "order": "rows", "lod": 0.0},
        # the cave configuration: 1024^3 at 50 %, DXT1, a full-HD frame in tile order
        {"name": "cast_1024_1080p", "kind": "cast", "R": 1024, "fill": 0.5, "shell": False, "color": "dxt1",
         "rays": "camera", "width": 1920, "height": 1080, "fov": 70.0, "order": "tiles", "lod": 0.0},
        # incoherent probes with a level-of-detail cone, an odd number of them
        {"name": "cast_lod_probes", "kind": "cast", "R": 512, "fill": 0.3, "shell": False, "color": "dxt1",
         "rays": "random", "count": 1000003, "lod": 0.002},
        # a window of odd size with compressed colours and normals
        {"name": "render_512_ragged", "kind": "render", "R": 512, "fill": 0.3, "color": "dxt1", "normals": True,
         "width": 1279, "height": 717, "fov": 70.0},
        # the city configuration: 2048^3, 4K primary rays and a shadow ray per hit
        {"name": "shadow_2048_4k", "kind": "shadow", "R": 2048, "width": 3840, "height": 2160},
        # eight small scenes in one launch: the batched form at its smallest
        {"name": "batch_8", "kind": "batch", "scenes": 8, "max_log_r": 8, "width": 317, "height": 211},
        # the batched frame with bounce rays: 64^3 to 1024^3, noise and city scenes, half of them DXT1
        {"name": "frame_24", "kind": "frame", "scenes": 24, "max_log_r": 10, "width": 1024, "height": 577},
        # the colour-fitting configuration: 512^3, 16 views of 512 x 512, per-voxel colours
        {"name": "train_rgb_16", "kind": "train", "R": 512, "views": 16, "width": 512, "height": 512, "attr": 0},
        # the backward pass of the DXT1 form over views of odd size
        {"name": "adjoint_dxt1", "kind": "adjoint", "R": 256, "views": 5, "width": 333, "height": 251, "attr": 1},
        # payloads of a scene's bricks after an edit
        {"name": "encode_150k", "kind": "encode", "bricks": 150001, "R": 512, "fill": 0.5},
        # a new procedural scene up to its first image
        {"name": "scene_512", "kind": "scene", "R": 512, "fill": 0.3, "color": "dxt1", "normals": True,
         "width": 640, "height": 360},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "cast", "cast", "probes", "render", "shadow", "batch", "frame", "train", "adjoint",
                       "encode", "scene"])
    width, height = _log(rng, 96, 1920), _log(rng, 64, 1080)
    if kind == "query":
        return {"kind": "query", "R": rng.choice([64, 128, 256, 512]), "fill": round(rng.uniform(0.05, 0.5), 3),
                "rays": _log(rng, 1, 5000)}
    if kind == "cast":
        return {"kind": "cast", "R": rng.choice([64, 192, 256, 512, 1024]), "fill": round(rng.uniform(0.05, 0.5), 3),
                "shell": rng.random() < 0.3, "color": rng.choice(["rgba8", "dxt1", "none"]), "rays": "camera",
                "width": width, "height": height, "fov": round(rng.uniform(45.0, 90.0), 1),
                "order": rng.choice(["rows", "tiles"]), "lod": rng.choice([0.0, 0.0, round(rng.uniform(0.0005, 0.01), 5)])}
    if kind == "probes":
        return {"kind": "cast", "R": rng.choice([128, 320, 512, 1024]), "fill": round(rng.uniform(0.05, 0.5), 3),
                "shell": rng.random() < 0.3, "color": rng.choice(["rgba8", "dxt1"]), "rays": "random",
                "count": _log(rng, 1000, 2000000), "lod": rng.choice([0.0, round(rng.uniform(0.0005, 0.01), 5)])}
    if kind == "render":
        return {"kind": "render", "R": rng.choice([64, 192, 256, 512]), "fill": round(rng.uniform(0.05, 0.5), 3),
                "color": rng.choice(["rgba8", "dxt1", "none"]), "normals": rng.random() < 0.5,
                "width": width, "height": height, "fov": round(rng.uniform(45.0, 90.0), 1)}
    if kind == "shadow":
        return {"kind": "shadow", "R": rng.choice([256, 512, 1024]), "width": _log(rng, 320, 3840),
                "height": _log(rng, 200, 2160)}
    if kind == "batch":
        return {"kind": "batch", "scenes": _log(rng, 1, 12), "max_log_r": rng.choice([7, 8, 9]),
                "width": _log(rng, 64, 800), "height": _log(rng, 64, 600)}
    if kind == "frame":
        return {"kind": "frame", "scenes": _log(rng, 2, 16), "max_log_r": rng.choice([8, 9]),
                "width": _log(rng, 128, 1000), "height": _log(rng, 96, 600)}
    if kind == "train":
        return {"kind": "train", "R": rng.choice([128, 256]), "views": _log(rng, 1, 16), "width": _log(rng, 96, 512),
                "height": _log(rng, 96, 512), "attr": rng.choice([0, 1])}
    if kind == "adjoint":
        return {"kind": "adjoint", "R": rng.choice([128, 256]), "views": _log(rng, 1, 16), "width": _log(rng, 96, 512),
                "height": _log(rng, 96, 512), "attr": rng.choice([0, 1])}
    if kind == "encode":
        return {"kind": "encode", "bricks": _log(rng, 100, 150000), "R": rng.choice([64, 128, 192, 256, 320, 512]),
                "fill": round(rng.uniform(0.05, 0.6), 3)}
    return {"kind": "scene", "R": rng.choice([64, 128, 192, 256, 320]), "fill": round(rng.uniform(0.05, 0.5), 3),
            "color": rng.choice(["rgba8", "dxt1"]), "normals": rng.random() < 0.5, "width": _log(rng, 96, 1000),
            "height": _log(rng, 64, 700)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------

def _rng(seed, salt=0):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, salt])


def _generator(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed((int(seed) & 0x7FFFFFFF) * 64 + salt)


def _noise(R):
    """Lattice spacing and octaves of the noise scenes at side R."""
    spacing = max(4, 64 * R // 1024)
    return spacing, 5 if spacing >= 64 else 3


def _noise_bits(vx, R, fill, seed, shell):
    spacing, octaves = _noise(R)
    return vx.synth_noise_dev(R, spacing, octaves, fill, int(seed), shell)


def _city_bits(R, seed, salt=0):
    """32 x 32 solid blocks of uniform random height between streets, as occupancy bits on the device."""
    pitch, street = R // 32, max(1, R // 256)
    low, high = (64, 1800) if R == 2048 else (max(1, R // 32), max(2, R * 1800 // 2048))
    heights = torch.from_numpy(_rng(seed, 70 + salt).integers(low, high + 1, size=(32, 32))).cuda().clamp(max=R)
    x = torch.arange(R, device="cuda")
    y = torch.arange(R, device="cuda")[:, None]
    shift = torch.arange(64, device="cuda")
    words = torch.zeros((32, pitch, R, R // 64), dtype=torch.int64, device="cuda")
    for block in range(32):
        solid = (x % pitch < pitch - street) & (y < heights[block][x // pitch])
        words[block, : pitch - street] = (solid.view(R, R // 64, 64).long() << shift).sum(-1)
    return words.reshape(-1)


def _color_kind(vx, name):
    return {"rgba8": vx.VX_COLOR_RGBA8, "dxt1": vx.VX_COLOR_DXT1, "none": vx.VX_COLOR_NONE}[name]


def _levels(R):
    return int(math.ceil(math.log2(R)))


def _scene(vx, bits, R, color, seed, normals=False):
    return vx.scene_from_dense_dev(bits, R, _levels(R), _color_kind(vx, color), int(seed) ^ 0xD7C1, normals)


def _tiles(width, height):
    """Pixel indices in 32 x 8 tiles of eight 8 x 4 pieces, the order the library recommends for primary rays."""
    tw, th = -(-width // 32), -(-height // 8)
    t = torch.arange(tw * th * 256, device="cuda")
    tile, warp, lane = t // 256, (t % 256) // 32, t % 32
    x = (tile % tw) * 32 + (warp % 4) * 8 + lane % 8
    y = (tile // tw) * 8 + (warp // 4) * 4 + lane // 8
    keep = (x < width) & (y < height)
    return (y * width + x)[keep]


def _camera_rays(vx, camera, width, height, order):
    rays = torch.from_numpy(vx.camera_rays(camera, width, height)).cuda()
    return rays[_tiles(width, height)].contiguous() if order == "tiles" else rays


def _hits(n):
    return torch.zeros((n, 4), dtype=torch.int32, device="cuda")


def _color_out(vx, name, n):
    if name == "none":
        return None
    return torch.zeros((n, 3), dtype=torch.float32, device="cuda") if name == "dxt1" else \
        torch.zeros((n, 1), dtype=torch.int32, device="cuda")


def _probe_rays(n, R, seed):
    """Origins in and around the grid, directions uniform on the sphere, some along an axis."""
    g = _generator(seed, 3)
    o = (torch.rand((n, 3), generator=g, device="cuda") * 1.5 - 0.25) * R
    d = torch.randn((n, 3), generator=g, device="cuda")
    axis = torch.nn.functional.one_hot(torch.randint(0, 3, (n,), generator=g, device="cuda"), 3).float()
    sign = torch.randint(0, 2, (n, 1), generator=g, device="cuda") * 2.0 - 1.0
    along = (torch.arange(n, device="cuda") % 13 == 5)[:, None]
    return torch.cat([o, torch.where(along, axis * sign, d)], 1).contiguous()


def _camera_for(W, bits, R, kind, seed, fov, width, height):
    if kind == "city":
        return W.look_camera([R * 0.5, R * 0.9, -R * 0.25], [0.05, -0.45, 1.0], fov, width, height)
    return W.empty_voxel_camera(bits, R, int(seed), fov, width, height)


def _scenes(vx, W, case, seed):
    """The scenes of a batched case and the primary rays of one camera each, with their offsets."""
    rng = _rng(case["scenes"], 11)  # the scenes' sides and the cameras' sizes belong to the case
    scenes, rays, begin = [], [], [0]
    for i in range(case["scenes"]):
        # the first scene has the largest side, the others are log-uniform down to 64
        R = 2 ** (case["max_log_r"] if i == 0 else int(rng.integers(6, case["max_log_r"] + 1)))
        kind = ("noise10", "noise50", "city")[i % 3]
        s = (int(seed) * 131 + i) & 0x7FFFFFFF
        bits = _city_bits(R, s) if kind == "city" else _noise_bits(vx, R, 0.1 if kind == "noise10" else 0.5, s, False)
        scenes.append(_scene(vx, bits, R, "dxt1" if i % 2 else "rgba8", s))
        # cameras between a third of the case's size and all of it
        f = 1.0 if i == 0 else float(rng.uniform(0.35, 1.0))
        w, h = max(8, int(case["width"] * f)), max(8, int(case["height"] * f))
        camera = _camera_for(W, bits, R, kind, s, 60.0 if kind == "city" else 70.0, w, h)
        rays.append(_camera_rays(vx, camera, w, h, "tiles"))
        begin.append(begin[-1] + w * h)
    offsets = torch.tensor(begin, dtype=torch.int64).to(torch.int32).cuda()
    return scenes, torch.cat(rays).contiguous(), offsets


def _orbit(W, rng, R, views, width, height):
    c, phase, cams = R / 2, rng.uniform(0, 2 * np.pi), []
    for v in range(views):
        th = phase + 2 * np.pi * v / views
        pos = [c + 0.95 * R * np.cos(th), c + R * rng.uniform(-0.3, 0.3), c + 0.95 * R * np.sin(th)]
        cams.append(W.look_camera(pos, [c - pos[0], c - pos[1], c - pos[2]], 60.0, width, height))
    return cams


def _surface_records(case, seed):
    """What a forward pass over a closed surface records: views of a sphere of voxels, as hit records
    (t, brick, node, voxel and flags), rendered and target images, and the DXT1 selectors.  Bricks are
    numbered over the whole grid.  Plain torch, so that the 64-bit gradient has the same inputs."""
    R, views, w, h = case["R"], case["views"], case["width"], case["height"]
    rng, bpa = _rng(seed, 21), R // 8
    parts = []
    for v in range(views):
        eye = rng.normal(size=3)
        eye = eye / np.linalg.norm(eye) * 0.95 * R
        fwd = -eye / np.linalg.norm(eye)
        right = np.cross(fwd, [0.0, 1.0, 0.0] if abs(fwd[1]) < 0.9 else [1.0, 0.0, 0.0])
        right /= np.linalg.norm(right)
        up = np.cross(right, fwd)
        e, f, r, u = (torch.from_numpy(a).cuda() for a in (eye, fwd, right, up))
        px = (torch.arange(w, device="cuda", dtype=torch.float64) + 0.5) / w * 2 - 1
        py = 1 - (torch.arange(h, device="cuda", dtype=torch.float64) + 0.5) / h * 2
        tan = math.tan(math.radians(30.0))
        d = f + (px * tan * w / h)[None, :, None] * r + (py * tan)[:, None, None] * u
        d = d / d.norm(dim=-1, keepdim=True)
        b, rad = (d * e).sum(-1), 0.42 * R
        disc = b * b - ((e * e).sum() - rad * rad)
        hit = disc > 0
        t = -b - disc.clamp(min=0).sqrt()
        p = e + d * t[..., None]
        cell = (p + R / 2).floor().long().clamp(0, R - 1)
        axis = p.abs().argmax(-1)
        neg = torch.gather(p, -1, axis[..., None])[..., 0] < 0
        brick = ((cell[..., 2] // 8) * bpa + cell[..., 1] // 8) * bpa + cell[..., 0] // 8
        voxel = (cell[..., 2] % 8) * 64 + (cell[..., 1] % 8) * 8 + cell[..., 0] % 8
        flags = 1 | (axis << 1) | (neg.long() << 3) | 16
        word = torch.where(hit, voxel | (flags << 16) | (7 << 24), torch.full_like(voxel, 0xFFFF))
        none = torch.full_like(voxel, -1)
        rec = torch.stack([torch.where(hit, t, torch.zeros_like(t)).float().view(torch.int32).long(),
                           torch.where(hit, brick, none), torch.where(hit, brick // 8, none), word], -1)
        parts.append(rec.reshape(-1, 4).to(torch.int32))
    g = _generator(seed, 22)
    n = views * w * h
    image = torch.rand((n, 3), generator=g, device="cuda")
    target = image + 0.05 * torch.randn((n, 3), generator=g, device="cuda")
    idx = torch.randint(-2 ** 31, 2 ** 31, (bpa ** 3 * 32,), generator=g, device="cuda", dtype=torch.int64).int()
    return torch.cat(parts).contiguous(), image, target, idx if case["attr"] else None


def _attr_size(case, bricks):
    return bricks * 512 * 3 if case["attr"] == 0 else bricks * 32 * 6


def _brick_occupancy(bits, R):
    """The 16 occupancy words of every brick that holds a voxel (x fastest, 8 voxels a byte row)."""
    b = R // 8
    rows = bits.view(torch.uint8).view(b, 8, b, 8, b).permute(0, 2, 4, 1, 3).reshape(-1, 64)
    return rows[(rows != 0).any(1)].contiguous().view(torch.int32).reshape(-1, 16).contiguous()


def prepare(case, seed):
    vx, W = _package()
    kind = case["kind"]
    s = int(seed) & 0x7FFFFFFF
    st = {"kind": kind, "vx": vx}
    if kind == "query":
        bits = _noise_bits(vx, case["R"], case["fill"], s, True)
        st["octree"] = vx.CudaOctree(_scene(vx, bits, case["R"], "none", s))
        rng, n = _rng(s, 1), case["rays"]
        st["origins"] = (rng.uniform(0.05, 0.95, size=(n, 3)) * case["R"]).astype(np.float32)
        st["directions"] = rng.normal(size=(n, 3)).astype(np.float32)
    elif kind == "cast":
        R = case["R"]
        bits = _noise_bits(vx, R, case["fill"], s, case["shell"])
        st["scene"] = _scene(vx, bits, R, case["color"], s)
        if case["rays"] == "random":
            st["rays"] = _probe_rays(case["count"], R, s)
        else:
            cam = W.empty_voxel_camera(bits, R, s, case["fov"], case["width"], case["height"])
            st["rays"] = _camera_rays(vx, cam, case["width"], case["height"], case["order"])
        n = st["rays"].shape[0]
        st["hits"], st["color"] = _hits(n), _color_out(vx, case["color"], n)
        st["lod"] = vx.LodParams(0.0, case["lod"]) if case["lod"] else None
    elif kind == "render":
        R, w, h = case["R"], case["width"], case["height"]
        bits = _noise_bits(vx, R, case["fill"], s, False)
        st["scene"] = _scene(vx, bits, R, case["color"], s, case["normals"])
        st["camera"] = W.empty_voxel_camera(bits, R, s, case["fov"], w, h)
        st["size"] = (w, h)
        st["image"] = torch.zeros(w * h, dtype=torch.int32, device="cuda")
    elif kind == "shadow":
        R, w, h = case["R"], case["width"], case["height"]
        st["scene"] = _scene(vx, _city_bits(R, s), R, "dxt1", s)
        cam = W.look_camera([R * 0.5, R * 0.9, -R * 0.25], [0.05, -0.45, 1.0], 60.0, w, h)
        st["rays"] = _camera_rays(vx, cam, w, h, "tiles")
        n = w * h
        st["light"] = W.light_dir(s)
        st["hits"], st["color"], st["shadow"] = _hits(n), _color_out(vx, "dxt1", n), _hits(n)
    elif kind in ("batch", "frame"):
        scenes, rays, begin = _scenes(vx, W, case, s)
        st["batch"], st["rays"], st["begin"] = vx.Batch(scenes), rays, begin
        n = rays.shape[0]
        st["hits"] = _hits(n)
        if kind == "frame":
            st["bounce"] = torch.zeros((2 * n, 6), dtype=torch.float32, device="cuda")
            st["bounce_hits"] = _hits(2 * n)
            stream = torch.cuda.Stream()
            stream.wait_stream(torch.cuda.current_stream())
            st["batch"].capture_frame_compact(rays, begin, st["hits"], st["bounce"], st["bounce_hits"], s,
                                              stream.cuda_stream)
            torch.cuda.current_stream().wait_stream(stream)
    elif kind == "train":
        R, w, h, views = case["R"], case["width"], case["height"], case["views"]
        bits = vx.synth_noise_dev(R, max(4, 32 * R // 512), 4 if R >= 512 else 3, 0.3, s, False)
        scene = _scene(vx, bits, R, "none", s)
        bricks = (R // 8) ** 3  # the pool holds every brick slot of the grid, so that an edited scene keeps it
        g = _generator(s, 31)
        attr = torch.rand(_attr_size(case, bricks), generator=g, device="cuda")
        idx = torch.randint(-2 ** 31, 2 ** 31, (bricks * 32,), generator=g, device="cuda",
                            dtype=torch.int64).int() if case["attr"] else None
        n = views * w * h
        st.update(scene=scene, cams=_orbit(W, _rng(s, 32), R, views, w, h), size=(w, h), attr_kind=case["attr"],
                  attr=attr, idx=idx, image=torch.zeros((n, 3), device="cuda"), record=_hits(n),
                  target=torch.zeros((n, 3), device="cuda"), grad=torch.zeros_like(attr),
                  loss=torch.zeros(1, device="cuda"))
        noisy = torch.randn(attr.shape, generator=g, device="cuda").mul_(0.05).add_(attr)
        vx.diff_forward_views(scene, st["cams"], w, h, case["attr"], noisy, idx, st["target"], st["record"])
        del noisy
    elif kind == "adjoint":
        record, image, target, idx = _surface_records(case, s)
        st.update(record=record, image=image, target=target, idx=idx, attr_kind=case["attr"],
                  grad=torch.zeros(_attr_size(case, (case["R"] // 8) ** 3), device="cuda"),
                  loss=torch.zeros(1, device="cuda"))
    elif kind == "encode":
        bits = _noise_bits(vx, case["R"], case["fill"], s, False)
        occ, n = _brick_occupancy(bits, case["R"]), case["bricks"]
        occ = occ[torch.arange(n, device="cuda") % occ.shape[0]].contiguous()
        # material ids of the noise scenes (30 to 40), in runs along x as strata give them
        g = _generator(s, 41)
        ids = torch.randint(30, 41, (n * 128,), generator=g, device="cuda", dtype=torch.int64).int()
        st.update(occ=occ, words=ids.repeat_interleave(4).contiguous(),
                  rgb=torch.zeros(n * 512 * 3, device="cuda"),
                  normals=torch.zeros(n * 64, dtype=torch.int64, device="cuda"),
                  colors=torch.zeros(n * 32, dtype=torch.int64, device="cuda"))
    elif kind == "scene":
        R, w, h = case["R"], case["width"], case["height"]
        # where the camera stands: in the middle of the grid's -z face, looking in
        st.update(R=R, fill=case["fill"], seed=s, color=case["color"], normals=case["normals"], size=(w, h),
                  camera=W.look_camera([R / 2 + 0.5, R / 2 + 0.5, -0.4 * R], [0.02, 0.01, 1.0], 60.0, w, h),
                  bits=torch.zeros(R * R * (R // 64), dtype=torch.int64, device="cuda"),
                  image=torch.zeros(w * h, dtype=torch.int32, device="cuda"), hits=_hits(w * h))
    else:
        raise ValueError("unknown kind of case: %r" % (kind,))
    return st


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------

def run(st):
    vx, kind = st["vx"], st["kind"]
    if kind == "query":
        hits = st["octree"].castRays(st["origins"], st["directions"])
        return hits.view(np.int32).reshape(-1, 4)
    if kind == "cast":
        st["scene"].cast_rays_dev(st["rays"], st["hits"], st["color"], lod=st["lod"])
        return [st["hits"]] if st["color"] is None else [st["hits"], st["color"]]
    if kind == "render":
        st["scene"].render_dev(st["camera"], *st["size"], image=st["image"])
        return st["image"]
    if kind == "shadow":
        st["scene"].cast_rays_dev(st["rays"], st["hits"], st["color"])
        st["scene"].cast_shadow_rays_dev(st["rays"], st["hits"], st["light"], st["shadow"])
        return st["hits"], st["color"], st["shadow"]
    if kind == "batch":
        st["batch"].cast(st["rays"], st["begin"], st["hits"])
        return st["hits"]
    if kind == "frame":
        st["batch"].launch_frame()
        return st["hits"], st["bounce_hits"]
    if kind == "train":
        w, h = st["size"]
        vx.diff_forward_views(st["scene"], st["cams"], w, h, st["attr_kind"], st["attr"], st["idx"], st["image"],
                              st["record"])
        st["grad"].zero_()
        st["loss"].zero_()
        vx.diff_backward(st["attr_kind"], st["idx"], st["record"], st["image"], st["target"], st["grad"], st["loss"])
        return st["image"], st["record"], st["grad"], st["loss"]
    if kind == "adjoint":
        st["grad"].zero_()
        st["loss"].zero_()
        vx.diff_backward(st["attr_kind"], st["idx"], st["record"], st["image"], st["target"], st["grad"], st["loss"])
        return st["grad"], st["loss"]
    if kind == "encode":
        vx.build_normals_dev(st["occ"], st["normals"])
        vx.material_rgb_dev(st["words"], st["rgb"])
        vx.build_dxt1_dev(st["rgb"], st["occ"], st["colors"])
        return st["normals"], st["colors"]
    spacing, octaves = _noise(st["R"])
    vx.synth_noise_dev(st["R"], spacing, octaves, st["fill"], st["seed"], False, st["bits"])
    scene = _scene(vx, st["bits"], st["R"], st["color"], st["seed"], st["normals"])
    scene.render_dev(st["camera"], *st["size"], image=st["image"], hits=st["hits"])
    return st["bits"], st["image"], st["hits"]


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------

# Operations of the shortest useful ray: normalisation, the box test and one brick.
_RAY_FLOPS = 120


def work(case):
    """Bytes: inputs read once and outputs written once (of a scene, what the rays touch depends on the
    view and is left out).  Flops: the arithmetic of a ray that ends at its first brick, or of the
    payload encoders' searches."""
    kind = case["kind"]
    if kind == "query":
        return {"bytes": 40 * case["rays"], "flops": _RAY_FLOPS * case["rays"]}
    if kind == "cast":
        n = case["count"] if case["rays"] == "random" else case["width"] * case["height"]
        out = {"rgba8": 4, "dxt1": 12, "none": 0}[case["color"]]
        return {"bytes": n * (24 + 16 + out), "flops": _RAY_FLOPS * n}
    if kind == "render":
        n = case["width"] * case["height"]
        return {"bytes": 4 * n, "flops": (_RAY_FLOPS + 40) * n}
    if kind == "shadow":
        n = case["width"] * case["height"]
        return {"bytes": n * (24 + 16 + 12 + 16), "flops": _RAY_FLOPS * n}
    if kind in ("batch", "frame"):
        # scenes after the first have (0.35 + 1) / 2 of its side on average: 0.49 of its pixels
        n = int(case["width"] * case["height"] * (1 + 0.49 * (case["scenes"] - 1)))
        if kind == "batch":
            return {"bytes": 40 * n, "flops": _RAY_FLOPS * n}
        return {"bytes": (40 + 32) * n, "flops": 2 * _RAY_FLOPS * n}
    if kind == "train":
        n = case["views"] * case["width"] * case["height"]
        pool = 4 * _attr_size(case, (case["R"] // 8) ** 3)  # the gradient, cleared
        return {"bytes": n * (12 + 16 + 12) + pool, "flops": _RAY_FLOPS * n}
    if kind == "adjoint":
        n = case["views"] * case["width"] * case["height"]
        return {"bytes": n * (16 + 12 + 12) + 4 * _attr_size(case, (case["R"] // 8) ** 3), "flops": 12 * n}
    if kind == "encode":
        bricks = case["bricks"]
        return {"bytes": bricks * (64 + 512 + 2048 + 256), "flops": bricks * 512 * 30}
    # scene: occupancy bits, the octree's and the payloads' arrays, the image and its hits
    bricks = int(0.75 * (case["R"] // 8) ** 3)
    colors = 256 if case["color"] == "dxt1" else 2048
    return {"bytes": case["R"] ** 3 // 8 + bricks * (64 + 16 + colors + (512 if case["normals"] else 0)) +
            20 * case["width"] * case["height"], "flops": 20 * case["R"] ** 3}


# ---------------------------------------------------------------------------
# Values in 64 bits
# ---------------------------------------------------------------------------

def exact(case, seed):
    """The adjoint's gradient and loss in 64 bits.  The other kinds return hits, images and payload
    blocks, whole numbers the binary32 traversal and the block formats define; the colours a cast
    writes beside its hits follow from them."""
    if case["kind"] != "adjoint":
        return None
    record, image, target, idx = _surface_records(case, int(seed) & 0x7FFFFFFF)
    diff = image.double() - target.double()
    grad = torch.zeros(_attr_size(case, (case["R"] // 8) ** 3), dtype=torch.float64, device="cuda")
    word = record[:, 3].long() & 0xFFFFFFFF
    flags, voxel = (word >> 16) & 0xFF, word & 0xFFFF
    hit = (flags & 1) == 1
    brick, voxel, flags = record[hit, 1].long(), voxel[hit], flags[hit]
    light = torch.tensor([1.0, 1.0, -1.0], dtype=torch.float64, device="cuda") / math.sqrt(3.0)
    facing = torch.where((flags & 8) != 0, -1.0, 1.0).double() * light[(flags >> 1) & 3]
    g = 2.0 * diff[hit] * (0.3 + 0.7 * facing.clamp(min=0.0))[:, None]
    if case["attr"] == 0:
        at = (brick * 512 + voxel) * 3
        for ch in range(3):
            grad.index_add_(0, at + ch, g[:, ch].contiguous())
    else:
        block = brick * 32 + (voxel >> 4)
        sel = (idx[block].long() >> (2 * (voxel & 15))) & 3
        w0 = torch.tensor([1.0, 0.0, 2.0 / 3.0, 1.0 / 3.0], dtype=torch.float64, device="cuda")[sel]
        w1 = torch.tensor([0.0, 1.0, 1.0 / 3.0, 2.0 / 3.0], dtype=torch.float64, device="cuda")[sel]
        for ch in range(3):
            grad.index_add_(0, block * 6 + ch, w0 * g[:, ch])
            grad.index_add_(0, block * 6 + 3 + ch, w1 * g[:, ch])
    return grad, (diff * diff).sum().reshape(1)

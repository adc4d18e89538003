"""Performance cases: what a program that uses this library has it do, through the public
entry points (the Python handle, and include/vrt.h where the handle has no device form).

A case is a dict of plain values.  `listed()` names the standing cases, `draw(rng)` gives
further ones over the same ranges, `prepare(case, seed)` builds what a program holds before
the call (resident worlds, a batch, device or pinned buffers), `run(state)` is one pass.

Every record is a packed bit format whose contract is bit-exact (include/vrt.h), so outputs
are returned as their 32-bit words: integers, to be equal word by word.  That includes the
distance of a record and the depth of a G-buffer, float32 values whose bits are part of the
contract.
"""
import ctypes
import math

import numpy as np
import torch

import voxelrt_gb300 as v
from voxelrt_gb300 import capi

SUN = tuple(c / math.sqrt(0.3 ** 2 + 0.8 ** 2 + 0.5 ** 2) for c in (0.3, 0.8, 0.5))
RESOLUTIONS = [(64, 64), (256, 256), (640, 360), (1280, 720)]  # the views of the uneven batch
DEVICE = "cuda:0"


def listed():
    return [
        # a thumbnail or a probe view: one launch, so the call and the longest ray count
        dict(name="frame_64", kind="frame", world="terrain", edge=256, width=64, height=64),
        # one frame of the renderer on the GPU's own traversal, with the G-buffer its shading reads
        dict(name="gbuffer_720p_glsl", kind="gbuffer", world="terrain", edge=512, width=1280, height=720, mode="glsl"),
        # one 1080p frame with sun shadows, a launch per view
        dict(name="shadow_1080p", kind="path", world="terrain", edge=1024, width=1920, height=1080, shadow=True,
             bounces=0, mode="cpu"),
        # many worlds with many cameras each (training environments): the headline workload, scaled
        dict(name="batch_uneven", kind="batch", world="mix", worlds=16, edge=384, max_views=16, width=0, height=0,
             shadow=False, bounces=0, mode="cpu"),
        # a few players in one large world: 1080p, primary and sun rays, one launch
        dict(name="batch_shadow_1080p", kind="batch", world="terrain", worlds=1, edge=1024, max_views=6, width=1920,
             height=1080, shadow=True, bounces=0, mode="cpu"),
        # path tracing: diffuse bounces, incoherent after the first hit
        dict(name="batch_bounces_720p", kind="batch", world="caves", worlds=1, edge=512, max_views=2, width=1280,
             height=720, shadow=False, bounces=4, mode="cpu"),
        # the GPU renderer's whole path (sun rays and bounces) with its anisotropic LODs, odd sizes
        dict(name="batch_path_aniso", kind="batch", world="terrain", worlds=2, edge=512, max_views=2, width=955,
             height=537, shadow=True, bounces=3, mode="aniso"),
        # a large set of explicit rays that the program made on the device (lidar, visibility)
        dict(name="cast_4m", kind="cast", world="mix", edge=512, rays=(1 << 22) + 13, mode="cpu", coherent=False),
        # a game's line-of-sight queries: few rays from host memory and back, each frame
        dict(name="cast_2000_host", kind="cast_host", world="terrain", edge=256, rays=2000, mode="cpu"),
        # moved cameras, and records delivered into pinned host memory (the end-to-end call)
        dict(name="batch_to_host", kind="batch_host", world="mix", worlds=6, edge=256, max_views=8, width=0, height=0,
             shadow=False, bounces=0, mode="cpu"),
        # an editor: a brush stroke, then the next frame
        dict(name="edit_frame", kind="edit", world="terrain", edge=512, edits=24, radius=14, width=640, height=360),
        # a world's sectors synced to the device (loading, streaming), then the first frame
        dict(name="load_frame", kind="load", world="terrain", edge=512, width=640, height=360),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _edge(rng, lo, hi):
    return max(lo, min(hi, 32 * round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 32)))


def _cost(case):
    """Rays of a pass, those of bounces four times (they are incoherent)."""
    return _n_records(case) * (4 if case.get("bounces") else 1)


def draw(rng):
    """One more case: sizes over the listed cases' ranges, odd ones among them, and no more
    rays than the largest of them."""
    most = max(_cost(c) for c in listed())
    while True:
        c = _draw(rng)
        if _cost(c) <= most:
            return c


def _draw(rng):
    kind = rng.choice(["frame", "gbuffer", "path", "batch", "batch", "batch", "cast", "cast_host", "batch_host", "edit",
                       "load"])
    world = rng.choice(["terrain", "mix"])
    edge = _edge(rng, 64, 512)
    width = _log(rng, 64, 1920)
    height = max(1, int(width * rng.uniform(0.5, 1.0)) if width < 1080 else 9 * width // 16)
    mode = rng.choice(["cpu", "cpu", "glsl", "aniso"])
    c = dict(kind=kind, world=world, edge=edge)
    if kind == "frame":
        c.update(width=width, height=height)
    elif kind == "gbuffer":
        c.update(width=width, height=height, mode=mode)
    elif kind == "path":
        c.update(width=width, height=height, mode=mode, shadow=rng.random() < 0.6, bounces=rng.choice([0, 0, 1, 3]))
    elif kind == "batch":
        c.update(mode=mode, shadow=rng.random() < 0.5, bounces=rng.choice([0, 0, 2, 4]))
        if rng.random() < 0.5:  # many views of mixed sizes
            c.update(worlds=_log(rng, 1, 12), edge=_edge(rng, 64, 256), max_views=_log(rng, 1, 8), width=0, height=0)
        else:
            c.update(worlds=rng.randint(1, 2), max_views=rng.randint(1, 2), width=width, height=height)
    elif kind == "cast":
        c.update(rays=_log(rng, 1000, 1 << 22), mode=mode, coherent=rng.random() < 0.3)
    elif kind == "cast_host":
        c.update(rays=_log(rng, 1, 20000), mode=mode)
    elif kind == "batch_host":
        c.update(worlds=_log(rng, 1, 6), edge=_edge(rng, 64, 256), max_views=_log(rng, 1, 8), width=0, height=0,
                 shadow=rng.random() < 0.5, bounces=0, mode=mode)
    elif kind == "edit":
        c.update(edge=_edge(rng, 128, 512), edits=_log(rng, 1, 64), radius=_log(rng, 2, 24), width=640, height=360)
    else:
        c.update(edge=_edge(rng, 64, 512), width=640, height=360)
    return c


def _height(edge):
    return min(edge, 256)


def _data(world, edge, seed):
    """Sectors of a world `edge` voxels long (terrain: at most 256 high)."""
    if world == "mix":
        return v.synth_mix(edge, seed)
    y = _height(edge)
    caves = dict(cave_octaves=3, cave_scale=64.0, cave_threshold=0.35, cave_seed=seed + 1) if world == "caves" else {}
    return v.synth_terrain((edge, y, edge), base=y * 0.42, amplitude=y * 0.25, seed=seed, **caves)


def _camera(rng, world, edge, seed, width, height):
    """Above the ground looking around (terrain), or anywhere looking anywhere (mix)."""
    if world == "mix":
        pos, tgt = rng.uniform(0, edge, 3), rng.uniform(0, edge, 3)
        if np.linalg.norm(tgt - pos) < 1.0:
            tgt = pos + np.array([1.0, 0.0, 0.0])
        return v.look_at(pos, tgt, float(rng.uniform(60, 90)), width, height)
    y = _height(edge)
    x, z = rng.uniform(0.1 * edge, 0.9 * edge, 2)
    h = v.terrain_height(x, z, (edge, y, edge), base=y * 0.42, amplitude=y * 0.25, seed=seed)
    top = min(h + rng.uniform(0.08, 0.24) * y, y - 2.0)
    yaw, pitch = rng.uniform(0, 2 * math.pi), math.radians(rng.uniform(-30, 10))
    d = (math.cos(pitch) * math.cos(yaw), math.sin(pitch), math.cos(pitch) * math.sin(yaw))
    return v.look_at((x, top, z), (x + d[0], top + d[1], z + d[2]), 90.0, width, height)


def _world(data):
    w = v.World(data.sectors, brick_capacity=data.n_bricks + 1024, device=0)
    w.upload(data)
    return w


def _view(cam, case, world=0):
    return v.make_view(cam, world=world, n_bounces=case["bounces"], shadow_dir=SUN if case["shadow"] else None,
                       glsl=case["mode"] == "glsl", aniso=case["mode"] == "aniso")


def _words(n, k):
    return torch.zeros((n, k), dtype=torch.int32, device=DEVICE)


def _projection(width, height):
    """A perspective projection, column-major (near 0.1, far 4096)."""
    f, n, r = 1.0, 0.1, 4096.0
    m = np.zeros((4, 4), np.float32)
    m[0, 0], m[1, 1] = f * height / width, f
    m[2, 2], m[2, 3], m[3, 2] = r / (n - r), n * r / (n - r), -1.0
    return m.T.copy().reshape(16)


def _rays(case, rng, size, seed):
    """Random rays as vrt_ray records, or (coherent) a fan of them from one point."""
    rays = v.random_rays(size, seed, case["rays"])
    if case.get("coherent"):
        n, y = case["rays"], size[1]
        th = np.linspace(0.0, 2 * math.pi, n, endpoint=False)
        el = np.deg2rad(rng.uniform(-50, -20) + rng.uniform(5, 25) * np.cos(th * 16))
        rays["origin"] = np.array([size[0] / 2, 0.85 * y, size[2] / 2], np.float32) + np.float32(0.37)
        rays["dir"] = np.stack([np.cos(th) * np.cos(el), np.sin(el), np.sin(th) * np.cos(el)], -1).astype(np.float32)
    return rays


def _strokes(case, rng, data, cam_target):
    """A brush stroke: spheres along a line on the ground, filled, carved and repainted."""
    e = np.zeros(case["edits"], v.EDIT_DTYPE)
    at = np.array(cam_target, float)
    step = rng.uniform(-1, 1, 3) * case["radius"] * 0.5
    for i in range(case["edits"]):
        e[i]["center"] = np.round(at).astype(np.int32)
        e[i]["radius"] = case["radius"]
        e[i]["material"] = 0 if i % 3 == 1 else int(rng.integers(1, 255))
        e[i]["mode"] = 1 if i % 3 == 2 else 0
        at = np.clip(at + step + rng.uniform(-1, 1, 3), 4, np.array(data.sectors) * 32 - 4)
    return e


def _layout(case):
    """Per world of a batch: its edge and the resolutions of its views.  Without a width they
    are drawn as the uneven batch draws them (edges log-uniform up to the case's, 1 to
    max_views views of mixed resolutions), the same for every seed of a case."""
    n, edge, most = case["worlds"], case["edge"], case["max_views"]
    if case["width"]:
        return [(edge, [(case["width"], case["height"])] * most)] * n
    rng = np.random.default_rng([n, edge, most])
    out = []
    for _ in range(n):
        e = max(64, 32 * round(math.exp(rng.uniform(math.log(64), math.log(edge))) / 32))
        out.append((e, [RESOLUTIONS[int(k)] for k in rng.integers(0, 4, rng.integers(1, most + 1))]))
    return out


def prepare(case, seed):
    seed = int(seed) & 0x3FFFFFFF
    rng = np.random.default_rng(seed)
    kind, edge = case["kind"], case["edge"]
    s = dict(kind=kind, case=case)
    if kind in ("batch", "batch_host"):
        views, datas = [], []
        for i, (e, sizes) in enumerate(_layout(case)):
            datas.append(_data(case["world"], e, seed * 1009 + i))
            for wh in sizes:
                views.append(_view(_camera(rng, case["world"], e, seed * 1009 + i, *wh), case, world=i))
        s["worlds"] = [_world(d) for d in datas]
        s["batch"] = v.Batch(s["worlds"], views)
        if kind == "batch":
            s["out"] = _words(s["batch"].total_records, 4)
        else:
            s["cams"] = [vw.cam for vw in views]
            s["pinned"] = torch.zeros((s["batch"].total_records, 3), dtype=torch.int32, pin_memory=True)
        return s
    data = _data(case["world"], edge, seed)
    s["world"] = w = _world(data)
    size = w.size
    if kind in ("cast", "cast_host"):
        rays = _rays(case, rng, size, seed + 1)
        s["mode"] = dict(glsl=case["mode"] == "glsl", aniso=case["mode"] == "aniso")
        if kind == "cast_host":
            s["rays"] = rays
        else:
            s["rays"] = torch.from_numpy(rays.view(np.int32).reshape(-1, 8)).to(DEVICE)
            s["out"] = _words(case["rays"], 4)
        return s
    cam = _camera(rng, case["world"], edge, seed, case["width"], case["height"])
    if kind == "load":
        s["data"] = data
    if kind == "edit":
        # the stroke lies where the camera looks: the first solid voxel of its centre ray
        hit = w.render_view(cam).reshape(case["height"], case["width"])[case["height"] // 2, case["width"] // 2]
        at = v.unpack_voxel(hit["voxel"]) if hit["voxel"] != v.MISS_VOXEL else np.array(size) * 0.45
        s["edits"] = _strokes(case, rng, data, at)
    if kind == "path":
        s["view"] = _view(cam, case)
        s["out"] = _words(v.view_records(s["view"]), 4)
    elif kind == "gbuffer":
        s["view"] = _view(cam, dict(case, shadow=False, bounces=0))
        s["palette"] = rng.integers(0, 1 << 16, 256).astype(np.uint32)
        s["proj"] = _projection(case["width"], case["height"])
        n = case["width"] * case["height"]
        s["texels"], s["depth"], s["out"] = _words(n, 1), _words(n, 1), _words(n, 4)
    else:
        s["cam"] = cam
        s["out"] = _words(case["width"] * case["height"], 4)
    return s


def run(s):
    kind = s["kind"]
    if kind == "frame":
        s["world"].render_view_device(s["cam"], s["out"])
        return s["out"]
    if kind == "path":
        capi.check(v.lib().vrt_render_path_device(s["world"].handle, ctypes.byref(s["view"]), capi.ptr(s["out"]), None))
        return s["out"]
    if kind == "gbuffer":
        capi.check(v.lib().vrt_render_gbuffer_device(
            s["world"].handle, ctypes.byref(s["view"]), capi.ptr(s["palette"]), capi.ptr(s["proj"]),
            capi.ptr(s["texels"]), capi.ptr(s["depth"]), capi.ptr(s["out"]), None))
        return s["texels"], s["depth"], s["out"]
    if kind == "batch":
        s["batch"].launch(s["out"], graph=True)
        return s["out"]
    if kind == "batch_host":
        s["batch"].update_cameras(s["cams"])
        return s["batch"].run_packed(s["pinned"])
    if kind == "cast":
        s["world"].cast_device(s["rays"], s["case"]["rays"], s["out"], **s["mode"])
        return s["out"]
    if kind == "cast_host":
        return s["world"].cast(s["rays"], **s["mode"]).view(np.int32).reshape(-1, 4)
    if kind == "edit":
        s["world"].edit(s["edits"])
    else:
        s["world"].upload(s["data"])
    s["world"].render_view_device(s["cam"], s["out"])
    return s["out"]


def _n_records(case):
    """Records and rays of a pass (at most one ray per record)."""
    kinds = 1
    if case.get("shadow") and case.get("bounces"):
        kinds = 2 + case["bounces"] + min(case["bounces"], 2)
    elif case.get("shadow") or case.get("bounces"):
        kinds = 1 + (1 if case.get("shadow") else case["bounces"])
    if "rays" in case:
        return case["rays"]
    if case["kind"] not in ("batch", "batch_host"):
        return kinds * case["width"] * case["height"]
    return kinds * sum(w * h for _, sizes in _layout(case) for w, h in sizes)


def _n_bricks(case):
    """Bricks of a terrain (about one per column of 8x8 voxels for every 8 voxels of height
    below the ground) or mixed world."""
    e, y = case["edge"], _height(case["edge"])
    return (e // 8) ** 3 if case["world"] == "mix" else (e // 8) ** 2 * max(1, int(0.48 * y / 8))


def work(case):
    """Bytes: records written once, explicit rays read once, for a load its bricks read once
    and stored once with what the traversal reads, for an edit the bricks of its spheres.
    How many bricks rays touch depends on the world; only the voxel a ray ends on is counted.
    Operations: direction, reciprocals and entry of a ray (about 60) and one DDA step."""
    n = _n_records(case)
    size = {"batch_host": 12 + 12, "cast": 16 + 32, "cast_host": 16 + 32, "gbuffer": 16 + 8}.get(case["kind"], 16)
    b = n * (size + 1)
    if case["kind"] == "load":
        b += _n_bricks(case) * 512 * 2
    if case["kind"] == "edit":
        b += case["edits"] * max(1, round(4.19 * (case["radius"] + 4) ** 3 / 512)) * 512
    return {"bytes": b, "flops": n * 90}


def exact(case, seed):
    """Records, texels and depths are bit formats, compared word by word: a traversal in 64
    bits ends rays on other steps and has no word of them in common by contract."""
    return None

"""The timed cases of the voxel ray tracer: what a program that uses the library has it do.

listed() names the cases, draw() gives more of the same ranges, prepare() makes what a
program holds before the call (worlds, cameras, images, renderers, servers), run() is one
pass through the public entry points, work() the bytes and operations no implementation
can do without.

Worlds are seeded terrain like the library's own scenes (two-octave value-noise heights in
[8, 40], grass/dirt/stone bands with jittered colours, caves where 3-D noise exceeds 0.7),
made on the GPU here so that the largest world takes a fraction of a second, or the
reference app's own level (initVoxels + fixDepthField).  Every output is an image, a voxel
word, an occupancy mask, an index or a count: whole numbers, which have to come out the
same bit for bit.  The light multipliers of the debug case are floats, but which of them a
pixel gets is decided by a binary32 voxel walk, so plain 64-bit arithmetic has no value
for them: exact() has none to give.
"""
from __future__ import annotations

import ctypes as C
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(ROOT, "voxel-rt_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import scenes  # noqa: E402
import serving  # noqa: E402
import vrt  # noqa: E402

DEV = "cuda"
SERVED = serving.RESOLUTIONS


# ---------------------------------------------------------------- cases

def listed():
    return [
        # The smallest scene: a preview or a thumbnail of a 64^3 world, 70 degrees, sun only.
        # Launch cost and the longest single ray count here.
        dict(name="frame_small", kind="frame", W=64, H=64, w=256, h=256, steps=256, lights=0, grazing=False),
        # The ordinary full frame: 1080p, sun + 16 local lights, 1024 steps.
        dict(name="frame_1080p", kind="frame", W=512, H=256, w=1920, h=1080, steps=1024, lights=16, grazing=False),
        # The largest frame: 4K over a 4 GiB world, camera one voxel above the ground looking
        # along it (long grazing rays, 4096 steps).
        dict(name="frame_4k_grazing", kind="frame", W=2048, H=256, w=3840, h=2160, steps=4096, lights=16, grazing=True),
        # Picking and validation: every side output (hit voxel, cast and occlusion bits, exact
        # step counts, light multipliers) of an odd-sized frame over an odd-sized world.
        dict(name="frame_outputs", kind="outputs", W=201, H=77, w=853, h=479, steps=384, lights=7, grazing=False),
        # A frame delivered to the host (a streaming or headless client): uniforms in, image in
        # page-locked memory when the call returns.  A laptop's odd 1366x768.
        dict(name="frame_to_host", kind="host", W=512, H=256, w=1366, h=768, steps=1024, lights=8, grazing=False),
        # The reference app between edits: its level with the depth field, 800x600, 384 steps.
        dict(name="level_frame", kind="level_frame", W=512, H=96, w=800, h=600, lights=3, steps_view=False),
        # The reference app's loop while the player digs: collision and gravity probes, a
        # removed sphere with the depth field refreshed around it, then the frame.
        dict(name="level_step", kind="level_step", W=512, H=96, w=800, h=600, lights=3, radius=7, probes=64),
        # Level start in the reference app: generate the level, apply a saved game's holes, and
        # compute the depth field of the whole world.
        dict(name="level_build", kind="level_build", W=512, H=96, holes=4),
        # Many cameras of uneven size over one world in one call (dataset rendering).
        dict(name="batch_64", kind="batch", W=512, H=256, views=64, lo=240, hi=1080, steps=1024, lights=16),
        # A burst of requests to the server over the four serving worlds: 90 % renders at
        # 360p/720p/1080p into the clients' page-locked buffers, 10 % edits.
        dict(name="serve_burst", kind="serve", requests=24, worlds=4),
        # A single edit of a plain terrain world (a server's or a tool's removeSphere).
        dict(name="edit_sphere", kind="edit", W=512, H=256, radius=8),
        # Loading geometry: a whole world from ordinary host memory (updateGeometry).
        dict(name="upload_world", kind="upload", W=256, H=256, first=0.0, part=1.0, device=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["frame", "frame", "frame", "outputs", "host", "level_frame", "level_frame", "level_step",
                       "level_build", "batch", "serve", "edit", "edit", "upload", "upload"])
    if kind in ("frame", "outputs", "host"):
        W = _log(rng, 48, 1024)
        h = _log(rng, 96, 1440 if kind == "frame" else 1080)
        return dict(kind=kind, W=W, H=rng.randint(48, 256), w=max(64, int(h * rng.uniform(1.0, 1.9))), h=h,
                    steps=_log(rng, 128, 4096), lights=rng.randint(0, 16), grazing=rng.random() < 0.3)
    if kind in ("level_frame", "level_step"):
        h = _log(rng, 120, 1080)
        c = dict(kind=kind, W=rng.randint(96, 512), H=rng.randint(56, 128), w=int(h * rng.uniform(1.0, 1.9)), h=h,
                 lights=rng.randint(0, 8))
        if kind == "level_frame":
            c["steps_view"] = rng.random() < 0.15
        else:
            c["radius"], c["probes"] = rng.randint(1, 12), _log(rng, 1, 4096)
        return c
    if kind == "level_build":
        return dict(kind=kind, W=rng.randint(64, 560), H=rng.randint(56, 128), holes=rng.randint(1, 8))
    if kind == "batch":
        lo = _log(rng, 64, 480)
        return dict(kind=kind, W=rng.choice([128, 200, 512]), H=rng.randint(64, 256), views=_log(rng, 2, 64), lo=lo,
                    hi=rng.randint(lo, 1080), steps=_log(rng, 256, 1024), lights=rng.randint(0, 16))
    if kind == "serve":
        return dict(kind=kind, requests=_log(rng, 4, 40), worlds=rng.randint(1, 4))
    if kind == "edit":
        return dict(kind=kind, W=_log(rng, 64, 1024), H=rng.randint(48, 256), radius=_log(rng, 1, 24))
    part = rng.choice([1.0, rng.random(), rng.random() * 0.01])
    return dict(kind="upload", W=_log(rng, 33, 512), H=rng.randint(33, 256), first=rng.random() * (1.0 - part), part=part,
                device=rng.random() < 0.5)


# ---------------------------------------------------------------- worlds and cameras

def _lattice(g, shape):
    return torch.rand(shape, generator=g, device=DEV)


def _blend(n, period, lo=0, hi=None):
    """Lattice index and smoothstep weight of cells [lo, hi) along one axis."""
    x = torch.arange(lo, n if hi is None else hi, device=DEV)
    f = (x % period).float() / period
    return x // period, f * f * (3.0 - 2.0 * f)


def _noise2(lat, zi, zf, xi, xf):
    a = lat[zi][:, xi] * (1 - xf) + lat[zi][:, xi + 1] * xf
    b = lat[zi + 1][:, xi] * (1 - xf) + lat[zi + 1][:, xi + 1] * xf
    return a * (1 - zf[:, None]) + b * zf[:, None]


class Terrain:
    """A seeded terrain world: its words on the device (z, y, x order) and column heights."""

    def __init__(self, W, H, seed):
        g = torch.Generator(device=DEV)
        g.manual_seed(seed)
        self.W, self.H = W, H
        n32, n8 = W // 32 + 2, W // 8 + 2
        l32, l8 = _lattice(g, (n32, n32)), _lattice(g, (n8, n8))
        l3 = _lattice(g, (n8, 7, n8))
        x32, f32 = _blend(W, 32)
        x8, f8 = _blend(W, 8)
        height = (8 + ((_noise2(l32, x32, f32, x32, f32) + 0.5 * _noise2(l8, x8, f8, x8, f8)) / 1.5 * 33).int())
        height = height.clamp(8, 40).clamp(max=H)
        self.words = torch.full((W, H, W), -1, dtype=torch.int32, device=DEV)
        Y = min(H, 40)
        yi, yf = _blend(Y, 8)
        y = torch.arange(Y, device=DEV)
        for z0 in range(0, W, 256):
            z1 = min(W, z0 + 256)
            zi, zf = _blend(W, 8, z0, z1)
            lz = l3[zi] * (1 - zf[:, None, None]) + l3[zi + 1] * zf[:, None, None]
            ly = lz[:, yi] * (1 - yf[:, None]) + lz[:, yi + 1] * yf[:, None]
            cave = ly[:, :, x8] * (1 - f8) + ly[:, :, x8 + 1] * f8
            depth = height[z0:z1, None, :] - 1 - y[:, None]
            j = torch.randint(-8, 9, (3, z1 - z0, Y, W), generator=g, device=DEV, dtype=torch.int32)
            grass, dirt = depth < 3, depth < 11
            r = (torch.where(grass, 10, torch.where(dirt, 120, 90)) + j[0]).clamp(0, 255)
            gr = (torch.where(grass, 130, torch.where(dirt, 100, 90)) + j[1]).clamp(0, 255)
            b = (torch.where(grass, 10, torch.where(dirt, 0, 90)) + j[2]).clamp(0, 255)
            word = 0x01000000 | (r << 16) | (gr << 8) | b
            self.words[z0:z1, :Y] = torch.where((depth >= 0) & (cave <= 0.7), word.int(), -1)
        self.height = height.cpu().numpy()

    def world(self):
        w = vrt.World(self.W, self.H)
        w.upload_device(self.words.data_ptr(), 0, w.num_words)
        return w

    def surface(self, rng, above, margin=0.0):
        lo, hi = int(self.W * margin), int(self.W * (1 - margin)) - 1
        x, z = rng.randint(lo, hi), rng.randint(lo, hi)
        return x, int(self.height[z, x]) + above, z


def _sun(rng, W, H):
    y, az = rng.uniform(0.05, 1.0), rng.uniform(0.0, 2.0 * math.pi)
    r = math.sqrt(1.0 - y * y)
    d = (r * math.cos(az), y, r * math.sin(az))
    return [c / 2.0 + 3.0 * W * d[i] for i, c in enumerate((W, H, W))]


def _lights(rng, ter, n):
    out = []
    for _ in range(n):
        x, y, z = ter.surface(rng, rng.randint(2, 6))
        out.append(((x + 0.5, y + 0.5, z + 0.5), [rng.uniform(0.5, 1.0) for _ in range(3)]))
    return out


def _camera(rng, ter, w, h, steps, lights, sun, grazing=False):
    """A camera just above the ground with the world's lights, as the benchmark scenes have it."""
    u = scenes.base_uniforms(w, h, steps, 70.0, 32.0)
    scenes.set_lights(u, lights)
    x, y, z = ter.surface(rng, 1 if grazing else 2, 0.25)
    scenes.aim(u, (x + 0.5, float(y), z + 0.5), rng.uniform(0.0, 360.0), -2.0 if grazing else rng.uniform(-30.0, 0.0))
    u.lightPos[:] = sun
    return u


def _level(W, H):
    w = vrt.World(W, H)
    w.init_reference()
    return w


def _level_camera(rng, c):
    """The app's uniforms (its sun, 384 steps, 90 degrees) from a seeded spot above the grass."""
    u = scenes.reference_scene_uniforms(rng.uniform(-60.0, -20.0))
    W = c["W"]
    u.aspectRatio = c["w"] / c["h"]
    scenes.aim(u, (rng.uniform(0.3, 0.7) * W, rng.uniform(44.0, 60.0), rng.uniform(0.2, 0.5) * W),
               rng.uniform(-60.0, 60.0), rng.uniform(-25.0, 10.0))
    for _ in range(c["lights"]):
        vrt.place_local_light(u, rng.uniform(0.2, 0.8) * W, rng.uniform(38.0, 50.0), rng.uniform(0.2, 0.8) * W,
                              rng.uniform(0.3, 0.9))
    u.viewDepthField = int(c.get("steps_view", False))
    return u


class _Device:
    """Device memory of a world for torch.as_tensor: the tensor holds this object, which
    holds the world, so the memory lives as long as the tensor does."""

    def __init__(self, world, ptr, n, typestr):
        self.world = world
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (int(ptr), False), "version": 2}


def _contents(world):
    """The world's voxel words and its occupancy masks (bricks, regions), where they lie."""
    i = world.info()
    sw, sh = (world.width + 63) // 64, (world.height + 63) // 64
    n = 64 * sw * sh * sw
    return [torch.as_tensor(_Device(world, i.d_words, int(i.num_words), "<i4"), device=DEV),
            torch.as_tensor(_Device(world, i.d_brick_mask, 64 * n, "<i8"), device=DEV),
            torch.as_tensor(_Device(world, i.d_region_mask, n, "<i8"), device=DEV)]


def _image(w, h):
    return torch.zeros(h * w * 4, dtype=torch.uint8, device=DEV)


# ---------------------------------------------------------------- state

def prepare(case, seed):
    rng = random.Random("%s %d" % (case["kind"], seed))
    s = dict(case)
    kind = case["kind"]
    if kind in ("frame", "outputs", "host"):
        ter = Terrain(case["W"], case["H"], seed)
        s["world"], s["r"] = ter.world(), vrt.Renderer()
        s["u"] = _camera(rng, ter, case["w"], case["h"], case["steps"], _lights(rng, ter, case["lights"]),
                         _sun(rng, case["W"], case["H"]), case["grazing"])
        n = case["w"] * case["h"]
        if kind == "host":
            s["img"] = torch.zeros(n * 4, dtype=torch.uint8, pin_memory=True)
        else:
            s["img"] = _image(case["w"], case["h"])
        if kind == "outputs":
            s["side"] = [torch.zeros(n, dtype=torch.int32, device=DEV) for _ in range(5)]
            s["side"].append(torch.zeros(n * 3, dtype=torch.float32, device=DEV))
            s["dbg"] = vrt.DebugOut(*[t.data_ptr() for t in s["side"]])
            s["stats"] = torch.zeros(vrt.STAT_COUNT, dtype=torch.int64, device=DEV)
    elif kind in ("level_frame", "level_step"):
        w = _level(case["W"], case["H"])
        w.fix_depth_field()
        s["world"], s["r"], s["u"], s["img"] = w, vrt.Renderer(), _level_camera(rng, case), _image(case["w"], case["h"])
        if kind == "level_step":
            # the player digs around: 64 centres in the ground, taken in turn
            s["at"] = 0
            s["centres"] = [(rng.randint(0, case["W"] - 1), rng.randint(28, 38), rng.randint(0, case["W"] - 1))
                            for _ in range(64)]
            xyz = np.array([[rng.randint(-2, case["W"] + 1), rng.randint(20, 60), rng.randint(-2, case["W"] + 1)]
                            for _ in range(case["probes"])], np.int32)
            s["xyz"] = torch.from_numpy(xyz).to(DEV)
            s["found"] = torch.zeros(case["probes"], dtype=torch.int32, device=DEV)
            s["contents"] = _contents(w)
    elif kind == "level_build":
        s["world"] = vrt.World(case["W"], case["H"])
        s["spheres"] = [(rng.randint(0, case["W"] - 1), rng.randint(20, 40), rng.randint(0, case["W"] - 1),
                         rng.randint(3, 9)) for _ in range(case["holes"])]
        s["contents"] = _contents(s["world"])
    elif kind == "batch":
        ter = Terrain(case["W"], case["H"], seed)
        s["world"], s["r"] = ter.world(), vrt.Renderer()
        lights, sun = _lights(rng, ter, case["lights"]), _sun(rng, case["W"], case["H"])
        sizes = random.Random(case["views"])  # the sizes belong to the case, the cameras to the seed
        s["views"], s["imgs"] = [], []
        for _ in range(case["views"]):
            h = _log(sizes, case["lo"], case["hi"])
            w = int(round(h * sizes.choice([4.0 / 3.0, 16.0 / 9.0])))
            u = _camera(rng, ter, w, h, case["steps"], lights[: rng.randint(0, case["lights"])], sun)
            s["imgs"].append(_image(w, h))
            s["views"].append(vrt.make_view(s["world"], u, w, h, s["imgs"][-1].data_ptr()))
    elif kind == "serve":
        _prepare_serve(s, case, seed, rng)
    elif kind == "edit":
        ter = Terrain(case["W"], case["H"], seed)
        s["world"] = ter.world()
        s["at"] = 0
        s["centres"] = [ter.surface(rng, -1) for _ in range(64)]
        s["contents"] = _contents(s["world"])
    elif kind == "upload":
        ter = Terrain(case["W"], case["H"], seed)
        n = case["W"] * case["H"] * case["W"]
        s["first"] = int(case["first"] * n)
        s["count"] = max(1, min(n - s["first"], int(case["part"] * n)))
        words = ter.words.reshape(-1)[s["first"]: s["first"] + s["count"]].clone()
        s["words"] = words if case["device"] else words.cpu().numpy()
        s["world"] = vrt.World(case["W"], case["H"])
        s["contents"] = _contents(s["world"])
    else:
        raise ValueError(kind)
    return s


class _Server(serving.Server):
    """A server that is closed with the state that holds it."""

    def __del__(self):
        self.close()


SERVE_WORLDS = [(256, 256), (512, 256), (1024, 256), (1024, 256)]


def _prepare_serve(s, case, seed, rng):
    plan = random.Random(1000 * case["requests"] + case["worlds"])  # request kinds and sizes belong to the case
    s["server"] = _Server(40 << 30, max_batch_pixels=1920 * 1080)
    s["world"], wids, scenery = [], [], []
    for k, (W, H) in enumerate(SERVE_WORLDS[: case["worlds"]]):
        ter = Terrain(W, H, seed * 7 + k)
        s["world"].append(ter.world())
        ter.words = None
        wids.append(s["server"].add_world(s["world"][-1]))
        scenery.append((ter, _lights(rng, ter, 16), _sun(rng, W, H)))
    s["requests"], s["imgs"], s["edits"] = [], [], []
    for tag in range(case["requests"]):
        k = plan.randrange(case["worlds"])
        ter, lights, sun = scenery[k]
        q = vrt.Request()
        q.world_id, q.user_tag = wids[k], tag
        if plan.random() < 0.9:
            w, h = plan.choice(SERVED)
            q.kind, q.width, q.height = vrt.REQ_RENDER, w, h
            q.uniforms = _camera(rng, ter, w, h, 1024, lights[: rng.randint(0, 16)], sun)
            s["imgs"].append(torch.zeros(w * h * 4, dtype=torch.uint8, pin_memory=True))
            q.host_rgba = s["imgs"][-1].data_ptr()
        else:
            q.kind, q.radius = vrt.REQ_EDIT, plan.randint(1, 8)
            s["edits"].append((q, [ter.surface(rng, -1) for _ in range(16)]))
        s["requests"].append(q)
    s["at"] = 0


# ---------------------------------------------------------------- one pass

def run(s):
    kind = s["kind"]
    if kind == "frame" or kind == "level_frame":
        s["r"].render(s["world"], s["u"], s["w"], s["h"], s["img"].data_ptr())
        return s["img"]
    if kind == "host":
        s["r"].render_to_host(s["world"], s["u"], s["w"], s["h"], s["img"].data_ptr())
        return s["img"]
    if kind == "outputs":
        s["stats"].zero_()
        s["r"].render(s["world"], s["u"], s["w"], s["h"], s["img"].data_ptr(), s["dbg"], s["stats"].data_ptr())
        # rays, iterations, hits and pixels; the counters after them describe the traversal
        # structure, not the frame
        return [s["img"], s["side"], s["stats"][:4]]
    if kind == "level_step":
        x, y, z = s["centres"][s["at"] % 64]
        s["at"] += 1
        w = s["world"]
        w.probe(s["xyz"].data_ptr(), s["probes"], s["found"].data_ptr())
        w.remove_sphere(x, y, z, s["radius"], 1)
        s["r"].render(w, s["u"], s["w"], s["h"], s["img"].data_ptr())
        return [s["found"], s["img"], s["contents"]]
    if kind == "level_build":
        w = s["world"]
        w.init_reference()
        for x, y, z, r in s["spheres"]:
            w.remove_sphere(x, y, z, r, 0)
        w.fix_depth_field()
        return s["contents"]
    if kind == "batch":
        s["r"].render_batch(s["views"])
        return s["imgs"]
    if kind == "serve":
        for q, centres in s["edits"]:
            q.cx, q.cy, q.cz = centres[s["at"] % 16]
        s["at"] += 1
        for q in s["requests"]:
            s["server"].submit(q)
        rays = [0] * len(s["requests"])
        for c in s["server"].drain():
            rays[c.user_tag] = c.rays
        return [s["imgs"], np.array(rays, np.int64)]
    if kind == "edit":
        x, y, z = s["centres"][s["at"] % 64]
        s["at"] += 1
        s["world"].remove_sphere(x, y, z, s["radius"], 0)
        return s["contents"]
    if kind == "upload":
        if s["device"]:
            s["world"].upload_device(s["words"].data_ptr(), s["first"], s["count"])
        else:
            s["world"].upload(s["words"], s["first"])
        return s["contents"]
    raise ValueError(kind)


# ---------------------------------------------------------------- what a pass cannot do without

# Per pixel of a frame: the image word, the colour word of a hit, and the walk: on the
# 1080p terrain frame the rays that can still hit something make 49 voxel steps per pixel,
# each three compares and one add, and about 100 operations set the pixel's rays up and
# shade it.
PIXEL_BYTES, PIXEL_FLOPS = 8, 49 * 4 + 100


def _frame(pixels):
    return {"bytes": PIXEL_BYTES * pixels, "flops": PIXEL_FLOPS * pixels}


def _edit_bytes(radius):
    """The sphere's words and a bit per voxel of its bounding box, written."""
    return int(4.19 * radius ** 3) * 4 + radius ** 3


def work(case):
    kind = case["kind"]
    if kind in ("frame", "outputs", "host", "level_frame", "level_step"):
        f = _frame(case["w"] * case["h"])
        if kind == "outputs":
            f["bytes"] += 8 * 4 * case["w"] * case["h"]
        if kind == "level_step":
            f["bytes"] += _edit_bytes(case["radius"]) + 8 * (case["radius"] + 3) ** 3 * 4 + 16 * case["probes"]
        return f
    if kind == "level_build":  # words and masks written
        n = case["W"] * case["H"] * case["W"]
        return {"bytes": 4 * n + n // 8, "flops": 0}
    if kind == "batch":
        sizes = random.Random(case["views"])
        px = 0
        for _ in range(case["views"]):
            h = _log(sizes, case["lo"], case["hi"])
            px += h * int(round(h * sizes.choice([4.0 / 3.0, 16.0 / 9.0])))
        return _frame(px)
    if kind == "serve":
        plan = random.Random(1000 * case["requests"] + case["worlds"])
        px, edits = 0, 0
        for _ in range(case["requests"]):
            plan.randrange(case["worlds"])
            if plan.random() < 0.9:
                w, h = plan.choice(SERVED)
                px += w * h
            else:
                edits += _edit_bytes(plan.randint(1, 8))
        f = _frame(px)
        f["bytes"] += edits
        return f
    if kind == "edit":
        return {"bytes": _edit_bytes(case["radius"]), "flops": 0}
    n = case["W"] * case["H"] * case["W"]
    n = max(1, min(n, int(case["part"] * n)))
    return {"bytes": 8 * n + n // 8, "flops": 0}


def exact(case, seed):
    """None: every output is a whole number, or (the light multipliers) hangs on a binary32
    voxel walk that 64-bit arithmetic would take elsewhere."""
    return None

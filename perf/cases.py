"""What a program has this library do, as measurable cases: whole bakes from host arrays
(`dl.bake`), bakes of a resident scene to the `.dynlight` payload (`dl.Session`), and the
non-allocating bounce filter on device buffers.

The scenes are the repository's seeded generators (`scenes.py`) at the sizes of the benchmark's
workloads and of slices of them, a room lit by every kind of light, and a clearing of alpha-tested
cards; a seed other than the first gives another scene of the same kind and size."""
import ctypes as C
import math
import warnings

import numpy as np
import torch

from __graft_entry__ import load_package

dl = load_package()
from dynlight_gb300 import scenes  # noqa: E402

warnings.filterwarnings("ignore", message="The given NumPy array is not writable")  # payloads are read


def listed():
    return [
        # an engine filtering one object's bounce window on its frame thread: launch latency
        dict(name="filter_window", kind="filter", width=61, height=45, map_size=128),
        # the same on the largest window the call takes
        dict(name="filter_largest", kind="filter", width=512, height=512, map_size=1024),
        # the smallest bake a level designer waits for: one room, point lights, direct light only
        dict(name="room_direct", kind="room", density=8.0, lights=4),
        # one room under every kind of light, with bounce and the maps for moving objects
        dict(name="room_every_light", kind="mixed", density=12.0, lights=5, sky_samples=64, sun_map=1024,
             probe_spacing=0.5, bounce_samples=32, bits=8, colored=False),
        # an interior level: 36 rooms, local lights with one bounce
        dict(name="rooms_bounce", kind="rooms", rooms=6, boxes=20, lights=64, samples=64, density=16.0, bits=8,
             colored=False),
        # a smaller one shipped compactly: dithered 5-bit colored bounce, an odd sample count
        dict(name="rooms_dithered", kind="rooms", rooms=3, boxes=12, lights=17, samples=45, density=14.0, bits=5,
             colored=True),
        # an interior under panels and tubes: soft shadows, no bounce
        dict(name="rooms_soft", kind="soft", rooms=6, boxes=20, lights=128, density=16.0),
        # a terrain tile baked from host arrays while editing: the whole call, upload and BVH included
        dict(name="terrain_tile", kind="terrain", grid=97, chunks=2, boxes=36, lights=2, sky_samples=256,
             sun_samples=32, bounce_samples=128, density=4.0, form="batched", whole=True),
        # the full outdoor level: soft sun with colored bounce, sky, point lights
        dict(name="terrain_level", kind="terrain", grid=512, chunks=8, boxes=2000, lights=32, sky_samples=256,
             sun_samples=32, bounce_samples=128, density=4.0, form="batched", whole=False),
        # a final bake whose bounce follows binary64, with sample counts that are no powers of two
        dict(name="terrain_bounce_refined", kind="terrain", grid=193, chunks=4, boxes=250, lights=8, sky_samples=200,
             sun_samples=24, bounce_samples=96, density=4.0, form="bounce_refined", whole=False),
        # decals and slivers under many mixed lights, every ray query refined
        dict(name="decals_refined", kind="stress", grid=193, decals=6000, slivers=900, boxes=80, lights=40,
             sky_samples=128, area_samples=32, bounce_samples=64, density=4.0, form="refined"),
        # foliage: alpha-tested cards under a sun, a sky and a lamp
        dict(name="foliage", kind="foliage", cards=600, side=24.0, texture=64, density=8.0, sky_samples=128,
             bounce_samples=64, bits=6, colored=True),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["filter", "room", "mixed", "rooms", "soft", "terrain", "terrain", "stress", "foliage"])
    if kind == "filter":
        width = log(5, 1024)
        height = min(log(5, 1024), 512 * 512 // width)
        return dict(kind=kind, width=width, height=height, map_size=max(width, height) + log(1, 1024))
    if kind == "room":
        return dict(kind=kind, density=round(rng.uniform(4.0, 24.0), 2), lights=log(1, 16))
    if kind == "mixed":
        return dict(kind=kind, density=round(rng.uniform(6.0, 20.0), 2), lights=log(1, 12),
                    sky_samples=rng.choice([16, 48, 64, 100, 256]), sun_map=log(64, 2048),
                    probe_spacing=round(rng.uniform(0.4, 1.5), 2), bounce_samples=rng.choice([12, 32, 50, 64]),
                    bits=rng.choice([4, 5, 6, 8]), colored=rng.random() < 0.5)
    if kind == "rooms":
        return dict(kind=kind, rooms=rng.randint(1, 5), boxes=log(2, 20), lights=log(2, 50),
                    samples=rng.choice([16, 33, 45, 64, 80]), density=round(rng.uniform(8.0, 16.0), 2),
                    bits=rng.choice([4, 5, 6, 8]), colored=rng.random() < 0.5)
    if kind == "soft":
        return dict(kind=kind, rooms=rng.randint(1, 5), boxes=log(2, 20), lights=log(4, 120),
                    density=round(rng.uniform(8.0, 16.0), 2))
    if kind == "terrain":
        grid = log(50, 400)
        return dict(kind=kind, grid=grid, chunks=2 if grid < 130 else rng.randint(2, 8),
                    boxes=min(36, grid * grid // 100) if grid < 130 else grid * grid // rng.randint(130, 600),
                    lights=rng.randint(1, 20), sky_samples=rng.choice([32, 64, 100, 128, 200, 256]),
                    sun_samples=rng.choice([16, 24, 32]), bounce_samples=rng.choice([20, 32, 64, 96, 128]),
                    density=round(rng.uniform(2.0, 4.0), 2),
                    form=rng.choice(["batched", "batched", "batched", "bounce_refined", "refined"]),
                    whole=grid < 130)
    if kind == "stress":
        grid = log(64, 256)
        return dict(kind=kind, grid=grid, decals=log(200, 8000), slivers=log(50, 1200), boxes=rng.randint(0, 120),
                    lights=log(4, 60), sky_samples=rng.choice([32, 100, 128]), area_samples=rng.choice([16, 25, 32]),
                    bounce_samples=rng.choice([32, 45, 64]), density=round(rng.uniform(2.0, 4.0), 2),
                    form=rng.choice(["batched", "refined"]))
    return dict(kind=kind, cards=log(20, 1500), side=round(rng.uniform(8.0, 32.0), 1), texture=log(8, 200),
                density=round(rng.uniform(4.0, 10.0), 2), sky_samples=rng.choice([32, 64, 100, 128]),
                bounce_samples=rng.choice([24, 32, 64, 100]), bits=rng.choice([4, 5, 6, 8]),
                colored=rng.random() < 0.5)


# ---- scenes -------------------------------------------------------------------------------------

def _sun(light_id, samples):
    return dl.BakeLight(id=light_id, position=(0.0, 0.0, 0.0), radius=1.0, illumination=dl.SINGLE_BOUNCE,
                        bounce=dl.BakeBounce(samples=samples),
                        shape=dl.LightShape.sun(scenes.rotation_arc((0, 0, 1), (0.35, 1.0, 0.25)), 0.53))


def _sky(light_id):
    return dl.BakeLight(id=light_id, position=(0.0, 0.0, 0.0), radius=1.0, shape=dl.LightShape.sky())


def _mixed(case, seed):
    inp, _ = scenes.small_room(seed=seed, lights=case["lights"])
    for light in inp.lights:
        light.illumination = dl.SINGLE_BOUNCE
        light.bounce = dl.BakeBounce(samples=case["bounce_samples"])
    rng = scenes.Rng(seed * 5 + 1)
    down = scenes.rotation_x(-math.pi / 2)
    inp.lights += [
        dl.BakeLight(id=800, position=(rng.uniform(-2, 2), 3.6, rng.uniform(-2, 2)), radius=7.0,
                     shape=dl.LightShape.rectangle(down, 1.5, 0.8)),
        dl.BakeLight(id=801, position=(rng.uniform(-3, 3), 3.0, rng.uniform(-3, 3)), radius=6.0,
                     shape=dl.LightShape.tube(scenes.rotation_y(rng.uniform(0, 3.0)), 2.0)),
        _sun(802, case["bounce_samples"]), _sky(803)]
    return inp, dl.BakeOptions(pixel_density=case["density"], sky_samples=case["sky_samples"],
                               sun_map_resolution=case["sun_map"], sky_probe_spacing=case["probe_spacing"],
                               bounce_compression=case["bits"], colored_bounce=case["colored"],
                               dynamic_geometry=dl.ANGULAR)


def _foliage(case, seed):
    """A square of ground, `cards` upright leaf cards with a cut-out texture in four meshes, and
    eight trunks."""
    rng = np.random.default_rng(seed)
    side, n = case["side"], case["cards"]
    ground = scenes.atlas_mesh(1, [scenes.grid_quad((-side / 2, 0, -side / 2), (side, 0, 0), (0, 0, side), 24, 24,
                                                    (0, 1, 0))], (0.3, 0.4, 0.2))
    meshes = [ground]
    size = case["texture"]
    y, x = np.mgrid[0:size, 0:size] / size
    leaf = (np.sin(x * 23.0 + seed % 7) * np.sin(y * 19.0) > -0.2).astype(np.uint8) * 255
    rgba = np.stack([leaf, leaf, leaf, leaf], -1)
    for m in range(4):
        count = max(1, n // 4)
        turn = rng.uniform(0, 2 * math.pi, count)
        base = np.stack([rng.uniform(-0.48, 0.48, count) * side, rng.uniform(0.1, 2.5, count),
                         rng.uniform(-0.48, 0.48, count) * side], -1)
        across = np.stack([np.cos(turn), np.zeros(count), np.sin(turn)], -1) * rng.uniform(0.4, 1.2, count)[:, None]
        up = np.stack([rng.uniform(-0.2, 0.2, count), np.ones(count), rng.uniform(-0.2, 0.2, count)], -1)
        corners = np.stack([base, base + across, base + across + up, base + up], 1)
        mesh = scenes._atlas_triangles(2 + m, corners, True, (0.2, 0.6, 0.2))
        mesh.uv0 = np.tile(np.float32([[0, 0], [1, 0], [1, 1], [0, 1]]), (count, 1))
        mesh.alpha = dl.AlphaTexture(size, size, rgba.reshape(-1), 0.5)
        meshes.append(mesh)
    for k in range(8):
        cx, cz = rng.uniform(-0.45, 0.45, 2) * side
        meshes.append(scenes.atlas_mesh(20 + k, scenes.box_parts((cx - 0.15, -0.1, cz - 0.15),
                                                                (cx + 0.15, 3.0, cz + 0.15)), (0.4, 0.3, 0.2)))
    lamp = dl.BakeLight(id=60, position=(0.0, 2.5, 0.0), radius=9.0, illumination=dl.SINGLE_BOUNCE,
                        bounce=dl.BakeBounce(samples=case["bounce_samples"]))
    lights = [_sun(61, case["bounce_samples"]), _sky(62), lamp]
    for light in lights:
        light.transparency = dl.TRANSPARENCY_ENABLED
    return dl.BakeInput(meshes, lights), dl.BakeOptions(
        pixel_density=case["density"], sky_samples=case["sky_samples"], bounce_compression=case["bits"],
        colored_bounce=case["colored"], area_light_samples=32, dynamic_geometry=dl.LIGHTING_ONLY)


def _scene(case, seed):
    """(input, options) of a bake case."""
    kind = case["kind"]
    if kind == "room":
        inp, opts = scenes.small_room(seed=seed, lights=case["lights"])
        opts.pixel_density = case["density"]
    elif kind == "mixed":
        inp, opts = _mixed(case, seed)
    elif kind == "rooms":
        inp, opts = scenes.room_grid(seed=seed, rooms=case["rooms"], boxes_per_room=case["boxes"],
                                     lights=case["lights"], samples=case["samples"])
        opts.pixel_density, opts.bounce_compression = case["density"], case["bits"]
        opts.colored_bounce = case["colored"]
    elif kind == "soft":
        inp, opts = scenes.soft_rooms(seed=seed, rooms=case["rooms"], boxes_per_room=case["boxes"],
                                      lights=case["lights"])
        opts.pixel_density = case["density"]
    elif kind == "terrain":
        inp, opts = scenes.outdoor(seed=seed, grid=case["grid"], chunks=case["chunks"], boxes=case["boxes"],
                                   point_lights=case["lights"], density=case["density"],
                                   sun_samples=case["sun_samples"], sky_samples=case["sky_samples"],
                                   bounce_samples=case["bounce_samples"])
    elif kind == "stress":
        inp, opts = scenes.precision_stress(seed=seed, grid=case["grid"], chunks=4, boxes=case["boxes"],
                                            decals=case["decals"], slivers=case["slivers"], lights=case["lights"],
                                            density=case["density"], area_samples=case["area_samples"],
                                            sky_samples=case["sky_samples"], bounce_samples=case["bounce_samples"])
    else:
        inp, opts = _foliage(case, seed)
    opts.seed = seed
    return inp, opts


def _whole(case):
    """Whether the case is the whole call from host arrays (few meshes), not a resident session."""
    return case.get("whole", case["kind"] in ("room", "mixed", "foliage"))


# ---- the filter's windows -----------------------------------------------------------------------

def _window(case, seed):
    """A gathered bounce map: smooth positive light with unlit patches (zeros)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    h, w = case["height"], case["width"]
    rough = torch.rand((1, 3, max(2, h // 16), max(2, w // 16)), generator=g, device="cuda")
    smooth = torch.nn.functional.interpolate(rough, size=(h, w), mode="bilinear", align_corners=True)[0]
    noise = torch.rand((3, h, w), generator=g, device="cuda")
    lit = torch.rand((h, w), generator=g, device="cuda") > 0.25
    return ((smooth + 0.2 * noise) * lit * (smooth.amax(0) > 0.3)).permute(1, 2, 0).contiguous()


def _place(case):
    """The window's corner in its map."""
    return (case["map_size"] - case["width"]) // 2, case["map_size"] - case["height"]


# ---- measuring ----------------------------------------------------------------------------------

def _buffer_words(case):
    """The words a program sets aside for the result: a level's budget, the same for every scene of
    the case's kind and size (the baked words' number depends on which texels are lit)."""
    kind, bits = case["kind"], 8.0 * (3 if case.get("colored", True) else 1)
    texels = lambda edge, n: n * (1.2 * edge * case["density"] + 11.0) ** 2  # noqa: E731  padded crops
    if kind in ("room", "mixed"):
        per = case["lights"] * (1.0 + (bits if kind == "mixed" else 0.0)) + (64.0 + bits if kind == "mixed" else 0.0)
        maps = case.get("sun_map", 0) ** 2 // 2 + (case["lights"] + 3) * 12288 + 65536
        return int(maps + (texels(10.0, 6) + texels(2.0, 60)) * per / 32)
    if kind in ("rooms", "soft"):
        rooms = case["rooms"] ** 2
        reach = min(case["lights"], 2.5 + 3.0 * case["lights"] / rooms)
        per = reach * (1.0 + bits) + 40.0 if kind == "rooms" else reach * 2.0 + 8.0
        return int(131072 + (texels(0.7, 850 * rooms) + texels(1.0, 12 * rooms * case["boxes"])) * per / 32)
    if kind in ("terrain", "stress"):
        tris = 2 * (case["grid"] - 1) ** 2 + 12 * case["boxes"]
        words = texels(1.0, tris) * 37.0 / 32 + tris * 16.0
        if kind == "stress":
            words = 3.0 * words + 60.0 * (2 * case["decals"] + 4 * case["slivers"]) * (8.0 + case["lights"] / 4)
        return int(131072 + 1.25 * words)
    return int(131072 + (texels(1.3, 2 * case["cards"] + 1200) + texels(3.0, 100)) * (14.0 + 2 * bits) / 32)


def prepare(case, seed):
    if case["kind"] == "filter":
        src = _window(case, seed)
        return dict(kind="filter", lib=dl.load_library(), src=src, out=torch.empty_like(src), size=case["map_size"],
                    at=_place(case), stream=torch.cuda.current_stream())
    inp, opts = _scene(case, seed)
    form = case.get("form", "batched")
    words = torch.zeros(_buffer_words(case), dtype=torch.int32)
    if _whole(case):
        dl.load_library()
        return dict(kind="whole", inp=inp, opts=opts, form=form, words=words)
    return dict(kind="resident", session=dl.Session(inp, opts, form=form), words=words)


def _put(words, at, part):
    """Appends a part of the result to the program's buffer, as one that fills its level file or its
    renderer's storage does."""
    part = torch.from_numpy(part.reshape(-1).view(np.int32))
    words[at:at + part.numel()].copy_(part)
    return at + part.numel()


def run(state):
    if state["kind"] == "filter":
        src, out = state["src"], state["out"]
        h, w = src.shape[:2]
        status = state["lib"].dl_filter_bounce_window_noalloc(
            C.c_void_p(src.data_ptr()), C.c_void_p(out.data_ptr()), w, h, state["at"][0], state["at"][1],
            state["size"], C.c_void_p(state["stream"].cuda_stream))
        if status:
            raise RuntimeError(state["lib"].dl_last_error().decode())
        return out
    words, at = state["words"], 0
    if state["kind"] == "whole":
        # the call and its result, every part of it, into the program's level buffer
        baked = dl.bake(state["inp"], state["opts"], form=state["form"])
        parts = [baked.light_bvh, baked.distance_cubes] + [m.texels for m in baked.sun_maps]
        parts += [baked.sky_probes.words] if baked.sky_probes is not None else []
        for part in parts + [m.triangles for m in baked.meshes]:
            at = _put(words, at, part)
        return dict(words=words, resolutions=np.array([m.resolution for m in baked.meshes]),
                    stats=np.array([v for _, v in sorted(baked.stats.items())]))
    session = state["session"]
    session.run()
    payload, crc = session.encode_payload()
    at = _put(words, at, np.frombuffer(payload, np.uint8))
    return dict(words=words, length=at, crc=crc)


def work(case):
    """A floor: the filter's exact traffic and arithmetic; for bakes, the scene read once and the
    packed words written once, and for each ray its direction and the slab tests and the one
    triangle test that a descent of a binary tree of the occluders takes."""
    if case["kind"] == "filter":
        n = case["width"] * case["height"]
        return dict(bytes=24.0 * n, flops=3.0 * n * 30)
    kind, d2 = case["kind"], case.get("density", 4.0) ** 2
    if kind in ("room", "mixed"):
        area, tris, hard = 360.0 + 5 * 9.0, 72, case["lights"] * 0.6
        soft = (16 * 2 + 30 + case["sky_samples"]) if kind == "mixed" else 0
        bounce = 2 * case["lights"] * 0.5 * case["bounce_samples"] if kind == "mixed" else 0
        bounce += 2 * case["bounce_samples"] if kind == "mixed" else 0
        photons = 6 * 512 * 512 * case["lights"] if kind == "mixed" else 0
    elif kind in ("rooms", "soft"):
        area, tris = case["rooms"] ** 2 * (240.0 + 7.0 * case["boxes"]), case["rooms"] ** 2 * 1230
        reach = min(case["lights"], 3.0 * case["lights"] / case["rooms"] ** 2)
        hard, soft = reach * 0.5, (reach * 8 if kind == "soft" else 0)
        bounce = reach * case["samples"] if kind == "rooms" else 0
        photons = 6 * 512 * 512 * case["lights"] if kind == "rooms" else 0
    elif kind in ("terrain", "stress"):
        area = 1.1 * (case["grid"] - 1) ** 2 + 20.0 * case["boxes"]
        tris = 2 * (case["grid"] - 1) ** 2 + 12 * case["boxes"] + 2 * case.get("decals", 0) + case.get("slivers", 0)
        hard, soft = 0.5, 16 + case["sky_samples"]
        bounce, photons = 1.2 * case["bounce_samples"], 0
    else:
        area, tris = case["side"] ** 2 + 0.8 * case["cards"], 1152 + 2 * case["cards"]
        hard, soft = 0.5, 16 + case["sky_samples"]
        bounce, photons = 2 * case["bounce_samples"], 6 * 512 * 512
    texels = area * d2
    rays = texels * (8 + hard + soft + bounce) + photons
    flops = rays * (50.0 + 24.0 * math.log2(tris) + 30.0)
    return dict(bytes=64.0 * tris + texels * 8.0, flops=flops)


def _exact_filter(case, seed):
    a = _window(case, seed).cpu().numpy()
    (x0, y0), last = _place(case), case["map_size"] - 1
    h, w = a.shape[:2]
    padded = np.zeros((h + 2, w + 2, 3), np.float32)
    padded[1:-1, 1:-1] = a
    out, done = np.zeros((h, w, 3)), np.zeros((h, w), bool)
    for dx, dy in ((0, 0), (-1, -1), (0, -1), (1, -1), (-1, 0), (1, 0), (-1, 1), (0, 1), (1, 1)):
        v = padded[1 + dy:1 + dy + h, 1 + dx:1 + dx + w]
        take = ~done & (v.max(-1) > 0)
        out[take] = v[take]
        done |= take
    taps = np.arange(-3, 4)
    weight = np.exp(-taps * taps / 50.0)
    weight /= weight.sum()
    for axis, start, size in ((1, x0, w), (0, y0, h)):
        total = np.zeros_like(out)
        for k, wk in zip(taps, weight):
            at = np.clip(np.arange(size) + start + k, 0, last) - start
            inside = ((at >= 0) & (at < size)).astype(float)
            v = np.take(out, np.clip(at, 0, size - 1), axis=axis)
            total += wk * v * (inside[None, :, None] if axis else inside[:, None, None])
        out = total
    return out


def exact(case, seed):
    """The filter in binary64; a bake's outputs are whole numbers."""
    return _exact_filter(case, seed) if case["kind"] == "filter" else None

"""The work that programs have this renderer do, as cases to time: single frames of three kinds of
scenes from icons to 3840x2160, a frame in host memory, a frame of solid and alpha-filtered layers, a
batch of mixed frames, the sprite engine's deferred-light frame, instances of dense models, and the
differentiable renderer's step in both of its modes.  Every pass clears what a frame loop clears and
draws through the package's public calls.

`exact` evaluates depth and height images, and the differentiable renderer's images and gradients, in
64 bits with plain torch.  Corners snap to 1/256 pixel and texture positions to 1/256 texel by the
path's own definition (a 32-bit position times 256, truncated), so those roundings are part of the
function; everything else is binary64.  The last row of an odd height and triangles crossing the near
plane follow rules of their own in the reference, and byte images are whole numbers: none of them
has a 64-bit value here.
"""
import dataclasses
import math

import numpy as np
import torch

import dfpsr_gb300 as dfpsr
from dfpsr_gb300 import scenes
from dfpsr_gb300.sprite_pass import BACKGROUND_HEIGHT, DeferredLightPass

FAR = 1000.0  # an orthogonal camera's depth buffer is cleared to its far distance
TILT, PIXELS_PER_TILE = -1.0, 64  # the sprite world's view in the dense-model cases


def listed():
    return [
        # an inventory icon or a preview: one small model, where launches and waits are the cost
        {"name": "icon_64x64", "kind": "frame", "scene": "torus", "width": 64, "height": 64, "size": 10, "threads": 0, "host": False},
        # a small orthogonal view with a light map drawn into page-locked host images, as a program that shows them on a window does
        {"name": "host_ortho_640x480", "kind": "frame", "scene": "ortho", "width": 640, "height": 480, "size": 60, "threads": 0, "host": True},
        # the benchmark's scene of large triangles with heavy overdraw
        {"name": "random_800x600", "kind": "frame", "scene": "random", "width": 800, "height": 600, "size": 20000, "threads": 0, "host": False},
        # the benchmark's headline: a dense terrain mesh at full HD, with the tile shape that the autotuner keeps for it
        {"name": "terrain_1920x1080", "kind": "frame", "scene": "terrain", "width": 1920, "height": 1080, "size": 512, "threads": 128, "host": False},
        # the largest single frame: two million triangles in 4k
        {"name": "terrain_3840x2160", "kind": "frame", "scene": "terrain", "width": 3840, "height": 2160, "size": 1024, "threads": 0, "host": False},
        # a frame of solid models and alpha-filtered particles through renderer_begin / giveTask / end, in an odd-sized window
        {"name": "layers_1281x719", "kind": "layers", "width": 1281, "height": 719, "size": 120, "particles": 1500},
        # many independent frames of mixed sizes in one call (thumbnails, training images)
        {"name": "batch_32_mixed", "kind": "batch", "frames": 32, "triangles": 200000, "threads": 128},
        # the sprite engine's frame at the size that the reference publishes its rate for
        {"name": "sprites_800x600", "kind": "sprites", "width": 800, "height": 600, "sprites": 900, "lights": 6, "cube": 256, "casters": 1000},
        # the benchmark's sprite frame: 4,096 sprites and 16 shadowed lights at full HD
        {"name": "sprites_1920x1080", "kind": "sprites", "width": 1920, "height": 1080, "sprites": 4096, "lights": 16, "cube": 512, "casters": 2000},
        # the sprite world's model instances of one frame
        {"name": "dense_64_instances", "kind": "dense", "width": 1920, "height": 1080, "instances": 64, "major": 80, "minor": 20, "high": False},
        # one optimisation step over the benchmark's 64 views: forward, loss, gradients with atomics
        {"name": "diff_64_views", "kind": "diff", "views": 64, "width": 256, "height": 256, "major": 250, "minor": 100, "texture": 512, "deterministic": False},
        # the reproducible step over a few odd-sized views
        {"name": "diff_sorted_9_views", "kind": "diff", "views": 9, "width": 201, "height": 150, "major": 120, "minor": 50, "texture": 256, "deterministic": True},
    ]


def _between(rng, low, high):
    """A whole number spread over the logarithm of the range."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "layers", "batch", "sprites", "dense", "diff"])
    width = _between(rng, 64, 2560)
    height = max(48, min(1600, int(width * rng.uniform(0.5, 1.0))))
    if kind == "frame":
        scene = rng.choice(["torus", "ortho", "random", "terrain"])
        low, high = {"torus": (8, 200), "ortho": (8, 120), "random": (300, 30000), "terrain": (48, 700)}[scene]
        if scene == "random":  # its overdraw grows with the pixels
            width, height = min(width, 1280), min(height, 960)
        return {"kind": kind, "scene": scene, "width": width, "height": height, "size": _between(rng, low, high),
                "threads": rng.choice([0, 128]), "host": scene == "ortho" and rng.random() < 0.5}
    if kind == "layers":
        return {"kind": kind, "width": min(width, 1920), "height": min(height, 1080), "size": _between(rng, 16, 160), "particles": _between(rng, 50, 2500)}
    if kind == "batch":
        return {"kind": kind, "frames": rng.randint(2, 28), "triangles": _between(rng, 4000, 150000), "threads": rng.choice([0, 128])}
    if kind == "sprites":
        return {"kind": kind, "width": max(128, min(width, 1920)), "height": max(96, min(height, 1080)), "sprites": _between(rng, 30, 4000),
                "lights": rng.randint(1, 12), "cube": rng.choice([64, 200, 256, 333, 512]), "casters": _between(rng, 100, 2000)}
    if kind == "dense":
        return {"kind": kind, "width": max(200, min(width, 1920)), "height": max(150, min(height, 1080)), "instances": _between(rng, 1, 60),
                "major": _between(rng, 12, 80), "minor": _between(rng, 8, 20), "high": rng.random() < 0.5}
    return {"kind": kind, "views": _between(rng, 1, 48), "width": rng.randint(64, 256), "height": rng.randint(64, 256), "major": _between(rng, 20, 250),
            "minor": _between(rng, 10, 100), "texture": rng.choice([64, 128, 256, 512]), "deterministic": rng.random() < 0.5}


# ------------------------------------------------------------------ inputs

def _textured_torus(rng, case, size):
    s = scenes.torus(2 * size, size, width=case["width"], height=case["height"])
    s.colors = rng.uniform(0.4, 1.0, size=s.colors.shape).astype(np.float32)
    s.colors[:, :, 3] = 1.0
    s.diffuse, s.diffuse_levels = scenes.noise_texture(rng, 256), 16
    s.model_to_world = np.concatenate([[0, 0, 0], scenes.random_rotation(rng).reshape(-1)]).astype(np.float32)
    return s


def _frame_scene(case, seed):
    rng = np.random.default_rng(seed)
    if case["scene"] == "random":
        return scenes.random_triangles(seed=seed, triangles=case["size"], width=case["width"], height=case["height"])
    if case["scene"] == "terrain":
        return scenes.terrain(seed=seed, grid=case["size"], width=case["width"], height=case["height"])
    s = _textured_torus(rng, case, case["size"])
    if case["scene"] == "ortho":
        s = scenes.with_variant(s, light=True, seed=seed)
        s.model_to_world = np.concatenate([[0, 0, 0], scenes.random_rotation(rng).reshape(-1)]).astype(np.float32)
        s.perspective, s.slope = False, 1.8
    return s


def _layer_scenes(case, seed):
    """A solid model, and clouds of small alpha-filtered triangles before and around it."""
    rng = np.random.default_rng(seed)
    solid = _textured_torus(rng, case, case["size"])
    clouds = []
    for k in range(2):
        n = case["particles"]
        cloud = scenes.random_triangles(seed=seed + 1 + k, triangles=n, width=case["width"], height=case["height"], texture_size=64)
        centers = rng.uniform(-1.2, 1.2, size=(n, 1, 3))
        cloud.positions = (centers + 0.12 * rng.normal(size=(n, 3, 3))).reshape(-1, 3).astype(np.float32)
        cloud.colors[:, :3, 3] *= np.float32(0.7)
        clouds.append(dataclasses.replace(cloud, filter=1, camera_location=solid.camera_location))
    return solid, clouds


def _light_scene(case, seed):
    m, _ = dfpsr.ortho_view(-0.7, PIXELS_PER_TILE, 0).arrays()
    return scenes.light_scene(seed=seed, width=case["width"], height=case["height"], sprites=case["sprites"], lights=case["lights"],
                              radius_px=(100, 400) if case["width"] >= 800 else (30, 200), caster_triangles=case["casters"],
                              cube_resolution=case["cube"], light_space=(m[9:18], m[0:9]))


def _dense_inputs(case, seed):
    rng = np.random.default_rng(seed)
    mesh = scenes.torus(case["major"], case["minor"], minor_radius=0.35)
    colors = rng.uniform(0.0, 1.0, size=mesh.colors.shape).astype(np.float32)
    ground = (scenes.value_noise(rng, 64) * 1.2 - 0.9).astype(np.float32)
    ground = np.tile(ground, (case["height"] // 64 + 1, case["width"] // 64 + 1))[:case["height"], :case["width"]]
    places = [((float(rng.uniform(0, case["width"])), float(rng.uniform(0, case["height"]))),
               np.concatenate([rng.uniform(-1, 1, 3), scenes.random_rotation(rng).reshape(-1)]).astype(np.float32))
              for _ in range(case["instances"])]
    return mesh, colors, np.ascontiguousarray(ground), places


def _diff_inputs(case, seed):
    p = scenes.diff_problem(seed=seed, views=case["views"], texture_size=case["texture"], major=case["major"], minor=case["minor"])
    p.mesh.width, p.mesh.height = case["width"], case["height"]
    generator = torch.Generator(device="cuda").manual_seed(seed)
    targets = torch.rand((case["views"], case["height"], case["width"], 4), device="cuda", generator=generator)
    return p, targets


def _batch_scenes(case, seed):
    """Frames of the benchmark's mixed batch: the sizes belong to the case, what is drawn to the seed."""
    sizes, rng = np.random.default_rng(case["frames"]), np.random.default_rng(seed)
    out = []
    for _ in range(case["frames"]):
        width, height = scenes.BATCH_RESOLUTIONS[int(sizes.integers(0, len(scenes.BATCH_RESOLUTIONS)))]
        triangles = int(round(math.exp(sizes.uniform(math.log(1000), math.log(case["triangles"])))))
        out.append(scenes.random_triangles(seed=int(rng.integers(0, 2**31 - 1)), triangles=triangles, width=width, height=height))
    return out


def _images(width, height, host):
    if host:
        return (torch.zeros((height, width), dtype=torch.int32).pin_memory().numpy(),
                torch.zeros((height, width), dtype=torch.float32).pin_memory().numpy())
    return torch.zeros((height, width), dtype=torch.int32, device="cuda"), torch.zeros((height, width), dtype=torch.float32, device="cuda")


def _clear(color, depth, far):
    if isinstance(color, np.ndarray):
        color.fill(0)
        depth.fill(far)
    else:
        color.zero_()
        depth.fill_(far)


def prepare(case, seed):
    ctx = dfpsr.Context(0)
    state = {"case": case, "ctx": ctx}
    if case.get("threads"):
        ctx.set_tuning(threads_per_tile=case["threads"], ctas_per_sm=1024 // case["threads"])
    kind = case["kind"]
    if kind == "frame":
        scene = _frame_scene(case, seed)
        state["model"] = dfpsr.Model(ctx, scene)
        state["far"] = 0.0 if scene.perspective else FAR
        state["images"] = _images(case["width"], case["height"], case["host"])
    elif kind == "layers":
        solid, clouds = _layer_scenes(case, seed)
        state["models"] = [dfpsr.Model(ctx, s) for s in (solid, *clouds)]
        state["renderer"] = ctx.renderer()
        state["images"] = _images(case["width"], case["height"], False)
    elif kind == "batch":
        frames = _batch_scenes(case, seed)
        state["models"] = [dfpsr.Model(ctx, s) for s in frames]
        state["images"] = [_images(s.width, s.height, False) for s in frames]
        state["batch"] = ctx.batch()
        for k, m in enumerate(state["models"]):
            state["batch"].add_frame(*state["images"][k])
            state["batch"].give_task(k, m)
    elif kind == "sprites":
        state["pass"] = DeferredLightPass(ctx, _light_scene(case, seed), reference_threads=8)
        # the tile shape that suits cube faces of a few short tiles each
        state["pass"].shadows.set_tuning({"threads_per_tile": 64, "ctas_per_sm": 16, "small_rows": 8, "small_width": 16})
    elif kind == "dense":
        mesh, colors, ground, places = _dense_inputs(case, seed)
        model = dfpsr.DenseModel(ctx, mesh.positions, mesh.poly_indices, colors)
        state["instances"] = [(model, origin, transform) for origin, transform in places]
        state["view"] = dfpsr.ortho_view(TILT, PIXELS_PER_TILE, 0)
        state["ground"] = torch.tensor(ground, device="cuda")
        state["height"] = torch.empty_like(state["ground"])
        state["diffuse"], state["normal"] = (torch.zeros(ground.shape, dtype=torch.int32, device="cuda") for _ in range(2))
    else:
        p, targets = _diff_inputs(case, seed)
        state["model"] = dfpsr.Model(ctx, p.mesh)
        state["diff"] = dfpsr.Diff(ctx, state["model"], case["texture"], case["texture"], p.ambient)
        state["cameras"] = []
        for location in p.cameras:
            camera = dfpsr.camera_struct(p.mesh)
            camera.location[:] = [float(v) for v in location]
            state["cameras"].append(camera)
        state["params"] = [torch.tensor(a, device="cuda") for a in (p.texture, p.vertex_colors, p.light)]
        state["grads"] = [torch.empty_like(a) for a in state["params"]]
        state["targets"] = targets
        state["rendered"], state["grad"] = torch.empty_like(targets), torch.empty_like(targets)
        state["visibility"] = torch.empty((*targets.shape[:3], 3), dtype=torch.int32, device="cuda")
        state["loss"] = torch.empty(1, device="cuda")
        state["transform"] = p.mesh.model_to_world
    return state


# ------------------------------------------------------------------ one pass

def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "frame":
        color, depth = state["images"]
        _clear(color, depth, state["far"])
        ctx.render(state["model"], state["model"].camera, color, depth)
        return {"color": color, "depth": depth}
    if kind == "layers":
        color, depth = state["images"]
        _clear(color, depth, 0.0)
        renderer = state["renderer"]
        renderer.begin(color, depth)
        for model in state["models"]:
            renderer.give_task(model)
        renderer.end()
        return {"color": color, "depth": depth}
    if kind == "batch":
        for color, depth in state["images"]:
            _clear(color, depth, 0.0)
        state["batch"].render()
        return [{"color": color, "depth": depth} for color, depth in state["images"]]
    if kind == "sprites":
        p = state["pass"]
        p.run()
        return {"output": p.output, "light": p.light, "diffuse": p.diffuse, "normal": p.normal, "height": p.height, "cubes": p.cubes}
    if kind == "dense":
        state["height"].copy_(state["ground"])
        state["diffuse"].zero_()
        state["normal"].zero_()
        ctx.dense_render_many(state["instances"], state["view"], state["height"], state["diffuse"], state["normal"], case["high"])
        return {"height": state["height"], "diffuse": state["diffuse"], "normal": state["normal"]}
    s = state
    s["diff"].forward(s["cameras"], s["transform"], *s["params"], s["rendered"], s["visibility"])
    s["diff"].l2_loss(s["rendered"], s["targets"], s["grad"], s["loss"])
    s["diff"].adjoint(case["views"], case["width"], case["height"], s["transform"], *s["params"], s["visibility"], s["grad"], *s["grads"],
                      case["deterministic"])
    return {"images": s["rendered"], "visibility": s["visibility"], "grad_images": s["grad"], "loss": s["loss"], "grad_texture": s["grads"][0],
            "grad_vertex_colors": s["grads"][1], "grad_light": s["grads"][2]}


# ------------------------------------------------------------------ what a pass cannot do without

def _frame_work(triangles, points, polygons, texels, pixels):
    """A model's arrays and its texture read once, the depth image read and both images written; some 200
    operations set a triangle up (projection, planes, edges) and some 100 shade a pixel."""
    return np.array([12 * points + 144 * polygons + 4 * triangles + 4 * texels + 12 * pixels, 200 * triangles + 100 * pixels], float)


def work(case):
    kind = case["kind"]
    if kind == "frame":
        n, pixels = case["size"], case["width"] * case["height"]
        if case["scene"] == "random":
            w = _frame_work(n, 3 * n, n, 256 * 256, pixels)
        elif case["scene"] == "terrain":
            w = _frame_work(2 * (n - 1) ** 2, n * n, (n - 1) ** 2, 1024 * 1024, pixels)
        else:
            w = _frame_work(4 * n * n, 2 * n * n, 2 * n * n, 256 * 256, pixels)
    elif kind == "layers":
        n, pixels = case["size"], case["width"] * case["height"]
        w = _frame_work(4 * n * n, 2 * n * n, 2 * n * n, 256 * 256, pixels) + 2 * _frame_work(case["particles"], 3 * case["particles"], case["particles"], 64 * 64, pixels)
    elif kind == "batch":
        # the mean of log-uniform triangle counts and of the four resolutions
        n = (case["triangles"] - 1000) / math.log(case["triangles"] / 1000)
        pixels = sum(a * b for a, b in scenes.BATCH_RESOLUTIONS) / len(scenes.BATCH_RESOLUTIONS)
        w = case["frames"] * _frame_work(n, 3 * n, n, 256 * 256, pixels)
    elif kind == "sprites":
        pixels = case["width"] * case["height"]
        # a sprite's three images per covered pixel, five frame images, the cubes written and read where
        # they are lit; a light touches the square around it: some 60 operations per pixel and light
        lit = case["lights"] * min(pixels, 500 * 500 if case["width"] >= 800 else 230 * 230)
        w = np.array([12 * 32 * 64 * 64 + 12 * pixels + 20 * pixels + 4 * 6 * case["cube"] ** 2 * case["lights"] + 4 * lit,
                      60 * lit + 40 * pixels + 2 * case["sprites"] * 64 * 64 + 200 * 6 * case["casters"] * case["lights"]], float)
    elif kind == "dense":
        n = 2 * case["major"] * case["minor"]
        w = np.array([108 * n + 24 * case["width"] * case["height"], case["instances"] * n * 200], float)
    else:
        pixels = case["views"] * case["width"] * case["height"]
        n = case["major"] * case["minor"]
        # images and visibility written; images, targets and visibility read; the gradient image written and read; parameters and their gradients
        w = np.array([pixels * (16 + 12 + 16 + 16 + 12 + 16 + 16) + 3 * 16 * (case["texture"] ** 2 + n) + 36 * n, 300 * pixels + 400 * n * case["views"]], float)
    return {"bytes": float(w[0]), "flops": float(w[1])}


# ------------------------------------------------------------------ 64 bits

def _world(positions, transform):
    t = torch.tensor(np.asarray(transform, np.float64), device="cuda")
    return torch.tensor(np.asarray(positions, np.float64), device="cuda") @ t[3:].reshape(3, 3) + t[:3]


def _fans(polygons):
    """Corner slots (polygon * 4 + corner) of every fan triangle, in order."""
    p = torch.tensor(polygons.astype(np.int64), device="cuda")
    k = torch.arange(len(p), device="cuda") * 4
    both = torch.stack([torch.stack([k, k + 1, k + 2], 1), torch.stack([k, k + 2, k + 3], 1)], 1)
    keep = torch.stack([torch.ones_like(k, dtype=torch.bool), p[:, 3] >= 0], 1)
    slots = both[keep]
    return slots, p.reshape(-1)[slots]


def _pairs(x0, y0, x1, y1, most=1 << 25):
    """(triangle, x, y) of every pixel of the triangles' bounds, in parts of bounded size."""
    w, h = (x1 - x0).clamp(min=0), (y1 - y0).clamp(min=0)
    area = w * h
    live = torch.nonzero(area).reshape(-1)
    ends = torch.cumsum(area[live], 0).cpu().numpy()
    at, done = 0, 0
    while at < len(ends):
        to = max(at + 1, int(np.searchsorted(ends, done + most, side="right")))
        ids = live[at:to]
        a = area[ids]
        t = torch.repeat_interleave(ids, a)
        k = torch.arange(len(t), device="cuda") - torch.repeat_interleave(torch.cumsum(a, 0) - a, a)
        yield t, x0[t] + k % w[t], y0[t] + k // w[t]
        done, at = int(ends[to - 1]), to


def _project(scene, location, points, transform):
    """Image position, depth and snapped position of every point."""
    c = torch.tensor(np.asarray(location, np.float64), device="cuda")
    camera = (_world(points, transform) - c[:3]) @ c[3:].reshape(3, 3).T
    ws = float(np.float32(scene.slope))
    hs = ws * scene.height / scene.width
    x, y, z = camera.unbind(1)
    if scene.perspective:
        sx, sy = (x * (0.5 / ws) / z + 0.5) * scene.width, (-y * (0.5 / hs) / z + 0.5) * scene.height
    else:
        sx, sy = (x * (0.5 / ws) + 0.5) * scene.width, (-y * (0.5 / hs) + 0.5) * scene.height
    screen = torch.stack([sx, sy], 1)
    return screen, z, (screen.float() * 256.0).to(torch.int64)


def _rasterise(scene, location, points, transform, corners, depth, winners=False):
    """Draws front-facing triangles into a 64-bit depth image (1/W grows towards a perspective camera, W
    shrinks towards an orthogonal one); optionally the earliest triangle of the nearest depth and its weights."""
    screen, z, flat = _project(scene, location, points, transform)
    f, s, w = flat[corners], screen[corners], z[corners]
    d = 1.0 / w if scene.perspective else w
    front = ((f[:, 2, 0] - f[:, 0, 0]) * (f[:, 1, 1] - f[:, 0, 1]) + (f[:, 2, 1] - f[:, 0, 1]) * (f[:, 0, 0] - f[:, 1, 0])) < 0
    low, high = f.amin(1).div(256, rounding_mode="floor") - 1, f.amax(1).div(256, rounding_mode="floor") + 2
    x0, y0 = low[:, 0].clamp(min=0), low[:, 1].clamp(min=0)
    x1, y1 = torch.where(front, high[:, 0].clamp(max=scene.width), x0), high[:, 1].clamp(max=scene.height)
    a, b, c = s.unbind(1)
    det = (b[:, 0] - a[:, 0]) * (c[:, 1] - a[:, 1]) - (c[:, 0] - a[:, 0]) * (b[:, 1] - a[:, 1])

    def covered():
        for t, x, y in _pairs(x0, y0, x1, y1):
            inside = torch.ones_like(t, dtype=torch.bool)
            for i in range(3):
                p, q = f[:, i], f[:, (i + 1) % 3]
                nx, ny = q[:, 1] - p[:, 1], p[:, 0] - q[:, 0]
                limit = -((p[:, 0] > q[:, 0]) | ((p[:, 0] == q[:, 0]) & (p[:, 1] > q[:, 1]))).to(torch.int64)
                inside &= (128 + 256 * x - p[t, 0]) * nx[t] + (128 + 256 * y - p[t, 1]) * ny[t] <= limit[t]
            t, x, y = t[inside], x[inside], y[inside]
            px, py = x + 0.5 - a[t, 0], y + 0.5 - a[t, 1]
            u = (px * (c[t, 1] - a[t, 1]) - py * (c[t, 0] - a[t, 0])) / det[t]
            v = (py * (b[t, 0] - a[t, 0]) - px * (b[t, 1] - a[t, 1])) / det[t]
            yield t, y * scene.width + x, d[t, 0] + u * (d[t, 1] - d[t, 0]) + v * (d[t, 2] - d[t, 0]), u, v

    image = depth.reshape(-1)
    for t, at, value, _, _ in covered():
        image.scatter_reduce_(0, at, value, "amax" if scene.perspective else "amin")
    if not winners:
        return depth
    first = torch.full_like(image, len(corners), dtype=torch.int64)
    for t, at, value, _, _ in covered():
        same = value == image[at]
        first.scatter_reduce_(0, at[same], t[same], "amin")
    wb, wc = torch.zeros_like(image), torch.zeros_like(image)
    for t, at, value, u, v in covered():
        mine = first[at] == t
        t, at, value, u, v = t[mine], at[mine], value[mine], u[mine], v[mine]
        wb[at], wc[at] = (u * d[t, 1] / value, v * d[t, 2] / value) if scene.perspective else (u, v)
    return first, wb, wc


def _scene_depth(scene):
    depth = torch.full((scene.height, scene.width), 0.0 if scene.perspective else FAR, dtype=torch.float64, device="cuda")
    return _rasterise(scene, scene.camera_location, scene.positions, scene.model_to_world, _fans(scene.poly_indices)[1], depth)


def _exact_heights(case, seed):
    if case["kind"] == "sprites":
        s = _light_scene(case, seed)
        image = torch.full((s.height, s.width), BACKGROUND_HEIGHT, dtype=torch.float64, device="cuda")
        types = [torch.tensor(h.astype(np.float64), device="cuda") for h in s.sprite_heights]
        for kind, left, top, offset in s.placements:
            h = types[int(kind)]
            x0, y0, x1, y1 = max(left, 0), max(top, 0), min(left + h.shape[1], s.width), min(top + h.shape[0], s.height)
            if x1 > x0 and y1 > y0:
                part = h[y0 - top:y1 - top, x0 - left:x1 - left] + float(np.array([offset], np.int32).view(np.float32)[0])
                image[y0:y1, x0:x1] = torch.maximum(image[y0:y1, x0:x1], part)
        return image
    mesh, _, ground, places = _dense_inputs(case, seed)
    # tile to screen: the rounded pixel offsets of a tile along x and z, and the pixels of a tile's height
    forward = np.array([0.707106781, TILT, 0.707106781])
    z = forward / np.linalg.norm(forward)
    x = np.cross([0.0, 1.0, 0.0], z)
    x /= np.linalg.norm(x)
    y = np.cross(z, x)
    along = [[math.trunc(x[k] * PIXELS_PER_TILE), math.trunc(-y[k] * PIXELS_PER_TILE), 0.0] for k in (0, 2)]
    to_screen = torch.tensor(np.array([along[0], [0.0, -float(math.trunc(PIXELS_PER_TILE / math.sqrt(TILT * TILT + 1))), 1.0], along[1]]), device="cuda")
    image = torch.tensor(ground.astype(np.float64), device="cuda")
    corners = _fans(mesh.poly_indices)[1]
    for origin, transform in places:
        p = (_world(mesh.positions, transform) @ to_screen + torch.tensor([*origin, 0.0], dtype=torch.float64, device="cuda"))[corners]
        a, b, c = p.unbind(1)
        det = (b[:, 0] - a[:, 0]) * (c[:, 1] - a[:, 1]) - (b[:, 1] - a[:, 1]) * (c[:, 0] - a[:, 0])
        front = (c[:, 0] - a[:, 0]) * (b[:, 1] - a[:, 1]) + (c[:, 1] - a[:, 1]) * (a[:, 0] - b[:, 0]) < 0
        low, high = p.amin(1).floor().to(torch.int64), p.amax(1).floor().to(torch.int64) + 1
        x0, y0 = low[:, 0].clamp(min=0), low[:, 1].clamp(min=0)
        x1, y1 = torch.where(front, high[:, 0].clamp(max=case["width"]), x0), high[:, 1].clamp(max=case["height"])
        for t, px, py in _pairs(x0, y0, x1, y1):
            ox, oy = px + 0.5 - a[t, 0], py + 0.5 - a[t, 1]
            wb = (ox * (c[t, 1] - a[t, 1]) - oy * (c[t, 0] - a[t, 0])) / det[t]
            wc = (oy * (b[t, 0] - a[t, 0]) - ox * (b[t, 1] - a[t, 1])) / det[t]
            wa = 1.0 - wb - wc
            inside = (wa >= -1e-5) & (wb >= -1e-5) & (wc >= -1e-5)
            h = (a[t, 2] * wa + b[t, 2] * wb + c[t, 2] * wc)[inside]
            image.reshape(-1).scatter_reduce_(0, (py * case["width"] + px)[inside], h, "amax")
    return image


def _exact_diff(case, seed):
    p, targets = _diff_inputs(case, seed)
    slots, corners = _fans(p.mesh.poly_indices)
    world = _world(p.mesh.positions, p.mesh.model_to_world)[corners]
    normal = torch.cross(world[:, 1] - world[:, 0], world[:, 2] - world[:, 0], dim=1)
    normal = normal / normal.norm(dim=1, keepdim=True)
    uv = torch.tensor(p.mesh.tex_coords.astype(np.float64), device="cuda").reshape(-1, 4)[:, :2][slots]
    params = [torch.tensor(a.astype(np.float64), device="cuda", requires_grad=True) for a in (p.texture, p.vertex_colors, p.light)]
    size, count = case["texture"], targets.numel()
    images, loss = torch.zeros(targets.shape, dtype=torch.float64, device="cuda"), 0.0
    grads = [torch.zeros_like(a) for a in params]
    for view, location in enumerate(p.cameras):
        depth = torch.zeros((case["height"], case["width"]), dtype=torch.float64, device="cuda")
        first, wb, wc = _rasterise(p.mesh, location, p.mesh.positions, p.mesh.model_to_world, corners, depth, winners=True)
        seen = torch.nonzero(first < len(corners)).reshape(-1)
        t = first[seen]
        w = torch.stack([1.0 - (wb[seen] + wc[seen]), wb[seen], wc[seen]], 1)
        texture, vertex, light = params
        taps = (((uv[t] * w[:, :, None]).sum(1).float() + 256.0) * (256.0 * size)).to(torch.int64) - 128
        near, part = (taps >> 8) & (size - 1), (taps & 255).double() / 256.0
        far = (near + 1) & (size - 1)
        texel = 0.0
        for x, fx in ((near[:, 0], 1.0 - part[:, 0]), (far[:, 0], part[:, 0])):
            for y, fy in ((near[:, 1], 1.0 - part[:, 1]), (far[:, 1], part[:, 1])):
                texel = texel + texture[y, x] * (fx * fy)[:, None]
        color = texel * (vertex[corners[t]] * w[:, :, None]).sum(1)
        lit = p.ambient + light[3] * (-(normal[t] @ light[:3])).clamp(min=0.0)
        image = torch.zeros((case["height"] * case["width"], 4), dtype=torch.float64, device="cuda")
        image = image.index_put((seen,), torch.cat([color[:, :3] * lit[:, None], color[:, 3:]], 1))
        part_loss = ((image - targets[view].double().reshape(-1, 4)) ** 2).sum() / count
        for total, g in zip(grads, torch.autograd.grad(part_loss, params)):
            total += g
        images[view] = image.detach().reshape(images[view].shape)
        loss += float(part_loss)
    return {"images": images, "visibility": None, "grad_images": 2.0 * (images - targets) / count,
            "loss": torch.tensor([loss], dtype=torch.float64, device="cuda"), "grad_texture": grads[0], "grad_vertex_colors": grads[1], "grad_light": grads[2]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "frame":
        depth = _scene_depth(_frame_scene(case, seed))
        return {"color": None, "depth": depth.cpu().numpy() if case["host"] else depth}
    if kind == "layers":  # alpha-filtered triangles write no depth
        return {"color": None, "depth": _scene_depth(_layer_scenes(case, seed)[0])}
    if kind == "batch":
        return [{"color": None, "depth": _scene_depth(s)} for s in _batch_scenes(case, seed)]
    if kind == "sprites":
        return {"output": None, "light": None, "diffuse": None, "normal": None, "height": _exact_heights(case, seed), "cubes": None}
    if kind == "dense":
        return {"height": _exact_heights(case, seed), "diffuse": None, "normal": None}
    return _exact_diff(case, seed)

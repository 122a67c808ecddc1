"""The two-pass triangle setup, which batches from 2^29 fan triangles on take, through the whole
pipeline: a context whose limit is lowered to nothing draws every kind of work with it, bit for bit
as the oracle does (tiles in parts, odd heights, clipped triangles, alpha-filtered runs, both
projections, depth-only tiles, buffers that overflow, and the differentiable renderer's views)."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

from dfpsr_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture
def two_pass(built):
    import dfpsr_gb300 as d
    c = d.Context(0)
    limit = C.CDLL(d.LIB_PATH).dsrg_internal_set_one_pass_limit  # not in the public header
    assert limit(c.handle, C.c_uint32(0)) == 0
    yield c
    c.close()


def _scene(w, h, triangles, near=False, **changes):
    s = scenes.random_triangles(seed=w * h, triangles=triangles, width=w, height=h, texture_size=32)
    if near:  # the camera among the triangles: many are clipped
        s.camera_location = scenes.camera_location((0.1, 0.2, -0.3), (0.0, 0.0, 1.0))
    return dataclasses.replace(s, **changes)


@pytest.mark.parametrize("resolve", [0, 1, 2])
@pytest.mark.parametrize("w,h,triangles,near", [(33, 17, 12000, False), (320, 201, 3000, True), (640, 480, 3000, False), (64, 64, 40, False)])
def test_two_pass_frames(two_pass, w, h, triangles, near, resolve):
    import dfpsr_gb300 as d
    from oracle import port
    s = _scene(w, h, triangles, near)
    rc, rz, info = port.render(s)
    model = d.Model(two_pass, s)
    two_pass.set_tuning(resolve=resolve)
    for counting in (True, False, False, False):  # the last one replays the phases' graphs
        two_pass.set_counting(counting)
        c, z = d.render_scene(two_pass, s, model=model)
        assert np.array_equal(c, rc) and np.array_equal(z.view(np.uint32), rz.view(np.uint32)), f"counting {counting}"
        assert not counting or two_pass.stats()["fragments"] == info["fragments"]


def test_two_pass_frame_of_mixed_tasks(two_pass):
    import dfpsr_gb300 as d
    from oracle import port
    tasks = [_scene(121, 83, 500 + 50 * i, filter=i & 1, perspective=i < 2, slope=0.6 if i < 2 else 1.3) for i in range(4)]
    tasks.append(_scene(121, 83, 9000, filter=1))
    rng = np.random.default_rng(4)
    color = rng.integers(0, 2**32, size=(83, 121), dtype=np.uint64).astype(np.uint32)
    depth = rng.uniform(0.0, 0.3, size=(83, 121)).astype(np.float32)
    o = port.OracleRenderer()
    o.begin(color, depth)
    for s in tasks:
        p = port.PreparedModel(s)
        o.give_task(p, s.model_to_world, p.cam)
    rc, rz, _ = o.end()
    models = [d.Model(two_pass, s) for s in tasks]
    for _ in range(3):
        c, z = color.copy(), depth.copy()
        r = d.Renderer(two_pass)
        r.begin(c, z)
        for m in models:
            r.give_task(m, m.camera)
        r.end()
        assert np.array_equal(c, rc) and np.array_equal(z.view(np.uint32), rz.view(np.uint32))
        r.destroy()


@pytest.mark.parametrize("w,h,triangles", [(35, 18, 15000), (200, 121, 400)])
def test_two_pass_depth_only(two_pass, ctx, w, h, triangles):
    import dfpsr_gb300 as d
    from oracle import port
    s = _scene(w, h, triangles)
    launches = {}
    for c in (two_pass, ctx):
        m = d.Model(c, s)
        for _ in range(3):
            z = np.zeros((h, w), np.float32)
            before = c.stats()["kernel_launches"]
            c.render_depth(m, m.camera, z)
            launches[c] = c.stats()["kernel_launches"] - before
            assert np.array_equal(z.view(np.uint32), port.render_depth(s)[0].view(np.uint32))
    assert launches[two_pass] > launches[ctx]  # the counting pass, its scan and the row scan: the setup is the other one


def test_two_pass_differentiable_views(two_pass, ctx):
    """The views' images and visibility are those of a context with the one-pass setup."""
    import torch
    from diff_harness import make_renderer
    problem = scenes.diff_problem(seed=6, views=3, size=80, texture_size=32, major=40, minor=20)
    out = []
    for c in (two_pass, ctx):
        model, renderer, cameras, params = make_renderer(c, problem)
        images = torch.empty((3, problem.height, problem.width, 4), dtype=torch.float32, device="cuda")
        visibility = torch.empty((3, problem.height, problem.width, 3), dtype=torch.int32, device="cuda")
        renderer.forward(cameras, problem.mesh.model_to_world, params["texture"], params["vertex_colors"], params["light"], images, visibility)
        out.append((images.cpu().numpy().view(np.uint32), visibility.cpu().numpy()))
    assert (out[0][1][..., 0] != -1).sum() > 1000
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])

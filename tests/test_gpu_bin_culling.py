"""GPU parity of frames whose large triangles are culled while binning, against the oracle, bit for bit.

A tile's threshold is the worst key of the large records that cover it completely; records whose
best key lies below it are not listed.  The scenes put many screen-filling triangles over one
another: parallel layers with exact depth ties (the earliest must win), planes crossing inside
tiles, an initial depth image in front of some of them; targets with partial tiles, odd heights
(whose bottom tile row is not culled) and large records over at most four tiles.
"""
import dataclasses

import numpy as np
import pytest

from dfpsr_gb300 import scenes
from test_gpu_render import run_case

pytestmark = pytest.mark.gpu


def _layers(w, h, n, seed, tilt, perspective):
    rng = np.random.default_rng(seed)
    s = scenes.random_triangles(seed=seed, triangles=n, width=w, height=h, texture_size=32)
    depth = rng.integers(-4, 5, size=(n, 1)) * 0.125  # few distinct depths: exact ties between layers
    corners = np.array([[-9.0, -7.0], [0.0, 9.0], [9.0, -7.0]])
    p = np.zeros((n, 3, 3))
    p[:, :, :2] = corners * rng.uniform(0.1, 1.0, size=(n, 1, 1)) + rng.uniform(-1.0, 1.0, size=(n, 1, 2))
    p[:, :, 2] = depth + tilt * rng.uniform(-1.0, 1.0, size=(n, 3))
    s.positions = p.reshape(-1, 3).astype(np.float32)
    if not perspective:
        s = dataclasses.replace(s, perspective=False, slope=2.0)
    return s


@pytest.mark.parametrize("perspective", [True, False])
@pytest.mark.parametrize("tilt", [0.0, 0.4])
@pytest.mark.parametrize("w,h", [(48, 32), (80, 75), (129, 64), (40, 17)])
def test_layers_over_one_another(ctx, w, h, tilt, perspective):
    s = _layers(w, h, 400, seed=w + h, tilt=tilt, perspective=perspective)
    run_case(ctx, s, f"{w}x{h} tilt {tilt}")
    rng = np.random.default_rng(1)
    depth = (rng.uniform(0.25, 0.4, (h, w)) if perspective else rng.uniform(2.4, 3.4, (h, w))).astype(np.float32)
    depth[::3, ::5] = 0.0 if perspective else 1000.0
    _prefilled(ctx, s, depth)


def _prefilled(ctx, s, depth):
    import dfpsr_gb300 as d
    from oracle import port
    color = np.full(depth.shape, 0x40302010, np.uint32)
    c, z = d.render_scene(ctx, s, color, depth)
    rc, rz, _ = port.render(s, color, depth)
    assert np.array_equal(c, rc)
    assert np.array_equal(z.view(np.uint32), rz.view(np.uint32))


@pytest.mark.parametrize("w,h", [(64, 48), (95, 33)])
def test_depth_only_layers(ctx, w, h):
    import dfpsr_gb300 as d
    from oracle import port
    s = _layers(w, h, 300, seed=w, tilt=0.3, perspective=True)
    z = np.zeros((h, w), np.float32)
    m = d.Model(ctx, s)
    ctx.render_depth(m, m.camera, z)
    rz = port.render_depth(s)[0]
    assert np.array_equal(z.view(np.uint32), rz.view(np.uint32))


@pytest.mark.parametrize("w,h,stride", [(64, 64, 64), (33, 31, 33), (70, 50, 75), (16, 16, 20), (7, 3, 8)])
@pytest.mark.parametrize("perspective", [True, False])
def test_depth_only_images_of_any_shape(ctx, w, h, stride, perspective):
    """Partial tiles, odd heights, row strides that are no multiple of 16 bytes, prefilled depths
    with infinities and NaN (never passed), signed zeros; page-locked host memory and device memory."""
    import torch
    import dfpsr_gb300 as d
    from oracle import port
    s = scenes.random_triangles(seed=w * 31 + h, triangles=500, width=w, height=h)
    if not perspective:
        s = dataclasses.replace(s, perspective=False, slope=1.5)
        s.positions = s.positions.copy()
        s.positions[::7, 2] = -3.0  # at the camera: linear depth zero
    rng = np.random.default_rng(w)
    initial = (rng.uniform(0.2, 0.4, (h, w)) if perspective else rng.uniform(1.0, 4.0, (h, w))).astype(np.float32)
    initial[0, ::3], initial[h // 2, 1::4], initial[-1, ::5], initial[h // 3, ::2] = np.inf, -np.inf, np.nan, -0.0
    expected = port.render_depth(s, initial)[0]
    m = d.Model(ctx, s)
    host = torch.zeros((h, stride), dtype=torch.float32).pin_memory()
    host[:, :w] = torch.from_numpy(initial)
    device = host.cuda()
    ctx.render_depth(m, m.camera, device[:, :w])
    ctx.render_depth(m, m.camera, host.numpy()[:, :w])
    for got in (device.cpu().numpy()[:, :w], host.numpy()[:, :w]):
        same = (got.view(np.uint32) == expected.view(np.uint32)) | (np.isnan(got) & np.isnan(expected))
        assert same.all(), np.argwhere(~same)[:5].tolist()
    assert (host.numpy()[:, w:] == 0).all() and bool((device[:, w:] == 0).all())


@pytest.mark.parametrize("perspective", [True, False])
@pytest.mark.parametrize("w,h", [(1000, 16), (16, 900), (700, 90), (333, 257)])
def test_slivers_over_many_tiles(ctx, w, h, perspective):
    """Triangles over many tiles whose edges are nearly horizontal, nearly vertical or exactly so, thin
    ones that touch few tiles of their bounds among them: the columns found for each row of tiles."""
    rng = np.random.default_rng(w * 7 + h)
    s = scenes.random_triangles(seed=w, triangles=300, width=w, height=h, texture_size=32)
    p = s.positions.reshape(-1, 3, 3).copy()
    k = np.arange(300)
    p[:, :, :2] = rng.uniform(-9.0, 9.0, (300, 3, 2))
    p[k % 6 == 0, 1, 1] = p[k % 6 == 0, 0, 1]                                  # a horizontal edge
    p[k % 6 == 1, 1, 0] = p[k % 6 == 1, 0, 0]                                  # a vertical edge
    for way, axis in ((2, 0), (3, 1)):                                         # slivers along each axis
        p[k % 6 == way, :, axis] = p[k % 6 == way, :1, axis] + rng.uniform(-0.01, 0.01, (50, 3))
    p[k % 6 == 4, 2, :2] = p[k % 6 == 4, :2, :2].mean(1) + rng.uniform(-0.02, 0.02, (50, 2))  # diagonal slivers
    s.positions = p.reshape(-1, 3).astype(np.float32)
    if not perspective:
        s = dataclasses.replace(s, perspective=False, slope=2.0)
    run_case(ctx, s, f"{w}x{h}")


def test_statistics_count_every_pair_whatever_is_culled(ctx):
    """binEntries counts the pairs of tiles and triangles that touch them, culled ones too, and is the same
    from run to run; with fragments counted nothing is culled and it is the same again."""
    import dfpsr_gb300 as d
    s = _layers(257, 131, 500, seed=3, tilt=0.3, perspective=True)
    seen = set()
    for _ in range(4):
        d.render_scene(ctx, s)
        seen.add(ctx.stats()["bin_entries"])
    ctx.set_counting(True)
    try:
        d.render_scene(ctx, s)
        seen.add(ctx.stats()["bin_entries"])
    finally:
        ctx.set_counting(False)
    assert len(seen) == 1 and seen.pop() > 500

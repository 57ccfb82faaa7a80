"""Renders take no longer with a world BVH and tail launches than without:
traversal limits other than the defaults keep a scene on the kernels that walk the instances, so the
same render is timed both ways in turn, the fastest of a few, and compared with it (films
as in test_tail.py).
"""
import time

import numpy as np
import pytest

from xitils_gb300 import scenes
from xitils_gb300.scene import SKY_UNIFORM, IntegratorParams, SceneDesc
from xitils_gb300.transform import scale, translate

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api_mod():
    import __graft_entry__ as g
    g.build()
    from xitils_gb300 import api
    return api


def _boxes(n, width, height, level):
    """A terrain under its sky with n boxes, moved there, many of which overlap; level: with
    their tops in one plane."""
    d = scenes.terrain(grid=129, width=width, height=height, spp=1, env_size=(128, 64))
    cpos, cidx = scenes.unit_cube_mesh()
    cube = d.add_mesh(cpos, cidx)
    grey = d.diffuse([0.6, 0.6, 0.6])
    rng = np.random.default_rng(3)
    for _ in range(n):
        x, z = rng.uniform(0.1, 0.9, 2)
        y = 0.2 if level else rng.uniform(0.15, 0.25)
        d.add_object(cube, grey, translate(float(x), float(y), float(z)) * scale(0.04, 0.04, 0.04))
    return d


def _both_ways(api, d, layout="binary"):
    ctx = api.Context(0)
    ctx.set_bvh_layout(layout)
    b = api.load_scene(ctx, d)
    best, films = [np.inf, np.inf], [None, None]
    for _ in range(6):
        for k, stack in enumerate((0, 63)):
            b.scene.set_traversal_limits(0, stack)
            rt = api.RenderTarget(ctx, d.width, d.height)
            t = time.perf_counter()
            rt.render(b.scene, d.spp, d.params)
            best[k] = min(best[k], time.perf_counter() - t)
            films[k] = rt.download()
    np.testing.assert_allclose(films[0], films[1], rtol=1e-4, atol=1e-6 * float(films[1].mean()))
    return best


def test_many_marked_rays(api_mod):
    """Level boxes that overlap: most rays hit two instances in the same place, and are traced
    again in the instance order. A world traversal and a second one of as much work as the other
    way's cost at most twice the time."""
    world, walked = _both_ways(api_mod, _boxes(2000, 2048, 2048, True))
    assert world < 2 * walked, (world, walked)


@pytest.mark.parametrize("n", [17, 300])
def test_no_large_tail_over_the_top_level(api_mod, n):
    """Without lights, 500,000 camera paths: many instances stay on the wavefront until 65,536
    paths are left."""
    world, walked = _both_ways(api_mod, _boxes(n, 724, 700, False))
    assert world < 1.25 * walked, (world, walked)


def _closed_room(width, height, max_depth):
    """A room lit by its sky through a gap in a wall, with clouds of triangles in it."""
    d = SceneDesc(name="closed_room", width=width, height=height, spp=1,
                  params=IntegratorParams(max_depth=max_depth, rr_start=5, rr_prob=0.9, seed=3))
    grey = d.diffuse([0.7, 0.7, 0.7])
    for q in ([[0, 0, 0], [0, 0, 1], [1, 0, 1], [1, 0, 0]], [[0, 1, 0], [1, 1, 0], [1, 1, 1], [0, 1, 1]],
              [[0, 0, 0], [0, 1, 0], [0, 1, 1], [0, 0, 1]], [[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0]],
              [[0, 0, 1], [0, 1, 1], [1, 1, 1], [1, 0, 1]], [[1, 0, 0], [1, 0, 1], [1, 0.5, 1], [1, 0.5, 0]],
              [[1, 0.8, 0], [1, 0.8, 1], [1, 1, 1], [1, 1, 0]]):
        d.add_object(d.add_mesh(*scenes.quad(*q)), grey)
    rng = np.random.default_rng(5)
    for k in range(5):
        c = rng.uniform(0.3, 0.7, 3) + rng.normal(scale=0.15, size=(6000, 1, 3))
        pos = (c + rng.normal(scale=0.02, size=(6000, 3, 3))).reshape(-1, 3).astype(np.float32)
        m = d.add_mesh(pos, np.arange(18000, dtype=np.int32))
        d.add_object(m, grey, translate(0.01 * k, 0, 0) if k % 2 else None)
    d.set_sky(SKY_UNIFORM, (0.8, 0.9, 1.0))
    d.set_camera(scenes.look_at((0.15, 0.6, 0.1), (0.6, 0.3, 0.8), (0, 1, 0)), 1.1, height / width)
    return d


@pytest.mark.parametrize("layout", ["binary", "wide8"])
@pytest.mark.parametrize("max_depth", [4, 10])
def test_no_large_tail_while_paths_stay(api_mod, max_depth, layout):
    """No lights either, but most paths live through a vertex: they stay on the wavefront until
    65,536 are left."""
    world, walked = _both_ways(api_mod, _closed_room(640, 420, max_depth), layout)
    assert world < 1.25 * walked, (world, walked)


def _metal_room(boxes, spp):
    """A closed room with a ceiling light, of metal, so that paths are long."""
    d = _closed_room(128, 127, 10)
    d.spp = spp
    d.meshes, d.objects = d.meshes[:7], d.objects[:7]
    metal = d.metal(0.3, [0.8, 0.7, 0.6])
    for o in d.objects:
        o.material = metal
    cpos, cidx = scenes.unit_cube_mesh()
    cube = d.add_mesh(cpos, cidx)
    rng = np.random.default_rng(4)
    for _ in range(boxes):
        c = rng.uniform(0.1, 0.9, 3)
        d.add_object(cube, metal, translate(*c) * scale(0.25, 0.25, 0.25))
    d.add_object(d.add_mesh(*scenes.quad([0.4, 0.99, 0.4], [0.6, 0.99, 0.4], [0.6, 0.99, 0.6], [0.4, 0.99, 0.6])), d.emission([8.0, 8.0, 8.0]))
    return d


@pytest.mark.parametrize("boxes,layout,spp", [(9, "binary", 4), (16, "binary", 4), (16, "binary", 1), (30, "binary", 1), (2, "wide8", 4), (4, "wide8", 4)])
def test_no_large_tail_over_the_top_level_or_wide_nodes(api_mod, boxes, layout, spp):
    """16,256 and 65,024 paths that stay: walked over a top-level BVH, or through 8-wide nodes, by one
    thread each, they are slower than on the wavefront until 8,192 are left."""
    world, walked = _both_ways(api_mod, _metal_room(boxes, spp), layout)
    assert world < 1.25 * walked, (world, walked)


@pytest.mark.parametrize("make,first_is_open", [(lambda: _boxes(0, 600, 500, False), True), (lambda: _closed_room(600, 500, 6), False)])
def test_calls_of_an_open_scene_are_alike(api_mod, make, first_is_open):
    """A scene's first call asks after a vertex whether its paths leave, a later one, or one into a film
    of such a scene, may know: the same paths and rays, and films as in test_tail.py."""
    api = api_mod
    ctx = api.Context(0)
    d = make()
    kept = api.RenderTarget(ctx, d.width, d.height)
    b = api.load_scene(ctx, d)
    films, counts = [], []
    for k in range(4):
        rt = kept if k in (1, 2) else api.RenderTarget(ctx, d.width, d.height)
        if k == 2:
            b = api.load_scene(ctx, d)  # a new scene into a film that knows
        rt.clear()
        rt.render(b.scene, d.spp, d.params)
        films.append(rt.download())
        s = b.scene.stats()
        counts.append((s["paths"], s["extension_rays"], s["shadow_rays"]))
    assert (counts[0][1] < 2 * counts[0][0]) == first_is_open
    assert all(c == counts[0] for c in counts)
    for f in films[1:]:
        np.testing.assert_allclose(f, films[0], rtol=1e-4, atol=1e-6 * float(films[0].mean()))

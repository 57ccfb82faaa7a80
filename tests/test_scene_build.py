"""xgb_scene_build with many objects: what their kind adds to it is small against the rest.

Times are of builds of the same objects with and without the property in question, a few of
each in turn, the fastest of each; the factors allowed are ten times what the kind
costs and a tenth of what a copy, a launch or a wait per object would.
"""
import time

import numpy as np
import pytest

from oracle.bindings import load_scene as load_cpu, relmse
from xitils_gb300 import scenes
from xitils_gb300.scene import IntegratorParams, SceneDesc
from xitils_gb300.transform import translate

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api_mod():
    import __graft_entry__ as g
    g.build()
    from xitils_gb300 import api
    return api


def _sheet(n, y):
    """2 n^2 triangles facing down."""
    x, z = np.meshgrid(np.linspace(0.3, 0.7, n + 1), np.linspace(0.3, 0.7, n + 1))
    pos = np.stack([x.ravel(), y + 0.02 * np.sin(20 * x.ravel()), z.ravel()], 1).astype(np.float32)
    i = (np.arange(n)[:, None] * (n + 1) + np.arange(n)[None]).ravel()
    idx = np.stack([i, i + 1, i + n + 2, i, i + n + 2, i + n + 1], 1).ravel().astype(np.int32)
    return pos, idx


def _fastest(builds):
    best = [np.inf] * len(builds)
    for _ in range(8):
        for k, b in enumerate(builds):
            t = time.perf_counter()
            b.scene.buildAccelerationStructure()
            best[k] = min(best[k], time.perf_counter() - t)
    return best


def _objects(n, emissive):
    d = SceneDesc()
    m = d.add_mesh(*_sheet(2, 0.5))
    mat = d.emission([1, 1, 1]) if emissive else d.diffuse([0.5, 0.5, 0.5])
    for k in range(n):
        d.add_object(m, mat, translate(0.01 * k, 0, 0))
    d.set_camera(scenes.translate(0, 0, -2), 1.0, 1.0)
    return d


def test_emitters_cost_no_copies_in_a_build(api_mod):
    ctx = api_mod.Context(0)
    emissive, plain = _fastest([api_mod.load_scene(ctx, _objects(1000, e)) for e in (True, False)])
    assert emissive < 10 * plain, (emissive, plain)


@pytest.mark.parametrize("n", [45, 46], ids=["4050_triangles", "4232_triangles"])
def test_emitter_tables(api_mod, n):
    """Two objects that share an emissive mesh, of either side of 4,096 triangles, built twice."""
    d = SceneDesc(name="sheets", width=40, height=32, spp=4,
                  params=IntegratorParams(max_depth=4, rr_start=8, rr_prob=0.9, seed=3))
    light = d.emission([3.0, 2.0, 1.0])
    m = d.add_mesh(*_sheet(n, 0.9))
    d.add_object(m, light)
    d.add_object(m, light, translate(0.1, -0.2, 0.3))
    d.add_object(d.add_mesh(*scenes.quad([-1, 0, -1], [-1, 0, 2], [2, 0, 2], [2, 0, -1])), d.diffuse([0.6, 0.5, 0.4]))
    d.set_camera(scenes.look_at((0.5, 0.5, -1.0), (0.5, 0.2, 0.5), (0, 1, 0)), 1.0, 32 / 40)
    api = api_mod
    ctx = api.Context(0)
    b = api.load_scene(ctx, d)
    want = load_cpu(d, "port").render_pcg(d)
    for _ in range(2):
        rt = api.RenderTarget(ctx, d.width, d.height)
        rt.render(b.scene, d.spp, d.params)
        assert relmse(rt.download(), want) <= 1e-4  # the bound of every comparison with the oracle
        b.scene.buildAccelerationStructure()


def _quads(n, moved):
    """n quads of their own, in place or moved there."""
    d = SceneDesc()
    pos, idx = scenes.quad([0, 0, 0], [0, 0, 1], [1, 0, 1], [1, 0, 0])
    grey = d.diffuse([0.5, 0.5, 0.5])
    m = d.add_mesh(pos, idx)
    for k in range(n):
        if moved:
            d.add_object(m, grey, translate(0, 0.01 * k, 0))
        else:
            d.add_object(m, grey)
    d.set_camera(scenes.translate(0, 0, -2), 1.0, 1.0)
    return d


def test_untransformed_instances_cost_no_launches_in_a_build(api_mod):
    ctx = api_mod.Context(0)
    placed, moved = _fastest([api_mod.load_scene(ctx, _quads(1000, m)) for m in (False, True)])
    assert placed < 5 * moved, (placed, moved)


@pytest.mark.parametrize("many", [False, True], ids=["few", "many"])
def test_meshes_of_every_size_side_by_side(api_mod, many):
    """The parts of a world BVH: meshes whose root is a leaf (1 and 4 triangles), the smallest
    with a node (5), larger ones, and moved ones between them, against the oracle."""
    rng = np.random.default_rng(6)
    d = SceneDesc(name="parts", width=48, height=40, spp=2, params=IntegratorParams(max_depth=4, rr_start=8, rr_prob=0.9, seed=3))
    sizes = [1, 5, 4, 4200, 2, 3] * (4 if many else 1) + [5, 1]
    for k, n in enumerate(sizes):
        c = rng.uniform(-1, 1, (1, 1, 3))
        pos = (c + rng.normal(scale=0.25, size=(n, 1, 3)) + rng.normal(scale=0.5 * n ** -0.5, size=(n, 3, 3))).reshape(-1, 3)
        m = d.add_mesh(pos.astype(np.float32), np.arange(3 * n, dtype=np.int32))
        mat = d.diffuse(rng.uniform(0.2, 0.9, 3))
        if k % 5 == 3 and many:
            d.add_object(m, mat, translate(*rng.uniform(-0.3, 0.3, 3)))
        else:
            d.add_object(m, mat)
    d.add_object(d.add_mesh(*scenes.quad([-1, 3, -1], [1, 3, -1], [1, 3, 1], [-1, 3, 1])), d.emission([8.0, 8.0, 8.0]))
    d.set_camera(scenes.look_at((0, 0.5, -4.0), (0, 0, 0), (0, 1, 0)), 0.9, 40 / 48)
    assert (len(d.objects) > 16) == many
    api = api_mod
    ctx = api.Context(0)
    got = api.render_desc(ctx, d)
    assert got.mean() > 0
    assert relmse(got, load_cpu(d, "port").render_pcg(d)) <= 1e-4  # as every comparison with the oracle

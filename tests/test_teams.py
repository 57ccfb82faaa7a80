"""Rays traced by teams of lanes (k_trace_team, launches of few rays) against one lane per ray.

A batch and the allocation-free render give small queues to teams; a profiled render of
the same scene keeps every launch on the per-lane kernels. The nearest hit comes from the
same triangle tests, and hits within rounding of each other are decided in the instance
order by both, so both follow the same paths: films differ by the order of their sums
alone (k float terms move by at most k ulp of their magnitude, far below the 1e-4 of
the pixel allowed here; one path with another hit is far above it). The sizes give a team of 32,
16 and 8 lanes (one, two and four rays per warp) and a warp with idle teams.
"""
import ctypes as C

import numpy as np
import pytest

from xitils_gb300 import scenes
from xitils_gb300.scene import IntegratorParams, SceneDesc
from xitils_gb300.transform import scale, translate

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api_mod():
    import __graft_entry__ as g
    g.build()
    from xitils_gb300 import api
    return api


def _boxes(n, w, h):
    """A terrain with n transformed boxes and a light."""
    d = scenes.terrain(grid=65, width=w, height=h, spp=1, env_size=(128, 64))
    cpos, cidx = scenes.unit_cube_mesh()
    cube = d.add_mesh(cpos, cidx)
    grey = d.diffuse([0.6, 0.6, 0.6])
    rng = np.random.default_rng(3)
    for _ in range(n):
        x, z = rng.uniform(0.1, 0.9, 2)
        d.add_object(cube, grey, translate(float(x), 0.2, float(z)) * scale(0.04, 0.04, 0.04))
    lp, li = scenes.quad([0.3, 0.6, 0.3], [0.7, 0.6, 0.3], [0.7, 0.6, 0.7], [0.3, 0.6, 0.7])
    d.add_object(d.add_mesh(lp, li), d.emission([3, 3, 3]))
    return d


def _coincident(w, h):
    """One mesh three times in the same place, in other colours and once through a
    transform: every ray is decided by the order."""
    t = scenes.terrain(grid=65, width=w, height=h, spp=1, env_size=(128, 64))
    m = t.meshes[0]
    d = SceneDesc(name="coincident", width=w, height=h, spp=1, params=IntegratorParams(max_depth=5, rr_start=9, seed=4))
    d.camera = t.camera
    mesh = d.add_mesh(m.pos, m.idx)
    d.add_object(mesh, d.diffuse([0.9, 0.2, 0.2]))
    d.add_object(mesh, d.diffuse([0.2, 0.9, 0.2]))
    d.add_object(mesh, d.diffuse([0.2, 0.2, 0.9]), translate(0.0, 1e-9, 0.0))
    lp, li = scenes.quad([0.3, 0.6, 0.3], [0.7, 0.6, 0.3], [0.7, 0.6, 0.7], [0.3, 0.6, 0.7])
    d.add_object(d.add_mesh(lp, li), d.emission([3, 3, 3]))
    return d


CASES = {
    "room_32_lanes": lambda: scenes.occluded_room(31, 23, 3, n_boxes=600),
    "room_16_lanes": lambda: scenes.occluded_room(91, 73, 1, n_boxes=600),
    "room_8_lanes": lambda: scenes.occluded_room(128, 128, 1, n_boxes=600),    # exactly the largest queue of teams
    "room_above": lambda: scenes.occluded_room(129, 128, 1, n_boxes=600),
    "one_instance": lambda: scenes.terrain(grid=65, width=61, height=40, spp=2, env_size=(128, 64)),
    "instances": lambda: _boxes(8, 61, 40),
    "top_level": lambda: _boxes(40, 61, 40),
    "coincident": lambda: _coincident(61, 40),
    "shell": lambda: scenes.shell_fabric(40, 32, 2, grid=24),
    "normal_mapped": lambda: scenes.mfnm_at_scale(36, 30, 3, grid=65, normal_res=64, env_size=(64, 32)),
}


@pytest.mark.parametrize("name", CASES)
def test_teams_equal_lanes(api_mod, name):
    api = api_mod
    from xitils_gb300.api import IntegratorParamsC

    ctx = api.Context(0)
    desc = CASES[name]()
    b = api.load_scene(ctx, desc)
    b.scene.set_profiling(True)
    rt = api.RenderTarget(ctx, desc.width, desc.height)
    rt.render(b.scene, desc.spp, desc.params)
    want, stats = rt.download(), b.scene.stats()
    assert stats["paths"] == desc.n_paths
    b.scene.set_profiling(False)
    films = [api.RenderTarget(ctx, desc.width, desc.height) for _ in range(2)]
    api.render_batch(ctx, [(b.scene, films[0], desc.params, 0, desc.spp)], queue_capacity=1 << 18, iterations_per_sync=4)
    p = desc.params
    pc = IntegratorParamsC(p.integrator, p.max_depth, p.rr_start, p.rr_prob, p.seed, 0)
    assert ctx.lib.xgb_render_noalloc(b.scene.h, C.byref(pc), films[1].h, 0, desc.spp, None) == 0
    for f in films:
        got = f.download()
        assert np.isfinite(got).all()
        np.testing.assert_allclose(got, want, rtol=1e-4, atol=1e-6 * float(np.abs(want).mean()) + 1e-30)

"""A bound on the steps of a ray (xgb_scene_set_traversal_limits) counts the steps of full
warps, however few rays a launch has and whatever its warps wait for without a bound. The
largest step count of any ray of these films was 15 (terrain 640 x 480), 3 (Cornell box),
18 (room 640 x 480), 5 and 7 (terrain and room, 16 x 8) when every lane took its next ray at
once and a warp tested triangles when none of its lanes was looking any more; neighbours in
a warp move a ray's count by a step or two, so the bounds here are a third above. With the
waits that an unbounded render has, the counts are 92, 10, 81, 7 and 11.
"""
import numpy as np
import pytest

from xitils_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api_mod():
    import __graft_entry__ as g
    g.build()
    from xitils_gb300 import api
    return api


def _terrain(w, h):
    return scenes.terrain(grid=129, width=w, height=h, spp=1, env_size=(128, 64))


def _room(w, h):
    return scenes.occluded_room(w, h, 1, n_boxes=400, max_depth=6)


CASES = {
    "terrain": (lambda: _terrain(640, 480), 20),
    "cornell": (lambda: scenes.cornell(640, 480, 1), 4),
    "room": (lambda: _room(640, 480), 24),
    "terrain_few_rays": (lambda: _terrain(16, 8), 6),
    "room_few_rays": (lambda: _room(16, 8), 9),
}


@pytest.mark.parametrize("batch", [False, True], ids=["render", "batch"])
@pytest.mark.parametrize("name", CASES)
def test_bound_of_full_warps(api_mod, name, batch):
    api = api_mod
    make, steps = CASES[name]
    ctx = api.Context(0)
    desc = make()
    b = api.load_scene(ctx, desc)
    films = []
    for limit in (steps, 0):
        b.scene.set_traversal_limits(max_steps=limit)
        rt = api.RenderTarget(ctx, desc.width, desc.height)
        if batch:
            api.render_batch(ctx, [(b.scene, rt, desc.params, 0, 1)], queue_capacity=4096, iterations_per_sync=4)
        else:
            rt.render(b.scene, 1, desc.params)
        films.append(rt.download())
    # the order of a pixel's float sums alone (see test_tail.py)
    np.testing.assert_allclose(films[0], films[1], rtol=1e-4, atol=1e-6 * float(films[1].mean()))

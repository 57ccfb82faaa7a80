"""A training render (guided, train=True) with its shadow rays on the second stream, against the
same launches one after the other (a profiled render). The light of a visible shadow ray goes
to its path's accumulator, which the next vertex reads: both ways every path adds the same
terms in the same order, so exactly the same records carry radiance and are trained on,
the paths and rays are equal, and the film differs by the order of its sums only (see
test_side_stream.py). The network is trained after the last path of a call: both ways render
with the same one.
"""
import numpy as np
import pytest

from xitils_gb300 import scenes

pytestmark = pytest.mark.gpu

CASES = {
    "cornell": (lambda: scenes.cornell(160, 120, 2), 0),
    "cornell_refill": (lambda: scenes.cornell(96, 80, 4), 4096),  # new paths join old ones
    "room": (lambda: scenes.occluded_room(96, 80, 3, n_boxes=400), 0),        # closest hits of the flat kernel, shadow rays of the world BVH's
    "room_teams": (lambda: scenes.occluded_room(64, 60, 2, n_boxes=1200), 0),  # teams of lanes for both
}


@pytest.fixture(scope="module")
def api_mod():
    import __graft_entry__ as g
    g.build()
    from xitils_gb300 import api
    return api


@pytest.mark.parametrize("name", CASES)
def test_training_beside_equals_in_turn(api_mod, name):
    api = api_mod
    make, capacity = CASES[name]
    ctx = api.Context(0)
    desc = make()
    desc.params.queue_capacity = capacity
    got = []
    for in_turn in (True, False):
        b = api.load_scene(ctx, desc)
        guide = api.Guide(ctx, seed=4)
        guide.set_training(64, 1 << 20)
        b.scene.setGuide(guide, 0.5, train=True)
        b.scene.set_profiling(in_turn)
        rt = api.RenderTarget(ctx, desc.width, desc.height)
        rt.render(b.scene, desc.spp, desc.params)
        s = b.scene.stats()
        got.append((rt.download(), (s["paths"], s["extension_rays"], s["shadow_rays"], s["guide_train_steps"])))
    assert got[0][1] == got[1][1]
    assert got[0][1][0] == desc.n_paths and got[0][1][3] > 10
    np.testing.assert_allclose(got[1][0], got[0][0], rtol=1e-4, atol=1e-6 * float(got[0][0].mean()))

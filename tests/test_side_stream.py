"""Shadow rays on a second stream, beside the rays to the next vertex, against the same
launches one after the other (a profiled render times each stage by itself).

Both follow every path through the same draws and decisions, the streams that a visible
light commits among them, so the counts of paths and rays are equal and a film differs
by the order of its sums only: k float terms move by at most k ulp of their magnitude, and
1e-4 of the pixel (plus a millionth of the image's mean) is far above that for the few
hundred terms here and far below one path's contribution.
"""
import threading

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


def _close(a, b):
    np.testing.assert_allclose(a, b, rtol=1e-4, atol=1e-6 * float(np.abs(b).mean()) + 1e-30)


CASES = {
    "cornell": lambda: scenes.cornell(301, 263, 2),
    "cornell_refill": lambda: scenes.cornell(64, 64, 5),   # a queue smaller than the call: new paths join old ones
    "room": lambda: scenes.occluded_room(96, 80, 3, n_boxes=400),
    "normal_mapped": lambda: scenes.mfnm_at_scale(61, 53, 3, grid=65, normal_res=64, env_size=(64, 32)),
    "shell": lambda: scenes.shell_fabric(40, 32, 2, grid=24),
    "one_pixel": lambda: scenes.cornell(1, 1, 1),
}


@pytest.mark.parametrize("name", CASES)
def test_beside_equals_in_turn(api_mod, name):
    ctx = api_mod.Context(0)
    desc = CASES[name]()
    if name == "cornell_refill":
        desc.params.queue_capacity = 4096
    b = api_mod.load_scene(ctx, desc)
    b.scene.set_traversal_limits(0, 63)  # no tail launch: every vertex on the wavefront
    got = []
    for in_turn in (True, False):
        b.scene.set_profiling(in_turn)
        rt = api_mod.RenderTarget(ctx, desc.width, desc.height)
        rt.render(b.scene, desc.spp, desc.params)
        s = b.scene.stats()
        got.append((rt.download(), (s["paths"], s["extension_rays"], s["shadow_rays"])))
    assert got[0][1] == got[1][1]
    assert got[0][1][0] == desc.n_paths
    _close(got[1][0], got[0][0])


def test_renders_of_several_threads(api_mod):
    """Each render in progress has a second stream of its own."""
    import torch

    ctx = api_mod.Context(0)
    descs = [scenes.cornell(281, 240, 2, seed=k) for k in range(12)]
    built = [api_mod.load_scene(ctx, d) for d in descs]
    alone = []
    for d, b in zip(descs, built):
        rt = api_mod.RenderTarget(ctx, d.width, d.height)
        rt.render(b.scene, d.spp, d.params)
        alone.append(rt.download())
    films = [api_mod.RenderTarget(ctx, d.width, d.height) for d in descs]
    torch.cuda.synchronize()
    errors = []

    def work(d, b, f):
        try:
            stream = torch.cuda.Stream()
            f.render(b.scene, d.spp, d.params, stream=stream.cuda_stream)
            stream.synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=a) for a in zip(descs, built, films)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for f, want in zip(films, alone):
        _close(f.download(), want)

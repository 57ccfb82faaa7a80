"""Surfaces in the same place: the instance order decides each of their hits, and it is the same
in the tail launch and in the wavefront's kernels, whichever of those a scene takes. Walls
of a shell-mapped scene stand two and three times with other colours; compared as in
test_tail.py, with its tolerance.
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


def _doubled_walls(method):
    d = scenes.shell_fabric(64, 50, 2, grid=24, tex_res=64, max_depth=6, method=method)
    rng = np.random.default_rng(2)
    walls = d.objects[:4]
    for o in walls + walls[:3]:
        d.add_object(o.mesh, d.diffuse(rng.uniform(0.1, 0.9, 3)), o.transform)
    assert len(d.objects) <= 16
    return d


@pytest.mark.parametrize("method", ["shell", "svbrdf"])
@pytest.mark.parametrize("layout", ["binary", "wide8"])
def test_tail_keeps_the_order(api_mod, layout, method):
    api = api_mod
    ctx = api.Context(0)
    ctx.set_bvh_layout(layout)
    desc = _doubled_walls(method)
    b = api.load_scene(ctx, desc)
    films, counts = [], []
    for stack in (63, 0):  # a bound of its own keeps a scene on the wavefront
        b.scene.set_traversal_limits(0, stack)
        rt = api.RenderTarget(ctx, desc.width, desc.height)
        rt.render(b.scene, desc.spp, desc.params)
        films.append(rt.download())
        s = b.scene.stats()
        counts.append((s["paths"], s["extension_rays"], s["shadow_rays"]))
    assert counts[0] == counts[1]
    np.testing.assert_allclose(films[1], films[0], rtol=1e-4, atol=1e-6 * float(films[0].mean()) + 1e-30)

"""The world BVH's traversal (k_trace_world) against the kernels that walk the instances.

A scene of more than 16 instances takes it for both kinds of rays, a large one of fewer
for its shadow rays. Traversal limits other than the defaults keep a scene of several
instances on the instance-order kernels, a small path queue keeps the call on wavefront iterations, so
the same render is made both ways. Hits are decided by the same triangle tests, and
where two instances lie within rounding of each other the ray is decided in the instance
order, so both ways follow the same paths: equal counts, and films that differ by the
order of their sums alone (see test_tail.py for the tolerance). The films are large
enough (260,000 paths in flight) that every lane of the persistent kernels takes several
rays.
"""
import numpy as np
import pytest

from xitils_gb300 import scenes
from xitils_gb300.scene import IntegratorParams, SceneDesc
from xitils_gb300.transform import scale, transformTRS, translate

pytestmark = pytest.mark.gpu
CAPACITY = 260_096


@pytest.fixture(scope="module")
def api_mod():
    import __graft_entry__ as g
    g.build()
    from xitils_gb300 import api
    return api


def _boxes(n, identity=False):
    """A terrain with n small boxes (with a transform each, or moved vertices)."""
    d = scenes.terrain(grid=65, width=600, height=500, spp=1, env_size=(128, 64))
    cpos, cidx = scenes.unit_cube_mesh()
    cube = d.add_mesh(cpos, cidx)
    grey = d.diffuse([0.6, 0.6, 0.6])
    rng = np.random.default_rng(3)
    for _ in range(n):
        x, z = rng.uniform(0.1, 0.9, 2)
        if identity:
            d.add_object(d.add_mesh(cpos * 0.05 + np.float32([x, 0.2, z]), cidx), grey)
        else:
            d.add_object(cube, grey, translate(float(x), 0.2, float(z)) * scale(0.04, 0.04, 0.04))
    lp, li = scenes.quad([0.3, 0.6, 0.3], [0.7, 0.6, 0.3], [0.7, 0.6, 0.7], [0.3, 0.6, 0.7])
    d.add_object(d.add_mesh(lp, li), d.emission([3, 3, 3]))
    return d


def _coincident(same_place, n=6):
    """Quads of different colours in the same place (or a rounding apart): every ray that
    hits them is decided by the instance order."""
    d = SceneDesc(name="coincident", width=600, height=500, spp=1,
                  params=IntegratorParams(max_depth=4, rr_start=8, rr_prob=0.9, seed=4))
    pos, idx = scenes.quad([-1, 0, -1], [-1, 0, 1], [1, 0, 1], [1, 0, -1])
    rng = np.random.default_rng(8)
    for k in range(n):
        m = d.diffuse(rng.uniform(0.1, 0.9, 3))
        step = 0.0 if same_place else k * 3e-8
        if k % 3 == 2:
            d.add_object(d.add_mesh(pos, idx), m, transformTRS((0, step, 0), (0, 90 * k, 0), (1, 1, 1)))
        else:
            d.add_object(d.add_mesh(pos + np.float32([0, step, 0]), idx), m)
    lp, li = scenes.quad([-0.3, 1, -0.3], [0.3, 1, -0.3], [0.3, 1, 0.3], [-0.3, 1, 0.3])
    d.add_object(d.add_mesh(lp, li), d.emission([5, 5, 5]))
    d.set_camera(scenes.look_at((0.3, 0.8, -1.6), (0.0, 0.0, 0.0), (0, 1, 0)), 0.9, 500 / 600)
    return d


CASES = {
    "cornell": lambda: scenes.cornell(451, 347, 2),
    "room": lambda: scenes.occluded_room(456, 400, 2, n_boxes=400, max_depth=8),
    "two_quads_only": lambda: _coincident(True),
    "a_rounding_apart": lambda: _coincident(False),
    "identity_boxes": lambda: _boxes(6, identity=True),
    "moved_boxes": lambda: _boxes(6),
    "sixteen": lambda: _boxes(14),
    "many": lambda: _boxes(40),
    "many_coincident": lambda: _coincident(True, 18),
    "many_identity": lambda: _boxes(23, identity=True),
    "materials": lambda: scenes.material_zoo(448, 340, 2, sky="latlong"),
    "normal_mapped": lambda: scenes.mfnm_at_scale(400, 350, 2, grid=129, normal_res=64, env_size=(64, 32)),
    "shell": lambda: scenes.shell_fabric(400, 350, 2, grid=24, max_depth=6),
}


def _render(api, ctx, b, desc, batch):
    rt = api.RenderTarget(ctx, desc.width, desc.height)
    p = desc.params
    if batch:
        api.render_batch(ctx, [(b.scene, rt, p, 0, desc.spp)], queue_capacity=CAPACITY, iterations_per_sync=4)
        return rt.download(), None
    q = IntegratorParams(p.integrator, p.max_depth, p.rr_start, p.rr_prob, p.seed, CAPACITY)
    rt.render(b.scene, desc.spp, q)
    s = b.scene.stats()
    return rt.download(), (s["paths"], s["extension_rays"], s["shadow_rays"])


@pytest.mark.parametrize("batch", [False, True], ids=["render", "batch"])
@pytest.mark.parametrize("name", CASES)
def test_world_equals_instance_order(api_mod, name, batch):
    api = api_mod
    ctx = api.Context(0)
    desc = CASES[name]()
    b = api.load_scene(ctx, desc)
    b.scene.set_traversal_limits(0, 63)
    want, n_want = _render(api, ctx, b, desc, batch)
    b.scene.set_traversal_limits(0, 0)
    got, n_got = _render(api, ctx, b, desc, batch)
    assert n_want == n_got
    assert np.isfinite(got).all() and got.mean() > 0
    np.testing.assert_allclose(got, want, rtol=1e-4, atol=1e-6 * float(np.abs(want).mean()))

"""The tail launch (one thread per path, tail.cuh) against the wavefront iterations.

Traversal limits other than the defaults keep a render on the wavefront kernels, so the
same call is made both ways. The two follow every path through the same random draws
and decisions and only add a pixel's contributions in another order: the counts of
paths and rays are equal, and a sum of k float terms moves by at most k ulp of its
magnitude, k <= 2 * (vertices of the pixel's paths). 1e-4 of the pixel (plus a millionth
of the image's mean, for sums that nearly cancel nothing here) is far above that for
the few hundred terms of these films and far below one path's contribution.
"""
import numpy as np
import pytest

from xitils_gb300 import scenes
from xitils_gb300.scene import NAIVE, IntegratorParams, SceneDesc
from xitils_gb300.transform import scale, translate

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api_mod():
    import __graft_entry__ as g
    g.build()
    from xitils_gb300 import api
    return api


def _boxes(n):
    """A terrain with n small boxes: more than 16 instances take the top-level BVH."""
    d = scenes.terrain(grid=65, width=40, height=31, spp=2, env_size=(128, 64))
    cpos, cidx = scenes.unit_cube_mesh()
    cube = d.add_mesh(cpos, cidx)
    grey = d.diffuse([0.6, 0.6, 0.6])
    rng = np.random.default_rng(3)
    for _ in range(n):
        x, z = rng.uniform(0.1, 0.9, 2)
        d.add_object(cube, grey, translate(float(x), 0.2, float(z)) * scale(0.04, 0.04, 0.04))
    return d


def _naive():
    d = scenes.cornell(21, 17, 3)
    d.params = IntegratorParams(integrator=NAIVE, max_depth=7, rr_start=3)
    return d


def _white_box():
    """A closed white box and no depth limit: paths of a thousand vertices, some of them
    longer than one tail launch follows a path."""
    d = SceneDesc(name="white_box", width=24, height=16, spp=2,
                  params=IntegratorParams(rr_start=5, rr_prob=0.9985, seed=9))
    cpos, cidx = scenes.unit_cube_mesh()
    d.add_object(d.add_mesh(cpos * 2.0, cidx), d.diffuse([1.0, 1.0, 1.0]))
    pos, idx = scenes.quad([-0.2, 0.9, -0.2], [0.2, 0.9, -0.2], [0.2, 0.9, 0.2], [-0.2, 0.9, 0.2])
    d.add_object(d.add_mesh(pos, idx), d.emission([0.05, 0.05, 0.05]))
    d.set_camera(scenes.look_at((0.0, 0.0, -0.9), (0.0, -0.1, 0.5), (0, 1, 0)), 1.2, 16 / 24)
    return d


CASES = {
    "one_pixel": (lambda: scenes.cornell(1, 1, 1), "binary"),
    "cornell_ragged": (lambda: scenes.cornell(37, 29, 1), "binary"),
    "cornell_limit": (lambda: scenes.cornell(256, 256, 1), "binary"),      # exactly the largest call it takes whole
    "cornell_above": (lambda: scenes.cornell(257, 256, 1), "binary"),      # iterations first, then the tail
    "room_no_depth_limit": (lambda: scenes.occluded_room(64, 48, 3, n_boxes=400), "binary"),
    "wide_nodes": (lambda: scenes.occluded_room(40, 40, 2, n_boxes=400), "wide8"),
    "terrain": (lambda: scenes.terrain(grid=65, width=48, height=40, spp=2, env_size=(128, 64)), "binary"),
    "top_level_bvh": (lambda: _boxes(17), "binary"),
    "materials": (lambda: scenes.material_zoo(48, 40, 2, sky="probe"), "binary"),
    "normal_mapped": (lambda: scenes.mfnm_at_scale(36, 30, 3, grid=65, normal_res=64, env_size=(64, 32)), "binary"),
    "shell": (lambda: scenes.shell_fabric(40, 32, 2, grid=24), "binary"),
    "svbrdf": (lambda: scenes.shell_fabric(40, 32, 2, grid=24, tex_res=64, method="svbrdf"), "binary"),
    "naive": (_naive, "binary"),
    "bounded_launch": (_white_box, "binary"),
}


@pytest.mark.parametrize("name", CASES)
def test_tail_equals_wavefront(api_mod, name):
    api = api_mod
    make, layout = CASES[name]
    ctx = api.Context(0)
    ctx.set_bvh_layout(layout)
    desc = make()
    b = api.load_scene(ctx, desc)
    fp64 = name == "room_no_depth_limit"
    got = {}
    for way, stack in (("wave", 63), ("tail", 0)):
        b.scene.set_traversal_limits(0, stack)
        rt = api.RenderTarget(ctx, desc.width, desc.height, fp64=fp64, aovs=not fp64)
        rt.render(b.scene, desc.spp, desc.params)
        planes = [rt.download()] + ([] if fp64 else [rt.download_aov("albedo"), rt.download_aov("normal")])
        s = b.scene.stats()
        got[way] = planes, (s["paths"], s["extension_rays"], s["shadow_rays"])
    assert got["wave"][1] == got["tail"][1]
    assert got["wave"][1][0] == desc.n_paths
    for w, t in zip(got["wave"][0], got["tail"][0]):
        assert np.isfinite(t).all()
        np.testing.assert_allclose(t, w, rtol=1e-4, atol=1e-6 * float(np.abs(w).mean()) + 1e-30)

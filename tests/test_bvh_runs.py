"""Meshes whose clusters hardly join in the PLOC rounds (bvh_build.cu): thousands of equal
boxes, strips whose triangles grow from one to the next, and boxes whose areas are NaN, in
which no two clusters choose each other. Alone (up to 2,048 clusters are one block's)
and in a soup of other triangles. The build ends with a tree that no ray overflows, and
every ray's hit equals a brute-force search in float64 (1e-5, far above a float's rounding
of these distances; a ray within rounding of an edge may be decided either way, 1 %) and
the LBVH's.
"""
import numpy as np
import pytest

from test_bvh_build import _nearest, _soup
from xitils_gb300 import scenes
from xitils_gb300.scene import SceneDesc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api_mod():
    import __graft_entry__ as g
    g.build()
    from xitils_gb300 import api
    return api


def _one_place(n):
    return np.tile(np.float32([[0.2, 0.3, 0.4], [0.7, 0.3, 0.4], [0.2, 0.8, 0.4]]), (n, 1))


def _collapsed(n):
    return np.tile(np.float32([[0.25, 0.5, 0.75]]), (3 * n, 1))


def _strip(n):
    """Coplanar triangles side by side, each a little larger than the one before."""
    x = np.exp(np.arange(n + 1) * 2e-3)
    a, b, z = x[:-1], x[1:], np.zeros(n)
    return np.stack([np.stack([a, z, z], 1), np.stack([b, z, z], 1), np.stack([a, b - a, z], 1)], 1).reshape(-1, 3).astype(np.float32)


def _rings(n):
    """Triples of which each prefers the next: the common box of the first and the last,
    NaN in x alike, has no area, and the middle one is nearer to the last."""
    t = np.float32([[[np.nan, 0, 0], [np.nan, 1, 0], [np.nan, 0, 1]], [[5, 0, 0], [5.1, 1, 0], [5, 0, 1]],
                    [[np.nan, 0.2, 0], [np.nan, 0.9, 0], [np.nan, 0.2, 0.9]]])
    up = np.float32([0, 3, 0]) * np.arange(n, dtype=np.float32)[:, None, None, None]
    return (t[None] + up).reshape(-1, 3)


def _in_soup(pos, n=2000):
    return np.concatenate([_soup(n, 5)[0], pos])


CASES = {
    **{f"one_place_{n}": (lambda n=n: _one_place(n), "both") for n in (16, 17, 18, 33, 300, 2049, 10_000)},
    "one_place_in_a_soup": (lambda: _in_soup(_one_place(300)), "both"),
    "many_in_a_soup": (lambda: _in_soup(_one_place(10_000)), "both"),
    "collapsed_in_a_soup": (lambda: _in_soup(_collapsed(10_000)), "both"),
    "strip": (lambda: _strip(10_000), "both"),
    "strip_of_one_block": (lambda: _strip(2000), "both"),
    "rings_of_one_block": (lambda: _rings(680), "binary"),
    "rings": (lambda: _rings(3000), "binary"),
}


@pytest.mark.parametrize("layout", ["binary", "wide8"])
@pytest.mark.parametrize("name", CASES)
def test_rounds_end(api_mod, name, layout):
    api = api_mod
    make, layouts = CASES[name]
    if layouts != "both" and layout != layouts:
        pytest.skip("boxes that are not finite are not quantised")
    pos = make()
    idx = np.arange(len(pos), dtype=np.int32)
    rng = np.random.default_rng(7)
    tri = pos.reshape(-1, 3, 3)
    tri = tri[np.isfinite(tri).all(axis=(1, 2))]
    size = (tri.max(axis=1) - tri.min(axis=1)).max(axis=1)
    tri, size = tri[size > 0], size[size > 0]
    k = rng.integers(0, len(tri), 200)
    to = (tri[k].astype(np.float64) * rng.dirichlet((1, 1, 1), 200)[:, :, None]).sum(1)
    o = to - rng.uniform(1, 5, (200, 1)) * size[k, None] * np.sign(rng.normal(size=(200, 3)))
    if name.startswith("rings"):
        o = to - np.float64([1.0, 0.1, 0.1]) * rng.uniform(0.5, 2, (200, 1))
    d = to - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.concatenate([o, d, np.full((200, 1), np.inf)], axis=1).astype(np.float32)
    got = {}
    for builder in ("ploc", "lbvh"):
        ctx = api.Context(0)
        ctx.set_bvh_builder(builder)
        ctx.set_bvh_layout(layout)
        s = SceneDesc()
        s.add_object(s.add_mesh(pos, idx), s.diffuse([0.5, 0.5, 0.5]))
        s.set_camera(scenes.translate(0, 0, -2), 1.0, 1.0)
        b = api.load_scene(ctx, s)
        got[builder] = b.scene.intersect(rays)[:, 0]
        assert (b.scene.occluded(rays) == np.isfinite(got[builder])).all()
    np.testing.assert_array_equal(got["ploc"], got["lbvh"])
    want = _nearest(pos, idx, rays)
    assert np.isfinite(want).mean() >= 0.5
    same = np.isclose(got["ploc"], want, rtol=1e-5, atol=1e-5)
    assert same.mean() >= 0.99

"""Ray queries of a scene of one instance (the persistent per-lane kernel) against the same
geometry in a scene of two instances (the top-level traversal): the second instance lies
where no ray goes. Ray counts around a warp, one ray, and enough rays that every lane takes
several; finite and infinite segments, with and without a transform. Both use the same
triangle tests in the same order, so the rows are equal."""
import numpy as np
import pytest

from xitils_gb300 import scenes
from xitils_gb300.transform import transformTRS, translate

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scenes_of(request):
    import __graft_entry__ as g
    g.build()
    from xitils_gb300 import api
    ctx = api.Context(0)
    out = {}
    for moved in (False, True):
        one = scenes.terrain(grid=97, width=16, height=16, spp=1, env_size=(16, 8))
        if moved:
            one.objects[0].transform = transformTRS((0.1, 0.0, -0.2), (5, 30, -10), (1.5, 1.0, 0.8))
        b1 = api.load_scene(ctx, one)
        cpos, cidx = scenes.unit_cube_mesh()
        one.add_object(one.add_mesh(cpos, cidx), one.objects[0].material, translate(0.0, -500.0, 0.0))
        out[moved] = b1, api.load_scene(ctx, one)
    return out


@pytest.mark.parametrize("moved", [False, True], ids=["identity", "transform"])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 1000, 300_001])
def test_one_instance_equals_two(scenes_of, n, moved):
    one, two = scenes_of[moved]
    rng = np.random.default_rng(n)
    o = rng.uniform((-0.3, 0.0, -0.3), (1.3, 0.6, 1.3), (n, 3))
    d = rng.normal(size=(n, 3)) * (1.0, 0.5, 1.0)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    far = np.where(rng.random((n, 1)) < 0.5, np.inf, rng.uniform(0.01, 1.0, (n, 1)))
    rays = np.concatenate([o, d, far], axis=1).astype(np.float32)
    a, b = one.scene.intersect(rays), two.scene.intersect(rays)
    np.testing.assert_array_equal(a, b)
    assert (a[a[:, 2] < 0, 3:] == 0).all() and (a[a[:, 2] < 0, 0] == rays[a[:, 2] < 0, 6]).all()
    occ = one.scene.occluded(rays)
    np.testing.assert_array_equal(occ, two.scene.occluded(rays))
    np.testing.assert_array_equal(occ != 0, a[:, 2] >= 0)


def test_limits_count_every_step(scenes_of):
    """With a limit on the steps a one-instance scene refuses what a two-instance scene
    refuses: a tree of 18,000 triangles cannot be descended in ten nodes and leaves."""
    from xitils_gb300 import api

    rng = np.random.default_rng(0)
    o = rng.uniform((0.2, 1.0, 0.2), (0.8, 1.0, 0.8), (64, 3))
    rays = np.concatenate([o, np.tile([0.0, -1.0, 0.0], (64, 1)), np.full((64, 1), np.inf)], axis=1).astype(np.float32)
    for b in scenes_of[False]:
        want = b.scene.intersect(rays)
        try:
            b.scene.set_traversal_limits(max_steps=10)
            with pytest.raises(api.XgbError):
                b.scene.intersect(rays)
        finally:
            b.scene.set_traversal_limits(0, 0)
        np.testing.assert_array_equal(b.scene.intersect(rays), want)

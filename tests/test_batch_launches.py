"""kernel_launches of a batch: the kernels of every wavefront iteration, those of the replayed
blocks among them. Per iteration plan, generate, closest hits, shade and shadow rays; teams of
lanes for both kinds of rays in scenes of 6,000 triangles and more; the marked rays of
scenes of many instances; and once per block a plan for the last shadow rays.
"""
import pytest

from xitils_gb300 import scenes
from xitils_gb300.transform import translate

pytestmark = pytest.mark.gpu
PER_SYNC = 4


@pytest.fixture(scope="module")
def api_mod():
    import __graft_entry__ as g
    g.build()
    from xitils_gb300 import api
    return api


def _many(moved):
    """A terrain of 512 triangles with 20 more copies of it, moved or not: 10,752 in all."""
    d = scenes.terrain(grid=17, width=40, height=30, spp=2, env_size=(64, 32))
    for k in range(20):
        if moved:
            d.add_object(0, d.objects[0].material, translate(0.0, -0.2 * k, 0.9))
        else:
            d.add_object(0, d.objects[0].material)
    return d


CASES = {  # kernels per iteration
    "one_instance": (lambda: [scenes.terrain(grid=17, width=40, height=30, spp=2, env_size=(64, 32))], 5),
    "few_instances": (lambda: [scenes.cornell(40, 30, 2)], 5),
    "few_and_one": (lambda: [scenes.cornell(40, 30, 2), scenes.terrain(grid=17, width=20, height=30, spp=2, env_size=(64, 32))], 5),
    "many_instances": (lambda: [_many(False)], 8),
    "many_moved": (lambda: [_many(True)], 8),
    "many_and_large": (lambda: [_many(True), scenes.occluded_room(40, 30, 2, n_boxes=400)], 6),
    "teams": (lambda: [scenes.occluded_room(40, 30, 2, n_boxes=600)], 7),
    "teams_one_instance": (lambda: [scenes.terrain(grid=65, width=40, height=30, spp=2, env_size=(64, 32))], 7),
}


@pytest.mark.parametrize("graph", [False, True], ids=["direct", "graph"])
@pytest.mark.parametrize("name", CASES)
def test_launch_count(api_mod, name, graph):
    api = api_mod
    make, per_iteration = CASES[name]
    ctx = api.Context(0)
    jobs, keep = [], []
    for d in make():
        b = api.load_scene(ctx, d)
        keep.append(b)
        jobs.append((b.scene, api.RenderTarget(ctx, d.width, d.height), d.params, 0, d.spp))
    api.render_batch(ctx, jobs, queue_capacity=512, iterations_per_sync=PER_SYNC, use_graph=graph)
    s = api.batch_stats(ctx)
    blocks = -(-s["iterations"] // PER_SYNC)
    assert blocks > 1
    assert s["kernel_launches"] == blocks * (PER_SYNC * per_iteration + 1)

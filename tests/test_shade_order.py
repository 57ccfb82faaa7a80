"""Shading with the hits of a chunk before its misses (shade.cuh) against the queue's order.

Large launches of a scene without emitters take the first way, launches of few paths the
second, which a small queue makes of the same call. Both follow every path through the
same random draws and decisions, so the counts of paths and rays are equal, and add a
pixel's contributions in another order: an FP64 sum of k terms, all of one sign, moves by
less than k 2^-52 of its value, the download rounds it to FP32 (2^-24 relative), so two
films differ by at most one rounding step, 2^-23 < 1.2e-7, plus that; 2e-7 covers both.
"""
import numpy as np
import pytest

from xitils_gb300 import scenes

pytestmark = pytest.mark.gpu

# two waves of chunks are 2 x 152 SMs x 5 blocks x 1024 paths = 1,556,480
SIZES = {
    "last_chunk_partial": (1253, 1249, 1),   # 1,564,997 paths: 325 in the last chunk
    "whole_chunks": (1024, 1024, 4),         # the second vertex is sorted too
    "two_over": (1025, 1025, 2),             # 2,101,250 paths: two in the last chunk
    "below": (1247, 1248, 1),                # 1,556,256: the queue's order both times
}


@pytest.mark.parametrize("name", SIZES)
def test_hits_first_equals_queue_order(name):
    import __graft_entry__ as g
    g.build()
    from xitils_gb300 import api
    w, h, spp = SIZES[name]
    ctx = api.Context(0)
    desc = scenes.terrain(grid=129, width=w, height=h, spp=spp, env_size=(128, 64))
    b = api.load_scene(ctx, desc)
    films, counts = [], []
    for capacity in (0, 1 << 19):
        desc.params.queue_capacity = capacity
        rt = api.RenderTarget(ctx, w, h, fp64=True)
        rt.render(b.scene, spp, desc.params)
        films.append(rt.download())
        s = b.scene.stats()
        counts.append((s["paths"], s["extension_rays"], s["shadow_rays"]))
    assert counts[0] == counts[1]
    assert counts[0][0] == w * h * spp
    assert np.isfinite(films[0]).all() and films[0].min() >= 0.0
    np.testing.assert_allclose(films[0], films[1], rtol=2e-7, atol=0.0)

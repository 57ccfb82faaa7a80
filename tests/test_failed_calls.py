"""Calls that fail part-way leave nothing behind: the work they had put on their stream is
over when they return, and the next call is not told of their error.
"""
import ctypes as C

import numpy as np
import pytest

from xitils_gb300 import scenes

pytestmark = pytest.mark.gpu
TOO_MANY = 1 << 24  # triangles: a mesh has fewer


@pytest.fixture(scope="module")
def api_mod():
    import __graft_entry__ as g
    g.build()
    from xitils_gb300 import api
    return api


def test_refused_mesh_leaves_no_copies_behind(api_mod):
    """A mesh of 2^24 triangles is refused when its arrays are already on their way to the
    device (pinned ones by themselves). The room rendered next, on a stream of its own, takes
    its queues from the same pool: the film and the counts are those of the room alone."""
    import torch
    api = api_mod
    ctx = api.Context(0)
    desc = scenes.occluded_room(160, 120, 2, n_boxes=400)
    idx = torch.empty(3 * TOO_MANY, dtype=torch.int32).pin_memory()
    idx.copy_(torch.arange(3 * TOO_MANY, dtype=torch.int32) % 3000)
    pos = torch.from_numpy(np.random.default_rng(1).uniform(0, 1, (3000, 3)).astype(np.float32)).pin_memory()
    stream = torch.cuda.Stream()
    films, counts = [], []
    for refused in (False, True, True):
        scene = api.load_scene(ctx, desc).scene  # without queues yet
        rt = api.RenderTarget(ctx, desc.width, desc.height)
        if refused:
            mesh = C.c_void_p()
            p = C.cast(pos.data_ptr(), C.POINTER(C.c_float))
            st = ctx.lib.xgb_mesh_create(ctx.h, 3000, p, None, None, None, None, 12, 8, 3 * TOO_MANY,
                                         C.cast(idx.data_ptr(), C.POINTER(C.c_int32)), C.byref(mesh))
            assert st != 0 and not mesh
        rt.render(scene, desc.spp, desc.params, 0, stream=stream.cuda_stream)
        films.append(rt.download(stream=stream.cuda_stream))
        s = scene.stats()
        counts.append((s["paths"], s["extension_rays"], s["shadow_rays"]))
    assert counts[1] == counts[0] and counts[2] == counts[0]
    for f in films[1:]:
        # the order of a pixel's float sums alone (see test_tail.py)
        np.testing.assert_allclose(f, films[0], rtol=1e-4, atol=1e-6 * float(films[0].mean()))


def test_refused_allocation_is_reported_once(api_mod):
    """A texture of 640 GB does not fit; the calls after it succeed."""
    api = api_mod
    ctx = api.Context(0)
    texel = (C.c_float * 3)(0.5, 0.5, 0.5)
    tex = C.c_void_p()
    assert ctx.lib.xgb_texture_create(ctx.h, 200_000, 200_000, 3, texel, 0, 0, C.byref(tex)) != 0 and not tex
    api.Texture(ctx, np.full((4, 4, 3), 0.25, np.float32))
    desc = scenes.terrain(grid=33, width=24, height=20, spp=1, env_size=(16, 8))
    b = api.load_scene(ctx, desc)
    rt = api.RenderTarget(ctx, desc.width, desc.height)
    rt.render(b.scene, desc.spp, desc.params)
    assert np.isfinite(rt.download()).all() and b.scene.stats()["paths"] == desc.n_paths

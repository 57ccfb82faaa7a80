"""The world BVH of a scene of several instances is a copy that may be left out: it leaves
the memory that a program had before for its queues, films and tensors.

The device is filled up to a known rest (one allocation, of the size that CUDA reports as
free less that rest). Two meshes of 1.2 million triangles have copies of 269 MB: with 1.6 GB
left they are not made; with 2.5 GB left they are, and a render or a batch whose queues
need 2.44 GB gives them back. Films equal those of the same calls with room for everything (the order
of a pixel's float sums alone, see test_tail.py).
"""
import gc

import numpy as np
import pytest

from xitils_gb300 import scenes
from xitils_gb300.scene import IntegratorParams, SceneDesc

pytestmark = pytest.mark.gpu
MB = 1 << 20


@pytest.fixture(scope="module")
def api_mod():
    import __graft_entry__ as g
    g.build()
    from xitils_gb300 import api
    return api


def _two_sheets(width, height, spp):
    n = 775
    x, z = np.meshgrid(np.linspace(-1, 1, n + 1), np.linspace(-1, 1, n + 1))
    i = (np.arange(n)[:, None] * (n + 1) + np.arange(n)[None]).ravel()
    idx = np.stack([i, i + n + 2, i + 1, i, i + n + 1, i + n + 2], 1).ravel().astype(np.int32)
    d = SceneDesc(name="two_sheets", width=width, height=height, spp=spp,
                  params=IntegratorParams(max_depth=3, rr_start=8, rr_prob=0.9, seed=2))
    for k in range(2):
        pos = np.stack([x.ravel(), 0.05 * np.sin(9 * x + 5 * z).ravel() - 0.5 * k, z.ravel()], 1).astype(np.float32)
        d.add_object(d.add_mesh(pos, idx), d.diffuse([0.5 + 0.2 * k, 0.6, 0.4]))
    lp, li = scenes.quad([-0.3, 1, -0.3], [0.3, 1, -0.3], [0.3, 1, 0.3], [-0.3, 1, 0.3])
    d.add_object(d.add_mesh(lp, li), d.emission([5, 5, 5]))
    d.set_camera(scenes.look_at((0.3, 0.8, -1.6), (0.0, 0.0, 0.0), (0, 1, 0)), 0.9, height / width)
    return d


class _Filled:
    """All of the device's memory but `rest` bytes (and what the context's pool holds unused)."""

    def __init__(self, rest):
        import torch
        torch.cuda.synchronize()
        gc.collect()
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info(0)[0]
        self.block = torch.empty(free - rest, dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        import torch
        self.block = None
        torch.cuda.empty_cache()


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info(0)[0]


@pytest.fixture(scope="module")
def sheets(api_mod):
    return _two_sheets(1024, 1024, 13)


def _build_without_copies(scene):
    with _Filled(1500 * MB):
        before = _free()
        scene.buildAccelerationStructure()
        assert before - _free() < 64 * MB


def _build_with_copies(scene):
    before = _free()
    scene.buildAccelerationStructure()
    assert before - _free() > 100 * MB  # the pool may hold up to 128 MB of them unused


def test_copies_leave_room(api_mod, sheets):
    ctx = api_mod.Context(0)
    b = api_mod.load_scene(ctx, sheets)
    _build_without_copies(b.scene)
    _build_with_copies(b.scene)


@pytest.mark.parametrize("batch", [False, True], ids=["render", "batch"])
def test_queues_take_the_place_of_the_copies(api_mod, sheets, batch):
    api = api_mod
    ctx = api.Context(0)
    scene = api.load_scene(ctx, sheets).scene
    rt = api.RenderTarget(ctx, sheets.width, sheets.height)
    p = sheets.params

    def call(spp, capacity):
        rt.clear()
        if batch:
            api.render_batch(ctx, [(scene, rt, p, 0, spp)], queue_capacity=capacity, iterations_per_sync=4)
        else:
            rt.render(scene, spp, IntegratorParams(p.integrator, p.max_depth, p.rr_start, p.rr_prob, p.seed, capacity))
        return rt.download()

    for _ in range(2):  # every kernel's local memory is there before the device is filled
        call(1, 65536)
        _build_without_copies(scene)
    capacity = 2329 * MB // (188 if batch else 208)  # bytes per path
    with _Filled(2400 * MB):
        _build_with_copies(scene)
        squeezed = call(sheets.spp, capacity)
    scene.buildAccelerationStructure()
    want = call(sheets.spp, capacity)
    assert np.isfinite(want).all() and want.mean() > 0
    np.testing.assert_allclose(squeezed, want, rtol=1e-4, atol=1e-6 * float(want.mean()))

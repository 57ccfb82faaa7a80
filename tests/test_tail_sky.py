"""Scenes without lights end in a tail launch from 524,288 paths on (xgb_kernels.h::tailMaxPaths):
exactly that many camera paths, which never see the wavefront, and a row more. Against the
wavefront alone, which traversal limits other than the defaults keep: the same paths and
rays, and a pixel's few contributions in the order of its path, so the films agree to the
rounding of their sums (1e-4 of a pixel, as in test_tail.py, is far above that and far
below one path's contribution).
"""
import numpy as np
import pytest

from xitils_gb300 import scenes
from xitils_gb300.scene import NAIVE, IntegratorParams

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("naive", [False, True], ids=["standard", "naive"])
@pytest.mark.parametrize("width,height,spp", [(1024, 512, 1), (1024, 513, 1), (257, 255, 8), (331, 397, 4)])
def test_large_tail_equals_wavefront(width, height, spp, naive):
    import __graft_entry__ as g
    g.build()
    from xitils_gb300 import api
    ctx = api.Context(0)
    desc = scenes.terrain(grid=129, width=width, height=height, spp=spp, env_size=(128, 64))
    params = IntegratorParams(integrator=NAIVE, max_depth=7, rr_start=3, seed=5) if naive else desc.params
    b = api.load_scene(ctx, desc)
    films, counts = [], []
    for stack in (63, 0):
        b.scene.set_traversal_limits(0, stack)
        rt = api.RenderTarget(ctx, width, height)
        rt.render(b.scene, spp, params)
        films.append(rt.download())
        s = b.scene.stats()
        counts.append((s["paths"], s["extension_rays"], s["shadow_rays"]))
    assert counts[0] == counts[1]
    assert counts[0][0] == width * height * spp
    assert np.isfinite(films[1]).all()
    np.testing.assert_allclose(films[1], films[0], rtol=1e-4, atol=1e-6 * float(films[0].mean()))

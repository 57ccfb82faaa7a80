"""The SVNDF fit at the edges of its two kernels' ranges (a warp or a block per texel):
the smallest and largest rate, maps just below and above 10,000 low texels, ragged
edges whose blocks have fewer samples than lanes, one sample per texel.

Against the oracle with correctly rounded functions; both take the sums in sample
order, so all texels but a few (where the C library's own square roots and divisions are
the same but an exponential of the oracle misses its rounding) agree: 99.5 % within 1e-3, the bound of
test_svndf.py.
"""
import numpy as np
import pytest

from oracle.bindings import CpuChecker
from xitils_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api_ctx():
    import __graft_entry__ as g
    g.build()
    from xitils_gb300 import api
    return api, api.Context(0)


CASES = [(1, (9, 7)), (2, (33, 31)), (3, (300, 300)), (3, (303, 301)), (8, (70, 45)), (9, (64, 50)), (13, (40, 53)),
         (16, (49, 33))]


@pytest.mark.parametrize("rate,shape", CASES)
def test_fit_matches_oracle(api_ctx, rate, shape):
    api, ctx = api_ctx
    rng = np.random.default_rng(rate)
    rgb = scenes.weave_displacement(max(shape))[: shape[0], : shape[1]]
    rgb = np.clip(rgb + rng.normal(scale=0.01, size=rgb.shape[:2] + (1,)), 0.0, 1.0).astype(np.float32)
    if rgb.shape[2] == 1:
        rgb = np.repeat(rgb, 3, axis=2)
    rgb = np.ascontiguousarray(rgb)
    lobes = api.Svndf(ctx, api.Texture(ctx, rgb, warpClamp=False), 0.05, rate, 7).lobes()
    _, want = CpuChecker("port_cr255").svndf_fit(rgb, 0.05, rate, 7, False)
    assert lobes.shape == want.shape
    assert np.isfinite(lobes).all()
    err = np.abs(lobes - want) / (np.abs(want) + 1e-3)
    assert (err.reshape(err.shape[0], err.shape[1], -1).max(-1) < 1e-3).mean() >= 0.995

"""The kernels that draw one filter image over another, at the edges of their
four pixels per thread, and turbulence with its shared lattice work, against the
oracle (0 differing pixels: integer and f64 arithmetic in the reference's order).
"""
import numpy as np
import pytest

import oracle
import resvg_gb300 as R
from filter_bench import _prim
from resvg_gb300 import _abi as A
from tests.helpers import diff_stats

pytestmark = pytest.mark.gpu


def _check(w, h, prims, merge=(), ts=(1, 0, 0, 1, 0, 0), seed=0):
    import torch
    rng = np.random.default_rng(seed)
    img = rng.integers(0, 256, (h, w, 4), dtype=np.uint8)
    img[..., 3] = np.where(img[..., 3] > 150, 255, np.where(img[..., 3] < 60, 0, img[..., 3]))
    img[..., :3] = np.minimum(img[..., :3], img[..., 3:4])
    filt = A.Filter()
    filt.x, filt.y, filt.w, filt.h = 0.0, 0.0, w / ts[0], h / ts[3]
    ref = oracle.filter_apply(img, filt, prims, merge, ts)
    t = torch.from_numpy(img).cuda()
    R.filter_apply(t, filt, prims, merge, ts)
    assert diff_stats(t.cpu().numpy(), ref) == (0, 0)


@pytest.mark.parametrize("w", [1, 3, 255, 256, 257, 1023, 1024, 1025, 1281])
@pytest.mark.parametrize("dx,dy", [(0, 0), (7, -3), (-300, 2), (5000, 0), (-1, 40)])
def test_offset_merge_and_shadow(gpu, w, dx, dy):
    h = 5
    src = A.IN_SOURCE_GRAPHIC
    _check(w, h, [_prim(w, h, A.FE_OFFSET, f=(dx, dy)),
                  _prim(w, h, A.FE_DROP_SHADOW, i=(200, 30, 60), f=(1.0, 2.5, dx, dy, 0.6)),
                  _prim(w, h, A.FE_BLEND, in1=0, in2=src, i=(A.BLEND["multiply"],)),
                  _prim(w, h, A.FE_MERGE, i=(0, 3))], (1, 2, 0), seed=w)


@pytest.mark.parametrize("octaves", [1, 2, 7])
@pytest.mark.parametrize("fractal,stitch", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("ts", [(1, 0, 0, 1, 0, 0), (1.5, 0, 0, 0.75, 0, 0)])
def test_turbulence(gpu, octaves, fractal, stitch, ts):
    w, h = 61, 43
    p = _prim(w / ts[0], h / ts[3], A.FE_TURBULENCE, i=(octaves, 11, stitch, fractal), f=(0.07, 0.031))
    _check(w, h, [p], ts=ts)

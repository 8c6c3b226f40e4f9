"""Coverage events at the edges of the event and raster kernels, against the
oracle: sub-scanlines with more crossings than a lane's column holds (31), rows
with more events than a header's count field (4,095), row pieces whose last
group is partial, ends that fall on piece boundaries, spans inside one pixel,
aliased fills.  Pixels are integers computed by integer rules: the tolerance is
0 differing pixels.
"""
import numpy as np
import pytest

import resvg_gb300 as R
from resvg_gb300 import _abi as A
from tests.helpers import base_path, diff_stats, plain_group, solid

pytestmark = pytest.mark.gpu

IDENT = (1, 0, 0, 1, 0, 0)


def _comb(w, h, teeth, seed):
    """A closed path that crosses every row 2 x teeth times: thin teeth at
    random, sometimes coinciding, positions."""
    g = np.random.default_rng(seed)
    xs = np.sort(g.uniform(0.0, w, size=2 * teeth))
    xs[::7] = np.round(xs[::7] * 4) / 4  # some ends exactly on sub-columns
    v, p = [A.MOVE], [0.0, 0.0]
    for k in range(teeth):
        a, b = xs[2 * k], xs[2 * k + 1]
        v += [A.LINE] * 4
        p += [a, 0.3, a + g.uniform(-0.6, 0.6), h - 0.2, b, h - 0.2, b, 0.4]
    v += [A.CLOSE]
    return v, p


def _tree(w, h, paths):
    t = R.Tree(w, h)
    root = t.add_group(-1, plain_group())
    for k, (v, p, rule, aa) in enumerate(paths):
        paint = solid(t, 40 + 60 * (k % 3), 200 - 50 * (k % 4), 30 * (k % 8))
        t.add_path(root, base_path(fill_paint=paint, fill_opacity=0.7 if k % 2 else 1.0, fill_rule=rule, anti_alias=aa), v, p)
    t.finalize()
    return t


def _check(oracle_mod, t, w, h, ts=IDENT):
    got = R.render(t, ts, w, h)
    ref = oracle_mod.render(t.view(), ts, w, h)
    assert diff_stats(got, ref) == (0, 0)
    assert got.any()


@pytest.mark.parametrize("aa", [1, 0])
@pytest.mark.parametrize("rule", [A.NONZERO, A.EVENODD])
@pytest.mark.parametrize("teeth", [2, 4, 8, 15, 16, 24, 40])
def test_crossings_per_row(gpu, oracle_mod, teeth, rule, aa):
    # 4 .. 80 crossings a sub-scanline: every sorting network, and past the column
    w, h = 190, 21
    _check(oracle_mod, _tree(w, h, [_comb(w, h, teeth, s) + (rule, aa) for s in range(3)]), w, h)


def test_more_events_than_the_header_counts(gpu, oracle_mod):
    # 4 sub-scanlines x 1,200 ends in a row: past the header's 12-bit count
    w, h = 1500, 3
    _check(oracle_mod, _tree(w, h, [_comb(w, h, 600, 1) + (A.EVENODD, 1)]), w, h)


@pytest.mark.parametrize("width", [31, 33, 63, 64, 65, 127, 129, 255, 257, 511, 512, 513, 1023, 1025, 2049])
@pytest.mark.parametrize("px", [0, 4, 8, 16])
def test_row_pieces(gpu, oracle_mod, width, px):
    h = 9
    tree = _tree(width, h, [_comb(width, h, k, k) + (A.NONZERO, 1) for k in (1, 3, 9)]
                 + [([A.MOVE, A.LINE, A.LINE, A.LINE, A.CLOSE], [-5, -5, width + 5, -5, width + 5, h + 5, -5, h + 5],
                     A.NONZERO, 1)])
    saved = R.get_tuning()
    R.set_tuning(0, px)
    try:
        _check(oracle_mod, tree, width, h)
        _check(oracle_mod, tree, width, h, (1.0, 0.02, 0.3, 1.0, -3.7, 0.2))
    finally:
        R.set_tuning(*saved)


def test_spans_inside_one_pixel(gpu, oracle_mod):
    """Slivers narrower than a pixel: opening and closing ends in one pixel on
    the 4th sub-scanline, touching slivers, and full pixels made of two spans."""
    paths = []
    for k in range(24):
        x, d = 1.0 + 1.375 * k, (0.25, 0.5, 0.75, 1.0)[k % 4]
        paths.append(([A.MOVE, A.LINE, A.LINE, A.LINE, A.CLOSE, A.MOVE, A.LINE, A.LINE, A.LINE, A.CLOSE],
                      [x, 0, x + d, 0, x + d, 8, x, 8, x + d, 0, x + d + 0.5, 0, x + d + 0.5, 8, x + d, 8],
                      A.EVENODD if k % 3 else A.NONZERO, 1))
    _check(oracle_mod, _tree(40, 8, paths), 40, 8)


def _contours(xs, widths, h, tilt=0.0):
    v, p = [], []
    for x, d in zip(xs, widths):
        v += [A.MOVE, A.LINE, A.LINE, A.LINE, A.CLOSE]
        p += [x, 0.0, x + d, 0.0, x + d + tilt, h, x + tilt, h]
    return v, p


@pytest.mark.parametrize("aa", [1, 0])
@pytest.mark.parametrize("rule", [A.NONZERO, A.EVENODD])
@pytest.mark.parametrize("count", [15, 16, 31, 301, 700])
def test_contours_beside_the_canvas(gpu, oracle_mod, count, rule, aa):
    """A view into a drawing: most contours lie left or right of the canvas (their
    edges run along the clip's sides), some reach into it, and the left ones leave
    a winding of zero or not."""
    w, h = 90, 6
    g = np.random.default_rng(count)
    paths = []
    for k in range(4):
        xs = np.concatenate([g.uniform(-400, -2, size=count), g.uniform(w, w + 300, size=count // 2),
                             g.uniform(-30, w - 5, size=3 + k)])
        widths = np.concatenate([g.uniform(0.2, 1.5, size=count + count // 2), g.uniform(1, 50, size=3 + k)])
        widths[::3] *= -1  # both directions
        if k % 2:
            xs = np.append(xs, -20.0)
            widths = np.append(widths, 20.0 + 3.3 * k)
        paths.append(_contours(xs, widths, float(h) - 0.3, tilt=0.4 * k) + (rule, aa))
    _check(oracle_mod, _tree(w, h, paths), w, h)


@pytest.mark.parametrize("aa", [1, 0])
@pytest.mark.parametrize("rule", [A.NONZERO, A.EVENODD])
@pytest.mark.parametrize("count", [16, 33, 64, 257, 4001])
def test_crossings_that_share_pixels(gpu, oracle_mod, count, rule, aa):
    """Hundreds of crossings of equal x, or within two pixels, on every
    sub-scanline.  The time grows with n log^2 n: 8,002 of them are no second's work."""
    import time
    w, h = 70, 3
    g = np.random.default_rng(count)
    same = _contours([20.125] * count, [7.25 + (rule == A.EVENODD and count % 2) * 0.5] * count, 3.0)
    near = _contours(33.0 + np.round(g.uniform(0, 2, size=count) * 16) / 16, g.uniform(0.05, 0.5, size=count), 2.7)
    tree = _tree(w, h, [same + (rule, aa), near + (rule, aa)])
    R.render(tree, IDENT, w, h)
    t0 = time.perf_counter()
    _check(oracle_mod, tree, w, h)
    assert time.perf_counter() - t0 < 20.0

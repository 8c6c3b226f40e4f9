"""Clip paths whose children are filled with gradients, against the oracle: an
aliased child clears its clip layer through a source of a transparent colour,
whatever its paint, and an anti-aliased one through the clear blend.  Pixels are
integers computed by integer rules: the tolerance is 0 differing pixels.
"""
import pytest

import resvg_gb300 as R
from resvg_gb300 import _abi as A
from tests.helpers import base_path, diff_stats, plain_group, rect_path, solid

pytestmark = pytest.mark.gpu

IDENT = (1, 0, 0, 1, 0, 0)


def _gradient(t, kind, opacity, stops=2):
    p = A.Paint()
    p.kind = {"linear": A.PAINT_LINEAR, "radial": A.PAINT_RADIAL, "conical": A.PAINT_RADIAL}[kind]
    p.x1, p.y1, p.x2, p.y2 = 2.0, 3.0, 40.0, 30.0
    p.cx, p.cy, p.r_ = 20.0, 20.0, 25.0
    p.fx, p.fy = (12.0, 15.0) if kind == "conical" else (20.0, 20.0)
    p.transform = A.Transform.identity()
    out = []
    for k in range(stops):
        s = A.Stop()
        s.offset, s.opacity = k / (stops - 1), opacity
        s.r, s.g, s.b = (250, 20 + 60 * (k % 3), 10) if k % 2 else (10, 90, 200)
        out.append(s)
    return t.add_paint(p, out)


@pytest.mark.parametrize("opacity", [1.0, 0.5])
@pytest.mark.parametrize("rule", [A.NONZERO, A.EVENODD])
@pytest.mark.parametrize("aa", [0, 1])
@pytest.mark.parametrize("kind", ["solid", "linear", "radial", "conical"])
def test_gradient_in_a_clip_path(gpu, oracle_mod, kind, aa, rule, opacity):
    w, h = 75, 60
    t = R.Tree(w, h)
    root = t.add_group(-1, plain_group())
    croot = t.add_group(-1, plain_group())
    paint = solid(t, 0, 0, 0) if kind == "solid" else _gradient(t, kind, opacity, 2 if rule == A.NONZERO else 5)
    # a rectangle, and a self-crossing contour over part of it
    v, p = rect_path(5, 6, 40, 40)
    t.add_path(croot, base_path(fill_paint=paint, fill_rule=rule, anti_alias=aa, fill_opacity=opacity), v, p)
    t.add_path(croot, base_path(fill_paint=paint, fill_rule=rule, anti_alias=aa),
               [A.MOVE, A.LINE, A.LINE, A.LINE, A.LINE, A.CLOSE],
               [50.3, 8.2, 70.7, 55.1, 40.4, 22.6, 72.9, 20.3, 44.8, 57.7])
    c = A.Clip()
    c.transform = A.Transform.identity()
    c.clip_path = -1
    c.root = croot
    g = t.add_group(root, plain_group(clip_path=t.add_clip(c)))
    v, p = rect_path(0, 0, w, h)
    t.add_path(g, base_path(fill_paint=solid(t, 30, 160, 90)), v, p)
    t.finalize()
    got = R.render(t, IDENT, w, h)
    ref = oracle_mod.render(t.view(), IDENT, w, h)
    assert ref[..., 3].any()
    assert diff_stats(got, ref) == (0, 0)


@pytest.mark.parametrize("opacity", [float("nan"), float("inf"), float("-inf"), -0.5, 2.0, 0.0])
def test_group_opacity_out_of_range(gpu, oracle_mod, opacity):
    """A layer whose opacity is no number, infinite or outside [0, 1] composites by
    the same arithmetic everywhere, its transparent pixels included."""
    w, h = 70, 20
    t = R.Tree(w, h)
    root = t.add_group(-1, plain_group())
    v, p = rect_path(2, 2, 60, 16)
    t.add_path(root, base_path(fill_paint=solid(t, 30, 160, 90), fill_opacity=0.8), v, p)
    g = t.add_group(root, plain_group(opacity=opacity, isolate=1))
    v, p = rect_path(20.5, 5.3, 20, 9)
    t.add_path(g, base_path(fill_paint=solid(t, 200, 60, 10), fill_opacity=0.5), v, p)
    t.finalize()
    ref = oracle_mod.render(t.view(), IDENT, w, h)
    assert diff_stats(R.render(t, IDENT, w, h), ref) == (0, 0)

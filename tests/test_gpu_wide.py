"""Surfaces and layers wider than 32,767 pixels, which filters, patterns and
isolated groups make on canvases within that limit: coverage past column 32,767,
layers that start or end far outside the canvas, aliased fills whose 16.16
coordinates wrap, and canvases at the limit, against the oracle.  Pixels are
integers computed by integer rules: the tolerance is 0 differing pixels.
"""
import pytest

import resvg_gb300 as R
from resvg_gb300 import svg
from tests.helpers import diff_stats

pytestmark = pytest.mark.gpu


def _check(oracle_mod, text, ts, w, h):
    tree = svg.load_svg(text)
    ref = oracle_mod.render(tree.view(), ts, w, h)
    assert ref[..., 3].any()
    assert diff_stats(R.render(tree, ts, w, h), ref) == (0, 0)


def _svg(w, h, defs, body):
    return ('<svg width="%d" height="%d" viewBox="0 0 %d %d" xmlns="http://www.w3.org/2000/svg"><defs>%s</defs>%s</svg>'
            % (w, h, w, h, defs, body))


# groups along a tile, every 1,000 pixels: an isolated group with an anti-aliased
# shape, and an aliased bar
def _marks(width, step=1000):
    out = []
    for x in range(0, width, step):
        out.append('<g opacity="0.7"><path d="M%d 2 L%d 13 L%d 9 Z" fill="#%02x4080"/></g>'
                   % (x + 20, x + 130, x + 10, (x // step * 5) % 256))
        out.append('<rect x="%d" y="4" width="35" height="6" fill="#2a6" shape-rendering="crispEdges"/>' % (x + 200))
    return "".join(out)


@pytest.mark.parametrize("view", [0, 30000])
@pytest.mark.parametrize("width", [32766, 32767, 32768, 32800, 45000])
def test_pattern_tile(gpu, oracle_mod, width, view):
    defs = ('<pattern id="p" patternUnits="userSpaceOnUse" width="%d" height="16">%s'
            '<rect x="30" y="13" width="%d" height="2" fill="#d33" shape-rendering="crispEdges"/></pattern>'
            % (width, _marks(width), width - 60))
    body = '<rect x="0" y="0" width="%d" height="16" fill="url(#p)"/>' % (view + 16000)
    _check(oracle_mod, _svg(16000, 16, defs, body), (1, 0, 0, 1, -view, 0), 16000, 16)


@pytest.mark.parametrize("view", [0, 4200, 33000, 65000, 69000])
def test_aliased_fills_in_a_tile_of_70000(gpu, oracle_mod, view):
    bars = "".join('<path d="M%d 1 L%d 1 L%d 15 L%d 15 Z" fill="#a%dc" fill-rule="%s" shape-rendering="crispEdges"/>'
                   % (a, b, b - 3, a + 5, k % 10, "evenodd" if k % 2 else "nonzero")
                   for k, (a, b) in enumerate([(100, 69900), (4000, 40000), (32000, 33500), (32766, 32769), (40000, 69000),
                                               (65500, 65560), (10, 32768), (69000, 69500)]))
    defs = ('<pattern id="p" patternUnits="userSpaceOnUse" width="70000" height="16">%s</pattern>' % bars)
    body = '<rect x="0" y="0" width="%d" height="16" fill="url(#p)"/>' % (view + 700)
    tree = svg.load_svg(_svg(700, 16, defs, body))
    ts = (1, 0, 0, 1, -view, 0)
    assert diff_stats(R.render(tree, ts, 700, 16), oracle_mod.render(tree.view(), ts, 700, 16)) == (0, 0)


def test_filter_surface_wider_than_the_canvas(gpu, oracle_mod):
    # the filtered layer spans five canvases; the canvas shows columns 32,000 ..
    # 48,000 of it
    w, h = 16000, 24
    marks = "".join('<g opacity="0.8"><path d="M%d 2 L%d 20 L%d 11 Z" fill="#%02x4080"/>'
                    '<rect x="%d" y="6" width="40" height="9" fill="#2a6" shape-rendering="crispEdges"/></g>'
                    % (x, x + 150, x - 40, (x * 7) % 256, x + 60) for x in range(100, 16000, 500))
    defs = ('<filter id="f" filterUnits="userSpaceOnUse" x="-40000" y="0" width="100000" height="24">'
            '<feOffset dx="1" dy="1"/></filter>')
    body = ('<g filter="url(#f)"><rect x="-40000" y="1" width="100000" height="3" fill="#cde"/>%s</g>' % marks)
    _check(oracle_mod, _svg(w, h, defs, body), (1, 0, 0, 1, 0, 0), w, h)


@pytest.mark.parametrize("rule", ["nonzero", "evenodd"])
def test_layers_that_start_and_end_outside(gpu, oracle_mod, rule):
    # isolated layers of up to five canvases, drawn from outside on both sides:
    # their fills are aliased, and most of their coordinates wrap
    w, h = 20000, 20
    shapes = [(-40000, 60000), (-39990, 15000), (-39000, 200), (-200, 12000), (-7300, 25000), (-7232, 19000), (300, 59000),
              (-7233, -7232), (12000, 26000)]
    body = "".join('<g opacity="0.6"><path d="M%d 2 L%d 1 L%d 18 L%d 19 Z M%d 5 L%d 4 L%d 12 Z" fill="#%02x6090" '
                   'fill-rule="%s"/><rect x="%d" y="8" width="300" height="3" fill="#d33"/></g>'
                   % (a, b, b - 7, a + 9, a + 50, b - 60, b - 500, 25 * k, rule, 1000 * k + 40)
                   for k, (a, b) in enumerate(shapes))
    _check(oracle_mod, _svg(w, h, "", body), (1, 0, 0, 1, 0, 0), w, h)


@pytest.mark.parametrize("w", [32735, 32736, 32766, 32767])
def test_widest_canvases(gpu, oracle_mod, w):
    body = ('<rect width="%d" height="6" fill="#cde"/>%s<path d="M%d 0 L%d 6 L%d 3 Z" fill="#a00" fill-opacity="0.6"/>'
            '<path d="M%d 1 L%d 5 L%d 2 Z" fill="#0a0" shape-rendering="crispEdges"/>'
            % (w, _marks(w, 3000), w - 90, w + 20, w - 3, w - 200, w, w - 100))
    _check(oracle_mod, _svg(w, 6, "", body), (1, 0, 0, 1, 0, 0), w, 6)

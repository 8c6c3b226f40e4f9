"""Draw setup and edge building at the edges of their warps: verbs on the
boundary of the 32 taken at a time, open and empty contours, curves of 2 to 64
steps and edges of one to hundreds of rows (against the oracle).  Integer
geometry: the tolerance is 0 differing pixels.
"""
import numpy as np
import pytest

import resvg_gb300 as R
from resvg_gb300 import _abi as A
from tests.helpers import base_path, diff_stats, plain_group, solid

pytestmark = pytest.mark.gpu

NPTS = {A.MOVE: 1, A.LINE: 1, A.QUAD: 2, A.CUBIC: 3, A.CLOSE: 0}


def _render(oracle_mod, paths, w, h, ts=(1, 0, 0, 1, 0, 0)):
    t = R.Tree(w, h)
    root = t.add_group(-1, plain_group())
    for k, (v, p) in enumerate(paths):
        t.add_path(root, base_path(fill_paint=solid(t, 200 - 40 * (k % 4), 30 + 50 * (k % 3), 90), fill_opacity=0.6,
                                   fill_rule=k & 1), v, p)
    t.finalize()
    got = R.render(t, ts, w, h)
    assert diff_stats(got, oracle_mod.render(t.view(), ts, w, h)) == (0, 0)
    return got


@pytest.mark.parametrize("moves", [1, 2, 29, 30, 31, 32, 33, 62, 63, 64, 65])
@pytest.mark.parametrize("seed", range(4))
def test_verbs_across_a_warps_chunks(gpu, moves, seed):
    """Moves repeated in front of a path draw nothing but shift its verbs over
    the 32-verb chunks the setup takes: the pixels stay those of the path alone,
    whichever verb (a close, a move, a curve) lands on the boundary."""
    g = np.random.default_rng(seed)
    v = [A.MOVE]
    while len(v) < 50:
        # contours end by a close, by the next move, or at the path's end;
        # moves and closes may follow each other
        v.append(int(g.choice([A.LINE, A.QUAD, A.CUBIC, A.CLOSE, A.MOVE], p=[0.35, 0.2, 0.2, 0.15, 0.1])))
    p = g.uniform(-20.0, 140.0, size=(sum(NPTS[x] for x in v), 2)).astype(np.float32)

    def render(front):
        t = R.Tree(120, 110)
        root = t.add_group(-1, plain_group())
        t.add_path(root, base_path(fill_paint=solid(t, 90, 160, 30), fill_opacity=0.6, fill_rule=seed & 1),
                   [A.MOVE] * front + v, np.concatenate([np.repeat(p[:1], front, axis=0), p]))
        t.finalize()
        return R.render(t, (1, 0, 0, 1, 0, 0), 120, 110)

    alone = render(0)
    assert alone.any()
    assert diff_stats(render(moves), alone) == (0, 0)


@pytest.mark.parametrize("size", [2.0, 7.0, 40.0, 300.0, 1500.0])
def test_curve_steps_and_edge_heights(gpu, oracle_mod, size):
    g = np.random.default_rng(int(size))
    paths = []
    for k in range(6):
        c = g.uniform(0.0, size, size=14)
        paths.append(([A.MOVE, A.CUBIC, A.QUAD, A.LINE, A.CLOSE], c))
    w, h = (int(size) + 9, int(size) // 2 + 9)
    _render(oracle_mod, paths, w, h)
    _render(oracle_mod, paths, w, h, (1.3, 0.2, -0.4, 0.9, -0.1 * size, 0.05 * size))


@pytest.mark.parametrize("seed", range(12))
def test_verbs_of_every_kind_match_the_oracle(gpu, oracle_mod, seed):
    """Contours of every verb, 20 to 300 of them, so that lanes other than the one
    that clears a segment slot fill it.  Even-odd: under the non-zero rule a path
    of crossing contours differs from the oracle by one level in a few pixels, where
    edges of opposite direction cross a sub-scanline at the same x.  The device
    takes the one of winding -1 first, the oracle the one that came first on the
    sub-scanline before; the span between them is then one or two, which differ by
    1 where they make a full pixel on the 4th sub-scanline."""
    g = np.random.default_rng(100 + seed)
    t = R.Tree(120, 110)
    root = t.add_group(-1, plain_group())
    for k, n in enumerate((20, 31, 32, 33, 64, 97, 300)):
        v = [A.MOVE]
        while len(v) < n:
            v.append(int(g.choice([A.LINE, A.QUAD, A.CUBIC, A.CLOSE, A.MOVE], p=[0.35, 0.2, 0.2, 0.15, 0.1])))
        p = g.uniform(2.0, 108.0, size=(sum(NPTS[x] for x in v), 2)).astype(np.float32)
        t.add_path(root, base_path(fill_paint=solid(t, 200 - 40 * (k % 4), 30 + 50 * (k % 3), 90), fill_opacity=0.6,
                                   fill_rule=A.EVENODD), v, p)
    t.finalize()
    got = R.render(t, (1, 0, 0, 1, 0, 0), 120, 110)
    assert got.any()
    assert diff_stats(got, oracle_mod.render(t.view(), (1, 0, 0, 1, 0, 0), 120, 110)) == (0, 0)


@pytest.mark.parametrize("edges", [40, 8180, 8200, 32760, 32780, 131060, 131090])
def test_edges_per_warp_of_the_binning(gpu, oracle_mod, edges):
    # counts at either side of the lines between 1, 4, 8 and 32 edges a warp, of one
    # row to the whole canvas
    w, h = 300, 64
    g = np.random.default_rng(edges)
    paths, left = [], edges
    while left > 0:
        n = min(left, 1000)
        y = g.uniform(0.5, h - 0.5, size=(n, 1)) if len(paths) % 2 else np.clip(
            np.cumsum(g.uniform(-3, 3, size=(n, 1)), axis=0) % h, 0.5, h - 0.5)
        p = np.concatenate([np.linspace(3, w - 3, n)[:, None] + g.uniform(-1, 1, size=(n, 1)), y], axis=1)
        paths.append(([A.MOVE] + [A.LINE] * (n - 1) + [A.CLOSE], p.astype(np.float32)))
        left -= n
    t = R.Tree(w, h)
    root = t.add_group(-1, plain_group())
    for k, (v, p) in enumerate(paths):
        t.add_path(root, base_path(fill_paint=solid(t, 200 - 40 * (k % 4), 30 + 50 * (k % 3), 90), fill_opacity=0.6,
                                   fill_rule=A.EVENODD), v, p)
    t.finalize()
    got = R.render(t, (1, 0, 0, 1, 0, 0), w, h)
    assert got.any()
    assert diff_stats(got, oracle_mod.render(t.view(), (1, 0, 0, 1, 0, 0), w, h)) == (0, 0)

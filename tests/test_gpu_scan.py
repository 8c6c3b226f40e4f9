"""Offsets by the scan in one block (up to 4,096 words) and by three launches
beyond: canvases whose (row, draw) slots end at either side of the limit and of
one word per thread, against the oracle.  Pixels are integers computed by integer
rules: the tolerance is 0 differing pixels.
"""
import pytest

import resvg_gb300 as R
from resvg_gb300 import _abi as A
from tests.helpers import base_path, diff_stats, plain_group, solid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("draws", [1, 3])
@pytest.mark.parametrize("slots", [1, 1022, 1023, 1024, 4094, 4095, 4096, 8191, 16382, 16383, 16384, 16400, 30000])
def test_slots_around_the_limits(gpu, oracle_mod, slots, draws):
    w, h = 6, max(1, slots // draws)
    t = R.Tree(w, h)
    root = t.add_group(-1, plain_group())
    for k in range(draws):
        # a slanted sliver over all rows: every slot holds two edges
        v = [A.MOVE, A.LINE, A.LINE, A.CLOSE]
        p = [0.3 + k, 0.0, 3.1 + k, float(h), 1.2 + k, float(h)]
        t.add_path(root, base_path(fill_paint=solid(t, 90 * k, 200, 40), fill_opacity=0.7, anti_alias=1), v, p)
    t.finalize()
    got = R.render(t, (1, 0, 0, 1, 0, 0), w, h)
    assert diff_stats(got, oracle_mod.render(t.view(), (1, 0, 0, 1, 0, 0), w, h)) == (0, 0)
    assert got.any()

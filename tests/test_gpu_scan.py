"""Offsets by the scan in one block (up to 4,096 words) and by three launches
beyond: canvases whose (row, draw) slots end at either side of the limit and of
one word per thread, against the oracle.  Pixels are integers computed by integer
rules: the tolerance is 0 differing pixels.
"""
import ctypes as C

import numpy as np
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


@pytest.mark.parametrize("n", [1, 5, 1000, 1024, 4096, 4097, 5000, 262144, 300000])
@pytest.mark.parametrize("total", [0, 1, 0xFFFFFFFE, 0xFFFFFFFF, 1 << 32, (1 << 32) + 5, 3 << 32, 1 << 40])
def test_totals_that_do_not_fit(gpu, n, total):
    """Counts whose sum passes 2^32 within one tile, within the 256 tiles summed at
    a time, or over all of them: never a wrapped total, which would size the lists
    too small."""
    L = R.lib()
    L.rgpu_test_scan.restype = C.c_int
    L.rgpu_test_scan.argtypes = [C.c_void_p, C.c_uint32, C.c_void_p, C.POINTER(C.c_uint32)]
    for heavy in {1, min(n, 3), min(n, 1024), n}:  # the counts the total is spread over
        if total // heavy >= 1 << 32:
            continue
        counts = np.zeros(n, np.uint64)
        at = np.linspace(0, n - 1, heavy).astype(np.int64)
        counts[at] = total // heavy
        counts[at[-1]] += total - int(counts.sum())
        if counts.max() >= 1 << 32:
            continue
        c32, out, tot = counts.astype(np.uint32), np.empty(n, np.uint32), C.c_uint32(7)
        assert L.rgpu_test_scan(c32.ctypes.data, n, out.ctypes.data, C.byref(tot)) == 0
        assert tot.value == min(total, 0xFFFFFFFF)
        if total < 0xFFFFFFFF:
            assert np.array_equal(out, (np.cumsum(counts) - counts).astype(np.uint32))

"""Submissions whose rows take more working memory than one pass may: rendered in
several passes over rows and streams, on every route (host, device, batch,
prepared and replayed, filters and patterns on several levels), against the
oracle.  The bound is lowered by a test hook, down to one row a pass, and an
allocation that fails makes the passes smaller.  Pixels are integers computed by
integer rules: the tolerance is 0 differing pixels.
"""
import ctypes as C

import numpy as np
import pytest

import resvg_gb300 as R
from resvg_gb300 import _abi as A
from resvg_gb300 import svg
from tests.helpers import base_path, diff_stats, plain_group, solid

pytestmark = pytest.mark.gpu

IDENT = (1, 0, 0, 1, 0, 0)


def _lib():
    L = R.lib()
    for n, args in (("rgpu_test_pass_bytes", [C.c_uint64]), ("rgpu_test_fail_allocations", [C.c_uint32]),
                    ("rgpu_trim", [])):
        getattr(L, n).restype = C.c_int
        getattr(L, n).argtypes = args
    return L


@pytest.fixture(params=[1, 5000, 60_000, 300_000])
def pass_bytes(request, gpu):
    L = _lib()
    L.rgpu_test_pass_bytes(request.param)
    yield request.param
    L.rgpu_test_pass_bytes(0)


LEVELS = """<svg viewBox="0 0 120 90" xmlns="http://www.w3.org/2000/svg"><defs>
  <pattern id="p" patternUnits="userSpaceOnUse" width="17" height="13"><rect width="9" height="8" fill="#2a6"/>
    <circle cx="12" cy="8" r="4" fill="#d33" fill-opacity="0.7"/></pattern>
  <pattern id="q" patternUnits="userSpaceOnUse" width="31" height="23"><rect width="25" height="19" fill="url(#p)"/></pattern>
  <filter id="f"><feGaussianBlur stdDeviation="2"/><feOffset dx="3" dy="2"/></filter>
  <clipPath id="c"><circle cx="60" cy="45" r="40"/></clipPath></defs>
  <rect width="120" height="90" fill="#cde"/>
  <g filter="url(#f)"><rect x="10" y="10" width="60" height="40" fill="url(#q)"/>
    <g filter="url(#f)" opacity="0.8"><circle cx="70" cy="50" r="25" fill="#36c"/></g></g>
  <g clip-path="url(#c)"><path d="M0 0 L120 30 L20 90 Z" fill="url(#p)" stroke="#000" stroke-width="2"/></g></svg>"""


def _trees():
    return [(R.Tree.generate(1, seed=5, index=0, scale=0.02), (0.2, 0, 0, 0.15, 0, 0), 205, 154),
            (R.Tree.generate(2, seed=1, index=0, scale=0.03), (0.1, 0, 0, 0.1, 0, 0), 205, 130),
            (svg.load_svg(LEVELS), (2.5, 0, 0, 2.5, 0, 0), 300, 225)]


def test_host_and_device_calls(pass_bytes, oracle_mod):
    import torch
    for tree, ts, w, h in _trees():
        if pass_bytes < 5000 and w * h > 40000:
            continue
        ref = oracle_mod.render(tree.view(), ts, w, h)
        assert ref.any()
        assert diff_stats(R.render(tree, ts, w, h), ref) == (0, 0)
        dev = torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
        R.render_device(tree, ts, w, h, dev.data_ptr(), 4 * w)
        torch.cuda.synchronize()
        assert diff_stats(dev.cpu().numpy(), ref) == (0, 0)


def test_batch_and_prepared_scene(pass_bytes, oracle_mod):
    import torch
    sets = _trees()[:2] if pass_bytes < 5000 else _trees()
    trees, ts, ws, hs = (list(x) for x in zip(*sets))
    refs = [oracle_mod.render(t.view(), x, w, h) for t, x, w, h in sets]
    pix = [torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda") for w, h in zip(ws, hs)]
    ptrs = [p.data_ptr() for p in pix]

    def check():
        torch.cuda.synchronize()
        for p, ref in zip(pix, refs):
            assert diff_stats(p.cpu().numpy(), ref) == (0, 0)
            p.zero_()

    R.render_batch(trees, ts, ws, hs, ptrs)
    check()
    sc = R.Scene(trees, ts, ws, hs, ptrs)
    stream = torch.cuda.Stream()
    for _ in range(4):  # sizing, capture, replays
        torch.cuda.synchronize()
        sc.render(stream.cuda_stream)
        sc.check()
        check()
    many = sc.info()
    _lib().rgpu_test_pass_bytes(0)
    one = R.Scene(trees, ts, ws, hs, ptrs)
    one.render(stream.cuda_stream)
    one.check()
    check()
    info = one.info()
    for k in ("binned_edges", "edges", "work_items", "segments"):
        assert many[k] == info[k]
    assert many["kernel_launches"] > info["kernel_launches"]


def test_failed_allocations_make_smaller_passes(gpu, oracle_mod):
    import torch
    L = _lib()
    L.rgpu_trim()

    def tree(h):
        t = R.Tree(64, h)
        root = t.add_group(-1, plain_group())
        g = np.random.default_rng(3)
        for k in range(40):
            p = (g.uniform(0, 1, size=(5, 2)) * (64, h)).astype(np.float32)
            t.add_path(root, base_path(fill_paint=solid(t, 9 * k % 255, 200 - 3 * k, 90), fill_opacity=0.6, fill_rule=k & 1),
                       [A.MOVE, A.LINE, A.LINE, A.LINE, A.LINE, A.CLOSE], p)
        t.finalize()
        return t

    small, large = tree(16), tree(1200)
    dev = torch.zeros((1200, 64, 4), dtype=torch.uint8, device="cuda")
    ref = oracle_mod.render(large.view(), IDENT, 64, 1200)
    R.render_device(small, IDENT, 64, 16, dev.data_ptr(), 256)
    launches = R.stats()["kernel_launches"]
    for fail in (1, 3):
        dev.zero_()
        torch.cuda.synchronize()
        L.rgpu_test_fail_allocations(fail)  # the slot buffers come first: the records fit those of the small render
        try:
            R.render_device(large, IDENT, 64, 1200, dev.data_ptr(), 256)
        finally:
            L.rgpu_test_fail_allocations(0)
        torch.cuda.synchronize()
        assert R.stats()["kernel_launches"] > launches + 4
        assert diff_stats(dev.cpu().numpy(), ref) == (0, 0)
        L.rgpu_trim()
        R.render_device(small, IDENT, 64, 16, dev.data_ptr(), 256)


def test_more_binned_edges_than_32_bits_number(gpu, oracle_mod):
    """4.4 G binned edges in 4.4 M slots: 1,000 paths, each a triangle in view and 500
    contours left of it over all 4,400 rows.  One pass cannot number them."""
    w, h, n = 64, 4400, 500
    t = R.Tree(w, h)
    root = t.add_group(-1, plain_group())
    g = np.random.default_rng(1)
    for k in range(1000):
        x, (y0, y1) = 64 * g.uniform(), np.sort(g.uniform(0, h, 2))
        xs = g.uniform(-300, -5, n)
        lo, hi = np.full(n, -1.0), np.full(n, h + 1.0)
        p = np.concatenate([[x, y0, x + 9, y1, x - 5, y1],
                            np.stack([xs, lo, xs + 2, lo, xs + 2, hi, xs, hi], 1).ravel()]).astype(np.float32)
        t.add_path(root, base_path(fill_paint=solid(t, k % 256, 99, 255 - k % 256), fill_opacity=0.5, fill_rule=k & 1),
                   [A.MOVE, A.LINE, A.LINE, A.CLOSE] + [A.MOVE, A.LINE, A.LINE, A.LINE, A.CLOSE] * n, p)
    t.finalize()
    got = R.render(t, IDENT, w, h)
    assert diff_stats(got, oracle_mod.render(t.view(), IDENT, w, h)) == (0, 0)
    _lib().rgpu_trim()

"""The differentiable renderer's row kernels at the edges of their splits: one
pixel to the widest canvas (lanes that scan 1 to 32 pixels), groups that the
canvas cuts, path counts around the 32 masks read at a time, and batches large
enough for two groups per warp, against the FP64 reference.

Tolerances: the FP32 forward within 2e-4 of FP64 (values in [0, 1]); a random
directional derivative within 1e-3 of the sum of its terms' magnitudes.
"""
import numpy as np
import pytest

from resvg_gb300 import soft

pytestmark = pytest.mark.gpu

KEYS = ("points", "colors", "stop_offsets", "stop_colors", "sigma", "opacity")


def _arrays(scenes, w, h, paths, seed):
    a = soft.make_scenes(seed=seed, scenes=scenes, size=max(w, h), paths=paths, min_segs=2, max_segs=5)
    s = np.array([w, h], np.float32) / max(w, h)
    a["width"], a["height"] = w, h
    # a margin on every side: lines left of, right of and above the canvas too
    a["points"] = ((a["points"] * 1.2 - 0.1 * max(w, h)) * s).astype(np.float32)
    a["grad_line"] = (a["grad_line"] * np.tile(s, 2)).astype(np.float32)
    return a


@pytest.mark.parametrize("scenes,w,h,paths", [
    (1, 1, 5, 2), (2, 31, 9, 3), (1, 32, 8, 1), (1, 33, 20, 33), (2, 65, 3, 64), (1, 127, 7, 32), (3, 255, 6, 5),
    (1, 257, 12, 31), (1, 511, 5, 2), (1, 513, 5, 3), (1, 1024, 4, 2), (8, 256, 128, 2), (9, 250, 128, 3)])
def test_rows_match_fp64(gpu, oracle_mod, scenes, w, h, paths):
    import torch
    a = _arrays(scenes, w, h, paths, seed=w + h)
    sc = soft.Scenes(a)
    image, blurred = soft.forward(sc)
    im64, bl64 = oracle_mod.soft_forward(a)
    assert np.abs(image.cpu().numpy() - im64).max() <= 2e-4
    assert np.abs(blurred.cpu().numpy() - bl64).max() <= 2e-4
    rng = np.random.default_rng(3)
    target = torch.from_numpy(rng.uniform(0, 1, size=im64.shape).astype(np.float32)).cuda()
    _, g = soft.mse(blurred, target)
    grads = soft.backward(sc, image, g)
    v = {k: rng.normal(size=a[k].shape) for k in KEYS}
    terms = np.concatenate([(grads[k].double().cpu().numpy() * v[k]).ravel() for k in KEYS])
    _, ref = oracle_mod.soft_dloss(a, target.cpu().numpy(), v)
    assert abs(terms.sum() - ref) <= 1e-3 * np.abs(terms).sum()


def test_rows_of_a_large_scene(gpu, oracle_mod):
    # more scratch than a slice holds: the rows of one scene in slices (280 and 10
    # forward, 56 rows at a time in the adjoint)
    test_rows_match_fp64(gpu, oracle_mod, 1, 1024, 290, 1400)


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("gradient", [0, 1])
def test_non_finite_paint_stays_in_its_coverage(gpu, bad, gradient):
    """A path with an infinite or NaN colour spoils the pixels it covers and no
    others: those keep the colours of a scene where it is transparent."""
    w, h = 70, 16
    a = soft.make_scenes(seed=5, scenes=1, size=w, paths=3, min_segs=2, max_segs=3)
    a["width"], a["height"] = w, h
    a["paint_kind"][:] = (0, gradient, 0)
    off = a["seg_offset"].astype(int)
    a["points"] = a["points"].astype(np.float32)
    a["points"][:, 1] *= h / w
    lo, hi = 3 * off[1], 3 * off[2]
    a["points"][lo:hi, 0] = 33.0 + (a["points"][lo:hi, 0] % 9.0)  # columns 33 .. 42 of a 32-pixel group
    b = {k: np.copy(v) if isinstance(v, np.ndarray) else v for k, v in a.items()}
    a["colors"][1], a["stop_colors"][1] = bad, bad
    b["colors"][1], b["stop_colors"][1] = 0.0, 0.0
    img, ref = (soft.forward(soft.Scenes(x))[0].cpu().numpy() for x in (a, b))
    for part in (slice(0, 33), slice(43, w)):
        assert np.isfinite(img[:, :, part]).all() and np.array_equal(img[:, :, part], ref[:, :, part])
    assert not np.isfinite(img[:, :, 33:43]).all()  # the covered ones are spoilt


def _failure_hooks():
    import ctypes as C
    import resvg_gb300 as R
    L = R.lib()
    L.rgpu_test_fail_allocations.argtypes = [C.c_uint32]
    return L


@pytest.mark.parametrize("fail", [1, 3, 6])
def test_short_memory_makes_smaller_slices(gpu, fail):
    """Failed allocations of the scratch halve the slices, down to one row; the
    results do not depend on them (but for the order of the gradients' sums)."""
    L = _failure_hooks()
    L.rgpu_trim()
    # no more lines, but more paths: nothing but the scratch grows
    few = dict(soft.make_scenes(seed=2, scenes=3, size=96, paths=2, min_segs=64, max_segs=64), height=41)
    many = dict(soft.make_scenes(seed=3, scenes=3, size=96, paths=32, min_segs=2, max_segs=4), height=41)
    assert many["seg_offset"][-1] <= few["seg_offset"][-1]

    def step(arrays):
        sc = soft.Scenes(arrays)
        image, blurred = soft.forward(sc)
        return image, blurred, soft.backward(sc, image, blurred)

    ref = step(many)
    L.rgpu_trim()
    step(few)
    L.rgpu_test_fail_allocations(fail)
    try:
        got = step(many)
    finally:
        L.rgpu_test_fail_allocations(0)
    assert np.array_equal(got[0].cpu().numpy(), ref[0].cpu().numpy())
    assert np.array_equal(got[1].cpu().numpy(), ref[1].cpu().numpy())
    for k in KEYS:
        a, b = got[2][k].cpu().numpy(), ref[2][k].cpu().numpy()
        assert np.abs(a - b).max() <= 1e-4 * max(1.0, np.abs(b).max())


def test_trim_gives_the_scratch_back(gpu):
    import torch
    L = _failure_hooks()
    a = soft.make_scenes(seed=4, scenes=4, size=512, paths=64, min_segs=2, max_segs=3)
    sc = soft.Scenes(a)
    image, blurred = soft.forward(sc)
    soft.backward(sc, image, blurred)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    assert L.rgpu_trim() == 0
    # 4 x 512^2 pixels x 64 paths x 20 bytes
    assert torch.cuda.mem_get_info()[0] - free >= 1_300_000_000
    again, _ = soft.forward(sc)
    assert torch.equal(again, image)


@pytest.mark.parametrize("count", [1, 2, 255, 256, 257, 262143, 262145, 3_000_001])
def test_loss_is_the_same_every_time(gpu, count):
    """The loss against float64, and to the bit on every call: its sum does not
    depend on the order in which blocks finish.  Tolerance: a thread's float sum of
    at most 12 squares, a factor 1 / count and the result each rounded to 24 bits:
    14 roundings of 2^-24."""
    import ctypes as C
    import resvg_gb300 as R
    import torch
    L = R.lib()
    soft._declare(L)
    g = torch.Generator(device="cuda").manual_seed(count)
    a = torch.rand(count, device="cuda", generator=g)
    b = torch.rand(count, device="cuda", generator=g)
    out = []
    for _ in range(4):
        loss, grad = torch.full((1,), 7.0, device="cuda"), torch.empty_like(a)
        torch.cuda.synchronize()
        assert L.rgpu_soft_mse(a.data_ptr(), b.data_ptr(), count, loss.data_ptr(), grad.data_ptr(), None) == 0
        out.append(float(loss))
        assert torch.equal(grad, 2.0 * (a - b) * np.float32(1.0 / np.float32(count)))
    assert len(set(out)) == 1
    # differences in float32, as the kernel takes them
    ref = float((a - b).double().pow(2).mean())
    assert abs(out[0] - ref) <= 14 * 2.0 ** -24 * ref

"""Workloads of the renderer through its public entry points, for timing.

A case is a dict of plain values.  `listed()` names the representative ones,
`draw(rng)` gives more of the same ranges, `prepare(case, seed)` makes what a
program holds before the call, `run(state)` is one pass, `work(case)` the bytes
and operations the pass cannot do without, and `exact(case, seed)` the result
in 64 bits where outputs are computed numbers (pixels are bytes and have none).

Kinds:
  host    resvg_render: one tree onto a host pixmap (flatten, upload, render,
          read back).
  device  rgpu_render_device: one tree onto a device pixmap.
  frame   a prepared scene replayed onto a cleared device pixmap.
  batch   rgpu_render_batch: many trees in one call, flattened each time.
  gallery many trees as one prepared scene, replayed.
  filter  a filter chain applied to a device image.
  soft    one optimisation step of the differentiable renderer: forward, MSE
          against a target, adjoint.
"""
import math

import numpy as np
import torch
import torch.utils.checkpoint

import resvg_gb300 as R
from resvg_gb300 import _abi as A
from resvg_gb300 import soft

# canvas sides of the seeded generator's scenes, by its config number
SIDE = {0: 512.0, 1: 1024.0, 2: 2048.0}


def listed():
    return [
        # an icon drawn by a toolbar or a thumbnailer: call latency
        {"name": "icon", "kind": "host", "config": 0, "scale": 0.03, "w": 48, "h": 48},
        # a page illustration with strokes, clips and a mask, at the odd size a
        # layout asks for
        {"name": "page", "kind": "host", "config": 1, "scale": 0.2, "w": 1021, "h": 767},
        # a drawing of plain fills redrawn by a viewer
        {"name": "drawing", "kind": "frame", "config": 0, "scale": 1.0, "w": 512, "h": 512},
        # a dense poster: gradients, strokes, nested clips, masks
        {"name": "poster", "kind": "frame", "config": 1, "scale": 1.0, "w": 1024, "h": 1024},
        # a large canvas whose content goes through a filter chain
        {"name": "filtered_poster", "kind": "frame", "config": 2, "scale": 1.0, "w": 2048, "h": 2048},
        # a server's request: a few dozen mixed drawings flattened and rendered in one call
        {"name": "batch", "kind": "batch", "scenes": 96},
        # mixed drawings kept as one prepared scene and redrawn
        {"name": "gallery", "kind": "gallery", "scenes": 256},
        # a user interface's shadowed and tinted layer, full HD
        {"name": "effects", "kind": "filter", "chain": "effects", "w": 1920, "h": 1080, "radius": 6.0},
        # procedural texture: noise, displacement, lighting, convolution, odd size
        {"name": "texture", "kind": "filter", "chain": "texture", "w": 1023, "h": 769, "radius": 3.0},
        # a small-sigma blur (the recursive filter) and a morphology on a large layer
        {"name": "soften", "kind": "filter", "chain": "soften", "w": 2048, "h": 2048, "radius": 1.5},
        # one image being fitted: a step of a few hundred microseconds to a millisecond
        {"name": "fit_one", "kind": "soft", "scenes": 1, "w": 200, "h": 150, "paths": 24},
        # a batch of fits at the differentiable form's own size
        {"name": "fit_batch", "kind": "soft", "scenes": 16, "w": 256, "h": 256, "paths": 64},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _ilog(rng, lo, hi):
    return max(lo, min(hi, int(round(_log(rng, lo, hi)))))


def draw(rng):
    kind = rng.choice(["host", "host", "device", "frame", "frame", "batch", "gallery", "filter", "filter", "soft",
                       "soft"])
    if kind in ("host", "device", "frame"):
        config = rng.choice([0, 0, 1, 1, 1, 2])
        top = 1024 if config < 2 else 2048
        w = _ilog(rng, 32, top)
        h = max(32, min(top, int(round(w * _log(rng, 0.5, 2.0)))))
        return {"kind": kind, "config": config, "scale": round(_log(rng, 0.03, 1.0), 4), "w": w, "h": h}
    if kind == "batch":
        return {"kind": kind, "scenes": _ilog(rng, 8, 96)}
    if kind == "gallery":
        return {"kind": kind, "scenes": _ilog(rng, 8, 192)}
    if kind == "filter":
        chain = rng.choice(["effects", "texture", "soften"])
        w = _ilog(rng, 64, 2048)
        h = max(48, min(2048, int(round(w * _log(rng, 0.5, 2.0)))))
        radius = rng.uniform(0.5, 1.9) if chain == "soften" else rng.uniform(2.0, 12.0)
        return {"kind": kind, "chain": chain, "w": w, "h": h, "radius": round(radius, 3)}
    w, h = _ilog(rng, 48, 640), _ilog(rng, 48, 640)
    paths = _ilog(rng, 4, 64)
    most = max(1, int(16 * 256 * 256 * 64 / (w * h * paths)))
    return {"kind": kind, "scenes": _ilog(rng, 1, min(16, most)), "w": w, "h": h, "paths": paths}


# ---------------------------------------------------------------- prepare

class _Render:
    """Trees and their device pixmaps (one buffer), on a stream of the program's own."""

    def __init__(self, kind, trees, transforms, sizes):
        self.kind, self.trees, self.transforms = kind, trees, transforms
        self.ws, self.hs = [w for w, _ in sizes], [h for _, h in sizes]
        offs, total = [], 0
        for w, h in sizes:
            offs.append(total)
            total += (w * h * 4 + 255) // 256 * 256
        self.pix = torch.zeros(total, dtype=torch.uint8, device="cuda")
        self.ptrs = [self.pix.data_ptr() + o for o in offs]
        self.stream = torch.cuda.Stream()
        self.scene = None
        if kind in ("frame", "gallery"):
            self.scene = R.Scene(trees, transforms, self.ws, self.hs, self.ptrs)
            for _ in range(2):  # sizes the work buffers, then captures the graph
                self.scene.render(self.stream.cuda_stream)
            self.scene.check()
        torch.cuda.synchronize()


def _tree(config, seed, index, scale, w, h):
    tree = R.Tree.generate(config, seed=seed, index=index, scale=scale)
    tree.view()
    side = SIDE[config]
    return tree, (w / side, 0, 0, h / side, 0, 0)


def _sides(scenes):
    """Square canvases of a set of drawings, log-uniform 64..1024, the same for every seed."""
    g = np.random.default_rng(scenes)
    return [(int(v), int(v)) for v in np.rint(np.exp(g.uniform(np.log(64.0), np.log(1024.0), size=scenes)))]


def _prim(w, h, kind, in1, in2=A.IN_SOURCE_GRAPHIC, i=(), f=(), linear=0):
    p = A.Primitive()
    p.kind, p.in1, p.in2, p.linear_rgb = kind, in1, in2, linear
    p.x, p.y, p.w, p.h = 0.0, 0.0, float(w), float(h)
    for k, v in enumerate(i):
        p.i[k] = int(v)
    for k, v in enumerate(f):
        p.f[k] = float(v)
    return p


def _chain(name, w, h, radius):
    """(primitives, merge inputs) of a filter; inputs name earlier primitives."""
    src = A.IN_SOURCE_GRAPHIC
    P = lambda *a, **k: _prim(w, h, *a, **k)  # noqa: E731
    if name == "effects":
        ct = P(A.FE_COMPONENT_TRANSFER, 2, i=[A.TF_LINEAR, A.TF_GAMMA, A.TF_TABLE, A.TF_IDENTITY, 0, 0, 3, 0])
        ct.f[0], ct.f[1] = 1.1, -0.05
        ct.f[16], ct.f[17], ct.f[18] = 1.0, 0.8, 0.0
        ct.f[32], ct.f[33], ct.f[34] = 0.0, 0.6, 1.0
        return [
            P(A.FE_DROP_SHADOW, src, i=(20, 30, 60), f=(radius, radius, 4, 6, 0.6)),
            P(A.FE_OFFSET, src, f=(3, -2)),
            P(A.FE_COLOR_MATRIX, 0, i=(A.CM_SATURATE,), f=(0.6,), linear=1),
            ct,
            P(A.FE_BLEND, 3, 1, i=(A.BLEND["multiply"],)),
            P(A.FE_MERGE, 4, i=(0, 2)),
        ], (4, 0)
    if name == "texture":
        return [
            P(A.FE_TURBULENCE, src, i=(3, 5, 0, 1), f=(0.03, 0.02)),
            P(A.FE_DISPLACEMENT_MAP, src, 0, i=(0, 1), f=(4.0 * radius,)),
            P(A.FE_DIFFUSE, 0, i=(A.LIGHT_DISTANT, 255, 240, 220), f=(radius, 1, 1, 0, 60, 50)),
            P(A.FE_CONVOLVE, 1, i=(3, 3, 1, 1, A.EDGE_DUPLICATE, 0), f=[1.0, 0.0, 0, -1, 0, -1, 5, -1, 0, -1, 0]),
            P(A.FE_COMPOSITE, 2, 3, i=(A.OP_ARITHMETIC,), f=(1.0, 0.2, 0.2, 0.0)),
        ], ()
    return [
        P(A.FE_BLUR, src, f=(radius, radius)),
        P(A.FE_MORPHOLOGY, 0, i=(1,), f=(2, 2)),
        P(A.FE_COMPOSITE, 1, src, i=(A.OP_OVER,)),
    ], ()


def _layer(w, h, seed):
    """A premultiplied layer as drawings have them: flat opaque areas,
    translucent ones with soft slopes, and transparency."""
    g = np.random.default_rng(seed)
    cells = 16
    a = g.choice([0.0, 0.0, 0.35, 0.7, 1.0, 1.0, 1.0], size=(cells, cells))
    c = g.uniform(0.0, 1.0, size=(cells, cells, 3))
    yi = (np.arange(h) * cells // h)[:, None]
    xi = (np.arange(w) * cells // w)[None, :]
    alpha = a[yi, xi]
    slope = 0.75 + 0.25 * np.cos(np.arange(w) * (2 * np.pi / 97.0))[None, :] * np.sin(np.arange(h) / 31.0)[:, None]
    rgb = c[yi, xi] * slope[..., None]
    a8 = np.rint(alpha * np.where(alpha < 1.0, slope, 1.0) * 255.0)
    out = np.empty((h, w, 4), np.uint8)
    out[..., 3] = a8
    out[..., :3] = np.floor(rgb * a8[..., None])
    return out


def _soft_arrays(case, seed):
    """Closed cubic loops, half solid and half 4-stop linear gradients, and one
    blur per scene (the differentiable form's own value ranges)."""
    S, P, w, h = case["scenes"], case["paths"], case["w"], case["h"]
    g = np.random.default_rng(seed)
    n = S * P
    segs = np.random.default_rng(n).integers(4, 17, size=n)  # the structure is the case's, the values the seed's
    off = np.concatenate([[0], np.cumsum(segs)]).astype(np.uint32)
    canvas = np.array([w, h], np.float32)
    f32 = np.float32
    a = {"scenes": S, "width": w, "height": h, "paths": P, "seg_offset": off,
         "points": (g.uniform(0, 1, size=(3 * int(off[-1]), 2)).astype(f32) * canvas).astype(f32),
         "paint_kind": (np.arange(n) % 2).astype(np.uint32),
         "colors": g.uniform(0, 1, size=(n, 4)).astype(f32),
         "stop_offsets": np.sort(g.uniform(0, 1, size=(n, 4)), axis=1).astype(f32),
         "stop_colors": g.uniform(0, 1, size=(n, 4, 4)).astype(f32),
         "grad_line": (g.uniform(0, 1, size=(n, 2, 2)) * canvas).astype(f32).reshape(n, 4),
         "sigma": g.uniform(0.5, 4.0, size=S).astype(f32),
         "opacity": g.uniform(0.3, 1.0, size=n).astype(f32)}
    a["colors"][:, 3] = g.uniform(0.3, 1.0, size=n)
    a["stop_colors"][:, :, 3] = g.uniform(0.3, 1.0, size=(n, 4))
    target = g.uniform(0, 1, size=(S, h // 8 + 2, w // 8 + 2, 4)).astype(f32)
    target = np.ascontiguousarray(np.repeat(np.repeat(target, 8, axis=1), 8, axis=2)[:, :h, :w])
    return a, target


def prepare(case, seed):
    kind = case["kind"]
    if kind == "host":
        tree, ts = _tree(case["config"], seed, 0, case["scale"], case["w"], case["h"])
        return ("host", tree, ts, case["w"], case["h"])
    if kind in ("device", "frame"):
        tree, ts = _tree(case["config"], seed, 0, case["scale"], case["w"], case["h"])
        return ("render", _Render(kind, [tree], [ts], [(case["w"], case["h"])]))
    if kind in ("batch", "gallery"):
        trees = [R.Tree.generate(3, seed=seed, index=i) for i in range(case["scenes"])]
        sizes = _sides(case["scenes"])
        ts = [(w / t.size[0], 0, 0, h / t.size[1], 0, 0) for t, (w, h) in zip(trees, sizes)]
        return ("render", _Render(kind, trees, ts, sizes))
    if kind == "filter":
        w, h = case["w"], case["h"]
        base = torch.from_numpy(_layer(w, h, seed)).cuda()
        filt = A.Filter()
        filt.x, filt.y, filt.w, filt.h = 0.0, 0.0, float(w), float(h)
        prims, merge = _chain(case["chain"], w, h, case["radius"])
        return ("filter", base, filt, prims, merge, torch.cuda.Stream())
    arrays, target = _soft_arrays(case, seed)
    return ("soft", soft.Scenes(arrays), torch.from_numpy(target).cuda())


# ---------------------------------------------------------------- run

def run(state):
    if state[0] == "host":
        _, tree, ts, w, h = state
        return R.render(tree, ts, w, h)
    if state[0] == "render":
        s = state[1]
        here = torch.cuda.current_stream()
        s.stream.wait_stream(here)
        with torch.cuda.stream(s.stream):
            s.pix.zero_()
        sh = s.stream.cuda_stream
        if s.kind == "device":
            R.render_device(s.trees[0], s.transforms[0], s.ws[0], s.hs[0], s.ptrs[0], 4 * s.ws[0], sh)
        elif s.kind == "batch":
            R.render_batch(s.trees, s.transforms, s.ws, s.hs, s.ptrs, sh)
        else:
            s.scene.render(sh)
        here.wait_stream(s.stream)
        return s.pix
    if state[0] == "filter":
        _, base, filt, prims, merge, stream = state
        here = torch.cuda.current_stream()
        img = base.clone()
        stream.wait_stream(here)
        img.record_stream(stream)
        R.filter_apply(img, filt, prims, merge, stream=stream.cuda_stream)
        here.wait_stream(stream)
        return img
    _, scenes, target = state
    image, blurred = soft.forward(scenes)
    loss, grad = soft.mse(blurred, target)
    grads = soft.backward(scenes, image, grad)
    return {"image": image, "blurred": blurred, "loss": loss, **{"d_" + k: v for k, v in grads.items()}}


# ---------------------------------------------------------------- work

# the generator's averages: a loop of 4..16 cubics, a stroked path of 1..3;
# the share of the canvas a loop covers; operations per covered pixel (blend,
# and a gradient's evaluation)
_LOOP_BYTES, _STROKE_BYTES, _COVER, _BLEND, _GRADIENT = 260, 90, 0.5, 16, 24


def _tree_work(config, scale, w, h):
    if config == 0:
        loops, strokes, grads = 200 * scale, 0, 0
    elif config == 1:
        loops, strokes, grads = 2000 * scale, 500 * scale, 1
    else:
        loops, strokes, grads = 500 * scale, 0, 0
    flops = loops * _COVER * w * h * (_BLEND + grads * _GRADIENT)
    filt = 4 * 16 * w * h if config == 2 else 0
    return 4 * w * h + loops * _LOOP_BYTES + strokes * _STROKE_BYTES, flops + filt


def work(case):
    kind = case["kind"]
    if kind in ("host", "device", "frame"):
        b, f = _tree_work(case["config"], case["scale"], case["w"], case["h"])
    elif kind in ("batch", "gallery"):
        # paths log-uniform 10..2000, a fifth stroked
        area = sum(w * h for w, h in _sides(case["scenes"])) / case["scenes"]
        paths = (2000.0 - 10.0) / math.log(200.0)
        b = case["scenes"] * (4 * area + paths * (0.8 * _LOOP_BYTES + 0.2 * _STROKE_BYTES))
        f = case["scenes"] * area * 0.8 * paths * _COVER * (_BLEND + 2 / 3 * _GRADIENT)
    elif kind == "filter":
        px = case["w"] * case["h"]
        per = {"effects": 10 * 8 + 6 * 20, "texture": 3 * 4 * 40 + 30 + 60 + 20, "soften": 4 * 4 * 8 + 4 * 10 + 20}
        b, f = 8 * px, px * per[case["chain"]]
    else:
        S, P, px = case["scenes"], case["paths"], case["w"] * case["h"]
        params = S * P * (10 * 3 * 2 + 4 + 4 + 16 + 4 + 1) * 4
        b = 2 * params + S * px * 16 * 3
        f = S * px * (P * _COVER * (40 + 90) + 8 * 25 * 5)
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------------------- exact

_FLAT, _RADIUS = 16, 12  # lines per cubic, blur taps each side


def _path_area(points, w, h):
    """Signed area of every pixel (h, w) inside a closed path of flattened cubics."""
    n = points.shape[0] // 3
    start = points[0::3]
    end = torch.roll(start, -1, 0)
    ctrl = torch.stack([start, points[1::3], points[2::3], end], 1)
    t = torch.arange(_FLAT, dtype=torch.float64, device=points.device) / _FLAT
    u = 1 - t
    bern = torch.stack([u ** 3, 3 * u * u * t, 3 * u * t * t, t ** 3], 1)
    v = torch.einsum("tk,nkc->ntc", bern, ctrl).reshape(n * _FLAT, 2)
    nx = torch.roll(v, -1, 0)
    x0, y0, x1, y1 = v[:, 0], v[:, 1], nx[:, 0], nx[:, 1]
    up = y1 > y0
    xa, ya = torch.where(up, x0, x1), torch.where(up, y0, y1)
    xb, yb = torch.where(up, x1, x0), torch.where(up, y1, y0)
    py = torch.arange(h, dtype=torch.float64, device=v.device)[:, None]
    lo, hi = torch.clamp(ya[None], min=py), torch.minimum(yb[None], py + 1)
    hit = (y0 != y1)[None] & (ya[None] < py + 1) & (yb[None] > py) & (hi > lo)
    den = torch.where(ya == yb, torch.ones_like(ya), yb - ya)[None]
    xl = torch.where(ya[None] >= py, xa[None].expand_as(lo), xa[None] + (xb - xa)[None] * ((py - ya[None]) / den))
    xh = torch.where(yb[None] <= py + 1, xb[None].expand_as(lo), xa[None] + (xb - xa)[None] * ((py + 1 - ya[None]) / den))
    sdy = torch.where(hit, torch.where(up, 1.0, -1.0)[None] * (hi - lo), torch.zeros_like(lo))
    left, right = torch.minimum(xl, xh), torch.maximum(xl, xh)
    rows = []
    px = torch.arange(w, dtype=torch.float64, device=v.device)[None, None, :]
    step = max(1, (1 << 24) // (w * n * _FLAT))
    for r in range(0, h, step):
        a, b = left[r:r + step, :, None] - px, right[r:r + step, :, None] - px
        d = b - a
        inside, full, none = (a >= 0) & (b <= 1), b <= 0, a >= 1
        safe = torch.where(inside | full | none | (d == 0), torch.ones_like(d), d)
        part = torch.where(a < 0, torch.where(b <= 1, 1 - b * b / (2 * safe), (0.5 - a) / safe),
                           (1 - a) * (1 - a) / (2 * safe))
        m = torch.where(full, torch.ones_like(d), torch.where(none, torch.zeros_like(d), torch.where(
            inside, 1 - (a + b) * 0.5, part)))
        rows.append((sdy[r:r + step, :, None] * m).sum(1))
    return torch.cat(rows, 0)


def _paint(kind, color, line, offs, stops, opacity, w, h):
    """Straight colour (h, w, 4) of a path at pixel centres, alpha times opacity."""
    if kind == 0:
        c = color.expand(h, w, 4)
    else:
        dev = color.device
        x = torch.arange(w, dtype=torch.float64, device=dev)[None, :] + 0.5
        y = torch.arange(h, dtype=torch.float64, device=dev)[:, None] + 0.5
        dx, dy = line[2] - line[0], line[3] - line[1]
        len2 = dx * dx + dy * dy
        t = ((x - line[0]) * dx + (y - line[1]) * dy) / len2 if float(len2) > 0 else torch.zeros(h, w, device=dev,
                                                                                               dtype=torch.float64)
        t = t.clamp(0, 1)
        i = (t >= offs[1]).long() + (t >= offs[2]).long()
        span = offs[i + 1] - offs[i]
        wt = torch.where(span > 0, (t - offs[i]) / torch.where(span > 0, span, torch.ones_like(span)),
                         torch.ones_like(t))[..., None]
        c = stops[i] + wt * (stops[i + 1] - stops[i])
        c = torch.where((t < offs[0])[..., None], stops[0], torch.where((t >= offs[3])[..., None], stops[3], c))
    return torch.cat([c[..., :3], c[..., 3:] * opacity], -1)


def _over(under, points, color, offs, stops, opacity, kind, line):
    h, w = under.shape[:2]
    area = _path_area(points, w, h).abs()
    cov = torch.where(area < 1, area, torch.ones_like(area))[..., None]
    c = _paint(kind, color, line, offs, stops, opacity, w, h)
    a = c[..., 3:]
    return cov * torch.cat([c[..., :3] * a, a], -1) + (1 - cov * a) * under


def _blur(img, sigma):
    j = torch.arange(-_RADIUS, _RADIUS + 1, dtype=torch.float64, device=img.device)
    k = torch.exp(-j * j / (2 * sigma * sigma))
    k = k / k.sum()
    for dim in (1, 0):
        n = img.shape[dim]
        pad = [0, 0] * 3
        pad[2 * (2 - dim)] = pad[2 * (2 - dim) + 1] = _RADIUS
        p = torch.nn.functional.pad(img, pad)
        img = sum(k[q] * p.narrow(dim, q, n) for q in range(2 * _RADIUS + 1))
    return img


def exact(case, seed):
    if case["kind"] != "soft" or case["scenes"] * case["paths"] * case["w"] * case["h"] > 70e6:
        return None
    arrays, target = _soft_arrays(case, seed)
    S, P, w, h = case["scenes"], case["paths"], case["w"], case["h"]
    names = ("points", "colors", "stop_offsets", "stop_colors", "sigma", "opacity")
    p = {k: torch.from_numpy(arrays[k]).cuda().double().requires_grad_() for k in names}
    lines = torch.from_numpy(arrays["grad_line"]).cuda().double()
    goal = torch.from_numpy(target).cuda().double()
    off, kinds = arrays["seg_offset"].astype(np.int64), arrays["paint_kind"]
    images, blurs, loss = [], [], 0.0
    for s in range(S):
        img = torch.zeros(h, w, 4, dtype=torch.float64, device="cuda")
        for j in range(s * P, (s + 1) * P):
            img = torch.utils.checkpoint.checkpoint(
                _over, img, p["points"][3 * off[j]:3 * off[j + 1]], p["colors"][j], p["stop_offsets"][j],
                p["stop_colors"][j], p["opacity"][j], int(kinds[j]), lines[j], use_reentrant=False)
        out = _blur(img, p["sigma"][s])
        part = ((out - goal[s]) ** 2).sum() / goal.numel()
        part.backward()
        loss += float(part.detach())
        images.append(img.detach())
        blurs.append(out.detach())
    return {"image": torch.stack(images), "blurred": torch.stack(blurs), "loss": loss,
            **{"d_" + k: p[k].grad for k in names}}

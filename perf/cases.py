"""The work a program has this library do, as cases to be timed: frames of vector scenes through the renderer's public
calls, batches of scenes, retained scenes and differentiable rendering steps.

A case is a dict of plain values; `kind` names the sort of scene and `call` what is done with it on every pass:

    redraw    the scene is on the GPU; one frame, its pixels copied to a device buffer (an animation loop, a compositor)
    frame     the recorded Canvas goes up, is rendered and read back into host memory (one call per image)
    batch     many small scenes uploaded together; one batched frame, every image read back into host memory
    retained  one node of a retained scene moves; its damage is redrawn and the frame read back
    diff      one training step of a differentiable scene: the loss and the gradients of points, colours and sigma
"""
from __future__ import annotations

import math

import numpy as np
import torch

import tileink_b200 as tk
from tileink_b200 import _native as N
from tileink_b200.diff import DiffScene


def listed():
    return [
        # a button or an icon: a dozen small fills, where launches and waits are the time
        {"name": "icon", "kind": "fills", "call": "redraw", "width": 97, "height": 80, "count": 12},
        # a small illustration rendered in one call, host records in and host image out
        {"name": "frame_640x360", "kind": "fills", "call": "frame", "width": 640, "height": 360, "count": 240},
        # a drawing of fills, strokes, gradients and clips redrawn in a window (odd sides: ragged tiles)
        {"name": "mixed_1283x717", "kind": "mixed", "call": "redraw", "width": 1283, "height": 717, "count": 2500},
        # the same sort of drawing recorded anew for every image, curves flattened on the GPU
        {"name": "mixed_frame_2048", "kind": "mixed", "call": "frame", "width": 2048, "height": 2048, "count": 6000},
        # the largest: a 4096 x 4096 map-like scene of 50,000 paths redrawn from GPU memory
        {"name": "mixed_4096_50k", "kind": "mixed", "call": "redraw", "width": 4096, "height": 4096, "count": 50000},
        # a full HD page of text set as glyph outlines, one call per page
        {"name": "page_20k_outlines", "kind": "outlines", "call": "frame", "width": 1920, "height": 1080,
         "count": 20000},
        # a window of text as runs of rasterized glyphs, every content kind
        {"name": "text_runs_1280x800", "kind": "runs", "call": "redraw", "width": 1280, "height": 800, "count": 400},
        # a user interface of analytic shapes: rects, circles, lines and their strokes and shadows
        {"name": "shapes_2048", "kind": "shapes", "call": "redraw", "width": 2048, "height": 2048, "count": 12500,
         "extended": False},
        # fills under a blurred group and a filter layer (colour filters, a chain blur, a drop shadow)
        {"name": "effects_1024", "kind": "effects", "call": "redraw", "width": 1024, "height": 1024, "count": 256,
         "sigma": 4.0},
        # thumbnails: many uneven scenes in one batched frame
        {"name": "batch_96", "kind": "batch", "call": "batch", "width": 0, "height": 0, "count": 96},
        # an editor: one of the nodes is dragged, the rest stays
        {"name": "retained_drag", "kind": "retained", "call": "retained", "width": 1000, "height": 760, "count": 60},
        # one optimisation step of 256 curve paths under a blur against a target image
        {"name": "diff_1024", "kind": "diff", "call": "diff", "width": 1024, "height": 1024, "count": 256,
         "sigma": 4.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fills", "mixed", "mixed", "outlines", "runs", "shapes", "effects", "batch", "retained", "diff"])
    c = {"kind": kind, "call": rng.choice(["redraw", "frame"]), "width": 0, "height": 0, "count": 0}
    if kind == "fills":
        c.update(width=_log(rng, 48, 900), height=_log(rng, 48, 900), count=_log(rng, 8, 600))
    elif kind == "mixed":
        c.update(width=_log(rng, 320, 4096), height=_log(rng, 320, 4096))
        c["count"] = max(40, _log(rng, 1, 10) * c["width"] * c["height"] // 6000)
    elif kind == "outlines":
        c.update(width=_log(rng, 240, 2560), height=_log(rng, 200, 1440))
        c["count"] = max(30, c["width"] * c["height"] // rng.randint(90, 900))
    elif kind == "runs":
        c.update(width=_log(rng, 200, 2000), height=_log(rng, 160, 1400))
        c["count"] = max(8, c["width"] * c["height"] // rng.randint(1500, 8000))
    elif kind == "shapes":
        c.update(width=_log(rng, 300, 2500), height=_log(rng, 300, 2500), extended=rng.random() < 0.4)
        c["count"] = max(30, c["width"] * c["height"] // rng.randint(350, 3000))
    elif kind == "effects":
        c.update(width=_log(rng, 200, 1900), height=_log(rng, 200, 1900), count=_log(rng, 20, 400),
                 sigma=round(rng.uniform(0.8, 14.0), 3))
    elif kind == "batch":
        c.update(call="batch", count=_log(rng, 8, 160))
    elif kind == "retained":
        c.update(call="retained", width=_log(rng, 300, 1600), height=_log(rng, 300, 1200), count=_log(rng, 10, 120))
    else:
        c.update(call="diff", width=_log(rng, 60, 1024), height=_log(rng, 60, 1024), count=_log(rng, 8, 256),
                 sigma=round(rng.choice([0.0, rng.uniform(0.7, 6.0)]), 3))
    return c


# --- scenes ---------------------------------------------------------------------------------------------------------

def _paint(rng, x, y, extent):
    """Half solid (most of them opaque), the rest two- and three-stop gradients."""
    u = rng.uniform()
    col = lambda a: (*(float(v) for v in rng.uniform(0, 1, 3)), a)  # noqa: E731
    if u < 0.35:
        return tk.Brush.solid(*col(1.0))
    if u < 0.6:
        return tk.Brush.solid(*col(float(rng.uniform(0.2, 0.9))))
    stops = [(0.0, col(1.0)), (0.55, col(float(rng.uniform(0.4, 1.0)))), (1.0, col(float(rng.uniform(0.3, 1.0))))]
    extend = int(rng.integers(0, 3))
    if u < 0.8:
        return tk.Brush.linear((x, y), (x + extent, y + 0.5 * extent), stops, extend)
    return tk.Brush.radial((x, y), 0.0, (x, y), float(extent), stops, extend)


def _runs(case, seed):
    """Text runs over rasterized glyph images of the six contents, some clipped to a column."""
    rng = np.random.default_rng(seed)
    w, h = case["width"], case["height"]
    c = tk.Canvas(w, h)
    c.set_clear_color(0xFFFFFFFF)
    fonts = []
    for k in range(48):
        gw, gh = int(rng.integers(4, 17)), int(rng.integers(6, 22))
        yy, xx = np.mgrid[0:gh, 0:gw]
        r = np.hypot((xx + 0.5 - gw / 2) / (gw / 2), (yy + 0.5 - gh / 2) / (gh / 2))
        cov = np.clip((1.1 - r) * 255 * rng.uniform(1.5, 4.0), 0, 255).astype(np.uint32)
        content = k % 6
        if content in (N.GLYPH_SUBPIXEL_MASK, N.GLYPH_LINEAR_SUBPIXEL_MASK):
            texels = np.roll(cov, -1, 1) | (cov << 8) | (np.roll(cov, 1, 1) << 16)
        elif content in (N.GLYPH_COLOR, N.GLYPH_LINEAR_COLOR):
            rgb = rng.integers(0, 256, 3)
            texels = (rgb[0] * cov // 255) | ((rgb[1] * cov // 255) << 8) | ((rgb[2] * cov // 255) << 16) | (cov << 24)
        else:
            texels = cov
        fonts.append((content, gw, c.add_glyph_image(int(rng.integers(0, 2)), gh - 3, texels.astype(np.uint32), content)))
    for k in range(case["count"]):
        x, y = int(rng.integers(0, max(1, w - 60))), int(rng.integers(14, h + 1))
        content = int(rng.integers(0, 6))
        own = [f for f in fonts if f[0] == content]
        glyphs = []
        for _ in range(int(rng.integers(6, 32))):
            _, gw, image = own[int(rng.integers(0, len(own)))]
            glyphs.append((image, x, y))
            x += gw + 1
            if x >= w:
                break
        clip = (0, 0, int(rng.integers(w // 2, w + 1)), h) if rng.uniform() < 0.1 else None
        try:
            c.push_glyph_run(glyphs, _paint(rng, float(glyphs[0][1]), float(y), 120.0), clip=clip)
        except ValueError:  # the clip leaves nothing of this run
            pass
    return c


def _shapes(case, seed):
    """Analytic shapes of 4 to 160 px in clusters; `extended` adds triangles, dashes, arcs, stars and callouts."""
    rng = np.random.default_rng(seed)
    w, h = case["width"], case["height"]
    c = tk.Canvas(w, h)
    c.set_clear_color(0xFFFFFFFF)
    centres = rng.uniform(0, 1, (200, 2)) * (w, h)
    n = case["count"]
    pick, off, size, kinds = rng.integers(0, 200, n), rng.normal(0, 300, (n, 2)), rng.uniform(4, 160, (n, 2)), 9
    if case["extended"]:
        kinds = 16
    for k in range(n):
        x, y = (float(v) for v in centres[pick[k]] + off[k])
        a, b = (float(v) for v in size[k])
        brush, kind, t = _paint(rng, x, y, max(a, b)), k % kinds, float(rng.uniform(1, 8))
        if kind < 2:
            c.push_rect(x, y, x + a, y + b, brush, radius=2.0 * t * kind)
        elif kind == 2:
            c.push_rect_stroke(x, y, x + a, y + b, t, brush, radius=t)
        elif kind == 3:
            c.push_circle(x, y, a / 2, brush)
        elif kind == 4:
            c.push_circle_stroke(x, y, a / 2, t, brush)
        elif kind == 5:
            c.push_line(x, y, x + a, y - b, t, brush, cap=k % 3)
        elif kind == 6:
            c.push_rect_shadow(x, y, x + a, y + b, brush, offset=(4, 4), expand=t, intensity=0.5, radius=8.0)
        elif kind == 7:
            c.push_circle_shadow(x, y, a / 2, brush, offset=(3, 3), expand=t, intensity=0.6)
        elif kind == 8:
            c.push_line_shadow(x, y, x + a, y + b, t, brush, offset=(2, 2), expand=3.0, intensity=0.5, cap=N.CAP_ROUND)
        elif kind == 9:
            c.push_dash_line(x, y, x + a, y + b, t, 8.0, 4.0, brush, cap=k % 3)
        elif kind == 10:
            c.push_triangle((x, y), (x + a, y + b / 3), (x + a / 2, y + b), brush, corner_radius=t / 2)
        elif kind == 11:
            c.push_checkerboard(x, y, x + a, y + b, 4.0 + t, brush, tk.Brush.solid(1, 1, 1, 1))
        elif kind == 12:
            c.push_sdf_arc(x, y, a / 2, t, 4.0, t, brush, cap=k % 3)
        elif kind == 13:
            c.push_star(x, y, a / 2, a * 0.2, brush, corner_radius=1.0, rotation=t)
        elif kind == 14:
            c.push_callout((x, y, x + a, y + b), 8.0, (k % 4, a / 2, min(a, b) / 3, 12.0, 2.0), brush)
        else:
            c.push_candlestick(x, y, y + b, y + b / 4, y + 3 * b / 4, 3 + k % 17, 1, brush)
    return c


def _blob(rng, x, y, r, n):
    p = tk.BezPath()
    ang = np.linspace(0, 2 * math.pi, n, endpoint=False)
    rad = r * rng.uniform(0.6, 1.0, n)
    px, py = x + rad * np.cos(ang), y + rad * np.sin(ang)
    p.move_to(px[0], py[0])
    for k in range(n):
        j = (k + 1) % n
        p.quad_to(x + 1.2 * r * math.cos(ang[k] + math.pi / n), y + 1.2 * r * math.sin(ang[k] + math.pi / n), px[j], py[j])
    return p.close()


def _effects(case, seed):
    """Half of the fills in a blurred group, half in a filter layer over the middle of the canvas."""
    rng = np.random.default_rng(seed)
    w, h, n = case["width"], case["height"], case["count"]
    c = tk.Canvas(w, h)
    c.set_clear_color(0xFFFFFFFF)

    def fills(count):
        for _ in range(count):
            x, y, r = float(rng.uniform(0, w)), float(rng.uniform(0, h)), float(rng.uniform(0.03, 0.2)) * min(w, h)
            c.push_path(_blob(rng, x, y, r, int(rng.integers(5, 12))), _paint(rng, x, y, r))

    c.push_blur_group(case["sigma"])
    fills(n // 2)
    c.pop_layer()
    table = np.concatenate([np.arange(256), (np.arange(256) ** 2) // 255, np.arange(256), np.arange(256)])
    reach = math.ceil(3.0 * case["sigma"]) + 8
    chain = [(N.FILTER_GRAYSCALE, 0.6), (N.FILTER_CONTRAST, 1.3), (N.FILTER_COMPONENT_TRANSFER, table),
             (N.FILTER_BLUR, (case["sigma"] / 2, case["sigma"] / 2)),
             (N.FILTER_DROP_SHADOW, (4, 4, case["sigma"] / 4, (0.1, 0.1, 0.2, 0.7)))]
    c.push_filter_layer(chain, (2.0 * reach, 2.0 * reach, w - 2.0 * reach, h - 2.0 * reach))
    fills(n - n // 2)
    c.pop_layer()
    return c


def _retained(case, seed):
    """A retained scene of `count` nodes, each a few blobs and a stroke."""
    rng = np.random.default_rng(seed)
    w, h = case["width"], case["height"]
    scene = tk.RetainedScene(w, h)
    scene.set_clear_color(0xFFFFFFFF)
    for node in range(1, case["count"] + 1):
        c = tk.Canvas(w, h)
        c.keep_commands()
        x, y = float(rng.uniform(0.1, 0.9)) * w, float(rng.uniform(0.1, 0.9)) * h
        for _ in range(4):
            c.push_path(_blob(rng, x, y, float(rng.uniform(15, 70)), 8), _paint(rng, x, y, 60.0))
        c.push_stroke(_blob(rng, x, y, 60.0, 8), tk.Brush.solid(0.1, 0.1, 0.1, 1.0), 2.0)
        scene.insert(node, c)
    return scene


def _diff_inputs(case, seed):
    """Closed paths of 12 cubics over the canvas as float32 points, their colours, and a smooth target image."""
    rng = np.random.default_rng(seed)
    w, h, n = case["width"], case["height"], case["count"]
    points = (rng.uniform(0, 1, (n, 37, 2)) * (w, h)).astype(np.float32)
    colors = np.concatenate([rng.uniform(0, 1, (n, 3)), rng.uniform(0.3, 1.0, (n, 1))], 1).astype(np.float32)
    yy, xx = np.mgrid[0:h, 0:w]
    f, ph = rng.uniform(1, 7, (4, 2)), rng.uniform(0, 6.28, 4)
    target = np.stack([0.5 + 0.5 * np.sin(f[k, 0] * xx / w + f[k, 1] * yy / h + ph[k]) for k in range(4)], -1)
    target[..., 3] = 1.0
    return points, colors, np.ascontiguousarray(target.astype(np.float32))


def _canvas(case, seed):
    kind, size = case["kind"], {"width": case["width"], "height": case["height"], "paths": case["count"]}
    if kind == "fills":
        return tk.generate(1, seed, **size)
    if kind == "mixed":
        return tk.generate(2, seed, device_flatten=True, **size)
    if kind == "outlines":
        return tk.generate(3, seed, device_flatten=True, **size)
    return {"runs": _runs, "shapes": _shapes, "effects": _effects}[kind](case, seed)


# --- what is measured -----------------------------------------------------------------------------------------------

def prepare(case, seed):
    call = case["call"]
    s = {"call": call, "renderer": tk.NativeRenderer(0)}
    if call == "batch":
        sizes = np.random.default_rng(case["count"])  # the sides and path counts belong to the case
        s["scenes"] = []
        for k in range(case["count"]):
            w, h, n = np.exp(sizes.uniform(np.log((64, 64, 10)), np.log((1024, 1024, 2000)))).round().astype(int)
            s["scenes"].append(tk.generate(4, seed, variant=k, width=int(w), height=int(h), paths=int(n)))
        s["renderer"].batch_upload(s["scenes"])
        pixels = sum(i.width * i.height for i in (s["renderer"].batch_info(k) for k in range(case["count"])))
        s["out"] = torch.empty(pixels, dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
    elif call == "retained":
        s["scene"], s["at"], s["node"] = _retained(case, seed), 0, 1 + seed % case["count"]
        s["renderer"].render_retained(s["scene"])
        s["out"] = torch.empty(case["width"] * case["height"], dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
    elif call == "diff":
        points, colors, s["target"] = _diff_inputs(case, seed)
        s["scene"] = DiffScene(case["width"], case["height"], points, colors, sigma=case["sigma"])
    elif call == "redraw":
        s["canvas"] = _canvas(case, seed)
        s["renderer"].upload(s["canvas"])
        s["out"] = torch.empty(case["height"], case["width"], dtype=torch.int32, device="cuda")
    else:
        s["canvas"] = _canvas(case, seed)
        s["out"] = torch.empty(case["width"] * case["height"], dtype=torch.int32, pin_memory=True).numpy().view(np.uint32)
    return s


def run(s):
    r, call = s["renderer"], s["call"]
    if call == "batch":
        r.batch_render()
        r.batch_readback(s["out"])
        return s["out"].view(np.uint8)
    if call == "retained":
        s["at"] = (s["at"] + 1) % 8
        s["scene"].set_transform(s["node"], (1.0, 0.0, 0.0, 1.0, 6.0 * s["at"], 3.0 * s["at"]))
        r.render_retained(s["scene"])
        return r.readback(s["out"]).view(np.uint8)
    if call == "diff":
        loss = r.diff_forward(s["scene"], s["target"])
        d_points, d_colors, d_sigma = r.diff_backward()
        return {"loss": loss, "points": d_points, "colors": d_colors, "sigma": float(d_sigma)}
    if call == "redraw":
        r.render()
        r.readback_rows(0, s["out"].shape[0], out=s["out"].data_ptr())
        return s["out"].view(torch.uint8)
    r.upload(s["canvas"])
    r.render()
    return r.readback(s["out"]).view(np.uint8)


def work(case):
    """Bytes: the recorded scene once (64 B a curve or shape with its share of the draw) and the image once. Operations:
    17 per pixel under a draw (coverage, four channels scaled and composited), estimated from the scene's statistics."""
    w, h, n, kind = case["width"], case["height"], case["count"], case["kind"]
    px, side = w * h, min(w, h) if w else 0
    if kind == "batch":  # scenes of 64..1024 px sides and 10..2000 paths, log-uniform: their means
        px, curves, covered = n * 346.0 ** 2, n * 375 * 24, n * 375 * 346.0 ** 2 * 0.5
    elif kind == "fills":
        curves, covered = n * 24, n * px * 0.5
    elif kind == "mixed":  # clusters of deviation 300 px in 4096: fills over ~3 deviations, strokes ~4 px wide
        sd = 300.0 * side / 4096.0
        curves, covered = n * 33, n * (0.6 * 5.0 * sd * sd + 0.4 * 34 * 2.0 * sd * 4.0) * 0.9
    elif kind == "outlines":  # 36 px em on average, wrapped over the page
        curves, covered = n * 45, n * 0.3 * 1500.0
    elif kind == "runs":
        curves, covered = n * 18, n * 18 * 140.0
    elif kind == "shapes":
        curves, covered = n, n * 82.0 * 82.0 * 0.6
    elif kind == "effects":  # the fills, then separable Gaussians over the canvas (both groups and the shadow)
        taps = 2 * (2 * math.ceil(3 * case["sigma"]) + 1) * 1.75
        curves, covered = n * 8, n * 0.03 * side * side + px * 8 * taps / 17.0
    elif kind == "retained":
        curves, covered = n * 40, 5 * 70.0 * 70.0 * 2
    else:  # forward and backward of every path over the canvas, float32 RGBA target, layer and gradient images
        taps = 2 * (2 * math.ceil(3 * case["sigma"]) + 1)
        return {"bytes": float(n * (37 * 8 + 16) * 2 + px * 16 * 3),
                "flops": float(n * px * 0.5 * 17 * 3 + px * 8 * taps * 3)}
    return {"bytes": float(64 * curves + 4 * px), "flops": float(17 * covered)}


# --- the differentiable step in 64 bits ---------------------------------------------------------------------------------

def _flat_weights(c, tol):
    """Flattening of one cubic: for every point after its start the four Bernstein-like weights of its control points.
    Quadratics by the parabola integral (R. Levien, Flattening quadratic Beziers, 2019), a cubic first split in equal
    parameter steps with the error bound sqrt(3)/36 |third difference| / m^3 at a tenth of the tolerance."""
    third = c[3] - 3 * c[2] + 3 * c[1] - c[0]
    v = math.sqrt(3.0) / 36.0 * math.hypot(*third) / (0.1 * tol)
    m = 1 if v <= 1 else math.ceil(round(v ** (1 / 3), 12))
    bern = lambda t: np.array([(1 - t) ** 3, 3 * (1 - t) ** 2 * t, 3 * (1 - t) * t * t, t ** 3])  # noqa: E731

    def slope(t):
        a, b, d = 3 * (1 - t) ** 2, 6 * (1 - t) * t, 3 * t * t
        return np.array([-a, a - b, b - d, d])

    integral = lambda x: x / (0.33 + math.sqrt(math.sqrt(0.67 ** 4 + 0.25 * x * x)))  # noqa: E731
    inverse = lambda x: x * (0.61 + np.sqrt(0.39 ** 2 + 0.25 * x * x))  # noqa: E731
    out = []
    for j in range(m):
        t0, t1 = j / m, (j + 1) / m
        q0, q2, step = bern(t0), bern(t1), (t1 - t0) / 3
        q1 = ((q0 + slope(t0) * step + q2 - slope(t1) * step) * 3 - q0 - q2) * 0.25
        p0, p1, p2 = q0 @ c, q1 @ c, q2 @ c
        dd = 2 * p1 - p0 - p2
        cross = (p2 - p0)[0] * dd[1] - (p2 - p0)[1] * dd[0]
        size = math.hypot(*dd)
        if size > 1e-12 and abs(cross) > 1e-12 * size * size:
            x0, x2 = (p1 - p0) @ dd / cross, (p2 - p1) @ dd / cross
            a0, a2 = integral(x0), integral(x2)
            count = 0.5 * abs(a2 - a0) * math.sqrt(abs(cross) / (size * abs(x2 - x0)) / (0.9 * tol))
            k = max(1, math.ceil(count))
            u = inverse(a0 + (a2 - a0) * np.arange(1, k) / k)
            t = (u - inverse(a0)) / (inverse(a2) - inverse(a0))
        elif size > 1e-12:
            k = max(1, math.ceil(math.sqrt(size / (4 * 0.9 * tol))))
            t = np.arange(1, k) / k
        else:
            t = np.zeros(0)
        out += [q0 * (1 - s) ** 2 + q1 * 2 * (1 - s) * s + q2 * s * s for s in t]
        out.append(q2)
    return out


def _area(a, b, w, h):
    """Signed area of every pixel left of the edges a -> b (torch, [lines, 2] each): the edges are cut at the pixel
    grid; every piece covers its cell in part and the cells to its right by its height."""
    with torch.no_grad():
        cuts = []
        for d in (0, 1):
            lo, hi = torch.minimum(a[:, d], b[:, d]), torch.maximum(a[:, d], b[:, d])
            n = (torch.ceil(hi) - torch.floor(lo) - 1).clamp(min=0).long()
            line = torch.repeat_interleave(torch.arange(len(a), device=a.device), n)
            k = torch.arange(len(line), device=a.device) - (torch.cumsum(n, 0) - n)[line]
            at = torch.floor(lo)[line] + 1 + k
            cuts.append((line, (at - a[line, d]) / (b[line, d] - a[line, d]), torch.full_like(line, d), at))
        ends = torch.arange(len(a), device=a.device)
        line = torch.cat([cuts[0][0], cuts[1][0], ends, ends])
        u = torch.cat([cuts[0][1], cuts[1][1], torch.zeros_like(a[:, 0]), torch.ones_like(a[:, 0])])
        axis = torch.cat([cuts[0][2], cuts[1][2], torch.full_like(ends, 2), torch.full_like(ends, 3)])
        at = torch.cat([cuts[0][3], cuts[1][3], torch.zeros_like(a[:, 0]), torch.zeros_like(a[:, 0])])
        order = torch.argsort(u, stable=True)
        order = order[torch.argsort(line[order], stable=True)]
        line, axis, at = line[order], axis[order], at[order]
    # the cuts' parameters again, with gradients
    d = b - a
    safe = torch.where(d == 0, torch.ones_like(d), d)
    u = torch.zeros_like(at)
    for k in (0, 1):
        u = torch.where(axis == k, (at - a[line, k]) / safe[line, k], u)
    u = torch.where(axis == 3, torch.ones_like(u), u)
    p = a[line] + u[:, None] * d[line]
    same = line[1:] == line[:-1]
    p0, p1 = p[:-1][same], p[1:][same]
    mid = 0.5 * (p0 + p1).detach()
    col, row = mid[:, 0].floor().long().clamp(0, w - 1), mid[:, 1].floor().long().clamp(0, h - 1)
    dy = p1[:, 1] - p0[:, 1]
    part = dy * (1.0 - (0.5 * (p0[:, 0] + p1[:, 0]) - col))
    flat = torch.zeros(h * (w + 1), dtype=torch.float64, device=a.device)
    flat = flat.index_add(0, row * (w + 1) + col, part).index_add(0, row * (w + 1) + col + 1, dy - part)
    return torch.cumsum(flat.view(h, w + 1), 1)[:, :w]


def exact(case, seed):
    if case["call"] != "diff":
        return None  # RGBA8 bytes
    points, colors, target = _diff_inputs(case, seed)
    w, h, sigma, dev = case["width"], case["height"], case["sigma"], "cuda" if torch.cuda.is_available() else "cpu"
    pts = torch.tensor(points, dtype=torch.float64, device=dev, requires_grad=True)
    col = torch.tensor(colors, dtype=torch.float64, device=dev, requires_grad=True)
    sg = torch.tensor(float(np.float32(sigma)), dtype=torch.float64, device=dev, requires_grad=True)
    layer = torch.zeros(4, h, w, dtype=torch.float64, device=dev)
    for p in range(case["count"]):
        ctrl, weights, first = points[p].astype(np.float64), [], []
        for k in range(12):
            got = _flat_weights(ctrl[3 * k:3 * k + 4], float(np.float32(0.1)))
            weights += got
            first += [3 * k] * len(got)
        wt, ix = torch.tensor(np.array(weights), device=dev), torch.tensor(first, device=dev)
        ring = (wt[:, :, None] * pts[p][ix[:, None] + torch.arange(4, device=dev)]).sum(1)
        ring = torch.cat([pts[p, :1], ring, pts[p, :1]])
        c = _area(ring[:-1], ring[1:], w, h).abs().clamp(max=1.0)
        a = col[p, 3]
        premul = torch.cat([col[p, :3] * a, a[None]])
        layer = premul[:, None, None] * c + layer * (1.0 - a * c)
    if sigma > 0:
        r = math.ceil(3.0 * sigma)
        k = torch.arange(-r, r + 1, dtype=torch.float64, device=dev)
        taps = torch.exp(-k * k / (2 * sg * sg))
        taps = taps / taps.sum()
        x = torch.nn.functional.conv2d(layer[:, None], taps.view(1, 1, 1, -1), padding=(0, r))
        layer = torch.nn.functional.conv2d(x, taps.view(1, 1, -1, 1), padding=(r, 0))[:, 0]
    image = layer + (1.0 - layer[3])  # over opaque white
    loss = ((image - torch.tensor(target, device=dev).double().permute(2, 0, 1)) ** 2).mean()
    loss.backward()
    return {"loss": loss.item(), "points": pts.grad.cpu(), "colors": col.grad.cpu(),
            "sigma": sg.grad.item() if sigma > 0 else 0.0}

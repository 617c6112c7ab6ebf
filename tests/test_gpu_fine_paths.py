"""Fine raster of path-only scenes (two pixels per thread, chunks of records and
segments staged per tile) at the edges of its tiles, chunks and slices, bit for
bit against the oracle."""
import math

import numpy as np
import pytest

import tileink_b200 as tk

from test_gpu_parity import compare_frame

pytestmark = pytest.mark.gpu

STOPS = [(0.0, (1.0, 0.1, 0.0, 1.0)), (0.3, (0.0, 0.7, 0.2, 0.4)), (1.0, (0.1, 0.2, 0.9, 1.0))]


def zigzag(x0, x1, y0, y1, n):
    """A closed band of n teeth between x0 and x1: n near-horizontal segments per side."""
    p = tk.BezPath().move_to(x0, y0)
    for k in range(1, n + 1):
        p.line_to(x1 if k & 1 else x0, y0 + (y1 - y0) * k / n)
    return p.line_to(x0 - 0.5, y1).line_to(x0 - 0.5, y0).close()


def rect(x0, y0, x1, y1):
    return tk.BezPath().move_to(x0, y0).line_to(x1, y0).line_to(x1, y1).line_to(x0, y1).close()


def slices(c, rng):
    # more segments, crossings and product blocks in a tile than one chunk holds
    for n in (139, 141, 279, 700):
        for rule in (tk.FILL_NONZERO, tk.FILL_EVEN_ODD):
            c.push_path(zigzag(0.7, 15.4, 0.2, 15.9, n), tk.Brush.solid(*rng.uniform(0, 1, 3), 0.6), fill_rule=rule)
            c.push_path(zigzag(3.2, 3.9, 0.1, 31.0, n), tk.Brush.linear((0, 0), (16, 9), STOPS), fill_rule=rule)


def many(c, rng):
    for k in range(150):  # several chunks of records; whole-tile and empty ones among them
        x, y = rng.uniform(-4, 24, 2)
        w, h = rng.uniform(0.3, 30, 2)
        c.push_path(rect(x, y, x + w, y + h), tk.Brush.solid(*rng.uniform(0, 1, 3), 1.0 if k % 3 else 0.5),
                    fill_rule=k & 1)


def gradients(c, rng):
    for extend in range(3):
        for k in range(8):
            a, b, d = rng.uniform(-8, 30, 2), rng.uniform(-8, 30, 2), rng.uniform(0, 25, 2)
            stops = STOPS if k & 1 else [(0.0, (0, 0, 0, 0)), (1.0, (*rng.uniform(0, 1, 3), 1.0))]
            brushes = [tk.Brush.linear(a, b if k else a, stops, extend),
                       tk.Brush.radial(a, float(d[0]), a if k < 2 else b, float(d[1]) if k else float(d[0]), stops, extend),
                       tk.Brush.radial(a, 0.0, a + (3.0, 0.0), 3.0, stops, extend)]
            t = None if k < 4 else (math.cos(k), math.sin(k) * 0.7, -math.sin(k), math.cos(k) * 1.3, 3.0, -2.0)
            for brush in brushes:
                x, y = rng.uniform(-6, 20, 2)
                c.push_path(rect(x, y, x + 19.3, y + 14.6), brush, transform=t)


def layers(c, rng):
    for depth in (1, 3, 6):
        for k in range(depth):
            c.push_clip_layer(zigzag(1.0 + k, 30.0, 0.5, 31.5 - k, 5 + k))
        c.push_path(rect(0, 0, 33, 33), tk.Brush.solid(0.2, 0.9, 0.1, 1.0))
        c.push_path(rect(-2, 5, 20, 18.5), tk.Brush.radial((8, 8), 0.0, (8, 8), 12.0, STOPS))
        c.push_opacity_layer(rect(2.5, 2.5, 28.0, 27.2), 0.55)
        c.push_path(zigzag(4.0, 27.0, 3.0, 20.0, 30), tk.Brush.solid(0.9, 0.1, 0.3, 0.8))
        c.pop_layer()
        for _ in range(depth):
            c.pop_layer()


@pytest.mark.parametrize("size", [(1, 1), (15, 17), (16, 16), (33, 31)])
@pytest.mark.parametrize("scene", [slices, many, gradients, layers])
def test_gpu_fine_paths_edges(renderer, scene, size):
    c = tk.Canvas(*size)
    c.set_clear_color(0xFF5A96C8)
    scene(c, np.random.default_rng(7))
    compare_frame(renderer, c)

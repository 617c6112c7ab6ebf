"""Fine raster of path-only scenes: chunks of one, two and three fills (quarter and half
rows per lane), records taken in slices of every length, and the instances with and
without opacity groups, bit for bit against the oracle."""
import numpy as np
import pytest

import tileink_b200 as tk
from tileink_b200 import NativeRenderer

from test_gpu_fine_paths import STOPS, rect, zigzag
from test_gpu_parity import compare_frame

pytestmark = pytest.mark.gpu


def star(rng, n, w, h):
    """A closed path of n edges anywhere over the canvas."""
    p = rng.uniform((-2, -2), (w + 2, h + 2), (n, 2)).tolist()
    path = tk.BezPath().move_to(*p[0])
    for q in p[1:]:
        path.line_to(*q)
    return path.close()


# 3 segments a path: all in one chunk; 30: few records a chunk; 600: slices whose crossings, not segments, are the limit
@pytest.mark.parametrize("edges", [3, 30, 61, 600])
@pytest.mark.parametrize("fills", [1, 2, 3, 4])
def test_gpu_fine_few_fills(renderer, fills, edges):
    rng = np.random.default_rng((fills, edges))
    c = tk.Canvas(37, 30)
    c.set_clear_color(0xFF5A96C8)
    for k in range(fills):
        brush = tk.Brush.linear((0, 0), (30, 9), STOPS) if k == 1 else tk.Brush.solid(*rng.uniform(0, 1, 3), 0.7)
        c.push_path(star(rng, edges, 37, 30), brush, fill_rule=k & 1)
    compare_frame(renderer, c)


# flat segments (one crossing each) and steep ones (up to 16) in one tile, around the 480 crossings that a slice holds
@pytest.mark.parametrize("steep", [29, 30, 31, 59, 90])
def test_gpu_fine_slice_lengths(renderer, steep):
    c = tk.Canvas(16, 16)
    p = tk.BezPath().move_to(0.4, 0.0)
    for k in range(1, steep + 1):
        p.line_to(0.4 + 15.0 * k / steep, 16.0 if k & 1 else 0.0)
    for k in range(60):
        p.line_to(15.5 if k & 1 else 0.5, 15.9 - 0.25 * k)
    c.push_path(p.close(), tk.Brush.solid(0.9, 0.2, 0.1, 0.8), fill_rule=tk.FILL_EVEN_ODD)
    c.push_path(zigzag(2.0, 14.0, 1.0, 15.0, 150), tk.Brush.solid(0.1, 0.3, 0.9, 0.6))
    compare_frame(renderer, c)


def grouped(opacity, w, h):
    rng = np.random.default_rng(5)
    c = tk.Canvas(w, h)
    c.set_clear_color(0xFFFFFFFF)
    c.push_clip_layer(rect(3.5, 2.5, w - 4.2, h - 3.1))
    c.push_path(rect(-1, -1, w + 1, h + 1), tk.Brush.solid(0.2, 0.4, 0.9, 1.0))  # a colour under a clip
    for depth in (1, 2, 5):  # up to more groups than are kept as floats
        for k in range(depth):
            if opacity:
                c.push_opacity_layer(star(rng, 9, w, h), 0.8 - 0.05 * k)
            else:
                c.push_clip_layer(star(rng, 9, w, h))
        for _ in range(3):
            c.push_path(star(rng, 12, w, h), tk.Brush.solid(*rng.uniform(0, 1, 3), 0.6))
        for _ in range(depth):
            c.pop_layer()
    c.pop_layer()
    c.push_path(star(rng, 20, w, h), tk.Brush.solid(0.9, 0.5, 0.1, 0.5))
    return c


@pytest.mark.parametrize("opacity", [False, True])
def test_gpu_fine_group_instances(renderer, opacity):
    compare_frame(renderer, grouped(opacity, 49, 35))


@pytest.mark.parametrize("with_groups", [(), (2,), (0, 1, 2)])
def test_gpu_fine_groups_in_a_batch(with_groups):
    """A batch takes the instance with groups as soon as one of its scenes has them."""
    scenes = [grouped(k in with_groups, 40 + 9 * k, 33) for k in range(3)]
    r, one = NativeRenderer(0), NativeRenderer(0)
    try:
        r.batch_upload(scenes)
        r.batch_render()
        for got, scene in zip(r.batch_readback(), scenes):
            assert np.array_equal(got, one.render_to_image(scene))
    finally:
        r.close()
        one.close()

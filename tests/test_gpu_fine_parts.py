"""Fine raster of path-only scenes: chunks of one, two and three fills (quarter and half
rows per lane) and records taken in slices of every length, bit for bit against the
oracle."""
import numpy as np
import pytest

import tileink_b200 as tk

from test_gpu_fine_paths import STOPS, zigzag
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

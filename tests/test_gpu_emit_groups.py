"""Segment emission of long paths whose lines jump over many tiles (groups of 32 lines
down to one) and of scenes whose paths are long but too many for whole CTAs, bit for
bit against the oracle (every stage)."""
import numpy as np
import pytest

import tileink_b200 as tk

from test_gpu_parity import compare_frame

pytestmark = pytest.mark.gpu


def zigzag(rng, n, w, h, reach):
    """A closed path of exactly n edges, each about `reach` px across the canvas and a few px down."""
    y = np.abs((rng.uniform(0, h) + 7.3 * np.arange(n)) % (2 * h - 2) - (h - 1))
    x0 = rng.uniform(0, max(1.0, w - reach), n)
    x = np.where(np.arange(n) % 2 == 0, x0, np.minimum(x0 + reach, w))
    path = tk.BezPath().move_to(x[0], y[0])
    for px, py in zip(x[1:], y[1:]):
        path.line_to(px, py)
    return path.close()


# tiles a line: under 4 (32 lines a group), 4 to 8, 8 to 16, ..., more than 128 (one line, and more pairs
# than are held); canvases inside and outside the cursor window, a last group of one line
@pytest.mark.parametrize("reach,width,height,n", [
    (20, 400, 320, 257), (60, 400, 320, 300), (140, 400, 320, 289), (260, 600, 300, 513),
    (520, 700, 200, 300), (900, 1000, 90, 259), (2200, 2300, 60, 257), (1400, 1500, 1100, 300)])
def test_gpu_emit_jumping_lines(renderer, reach, width, height, n):
    rng = np.random.default_rng(reach)
    c = tk.Canvas(width, height)
    for k, lines in enumerate((n, 40, n + 1)):
        c.push_path(zigzag(rng, lines, width, height, reach), tk.Brush.solid(*rng.uniform(0, 1, 3), 0.5), fill_rule=k & 1)
    compare_frame(renderer, c)


# 256 lines each: whole CTAs up to 3,157 paths, a warp per path beyond
@pytest.mark.parametrize("paths", [3150, 3165])
def test_gpu_emit_many_long_paths(renderer, paths):
    rng = np.random.default_rng(paths)
    c = tk.Canvas(256, 240)
    steps = rng.uniform(-4, 4, (8, 256, 2)).cumsum(1)
    for k in range(paths):
        p = np.clip(rng.uniform((0, 0), (256, 240)) + steps[k % 8], 0.5, (255, 239)).tolist()
        path = tk.BezPath().move_to(*p[0])
        for q in p[1:]:
            path.line_to(*q)
        c.push_path(path.close(), tk.Brush.solid(0.2, 0.4, 0.8, 0.01))
    compare_frame(renderer, c)

"""Segment emission of long paths by whole CTAs at the edges of its groups and of
the cursor window, bit for bit against the oracle (every stage)."""
import numpy as np
import pytest

import tileink_b200 as tk

from test_gpu_parity import compare_frame

pytestmark = pytest.mark.gpu


def polyline(rng, n, w, h, step):
    """A closed path of exactly n edges: jumps anywhere (step None) or walks of up to `step` px."""
    p = rng.uniform((0, 0), (w, h))
    path = tk.BezPath().move_to(*p)
    for _ in range(n - 1):
        q = rng.uniform((0, 0), (w, h)) if step is None else np.clip(p + rng.uniform(-step, step, 2), 1, (w - 1, h - 1))
        path.line_to(*q)
        p = q
    return path.close()


@pytest.mark.parametrize("width,height,step,counts", [
    (96, 80, 6.0, (255, 256, 257, 287, 1, 33, 511, 513)),   # groups and turns, short paths behind long ones
    (300, 240, 40.0, (256, 600, 3000, 12)),                 # many lines per tile and path
    (1300, 1200, None, (256, 300, 40)),                     # more pairs a group than are held; 6,150 tiles: no window
    (1300, 1040, None, (260,)),                             # 5,330 tiles: inside the window
])
def test_gpu_emit_long_paths(renderer, width, height, step, counts):
    rng = np.random.default_rng(len(counts))
    c = tk.Canvas(width, height)
    for k, n in enumerate(counts):
        c.push_path(polyline(rng, n, width, height, step), tk.Brush.solid(*rng.uniform(0, 1, 3), 0.5), fill_rule=k & 1)
    compare_frame(renderer, c)

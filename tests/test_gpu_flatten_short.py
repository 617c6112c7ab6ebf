"""Device flattening of elements of a few lines (a thread each) beside long ones
(a warp each): the host Canvas's lines bit for bit."""
import numpy as np
import pytest

import tileink_b200 as tk
from tileink_b200 import _native as N

pytestmark = pytest.mark.gpu


def scene(n, long_every, device):
    """n + 1 elements or so: short quadratics, every `long_every`-th a curve across the canvas, some degenerate."""
    rng = np.random.default_rng(n)
    c = tk.Canvas(400, 300)
    c.set_device_flatten(device)
    if not device:
        c.set_host_segment_plan(False)
    k = 0
    while k < n:
        x, y = (float(v) for v in rng.uniform(20, 260, 2))
        p = tk.BezPath().move_to(x, y)
        for _ in range(min(n - k, int(rng.integers(1, 9)))):
            if long_every and k % long_every == 0:
                p.cubic_to(*(float(v) for v in rng.uniform(0, 300, 6)))
            elif k % 7 == 3:
                p.quad_to(x, y, x, y)  # no edge, or the way back to (x, y)
            else:
                q = rng.uniform(-1, 1, 4) * rng.choice([1.0, 6.0, 14.0])
                p.quad_to(x + q[0], y + q[1], x + q[2], y + q[3])
            k += 1
        c.push_path(p.close(), tk.Brush.solid(0.2, 0.4, 0.6, 0.5))
    return c


@pytest.mark.parametrize("n,long_every", [(1, 0), (31, 0), (33, 0), (700, 0), (640, 33), (97, 2)])
def test_gpu_flatten_short_elements(renderer, n, long_every):
    host = scene(n, long_every, False).scene_arrays()
    renderer.upload(scene(n, long_every, True))
    renderer.render()
    lines, paths = renderer.debug(N.STAGE_LINES), renderer.debug(N.STAGE_PATHS)
    assert len(lines) == len(host["lines"])
    for a, b in zip(host["paths"], paths):
        assert a["line_count"] == b["line_count"]
        want = host["lines"][a["line_start"]:a["line_start"] + a["line_count"]]
        assert lines[b["line_start"]:b["line_start"] + b["line_count"]].tobytes() == want.tobytes()

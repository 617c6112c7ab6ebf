"""Device flattening of runs of long elements among short ones (listed by the threads
that meet them, a warp each): the host Canvas's lines bit for bit."""
import numpy as np
import pytest

import tileink_b200 as tk
from tileink_b200 import _native as N

pytestmark = pytest.mark.gpu


def scene(short, run, device):
    """`short` small quadratics, then `run` curves across the canvas in a row, then `short` again."""
    rng = np.random.default_rng((short, run))
    c = tk.Canvas(400, 300)
    c.set_device_flatten(device)
    if not device:
        c.set_host_segment_plan(False)
    for n, reach in ((short, 4.0), (run, 300.0), (short, 4.0)):
        while n > 0:
            x, y = (float(v) for v in rng.uniform(20, 260, 2))
            p = tk.BezPath().move_to(x, y)
            for _ in range(min(n, 40)):
                q = rng.uniform(-1, 1, 6) * reach
                if reach > 4.0:
                    p.cubic_to(x + q[0], y + q[1], x + q[2], y + q[3], x + q[4], y + q[5])
                else:
                    p.quad_to(x + q[0], y + q[1], x + q[2], y + q[3])
                n -= 1
            c.push_path(p.close(), tk.Brush.solid(0.2, 0.4, 0.6, 0.5))
    return c


# no long element, one, a warp's, more than a warp's; more elements than threads (148 x 16 x 128)
@pytest.mark.parametrize("short,run", [(500, 0), (400, 1), (900, 32), (2000, 75), (160000, 200)])
def test_gpu_flatten_runs_of_long_elements(renderer, short, run):
    host = scene(short, run, False).scene_arrays()
    renderer.upload(scene(short, run, True))
    renderer.render()
    lines, paths = renderer.debug(N.STAGE_LINES), renderer.debug(N.STAGE_PATHS)
    assert len(lines) == len(host["lines"]) and len(paths) == len(host["paths"])
    for a, b in zip(host["paths"], paths):
        assert a["line_count"] == b["line_count"]
        want = host["lines"][a["line_start"]:a["line_start"] + a["line_count"]]
        assert lines[b["line_start"]:b["line_start"] + b["line_count"]].tobytes() == want.tobytes()

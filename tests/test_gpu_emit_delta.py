"""Delta uploads that replace long paths: their segments are emitted again by whole CTAs
over a list of paths, and every stage equals a full upload of the same scene."""
import numpy as np
import pytest

import tileink_b200 as tk
from tileink_b200 import NativeRenderer, _native as N

from test_gpu_emit import polyline
from test_gpu_retained import array_scene, same_scan_and_frame

pytestmark = pytest.mark.gpu


def backwards(arrays, paths):
    """The scene with the lines of some paths in reverse order: the same records, other segments."""
    out = {k: (v.copy() if isinstance(v, np.ndarray) else v) for k, v in arrays.items()}
    for p in paths:
        s, n = int(out["paths"][p]["line_start"]), int(out["paths"][p]["line_count"])
        out["lines"][s:s + n] = out["lines"][s:s + n][::-1].copy()
    return out


# lines around 256 and far above beside short ones; a path of more tiles than the cursor window; jumping lines
@pytest.mark.parametrize("width,height,step,counts,moved", [
    (96, 80, 6.0, (255, 40, 257, 3100, 7, 256, 30), (0, 2, 3)),
    (96, 80, 6.0, (255, 40, 257, 3100, 7, 256, 30), (1, 4, 5)),
    (1300, 1200, 30.0, (300, 20, 5000, 260), (0, 2)),
    (300, 240, None, (40, 600, 270, 9), (0, 1, 2)),
])
@pytest.mark.parametrize("device_plan", [False, True])
def test_gpu_delta_of_long_paths(width, height, step, counts, moved, device_plan):
    rng = np.random.default_rng(counts[0])
    c = tk.Canvas(width, height)
    c.set_host_segment_plan(not device_plan)
    for k, n in enumerate(counts):
        c.push_path(polyline(rng, n, width, height, step), tk.Brush.solid(0.1 * (k % 9), 0.4, 0.7, 0.5), fill_rule=k & 1)
    arrays = c.scene_arrays()
    r, full = NativeRenderer(0), NativeRenderer(0)
    try:
        r.upload(array_scene(arrays, device_plan))
        r.render()
        for changed in (moved, moved[1:]):
            arrays = backwards(arrays, changed)
            assert r.upload_delta(array_scene(arrays, device_plan), changed) == len(changed)
            r.render()
            same_scan_and_frame(r, full, array_scene(arrays, device_plan))
    finally:
        r.close()
        full.close()

"""Coarse's two candidate walks (a warp per tile; a thread per tile on very large
canvases) at the edges of their steps: candidates around 32 and 256, batches that
start, close and are rejected inside a step, SDF and glyph particles. Every stage
bit for bit against the oracle."""
import numpy as np
import pytest

import oracle
import tileink_b200 as tk
from tileink_b200 import _native as N

from test_gpu_parity import compare_frame

pytestmark = pytest.mark.gpu

LARGE = (4096, 2048)  # 32,768 tiles: a thread per tile


def rect(x0, y0, x1, y1):
    return tk.BezPath().move_to(x0, y0).line_to(x1, y0).line_to(x1, y1).line_to(x0, y1).close()


def brush(rng, k):
    return tk.Brush.solid(*rng.uniform(0, 1, 3), 1.0 if k % 3 == 0 else 0.4)


def fills(c, rng, n, extent=70.0):
    for k in range(n):
        x, y = rng.uniform(-10, extent, 2)
        c.push_path(rect(x, y, x + rng.uniform(1, 60), y + rng.uniform(1, 60)), brush(rng, k), fill_rule=k & 1)


def clipped(c, rng, n, extent=70.0):
    """Groups of one to three draws under up to three clip layers, some of which miss most tiles."""
    for k in range(n):
        depth = k % 4
        for d in range(depth):
            x, y = rng.uniform(-20, extent, 2)
            c.push_clip_layer(rect(x, y, x + 50 - 10 * d, y + 45))
        fills(c, rng, 1 + k % 3, extent)
        for _ in range(depth):
            c.pop_layer()


def mixed(c, rng, n, extent=70.0):
    image = c.add_glyph_image(0, 9, np.full((10, 8), 200, np.uint32), N.GLYPH_MASK)
    for k in range(n):
        x, y = (float(v) for v in rng.uniform(-10, extent, 2))
        if k % 5 == 0:
            c.push_rect(x, y, x + 70, y + 50, brush(rng, k))  # covers whole tiles
        elif k % 5 == 1:
            c.push_circle_stroke(x, y, 20.0, 3.0, brush(rng, k))
        elif k % 5 == 2:
            c.push_glyph_run([(image, int(x) + 9 * g, int(y) + 12) for g in range(5)], brush(rng, k))
        elif k % 5 == 3:
            c.push_clip_sdf_rect_layer(x, y, x + 40, y + 40, 3.0)
            fills(c, rng, 2, extent)
            c.pop_layer()
        else:
            fills(c, rng, 1, extent)


@pytest.mark.parametrize("scene,n", [(fills, 31), (fills, 33), (fills, 257), (fills, 600), (clipped, 40), (clipped, 150),
                                     (mixed, 90)])
@pytest.mark.parametrize("size", [(70, 66), LARGE])
def test_gpu_coarse_walk(renderer, scene, n, size):
    if size == LARGE and n in (31, 33):
        pytest.skip("the thread walk has no such step")
    c = tk.Canvas(*size)
    c.set_clear_color(0xFF405060)
    scene(c, np.random.default_rng(n), n)
    if c.scene_desc().glyph_run_count == 0:
        compare_frame(renderer, c)
        return
    img = renderer.render_to_image(c)
    ref = oracle.OracleRun(c.scene_desc(), threads=8)
    for p in range(ref.pass_count):
        assert np.array_equal(renderer.debug(N.STAGE_TILES, p), ref.get(oracle.OR_PASS_TILES, N.TILE_DTYPE, p))
        assert np.array_equal(renderer.debug(N.STAGE_PTCL, p), ref.get(oracle.OR_PASS_PTCL, N.PTCL_DTYPE, p))
    assert np.array_equal(img, ref.get(oracle.OR_IMAGE, np.uint32).view(np.uint8).reshape(img.shape))

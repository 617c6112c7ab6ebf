"""The differentiable kernels' walk of a tile's records in chunks of 16: fully
transparent paths in front leave the image and every other path's gradient as they
are, but move each record to another place of its chunk."""
import numpy as np
import pytest

from tileink_b200 import diff

pytestmark = pytest.mark.gpu


def scene(n, pad, cubics):
    """n paths (the first ones with many segments per tile) behind `pad` transparent ones, on a canvas of partial tiles."""
    rng = np.random.default_rng((n, cubics))
    pts = rng.uniform(-8, 48, (n, 1 + 3 * cubics, 2)).astype(np.float32)
    cols = rng.uniform(0.2, 0.9, (n, 4)).astype(np.float32)
    front = np.random.default_rng(pad).uniform(0, 40, (pad, 1 + 3 * cubics, 2)).astype(np.float32)
    pts, cols = np.concatenate([front, pts]), np.concatenate([np.zeros((pad, 4), np.float32), cols])
    return diff.DiffScene(41, 23, pts, cols, sigma=1.0)


# 1 to 3 chunks; 40 cubics: records of more segments than the 32 whose rows are staged at a time
@pytest.mark.parametrize("n,cubics", [(1, 2), (9, 2), (17, 3), (5, 40)])
def test_gpu_diff_record_chunks(renderer, n, cubics):
    target = np.random.default_rng(n).uniform(0, 1, (23, 41, 4)).astype(np.float32)
    want = None
    for pad in (0, 1, 7, 14, 15, 16, 31):
        loss, img = renderer.diff_forward(scene(n, pad, cubics), target, return_image=True)
        dp, dc, ds = renderer.diff_backward()
        got = (img, np.asarray(dp).reshape(pad + n, -1)[pad:], np.asarray(dc).reshape(pad + n, 4)[pad:], ds)
        if want is None:
            want = got
            continue
        assert np.array_equal(got[0], want[0])
        # the same terms (at most 943 pixels x 2 edges each) summed in another order, in f32
        for a, b in zip(got[1:], want[1:]):
            assert np.abs(np.subtract(a, b)).max() <= 1e-4 * np.abs(b).max()

"""A target pixel that is not a finite number reaches the gradients of the paths of its
own tile and no others': the records of a tile that are no fills add nothing."""
import numpy as np
import pytest

from tileink_b200 import diff

pytestmark = pytest.mark.gpu


def scene():
    """One path of two cubics in each 16-pixel tile of a row of four."""
    rng = np.random.default_rng(3)
    pts = rng.uniform(2, 14, (4, 7, 2)).astype(np.float32)
    pts[:, :, 0] += 16.0 * np.arange(4, dtype=np.float32)[:, None]
    return diff.DiffScene(64, 16, pts, rng.uniform(0.2, 0.9, (4, 4)).astype(np.float32), sigma=0.0)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("tile", [1, 3])
def test_gpu_diff_nonfinite_pixel(renderer, value, tile):
    target = np.random.default_rng(1).uniform(0, 1, (16, 64, 4)).astype(np.float32)
    target[8, 16 * tile + 8] = value
    renderer.diff_forward(scene(), target)
    for grad in renderer.diff_backward()[:2]:
        finite = np.isfinite(np.asarray(grad).reshape(4, -1)).all(axis=1)
        assert all(finite[k] for k in range(4) if k != tile)

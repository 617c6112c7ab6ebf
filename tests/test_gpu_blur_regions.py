"""The shared-memory blur on regions around the number of tiles from which a thread has
four pixels, against the oracle's pass byte for byte."""
import numpy as np
import pytest

import oracle
from helpers import blur_source
from tileink_b200 import _native as N

pytestmark = pytest.mark.gpu


# 90 and 100 tiles of 32x32, 102 in two ragged rows, 98 and 102 in two ragged columns
@pytest.mark.parametrize("width,height", [(320, 288), (320, 320), (1605, 33), (33, 1553), (35, 1603)])
@pytest.mark.parametrize("axis", [0, 1])
def test_gpu_blur_region_sizes(renderer, width, height, axis):
    src, untouched = blur_source(width, height), np.full(width * height, 0x71251F1D, np.uint32)
    for r in (1, 2, 3, 4, 5, 9, 15, 16):
        for region, source in (((0, 0, width, height), (0, 0, width, height)),
                               ((1, 2, width - 2, height - 3), (7, 9, width - 2, height - 3))):
            sigma = np.float32(r / 3.0 - 0.01)
            out = renderer.stage_blur(src, untouched, width, height, region, source, sigma, axis)
            want = untouched.copy()
            reg, bounds = np.array(region, np.uint32), np.array(source, np.uint32)
            oracle.lib().or_blur_pass(N.ptr(src), N.ptr(want), width, height, N.ptr(reg), N.ptr(bounds), sigma, axis)
            assert np.array_equal(out, want), (r, region)

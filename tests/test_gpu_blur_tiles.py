"""The shared-memory blur's 32x32 tiles, four pixels a thread: every radius it takes,
on sizes around the tile, against the oracle's pass byte for byte."""
import numpy as np
import pytest

import oracle
from helpers import blur_source
from tileink_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height", [(31, 33), (32, 32), (97, 70)])
@pytest.mark.parametrize("axis", [0, 1])
def test_gpu_blur_every_radius(renderer, width, height, axis):
    src, untouched = blur_source(width, height), np.full(width * height, 0x71251F1D, np.uint32)
    for r in range(1, 17):
        for region, source in (((0, 0, width, height), (0, 0, width, height)),
                               ((3, 1, width - 5, height - 2), (7, 9, width - 2, height - 3))):
            sigma = np.float32(r / 3.0 - 0.01)
            out = renderer.stage_blur(src, untouched, width, height, region, source, sigma, axis)
            want = untouched.copy()
            reg, bounds = np.array(region, np.uint32), np.array(source, np.uint32)
            oracle.lib().or_blur_pass(N.ptr(src), N.ptr(want), width, height, N.ptr(reg), N.ptr(bounds), sigma, axis)
            assert np.array_equal(out, want), (r, region)

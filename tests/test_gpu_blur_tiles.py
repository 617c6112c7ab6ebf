"""The blurs on 32x32 shared-memory tiles (up to radius 16; paired taps up to radius
48): radii, regions and bounds on sizes around the tile, against the oracle's pass
byte for byte."""
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


@pytest.mark.parametrize("width,height", [(33, 31), (97, 130), (130, 97)])
@pytest.mark.parametrize("axis", [0, 1])
def test_gpu_blur_wide(renderer, width, height, axis):
    src, untouched = blur_source(width, height), np.full(width * height, 0x71251F1D, np.uint32)
    for r in (17, 18, 24, 33, 42, 47, 48, 49):
        for region, source in (((0, 0, width, height), (0, 0, width, height)),
                               ((3, 1, width - 5, height - 2), (7, 9, width - 2, height - 3)),
                               ((0, 0, width, height), (14, 13, 16, 15))):
            sigma = np.float32(r / 3.0 - 0.01)
            out = renderer.stage_blur(src, untouched, width, height, region, source, sigma, axis)
            want = untouched.copy()
            reg, bounds = np.array(region, np.uint32), np.array(source, np.uint32)
            oracle.lib().or_blur_pass(N.ptr(src), N.ptr(want), width, height, N.ptr(reg), N.ptr(bounds), sigma, axis)
            assert np.array_equal(out, want), (r, region, source)

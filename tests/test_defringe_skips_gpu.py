"""Defringe skips the seeds of pixels without an edge only where no factor of a seed
can be NaN.  An infinite red sample in one corner forbids the skips in the whole
image, so the pixels that it cannot reach (two blurs, a line, a blur: 44) must have
the same bits with and without it, at thresholds and strengths at the ends of what
a caller may pass."""
import numpy as np
import pytest

import libraw_enhanced_b200 as lre
from libraw_enhanced_b200 import scenes

pytestmark = pytest.mark.gpu

INF = float("inf")


@pytest.fixture(scope="module")
def acc():
    a = lre.CudaAccelerator(0)
    yield a
    a.close()


@pytest.mark.parametrize("edge", [0.1, 0.5, 1e-40, INF])
@pytest.mark.parametrize("chroma", [0.15, 0.0, -0.1, 1e-45, INF])
@pytest.mark.parametrize("strength", [8.0, 0.0, 1e30])
@pytest.mark.parametrize("green", [False, True])
def test_skips_change_nothing(acc, edge, chroma, strength, green):
    rgb = scenes.inject_fringing(np.clip(scenes.scene_rgb(160, 240, 151) * 1.1, 0, 1)).astype(np.float32)
    rgb[100:130, 150:200] = 0.4  # no edge, no excess
    other = rgb.copy()
    other[0, 0, 0] = INF
    a, b = (acc.defringe(np.ascontiguousarray(x), 10.0, edge, chroma, strength, green) for x in (rgb, other))
    a, b = (x[45:, 45:].copy().view(np.int32) for x in (a, b))
    assert np.array_equal(a, b)

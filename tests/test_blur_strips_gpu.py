"""Defringe on the strip blur at the edges of its strips (128 columns) and
batches (2 ks + 1 rows), at every compiled tap radius and at radii that take
the tile kernel: the same bits whatever the chunk height, and, where the
reference is built, within the stage's tolerance of it."""
import numpy as np
import pytest

import oracle
from libraw_enhanced_b200 import scenes
from tests._util import assert_parity

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def acc():
    import libraw_enhanced_b200 as m

    a = m.CudaAccelerator(0)
    yield a
    a.close()


def image(h, w, seed):
    rgb = scenes.scene_rgb(max(h, 64), max(w, 64), seed) * np.float32(1.1)
    return np.ascontiguousarray(scenes.inject_fringing(np.clip(rgb, 0, 1))[:h, :w]).astype(np.float32)


@pytest.mark.parametrize("radius", [1.0, 2.0, 2.6, 4.0, 5.5, 7.0, 8.0, 9.3, 10.0, 12.0, 14.2, 15.0, 20.0])
@pytest.mark.parametrize("h,w", [(1, 5), (21, 128), (43, 129), (64, 256), (190, 131), (300, 404)])
def test_chunk_height_does_not_change_defringe(acc, h, w, radius):
    img = image(h, w, 110)
    try:
        acc.set_tuning(blur_tile=64)
        a = acc.defringe(img, radius, strength=8.0, defringe_green=True)
        acc.set_tuning(blur_tile=32)
        b = acc.defringe(img, radius, strength=8.0, defringe_green=True)
    finally:
        acc.set_tuning()
    assert np.array_equal(a, b)
    if oracle.ref_available():
        assert_parity(a, oracle.defringe(img, radius, 0.1, 0.15, 8.0, True), what=f"{w}x{h} r{radius}")


def test_wide_and_narrow_copies_agree(acc):
    """A strip inside an image whose rows are 16-byte aligned is staged by
    16-byte copies, every other strip sample by sample: the columns that the
    odd-width crop shares with the even-width image, away from the cut, are
    the same."""
    img = image(120, 1024, 111)
    # the brightest sample is in both, so both are normalised alike
    img[60, 200] = img.max()
    full = acc.defringe(img, 6.0, strength=8.0)
    crop = acc.defringe(np.ascontiguousarray(img[:, :1021]), 6.0, strength=8.0)
    assert (full != img).any()
    assert np.abs(full[:, :900] - crop[:, :900]).max() <= 1e-4

"""Defringe at tap radii that take the tile blur, up to the largest accepted
radius: it runs, an output does not depend on where in a tile it lies, and,
where the reference is built, the result is within the stage's tolerance of
it."""
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


@pytest.mark.parametrize("radius", [15.5, 30.0, 30.5, 31.0, 31.5, 32.0])
@pytest.mark.parametrize("h,w", [(33, 31), (130, 203)])
def test_accepted_radii_run(acc, h, w, radius):
    img = image(h, w, 112)
    out = acc.defringe(img, radius, strength=8.0, defringe_green=True)
    assert np.isfinite(out).all()
    assert np.array_equal(out, acc.defringe(img, radius, strength=8.0, defringe_green=True))
    if oracle.ref_available():
        assert_parity(out, oracle.defringe(img, radius, 0.1, 0.15, 8.0, True), what=f"{w}x{h} r{radius}")


@pytest.mark.parametrize("radius", [30.0, 30.5, 32.0])
def test_place_in_the_tile_does_not_matter(acc, radius):
    """Columns of a row alike, so that every output of a row is the same sum,
    whichever tile and lane it came through.  The edge magnitude of the first
    and last column is 0 by definition; what that changes reaches two blurs and
    a line further (32 + 32 + 14 + 32 columns)."""
    rng = np.random.default_rng(113)
    rows = np.clip(rng.random((150, 1, 3)) * np.array([1.0, 0.6, 1.0]), 0, 1).astype(np.float32)
    img = np.ascontiguousarray(np.repeat(rows, 300, axis=1))
    out = acc.defringe(img, radius, edge_threshold=0.01, strength=10.0)
    inner = out[:, 112:-112]
    assert np.array_equal(inner, np.repeat(inner[:, :1], inner.shape[1], axis=1))
    assert (inner != img[:, 112:-112]).any()

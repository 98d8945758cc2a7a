"""The plane-resident X-Trans kernel against the row-scan kernel, which runs the
reference's scans a row per thread: the same operations in the same order, so
the same bytes.  Sizes: one partial tile (17 computed rows, the fewest), tiles
that end at, before and after the image's frame, tiles wider than the image's
rest; layouts: the standard one, its shifts, red and blue exchanged, transposed."""
import numpy as np
import pytest

from libraw_enhanced_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def acc():
    import libraw_enhanced_b200 as m

    a = m.CudaAccelerator(0)
    yield a
    a.close()


STD = np.array(scenes.XTRANS_STD, dtype=np.int8).reshape(6, 6)
LAYOUTS = {
    "standard": STD,
    "down1": np.roll(STD, 1, 0),
    "down2right3": np.roll(STD, (2, 3), (0, 1)),
    "right5": np.roll(STD, 5, 1),
    "swapped": np.array([2, 1, 0], dtype=np.int8)[STD],
    "transposed": STD.T,
    # (d) finds a colour at two columns from a solitary green that is no sample
    # there, so the plane is cleared for each direction
    "irregular": np.array([int(c) for c in "011211102120011211211011120102211011"], dtype=np.int8).reshape(6, 6),
}


@pytest.mark.parametrize("layout", sorted(LAYOUTS))
@pytest.mark.parametrize("h,w", [(23, 23), (24, 120), (117, 131), (120, 23), (121, 218), (215, 120), (219, 330)])
def test_planes_equal_row_scans(acc, monkeypatch, layout, h, w):
    xt = np.ascontiguousarray(LAYOUTS[layout])
    rng = np.random.default_rng(h * 1000 + w)
    mosaic = np.zeros((h, w, 3), np.float32)
    y, x = np.mgrid[:h, :w]
    mosaic[y, x, xt[y % 6, x % 6]] = (rng.random((h, w)) * 0.8 + 0.1 + 0.1 * np.sin(x / 3) * np.cos(y / 5)).astype(np.float32)
    pat = xt.reshape(-1).tolist()
    planes = acc.demosaic_xtrans_3pass(mosaic, pat)
    monkeypatch.setenv("LRE_XTRANS_ROWSCAN", "1")
    rows = acc.demosaic_xtrans_3pass(mosaic, pat)
    # (as bits: the irregular layout leaves frame pixels without a neighbour of one colour)
    assert np.array_equal(planes.view(np.int32), rows.view(np.int32))

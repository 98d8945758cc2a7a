"""AMaZE with one, two, four and eight CTAs per tile: an image of few tiles
takes a cluster per tile, so a crop is demosaiced by another form than the
image it was cut from.  A tile's result depends on its own samples and its
place in the tile grid only, so the crop's tiles that lie inside it, aligned
with the image's grid, come out the same, bit for bit.  Cut at the top left,
the grids agree; the crop's last tile row and column see its own frame."""
import pytest

from libraw_enhanced_b200 import scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

WB = (2.0, 1.0, 1.5, 1.0)


@pytest.fixture(scope="module")
def acc():
    import libraw_enhanced_b200 as m

    a = m.CudaAccelerator(0)
    yield a
    a.close()


@pytest.fixture(scope="module")
def whole(acc):
    import libraw_enhanced_b200 as lre

    h, w = 2000, 2600  # 336 tiles: one CTA each
    m = torch.from_numpy(scenes.bayer_scene(h, w, 130)).cuda()
    out = {}
    for cfa, f in lre.FILTERS.items():
        o = torch.empty((h, w, 3), device="cuda")
        torch.cuda.synchronize()
        acc.dev_demosaic_bayer_amaze(m, o, w, h, f, WB)
        acc.synchronize()
        out[cfa] = o
    return m, out


# tiles of the crop: 6, 15, 16 (eight CTAs), 20, 30 (four), 35, 72 (two), 80, 120 (one)
@pytest.mark.parametrize("h,w", [(192, 256), (341, 511), (400, 420), (500, 560), (600, 700), (620, 800), (1000, 1100),
                                 (1000, 1200), (1270, 1390)])
@pytest.mark.parametrize("cfa", ["RGGB", "GBRG"])
def test_crop_equals_whole(acc, whole, h, w, cfa):
    import libraw_enhanced_b200 as lre

    m, out = whole
    crop = m[:h, :w].contiguous()
    got = torch.empty((h, w, 3), device="cuda")
    torch.cuda.synchronize()
    acc.dev_demosaic_bayer_amaze(crop, got, w, h, lre.FILTERS[cfa], WB)
    acc.synchronize()
    # outputs of the tiles that end at least their apron before the crop's frame
    rows, cols = (h - 16) // 128 * 128 - 16, (w - 16) // 128 * 128 - 16
    if rows > 0 and cols > 0:
        assert torch.equal(got[:rows, :cols], out[cfa][:rows, :cols])
    again = torch.empty_like(got)
    acc.dev_demosaic_bayer_amaze(crop, again, w, h, lre.FILTERS[cfa], WB)
    acc.synchronize()
    assert torch.equal(got, again)

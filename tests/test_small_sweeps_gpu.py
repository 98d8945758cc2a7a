"""Small planes run the in-order passes in order at once (blocks would take longer),
larger ones on blocks: seen in the number of launches, which is that of the in-order
form for the small ones.  The bits are the same either side of the line."""
import pytest

from libraw_enhanced_b200 import scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

F = scenes.FILTERS["RGGB"]


@pytest.fixture(scope="module")
def acc():
    import libraw_enhanced_b200 as m

    a = m.CudaAccelerator(0)
    yield a
    a.close()


def launches(acc, run, shape):
    out, n = [], []
    for limit in (0, 4_000_000_000):
        acc.set_wait_limit(limit)
        o = torch.zeros(shape, device="cuda")
        torch.cuda.synchronize()
        n0 = acc.launch_count
        run(o)
        n.append(acc.launch_count - n0)
        out.append(o.view(torch.int32))
    acc.set_wait_limit(0)
    assert torch.equal(*out)
    return n


# 2 w + 5 h against 1000 (DCB) and, with AAHD's margins of four, 950
@pytest.mark.parametrize("h,w,small", [(64, 64, True), (128, 128, True), (99, 250, True), (100, 250, False),
                                       (256, 256, False)])
def test_dcb(acc, h, w, small):
    raw = torch.from_numpy(scenes.bayer_scene(h, w, 160) * 4095).cuda()
    a, b = launches(acc, lambda o: acc.dev_demosaic_bayer_dcb(raw, o, w, h, F, 4095.0, 1, True), (h, w, 3))
    assert (a == b) == small and a >= b


@pytest.mark.parametrize("h,w,small", [(64, 64, True), (96, 200, True), (128, 140, False), (256, 256, False)])
def test_aahd(acc, h, w, small):
    raw = torch.from_numpy(scenes.bayer_scene(h, w, 161) * 16383).cuda()
    a, b = launches(acc, lambda o: acc.dev_demosaic_bayer_aahd(raw, o, w, h, F, 16383.0), (h, w, 3))
    # the other pass, hide_hots, has its line at 800
    if 2 * (w + 8) + 5 * (h + 8) < 800:
        assert (a == b) == small
    assert a >= b and (a > b or small)

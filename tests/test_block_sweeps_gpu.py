"""The in-order passes (DCB's and AAHD's sweeps, highlight recovery's LoCA
lift) on independent blocks against the same passes in order.

A wait limit set on the context selects the in-order form (the one that
waits), so both forms run here on the same inputs and must agree bit for bit:
at the edges of the blocks (192 or 128 owned rows, steps in multiples of 64),
on frames smaller than a block's overlap, and on inputs whose changes reach
farther than the overlap, where blocks disagree, are repaired, or give way to
the in-order sweep."""
import numpy as np
import pytest

from libraw_enhanced_b200 import scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def acc():
    import libraw_enhanced_b200 as m

    a = m.CudaAccelerator(0)
    yield a
    a.close()


def both_forms(acc, run, shape):
    outs = []
    for limit in (0, 4_000_000_000):
        acc.set_wait_limit(limit)
        try:
            out = torch.zeros(shape, device="cuda")
            torch.cuda.synchronize()
            run(out)
            acc.synchronize()
            outs.append(out.view(torch.int32))
        finally:
            acc.set_wait_limit(0)
    return outs


def mosaic(h, w, seed, scale):
    m = scenes.bayer_scene(max(h, 64), max(w, 64), seed)[:h, :w] * np.float32(scale)
    return torch.from_numpy(np.ascontiguousarray(m)).cuda()


SIZES = [(13, 17), (64, 65), (191, 130), (192, 257), (193, 64), (385, 700), (1000, 333)]


@pytest.mark.parametrize("h,w", SIZES)
@pytest.mark.parametrize("cfa", ["RGGB", "GRBG"])
def test_dcb_blocks(acc, h, w, cfa):
    raw = mosaic(h, w, 101, 4095.0)
    f = scenes.FILTERS[cfa]
    a, b = both_forms(acc, lambda o: acc.dev_demosaic_bayer_dcb(raw, o, w, h, f, 4095.0, 2, True), (h, w, 3))
    assert torch.equal(a, b)


@pytest.mark.parametrize("h,w", SIZES)
def test_aahd_blocks(acc, h, w):
    raw = mosaic(h, w, 102, 16383.0)
    g = torch.Generator(device="cuda").manual_seed(h)
    hot = torch.rand(raw.shape, generator=g, device="cuda") < 0.01  # the hot-pixel sweep has work
    raw = torch.where(hot, torch.full_like(raw, 60000.0), raw).contiguous()
    f = scenes.FILTERS["RGGB"]
    a, b = both_forms(acc, lambda o: acc.dev_demosaic_bayer_aahd(raw, o, w, h, f, 16383.0), (h, w, 3))
    assert torch.equal(a, b)


@pytest.mark.parametrize("h,w", SIZES + [(4, 9), (128, 640), (129, 2100)])
@pytest.mark.parametrize("thr", [0.6, 1.0])
def test_highlight_blocks(acc, h, w, thr):
    rgb = scenes.scene_rgb(max(h, 64), max(w, 64), 103)[:h, :w] * np.array([2.0, 1.15, 1.6], np.float32)
    rng = np.random.default_rng(h + w)
    rgb = (rgb + rng.normal(0, 0.03, rgb.shape)).astype(np.float32)
    img = torch.from_numpy(np.ascontiguousarray(rgb)).cuda()
    a, b = both_forms(acc, lambda o: acc.dev_recover_highlights(img, o, w, h, thr), (h, w, 3))
    assert torch.equal(a, b)


@pytest.mark.parametrize("step", [97, 400])
def test_dcb_far_reaching_changes(acc, step):
    """Samples of 1e30 among samples of 1: what they change decays by less
    than 2^-80 over a block's overlap, so the blocks below and to the right of
    them cannot have the in-order values from their own overlap."""
    h, w = 900, 1500
    raw = mosaic(h, w, 104, 1.0) + 0.01
    raw[5::step, 7::step] = 1e30
    f = scenes.FILTERS["RGGB"]
    a, b = both_forms(acc, lambda o: acc.dev_demosaic_bayer_dcb(raw, o, w, h, f, 1e32, 1, True), (h, w, 3))
    assert torch.equal(a, b)

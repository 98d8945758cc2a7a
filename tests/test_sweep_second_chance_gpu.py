"""Frames on which blocks of the in-order passes disagree with their neighbours:
chains of sites that each pass a change on whole, over more rows or steps than a
block's overlap.  The context's counters show that blocks were repeated (and, for
the direction refinement, which also writes behind its walk, that the pass ran in
order), and the bits are those of the in-order form."""
import numpy as np
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


def both(acc, run, shape):
    """Runs both forms; returns (blocks repeated, passes in order) of the block form."""
    out, ref = torch.zeros(shape, device="cuda"), torch.zeros(shape, device="cuda")
    torch.cuda.synchronize()
    c0 = acc.sweep_counts()
    run(out)
    c1 = acc.sweep_counts()
    acc.set_wait_limit(4_000_000_000)
    try:
        run(ref)
        assert acc.sweep_counts() == c1  # sent in order by the limit: not counted
    finally:
        acc.set_wait_limit(0)
    assert torch.equal(out.view(torch.int32), ref.view(torch.int32))
    return c1[0] - c0[0], c1[1] - c0[1]


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()


def test_noise_needs_no_second_chance(acc):
    raw = dev(scenes.bayer_scene(700, 900, 140) * 16383 + np.random.default_rng(1).random((700, 900)) * 40)
    assert both(acc, lambda o: acc.dev_demosaic_bayer_dcb(raw, o, 900, 700, F, 16383.0, 1, True), (700, 900, 3)) == (0, 0)
    assert both(acc, lambda o: acc.dev_demosaic_bayer_aahd(raw, o, 900, 700, F, 16383.0), (700, 900, 3)) == (0, 0)


@pytest.mark.parametrize("side", [60, 120, 250])
def test_dcb_clipped_areas(acc, side):
    """A clipped area is flat, and a mean of equal values keeps a difference of
    a unit in the last place that noise would let decay."""
    h, w = 900, 1300
    a = np.random.default_rng(2).random((h, w)) * 1000 + 8000
    for y, x in ((50, 100), (300, 400), (600, 900)):
        a[y:y + side, x:x + side] = 16383
    raw = dev(a)
    n = both(acc, lambda o: acc.dev_demosaic_bayer_dcb(raw, o, w, h, F, 16383.0, 2, True), (h, w, 3))
    assert n[0] > 0


@pytest.mark.parametrize("at", [(100, 100), (60, 61), (250, 500)])
@pytest.mark.parametrize("iterations,enhance", [(1, True), (2, False)])
def test_dcb_flat_frame_with_an_impulse(acc, at, iterations, enhance):
    h, w = 600, 900
    a = np.full((h, w), 1000.0)
    a[at] = 16000.0
    raw = dev(a)
    n = both(acc, lambda o: acc.dev_demosaic_bayer_dcb(raw, o, w, h, F, 16383.0, iterations, enhance), (h, w, 3))
    assert n[0] > 0


@pytest.mark.parametrize("length", [60, 130, 400])
@pytest.mark.parametrize("down", [False, True])
def test_aahd_rows_of_dead_sites(acc, length, down):
    """Each dead site is brighter than the one before it and so dead only once
    that one has been replaced."""
    h, w = 900, 1500
    a = np.full((h, w), 10000.0)
    rng = np.random.default_rng(3)
    for q in range(8):
        y, x = 2 * int(rng.integers(20, 40)), 2 * int(rng.integers(20, 100))
        y, x = (y, x + 160 * q) if down else (y + 100 * q, x)
        for i in range(length):
            r, c = (y + 2 * i, x) if down else (y, x + 2 * i)
            if r < h and c < w:
                a[r, c] = 1 + i
    raw = dev(a)
    assert both(acc, lambda o: acc.dev_demosaic_bayer_aahd(raw, o, w, h, F, 16383.0), (h, w, 3))[0] > 0


def test_aahd_directions_run_in_order(acc):
    """One-pixel columns whose direction flags are turned from the top down."""
    h, w = 520, 400
    a = np.full((h, w), 500.0)
    for x in range(40, w - 50, 50):
        a[20:h - 20, x] = np.tile((5000.0, 1000.0, 1000.0, 5000.0), h // 4 + 1)[:h - 40]
    raw = dev(a)
    n = both(acc, lambda o: acc.dev_demosaic_bayer_aahd(raw, o, w, h, F, 16383.0), (h, w, 3))
    assert n[0] > 0 and n[1] == 1


@pytest.mark.parametrize("radius", [80, 100, 200])
@pytest.mark.parametrize("cast", [1.1, 1.3])
def test_loca_flat_highlights(acc, radius, cast):
    """A flat clipped area with a cast: a lifted pixel makes its neighbours differ
    from theirs, so the lift runs through the whole area."""
    h, w = 600, 900
    g = torch.Generator(device="cuda").manual_seed(3)
    img = torch.rand((h, w, 3), generator=g, device="cuda") * 0.2 + 0.72
    img[..., 1] /= cast
    img[5:15] = torch.tensor((0.9, max(0.805, 0.9 / cast), 0.9), device="cuda")
    yy, xx = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"), indexing="ij")
    for cy, cx in ((150, 150), (200, 450), (380, 300), (420, 700)):
        img[(yy - cy) ** 2 + (xx - cx) ** 2 < radius ** 2] = torch.tensor((2.0, 1.15, 2.0), device="cuda")
    assert both(acc, lambda o: acc.dev_recover_highlights(img, o, w, h, 0.8), (h, w, 3))[0] > 0


def test_develop_with_disagreeing_blocks(acc):
    """Through the host develop, whose sweeps report through a flag of the context."""
    import libraw_enhanced_b200 as lre

    h, w = 600, 900
    a = np.full((h, w), 0.06, np.float32)
    a[100, 100] = 0.9
    p = lre.develop_params(cfa="RGGB", demosaic_algorithm=4, highlight_recovery=1, highlight_threshold=0.5)
    c0 = acc.sweep_counts()
    got = acc.develop(a, p)
    assert acc.sweep_counts()[0] > c0[0]
    acc.set_wait_limit(4_000_000_000)
    try:
        assert np.array_equal(got, acc.develop(a, p))
    finally:
        acc.set_wait_limit(0)

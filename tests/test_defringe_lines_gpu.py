"""Defringe's line search at every place of its tiles: a pixel's result depends on
its surroundings within the filter's reach only, so a crop that moves the tile
grid over the picture leaves the pixels beyond that reach as they are, bit for
bit.  Runs of four pixels leave the tile sideways by up to six, and begin in
each of its rows and columns, as the grid moves; the correction's warps pack
other pixels together, and end within a group of four at odd widths."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def acc():
    import libraw_enhanced_b200 as m

    a = m.CudaAccelerator(0)
    yield a
    a.close()


def fringed(h, w, seed):
    """Bright lines and blocks on a dark ground, red and blue spread by a pixel or two."""
    r = np.random.default_rng(seed)
    g = np.full((h, w), 0.05)
    for _ in range(60):
        y, x, s = r.integers(0, h), r.integers(0, w), r.integers(3, 30)
        if r.random() < 0.5:
            g[y:y + s, x:x + r.integers(2, 30)] = r.uniform(0.5, 1)
        else:
            dy, dx = r.integers(-2, 3, 2)
            for k in range(s * 2):
                yy, xx = y + dy * k // 2, x + dx * k // 2
                if 0 <= yy < h - 1 and 0 <= xx < w - 1:
                    g[yy:yy + 2, xx:xx + 2] = 0.9
    spread = np.maximum.reduce([np.roll(np.roll(g, a, 0), b, 1) for a in (-2, 0, 2) for b in (-2, 0, 2)])
    img = np.stack([0.6 * g + 0.35 * spread, g, 0.5 * g + 0.5 * spread], 2) + r.uniform(0, 0.01, (h, w, 3))
    img[h // 2, w // 2, 1] = 1.5  # the largest green, in every crop
    return img.astype(np.float32)


def run(acc, img, radius):
    h, w, _ = img.shape
    x = torch.from_numpy(np.ascontiguousarray(img)).cuda()
    out = torch.empty_like(x)
    torch.cuda.synchronize()
    acc.dev_defringe(x, out, w, h, radius)
    acc.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("dy,dx", [(0, 1), (1, 0), (2, 3), (5, 30), (13, 17), (31, 6), (16, 25)])
@pytest.mark.parametrize("radius", [4.0, 10.0])
def test_crop_moves_the_tiles(acc, dy, dx, radius):
    img = fringed(260, 330, 5)
    whole, crop = run(acc, img, radius), run(acc, img[dy:, dx:], radius)
    reach = 3 * 10 + 14 + 2  # three blurs, the longest line, the gradients
    m = reach + 2
    a, b = whole[dy + m:-m, dx + m:-m], crop[m:-m, m:-m]
    assert (np.abs(a - img[dy + m:-m, dx + m:-m]).max(2) > 1e-3).mean() > 0.05  # fringes are corrected there
    assert np.array_equal(a, b)

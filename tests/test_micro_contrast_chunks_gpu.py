"""Micro-contrast: an image's rows are split into chunks by the time that the fullest SM
takes.  The split must not change a bit, and must not leave a size slow: halving the
chunks until there were eight blocks per SM left 1.5 MP at 1.2 times the time per pixel
of 3 MP, and 0.28 MP (18 rows staged for ten written, four blocks on some SMs) slower
than a block per tile."""
import time

import pytest

import libraw_enhanced_b200 as lre

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def acc():
    with lre.CudaAccelerator(0) as a:
        yield a


def image(h, w, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand((h, w, 3), generator=g, device="cuda") * 0.9


def run(acc, img):
    h, w = img.shape[:2]
    out = torch.empty_like(img)
    torch.cuda.synchronize()
    acc.dev_enhance_micro_contrast(img, out, w, h, 0.3, 8.0, 0.4)
    acc.synchronize()
    return out


# one row, less than a period, the edges of two to five periods, and sizes whose own
# split has two, three, four and more of them
@pytest.mark.parametrize("h,w", [(1, 1), (1, 200), (9, 65), (10, 64), (11, 63), (19, 130), (20, 64), (28, 64), (29, 64),
                                 (37, 300), (341, 511), (530, 530), (400, 800), (700, 900), (1024, 1536)])
@pytest.mark.parametrize("more_h,more_w", [(0, 6000), (3000, 0), (700, 1500)])
def test_split_leaves_the_bits(acc, h, w, more_h, more_w):
    """An image continued by its last column and row, as the stage itself continues it,
    is split in another way."""
    img = image(h, w, 301)
    img[h // 2, w // 2] = 40.0  # the largest deviation lies inside (or, with one row or column, is continued)
    wide = torch.cat([img, img[:, -1:].expand(h, more_w, 3)], 1)
    wide = torch.cat([wide, wide[-1:].expand(more_h, w + more_w, 3)], 0).contiguous()
    a, b = run(acc, img), run(acc, wide)[:h, :w]
    assert torch.equal(a.view(torch.int32), b.contiguous().view(torch.int32))


def test_middle_sizes_cost_no_more_per_pixel(acc):
    def per_pixel(h, w):
        img = image(h, w, 302)
        out = torch.empty_like(img)
        torch.cuda.synchronize()
        best = 1e9
        for _ in range(12):
            t0 = time.perf_counter()
            for _ in range(10):
                acc.dev_enhance_micro_contrast(img, out, w, h, 0.3, 8.0, 0.4)
            acc.synchronize()
            best = min(best, time.perf_counter() - t0)
        return best / (10 * h * w)

    middle, large = per_pixel(1024, 1536), per_pixel(1500, 2000)
    assert middle < 1.1 * large, f"{middle * 1e12:.1f} ps, {large * 1e12:.1f} ps"

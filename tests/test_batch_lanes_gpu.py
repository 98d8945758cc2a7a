"""Small images on many lanes: each image by itself could fill the GPU with
clusters of CTAs, so lanes must leave room for one another.  Eight lanes take
well under the time of one (with every image in clusters of eight they took 0.80
of it), and the bits do not depend on the number of lanes."""
import time

import pytest

import libraw_enhanced_b200 as lre
from libraw_enhanced_b200 import scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N = 32
P = lre.develop_params(cfa="RGGB", cam_mul=(2.0, 1.0, 1.5, 1.0), tone_mapping=1)


def run(lanes, h, w):
    mosaics = [torch.from_numpy(scenes.bayer_scene(h, w, 120 + i % 3)).cuda() for i in range(N)]
    outs = [torch.empty((h, w, 3), device="cuda") for _ in range(N)]
    torch.cuda.synchronize()
    b = lre.Batch(0, lanes=lanes, autotune=False)
    try:
        took = []
        for k in range(15):
            t0 = time.perf_counter()
            b.dev_run(mosaics, outs, [P] * N)
            if k >= 3:
                took.append(time.perf_counter() - t0)
    finally:
        b.close()
    return min(took), outs


def test_lanes_share_the_gpu():
    one, a = run(1, 341, 511)
    eight, b = run(8, 341, 511)
    assert all(torch.equal(x, y) for x, y in zip(a, b))
    assert eight < 0.6 * one, f"{N} images of 511x341: {one * 1e6:.0f} us on one lane, {eight * 1e6:.0f} us on eight"


@pytest.mark.parametrize("h,w", [(120, 200), (341, 511), (600, 700), (768, 1024)])
def test_bits_do_not_depend_on_the_lanes(h, w):
    first = None
    for lanes in (1, 2, 3, 4, 8):
        outs = run(lanes, h, w)[1]
        first = first or outs
        assert all(torch.equal(x, y) for x, y in zip(first, outs))

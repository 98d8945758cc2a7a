"""Small images on many lanes: each image by itself could fill the GPU with
clusters of CTAs, so lanes must leave room for one another.  Eight lanes take
well under the time of one (with every image in clusters of eight they took 0.80
of it), and the bits do not depend on the number of lanes."""
import functools
import threading
import time

import pytest

import libraw_enhanced_b200 as lre
from libraw_enhanced_b200 import scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N = 32
P = lre.develop_params(cfa="RGGB", cam_mul=(2.0, 1.0, 1.5, 1.0), tone_mapping=1)


@functools.lru_cache(None)
def scene(h, w, seed):
    return torch.from_numpy(scenes.bayer_scene(h, w, seed))


def run(lanes, h, w):
    mosaics = [scene(h, w, 120 + i % 3).cuda() for i in range(N)]
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


def test_threads_share_the_gpu():
    """The same for threads that keep a context each."""
    h, w, n = 341, 511, 100

    def took(threads):
        accs = [lre.CudaAccelerator(0) for _ in range(threads)]
        mos = [scene(h, w, 120).cuda() for _ in accs]
        outs = [torch.empty((h, w, 3), device="cuda") for _ in accs]
        torch.cuda.synchronize()

        def work(i, n):
            for _ in range(n):
                accs[i].dev_develop(mos[i], outs[i], w, h, P)
            accs[i].synchronize()

        best = 1e9
        for n_dev in (10, n, n, n, n):
            ts = [threading.Thread(target=work, args=(i, n_dev)) for i in range(threads)]
            t0 = time.perf_counter()
            for t in ts:
                t.start()
            for t in ts:
                t.join()
            best = min(best, (time.perf_counter() - t0) / (n_dev * threads))
        assert all(torch.equal(o, outs[0]) for o in outs)
        for a in accs:
            a.close()
        return best

    one, eight = took(1), took(8)
    assert eight < 0.6 * one, f"an image on one thread {one * 1e6:.0f} us, on eight {eight * 1e6:.0f} us"

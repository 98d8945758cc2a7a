"""The radius-6 guided filter at the edges of its warps (112 output columns of
128, four per lane) and row chunks (multiples of 8): against the filter in
double precision with numpy, and its 16-bit form against the separate
quantisation.

The filter's sums are double and its planes float, so the result is within a
few float roundings of the double one: 1e-5 on data in [0, 1]."""
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


def box(x, r=6):
    for ax in (0, 1):
        n = x.shape[ax]
        s = np.concatenate([np.zeros_like(np.take(x, [0], ax)), np.cumsum(x, ax)], ax)
        i = np.arange(n)
        hi, lo = np.minimum(i + r + 1, n), np.maximum(i - r, 0)
        x = (np.take(s, hi, ax) - np.take(s, lo, ax)) / (hi - lo).reshape((-1, 1) if ax == 0 else (1, -1))
    return x


def axial64(img, eps=1e-4, strength=0.3):
    norm = max(1e-6, float(img[..., 1].max()))
    R, G, B = (img[..., c].astype(np.float64) / norm for c in range(3))
    mi = box(G)
    vi = box(G * G) - mi * mi
    e = np.zeros_like(G)
    if min(G.shape) > 2:
        e[1:-1, 1:-1] = np.hypot(G[1:-1, 2:] - G[1:-1, :-2], G[2:, 1:-1] - G[:-2, 1:-1])
    t = np.clip((box(e) - 0.01) / 0.05, 0, 1)
    w = strength * t * t * (3 - 2 * t)
    out = img.astype(np.float64).copy()
    for c, X in ((0, R), (2, B)):
        mp = box(X)
        a = (box(G * X) - mi * mp) / (vi + eps)
        q = box(a) * G + box(mp - a * mi)
        out[..., c] = (X * (1 - w) + q * w) * norm
    return out


def image(h, w):
    return np.ascontiguousarray(scenes.scene_rgb(max(h, 64), max(w, 64), 120)[:h, :w])


@pytest.mark.parametrize("h,w", [(1, 1), (5, 9), (7, 112), (8, 113), (9, 128), (40, 447), (41, 448), (33, 452), (150, 225),
                                 (300, 1000)])
def test_axial_radius_6_edges(acc, h, w):
    img = image(h, w)
    got = acc.ca_axial_cleanup(img)
    assert np.array_equal(got[..., 1], img[..., 1])
    assert np.abs(got - axial64(img)).max() <= 1e-5


@pytest.mark.parametrize("order,tone", [(0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("h,w", [(96, 144), (75, 131)])
def test_axial_writes_the_codes(acc, h, w, order, tone):
    import libraw_enhanced_b200 as lre

    m = scenes.bayer_scene(h, w, 121)
    kw = dict(cfa="RGGB", cam_mul=(2.0, 1.0, 1.5, 1.0), stage_order=order, tone_mapping=tone, axial_ca_correction=1,
              defringe=order)
    f = acc.develop(m, lre.develop_params(**kw))
    u = acc.develop(m, lre.develop_params(output_bits=16, **kw))
    assert np.array_equal(u, acc.quantize(f))

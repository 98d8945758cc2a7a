"""Lateral CA against a numpy restatement of it: cells at the image's edge and
inside (with and without clamps), cells wider than the multiply-high division
takes, odd sides (a last column or row without a box), rows of pairs and of
odd width, one level and several, images narrower than a warp."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
f32 = np.float32


@pytest.fixture(scope="module")
def acc():
    import libraw_enhanced_b200 as m

    a = m.CudaAccelerator(0)
    yield a
    a.close()


def bilinear(p, x, y):
    h, w = p.shape
    x = np.minimum(np.maximum(x, f32(0)), f32(w - 1))
    y = np.minimum(np.maximum(y, f32(0)), f32(h - 1))
    x0, y0 = x.astype(np.int64), y.astype(np.int64)
    x1, y1 = np.minimum(x0 + 1, w - 1), np.minimum(y0 + 1, h - 1)
    fx, fy = x - x0.astype(f32), y - y0.astype(f32)
    one = f32(1)
    return ((p[y0, x0] * (one - fx) + p[y0, x1] * fx) * (one - fy) +
            (p[y1, x0] * (one - fx) + p[y1, x1] * fx) * fy)


def box(p):
    h, w = p.shape[0] // 2 * 2, p.shape[1] // 2 * 2
    p = p[:h, :w]
    return f32(0.25) * (p[::2, ::2] + p[::2, 1::2] + p[1::2, ::2] + p[1::2, 1::2])


def cell_step(G, T, x0, x1, y0, y1, dx, dy, iters, max_shift):
    ys, xs = np.mgrid[y0 + 1:y1 - 1, x0 + 1:x1 - 1]
    gx = (G[ys, xs + 1] - G[ys, xs - 1]).astype(np.float64)
    gy = (G[ys + 1, xs] - G[ys - 1, xs]).astype(np.float64)
    a, b, d, conf = (gx * gx).sum(), (gx * gy).sum(), (gy * gy).sum(), 0.0
    if xs.size < 32:
        return dx, dy, f32(0)
    for _ in range(iters):
        e = (bilinear(T, xs.astype(f32) + dx, ys.astype(f32) + dy) - G[ys, xs]).astype(np.float64)
        bx, by = -(gx * e).sum(), -(gy * e).sum()
        det, tr = a * d - b * b, a + d
        conf = f32(0.5 * (tr - np.sqrt(max(0.0, tr * tr - 4 * det))))
        if det <= 1e-12:
            break
        sx, sy = (d * bx - b * by) / det, (-b * bx + a * by) / det
        dx = f32(min(max(f32(dx + f32(sx)), f32(-max_shift)), f32(max_shift)))
        dy = f32(min(max(f32(dy + f32(sy)), f32(-max_shift)), f32(max_shift)))
        if abs(sx) < 0.005 and abs(sy) < 0.005:
            break
    return dx, dy, f32(max(0, conf))


def smooth(m):
    h, w = m.shape
    out = np.empty_like(m)
    for y in range(h):
        for x in range(w):
            acc = f32(0)
            box9 = m[max(0, y - 1):y + 2, max(0, x - 1):x + 2].ravel()
            for v in box9:
                acc = f32(acc + v)
            out[y, x] = acc / f32(box9.size)
    return out


def place(n_px, cell, n):
    g = np.arange(n_px).astype(f32) / f32(cell) - f32(0.5)
    g0 = np.maximum(np.minimum(np.maximum(np.floor(g).astype(np.int64), 0), n - 2), 0)
    return g0, np.minimum(g0 + 1, n - 1), np.clip(g - g0.astype(f32), f32(0), f32(1)).astype(f32)


def lateral(rgb, cell, iters, max_shift, min_conf, levels):
    h, w, _ = rgb.shape
    while levels > 1 and (w >> (levels - 1) < 32 or h >> (levels - 1) < 32):
        levels -= 1
    mw, mh = max(2, -(-w // cell)), max(2, -(-h // cell))
    pyr = [[np.ascontiguousarray(rgb[..., c]) for c in range(3)]]
    for _ in range(levels - 1):
        pyr.append([box(p) for p in pyr[-1]])
    out = rgb.copy()
    for c in (0, 2):
        dx, dy, cf = (np.zeros((mh, mw), f32) for _ in range(3))
        for L in range(levels - 1, -1, -1):
            G, T = pyr[L][1], pyr[L][c]
            H, W = G.shape
            down, up = f32(1 / (1 << L)), f32(1 << L)
            limit = f32(f32(max_shift) * down + f32(1 << L) * f32(0.5))
            cw, ch = f32(W) / f32(mw), f32(H) / f32(mh)
            for y in range(mh):
                for x in range(mw):
                    x0, x1 = int(f32(x) * cw), min(int(f32(x + 1) * cw), W)
                    y0, y1 = int(f32(y) * ch), min(int(f32(y + 1) * ch), H)
                    a, b = f32(dx[y, x] * down), f32(dy[y, x] * down)
                    if x1 > x0 + 4 and y1 > y0 + 4:
                        a, b, cf[y, x] = cell_step(G, T, x0, x1, y0, y1, a, b, iters, limit)
                    dx[y, x], dy[y, x] = f32(a * up), f32(b * up)
        if cf.max() > 0:
            low = cf < f32(cf.max() * f32(min_conf))
            dx[low], dy[low] = 0, 0
        lim = f32(f32(max_shift) * f32(1 << (levels - 1)))
        x0, x1, fx = place(w, cell, mw)
        y0, y1, fy = (v[:, None] for v in place(h, cell, mh))
        one = f32(1)
        s = []
        for m in (smooth(dx), smooth(dy)):
            v = ((m[y0, x0] * (one - fx) + m[y0, x1] * fx) * (one - fy) + (m[y1, x0] * (one - fx) + m[y1, x1] * fx) * fy)
            s.append(np.clip(v, -lim, lim).astype(f32))
        ys, xs = np.mgrid[:h, :w]
        out[..., c] = bilinear(pyr[0][c], xs.astype(f32) + s[0], ys.astype(f32) + s[1])
    return out


def scene(h, w, seed):
    """Smooth waves, red and blue displaced by up to two pixels."""
    r = np.random.default_rng(seed)
    y, x = np.mgrid[:h, :w].astype(np.float64)
    out = np.zeros((h, w, 3))
    for c, (ox, oy) in enumerate(((1.3, -0.8), (0, 0), (-2.0, 0.6))):
        rr = np.random.default_rng(seed + 1)
        for _ in range(6):
            kx, ky, ph = rr.uniform(-.25, .25), rr.uniform(-.25, .25), rr.uniform(0, 6)
            out[..., c] += 0.08 * np.sin(kx * (x + ox) + ky * (y + oy) + ph)
    return (out + 0.5 + r.uniform(-.002, .002, out.shape)).astype(f32)


@pytest.mark.parametrize("h,w,cell,levels", [
    (70, 3402, 3402, 1),     # cells of 1701 columns: the division itself
    (70, 3401, 1700, 1),     # three columns of cells on either side of it, odd rows
    (17, 19, 16, 3), (33, 31, 16, 2), (64, 64, 16, 2), (97, 130, 32, 3), (131, 257, 96, 3),
    (200, 96, 33, 2), (260, 515, 96, 3)])
def test_against_numpy(acc, h, w, cell, levels):
    img = scene(h, w, 1000 + h + w)
    got = np.asarray(acc.ca_register_lateral(img, cell, 3, 6.0, 0.02, levels))
    ref = lateral(img, cell, 3, 6.0, 0.02, levels)
    assert np.array_equal(got[..., 1], img[..., 1])
    # The sums' order differs (in double): a shift may round to the next float,
    # and a position x + shift then to the next one of its size: a neighbours'
    # difference times that spacing in each direction.  On top the rounding of
    # the three means: three half-ulps of values below 2.
    slope = max(np.abs(np.diff(img, axis=0)).max(), np.abs(np.diff(img, axis=1)).max())
    tol = 2 * 2 * slope * np.spacing(f32(max(h, w))) + 4e-7
    assert np.abs(got - ref).max() <= tol

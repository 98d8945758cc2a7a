"""The calls a user of the develop backend makes, as timed cases.

Each case is one pass through a public entry point of ``libraw_enhanced_b200``:
whole develops of a CFA mosaic (plain, with every correction, 16-bit, X-Trans,
and from page-locked host buffers), and the stages that a program calls by
themselves (DCB and AAHD demosaics, highlight recovery, the detail-preserving
tone map, micro-contrast, defringe).  Sizes run from a thumbnail to the 51 MP
sensor; inputs are seeded scenes with sensor noise, clipped highlights and
purple fringes, made on the GPU.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

import libraw_enhanced_b200 as lre
from libraw_enhanced_b200 import scenes

DEV = "cuda"
XTRANS = scenes.XTRANS_STD

# Pixels of the largest case of each kind.
LARGEST = {
    "develop": 8736 * 5856,
    "xtrans": 6240 * 4160,
    "host": 8256 * 5504,
    "dcb": 6000 * 4000,
    "aahd": 6000 * 4000,
    "highlights": 6000 * 4000,
    "detail": 8256 * 5504,
    "micro": 8256 * 5504,
    "defringe": 8256 * 5504,
}


def listed():
    return [
        # A browser's thumbnail of an embedded small raw: demosaic and tone
        # map, nothing else.  The smallest call: launches and one tile's time.
        dict(name="develop_thumb", kind="develop", w=511, h=341, cfa="RGGB", order=0, tone=1, lateral=False,
             axial=False, defringe=False, bits=32),
        # An editor's preview with every correction on, in the order of the
        # reference's process_raw_to_rgb.
        dict(name="develop_preview", kind="develop", w=1536, h=1024, cfa="RGGB", order=0, tone=1, lateral=True,
             axial=True, defringe=True, bits=32),
        # A 24 MP export to 16 bits (the batched develop's options).
        dict(name="develop_24mp_u16", kind="develop", w=6000, h=4000, cfa="GBRG", order=1, tone=0, lateral=False,
             axial=True, defringe=True, bits=16),
        # The headline workload: 51 MP AMaZE, defringe, axial CA, ACES.
        dict(name="develop_51mp", kind="develop", w=8736, h=5856, cfa="RGGB", order=1, tone=1, lateral=False,
             axial=True, defringe=True, bits=32),
        # The X-Trans workload: 3-pass demosaic and lateral CA.
        dict(name="xtrans_26mp", kind="xtrans", w=6240, h=4160, passes=3, tone=0, lateral=True),
        # A caller with mosaics in page-locked host memory: upload, develop,
        # download, one call.
        dict(name="host_24mp", kind="host", w=6000, h=4000, cfa="RGGB", order=1, tone=1, lateral=False, axial=True,
             defringe=True, bits=32),
        # The other demosaics that the develop routes to, called alone.
        dict(name="dcb_24mp", kind="dcb", w=6000, h=4000, cfa="RGGB", iterations=1, enhance=True),
        dict(name="aahd_12mp", kind="aahd", w=4032, h=3024, cfa="GRBG"),
        # Clipped skies: about a quarter of the frame above the threshold.
        dict(name="highlights_24mp", kind="highlights", w=6000, h=4000, threshold=1.0),
        # The detail-preserving tone map of a 45 MP frame.
        dict(name="detail_45mp", kind="detail", w=8256, h=5504),
        # enhance_micro_contrast as RawImage calls it on a 12 MP frame.
        dict(name="micro_12mp", kind="micro", w=4032, h=3024, threshold=0.5, strength=8.0, target=0.06),
        # RawImage.defringe of a 26 MP crop with odd sides, a smaller radius
        # than the default and green correction on.
        dict(name="defringe_26mp_odd", kind="defringe", w=5101, h=5099, radius=7.0, strength=6.0, green=True),
    ]


def _size(rng, kind):
    """Width and height: pixels log-uniform up to the kind's largest, aspect
    1:1 to 16:9 in either orientation, odd sides among them."""
    n = math.exp(rng.uniform(math.log(200e3), math.log(LARGEST[kind])))
    a = rng.choice([1.0, 4 / 3, 3 / 2, 16 / 9])
    w, h = math.sqrt(n * a), math.sqrt(n / a)
    if rng.random() < 0.25:
        w, h = h, w
    w, h = max(64, int(w)), max(64, int(h))
    if rng.random() < 0.5:
        w, h = w & ~1, h & ~1
    return w, h


def draw(rng):
    kind = rng.choice(["develop"] * 4 + ["xtrans", "host", "dcb", "aahd", "highlights", "detail", "micro"] +
                      ["defringe"] * 2)
    w, h = _size(rng, kind)
    c = dict(kind=kind, w=w, h=h)
    if kind in ("develop", "dcb", "aahd", "host"):
        c["cfa"] = rng.choice(["RGGB", "BGGR", "GRBG", "GBRG"])
    if kind in ("develop", "host"):
        bits = rng.choice([32, 32, 16])
        c.update(order=rng.choice([0, 1]), tone=rng.choice([0, 1, 1]), axial=rng.random() < 0.7,
                 defringe=rng.random() < 0.7, bits=bits)
        c["lateral"] = bits == 32 and c["order"] == 0 and rng.random() < 0.5
    elif kind == "xtrans":
        c.update(passes=rng.choice([1, 3, 3]), tone=rng.choice([0, 1]), lateral=rng.random() < 0.7)
    elif kind == "dcb":
        c.update(iterations=rng.choice([1, 1, 2]), enhance=rng.random() < 0.7)
    elif kind == "highlights":
        c["threshold"] = rng.choice([0.95, 1.0, 1.1])
    elif kind == "micro":
        c.update(threshold=rng.choice([0.4, 0.5, 0.7]), strength=rng.choice([4.0, 8.0]), target=0.06)
    elif kind == "defringe":
        c.update(radius=rng.choice([4.0, 6.0, 8.5, 10.0, 10.0, 14.0]), strength=rng.choice([4.0, 10.0, 16.0]),
                 green=rng.random() < 0.4)
    return c


# ---------------------------------------------------------------- inputs
def _scene(h, w, seed):
    """Linear RGB (3, h, w) in [0, 1]: the seeded scene, upscaled, with purple
    fringes (R and B blurred) along edges next to bright areas."""
    small = torch.from_numpy(scenes.scene_rgb(384, 576, seed)).to(DEV)
    big = F.interpolate(small.permute(2, 0, 1)[None], size=(h, w), mode="bilinear", align_corners=False)[0]
    luma = 0.2126 * big[0] + 0.7152 * big[1] + 0.0722 * big[2]
    p = F.pad(luma[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
    mag = (p[1:-1, 2:] - p[1:-1, :-2]).abs() + (p[2:, 1:-1] - p[:-2, 1:-1]).abs()
    near = F.max_pool2d(luma[None, None], 5, 1, 2)[0, 0]
    wgt = ((mag > 0.05) & (near > 0.6)).float()[None, None]
    wgt = F.avg_pool2d(wgt, 5, 1, 2)[0, 0].mul_(2).clamp_(0, 1)
    x = torch.arange(-6, 7, device=DEV, dtype=torch.float32)
    k = torch.exp(-0.5 * (x / 2) ** 2)
    k = k / k.sum()
    for c in (0, 2):
        b = F.conv2d(F.pad(big[c][None, None], (6, 6, 0, 0), mode="replicate"), k.view(1, 1, 1, -1))
        b = F.conv2d(F.pad(b, (0, 0, 6, 6), mode="replicate"), k.view(1, 1, -1, 1))[0, 0]
        big[c] += (b * 1.1 - big[c]) * wgt
    return big.clamp_(0, 1)


def _noise(x, seed):
    """Poisson-Gaussian sensor noise, gain 1/4000 and read sigma 0.002."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed + 7919)
    x = torch.poisson(x * 4000.0, generator=g) / 4000.0
    x += torch.randn(x.shape, generator=g, device=DEV) * 0.002
    return x.clamp_(0, 1)


def _wb(seed):
    r = np.random.RandomState(seed % (1 << 31))
    return (float(r.uniform(1.5, 2.5)), 1.0, float(r.uniform(1.2, 2.0)), 1.0)


def _mosaic(case, seed, wb, top=1.0):
    """Dense CFA mosaic (h, w), white-balanced, scaled to `top`."""
    h, w = case["h"], case["w"]
    pat = XTRANS if case["kind"] == "xtrans" else case["cfa"]
    n = 6 if case["kind"] == "xtrans" else 2
    idx = torch.from_numpy(scenes.cfa_map(n, n, pat)).to(DEV).repeat(-(-h // n), -(-w // n))[:h, :w]
    x = torch.gather(_scene(h, w, seed), 0, torch.where(idx == 3, 1, idx)[None])[0]
    gains = torch.tensor(wb, dtype=torch.float32, device=DEV)
    return (_noise(x, seed) * gains[idx] * top).contiguous()


def _rgb(case, seed, gain):
    """RGB image (h, w, 3) as the demosaic hands it on: white-balanced, some
    of it above 1 where `gain` lifts it there."""
    x = _noise(_scene(case["h"], case["w"], seed), seed)
    x *= torch.tensor(gain, dtype=torch.float32, device=DEV).view(3, 1, 1)
    return x.permute(1, 2, 0).contiguous()


def _image(case, seed):
    kind = case["kind"]
    if kind == "highlights":
        return _rgb(case, seed, (2.0, 1.15, 1.6))
    if kind in ("detail", "micro"):
        return _rgb(case, seed, (1.3, 1.2, 1.25))
    return _rgb(case, seed, (1.0, 1.0, 1.0))


def _params(case, wb):
    p = dict(cam_mul=wb, tone_mapping=case["tone"], lateral_ca_correction=int(case["lateral"]))
    if case["kind"] == "xtrans":
        return lre.develop_params(cfa=XTRANS, xtrans_passes=case["passes"], **p)
    return lre.develop_params(cfa=case["cfa"], stage_order=case["order"], axial_ca_correction=int(case["axial"]),
                              defringe=int(case["defringe"]), output_bits=case["bits"], **p)


# ---------------------------------------------------------------- the passes
def prepare(case, seed):
    h, w, kind = case["h"], case["w"], case["kind"]
    s = dict(case, acc=lre.default_accelerator())
    if kind in ("develop", "xtrans", "host"):
        wb = _wb(seed)
        s["params"] = _params(case, wb)
        s["inp"] = _mosaic(case, seed, wb)
        # 16-bit codes in an int16 buffer of the same bits (torch has few uint16 operations)
        kept = torch.float32 if case.get("bits", 32) == 32 else torch.int16
        s["out"] = torch.empty((h, w, 3), dtype=kept, device="cpu" if kind == "host" else DEV,
                               pin_memory=kind == "host")
        if kind == "host":
            host = torch.empty((h, w), dtype=torch.float32, pin_memory=True)
            host.copy_(s["inp"])
            s["keep"] = (host, s["out"])
            s["inp"], s["out"] = host.numpy(), s["out"].numpy()
    elif kind in ("dcb", "aahd"):
        s["inp"] = _mosaic(case, seed, _wb(seed), 16383.0)  # 14-bit raw range
        s["out"] = torch.empty((h, w, 3), dtype=torch.float32, device=DEV)
    else:
        s["inp"] = _image(case, seed)
        s["out"] = torch.empty_like(s["inp"])
    torch.cuda.synchronize()  # the library has a stream of its own
    return s


def run(s):
    acc, kind, w, h, inp, out = s["acc"], s["kind"], s["w"], s["h"], s["inp"], s["out"]
    if kind in ("develop", "xtrans"):
        acc.dev_develop(inp, out, w, h, s["params"])
    elif kind == "host":
        acc.develop(inp, s["params"], out=out)
    elif kind == "dcb":
        acc.dev_demosaic_bayer_dcb(inp, out, w, h, lre.FILTERS[s["cfa"]], 16383.0, s["iterations"], s["enhance"])
    elif kind == "aahd":
        acc.dev_demosaic_bayer_aahd(inp, out, w, h, lre.FILTERS[s["cfa"]], 16383.0)
    elif kind == "highlights":
        acc.dev_recover_highlights(inp, out, w, h, s["threshold"])
    elif kind == "detail":
        acc.dev_detail_tonemap(inp, out, w, h)
    elif kind == "micro":
        acc.dev_enhance_micro_contrast(inp, out, w, h, s["threshold"], s["strength"], s["target"])
    else:
        acc.dev_defringe(inp, out, w, h, s["radius"], 0.1, 0.15, s["strength"], s["green"])
    return out


# Arithmetic operations per pixel of each algorithm's formulas (estimates, each
# quantity formed once).
OPS = {"amaze": 600, "xtrans3": 1800, "xtrans1": 40, "dcb": 250, "aahd": 350, "highlights": 60, "detail": 60,
       "micro": 250, "axial": 90, "lateral": 120, "tone": 33}


def _defringe_ops(radius):
    ks = math.ceil(3 * max(radius / 3, 0.5))
    return 8 * 2 * 2 * (2 * ks + 1) + 300  # eight separable blurs and the classification


def work(case):
    n, kind = case["w"] * case["h"], case["kind"]
    if kind in ("develop", "host"):
        ops = OPS["amaze"] + (OPS["tone"] if case["tone"] else 0) + (OPS["lateral"] if case["lateral"] else 0)
        ops += (OPS["axial"] if case["axial"] else 0) + (_defringe_ops(10.0) if case["defringe"] else 0)
        return {"bytes": n * (4 + 3 * case["bits"] // 8), "flops": n * ops}
    if kind == "xtrans":
        ops = OPS["xtrans%d" % case["passes"]] + (OPS["tone"] if case["tone"] else 0)
        return {"bytes": n * 16, "flops": n * (ops + (OPS["lateral"] if case["lateral"] else 0))}
    if kind == "defringe":
        return {"bytes": n * 24, "flops": n * _defringe_ops(case["radius"])}
    return {"bytes": n * (16 if kind in ("dcb", "aahd") else 24), "flops": n * OPS[kind]}


# ---------------------------------------------------------------- 64 bits
def _box64(x, r):
    """Mean over the (2r+1)^2 window, cut at the frame."""
    for dim in (0, 1):
        n = x.shape[dim]
        s = F.pad(x.cumsum(dim), (1, 0, 0, 0) if dim else (0, 0, 1, 0))
        i = torch.arange(n, device=x.device)
        hi, lo = (i + r + 1).clamp(max=n), (i - r).clamp(min=0)
        cnt = (hi - lo).double().view(*((1, -1) if dim else (-1, 1)))
        x = (s.index_select(dim, hi) - s.index_select(dim, lo)) / cnt
    return x


def _detail64(rgb):
    guide = rgb.amax(2).clamp(min=0)
    m = _box64(guide, 12)
    var = (_box64(guide * guide, 12) - m * m).clamp(min=0)
    a = var / (var + 0.0025)
    base = (_box64(a, 12) * guide + _box64(m * (1 - a), 12)).clamp(min=1e-6)
    mapped = base * (2.51 * base + 0.03) / (base * (2.43 * base + 0.59) + 0.14)
    gain = (mapped / base).clamp(0, 1)
    t = ((base - 0.55) / 0.35).clamp(0, 1)
    t = t * t * (3 - 2 * t)
    return rgb * (1 + (gain - 1) * t)[..., None]


def _micro64(rgb, threshold, strength, target):
    x = torch.arange(-4, 5, device=rgb.device, dtype=torch.float64)
    k = torch.exp(-x * x / (2 * (5 / 3.7) ** 2))
    k = k / k.sum()

    def blur(v):
        v = F.pad(v.permute(2, 0, 1)[:, None], (4, 4, 4, 4), mode="replicate")
        v = sum(k[i] * v[..., i:v.shape[-1] - 8 + i] for i in range(9))
        v = sum(k[i] * v[..., i:v.shape[-2] - 8 + i, :] for i in range(9))
        return v[:, 0].permute(1, 2, 0)

    mean = blur(rgb)
    std = (blur(rgb * rgb) - mean * mean).clamp(min=0).sqrt()
    contrast = std / std.max()
    lift = torch.where(contrast < target, strength * (target - contrast) / target, 0.0)
    out = mean + (rgb - mean) * (1 + lift)
    out = out / out.amax(2, keepdim=True).clamp(min=1)
    return torch.where(rgb[..., 1:2] >= float(np.float32(threshold)), out, rgb)


def exact(case, seed):
    if case["kind"] == "detail":
        return _detail64(_image(case, seed).double())
    if case["kind"] == "micro":
        return _micro64(_image(case, seed).double(), case["threshold"], case["strength"], case["target"])
    return None  # demosaics, recovery and defringe decide by thresholds at every pixel

"""AAHD on a workspace that holds another image's planes: only the margins are
cleared, so nothing inside may be read before it is written.  The same bits as
on a fresh context, for each Bayer layout, with zeros and negative zeros among
the samples, at sizes around the margin and the tiles."""
import numpy as np
import pytest

from libraw_enhanced_b200 import scenes

pytestmark = pytest.mark.gpu


def mosaic(h, w, seed):
    m = np.round(scenes.bayer_scene(h, w, seed) * 16000).astype(np.float32)
    r = np.random.default_rng(seed)
    m[r.random((h, w)) < 0.02] = 0.0
    m[r.random((h, w)) < 0.01] = -0.0
    return m


@pytest.mark.parametrize("cfa", ["RGGB", "BGGR", "GRBG", "GBRG"])
@pytest.mark.parametrize("h,w", [(8, 8), (9, 13), (31, 33), (64, 130), (203, 157)])
def test_dirty_workspace(cfa, h, w):
    import torch

    import libraw_enhanced_b200 as lre

    f = lre.FILTERS[cfa]
    x = torch.from_numpy(mosaic(h, w, h + w)).cuda()
    big = torch.full((600, 700), 15000.0, device="cuda") + 500 * torch.rand((600, 700), device="cuda")
    big_out = torch.empty((600, 700, 3), device="cuda")
    outs = []
    for dirty in (False, True):
        a = lre.CudaAccelerator(0)
        if dirty:
            for filters in (f, lre.FILTERS["GRBG"]):
                a.dev_demosaic_bayer_aahd(big, big_out, 700, 600, filters, 16383.0)
        o = torch.empty((h, w, 3), device="cuda")
        torch.cuda.synchronize()
        a.dev_demosaic_bayer_aahd(x, o, w, h, f, 16383.0)
        a.synchronize()
        outs.append(o.cpu().numpy().view(np.int32))
        a.close()
    assert np.array_equal(*outs)

"""Lateral CA with few cells: cells of 400 pixels on 1.6 MP leave the GPU a CTA on
every sixth SM, and such a call had become slower when the estimate's registers were
bounded for five CTAs per SM.  In units of the same image with cells of 96: 7.0 then,
4.9 with a form for few CTAs."""
import time

import pytest

import libraw_enhanced_b200 as lre

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_few_large_cells():
    h, w = 1024, 1536
    g = torch.Generator(device="cuda").manual_seed(170)
    img = torch.rand((h, w, 3), generator=g, device="cuda")
    img = torch.nn.functional.avg_pool2d(img.permute(2, 0, 1)[None], 5, 1, 2)[0].permute(1, 2, 0).contiguous()
    out = torch.empty_like(img)
    torch.cuda.synchronize()
    with lre.CudaAccelerator(0) as acc:
        def took(cell, iters):
            best = 1e9
            for _ in range(8):
                t0 = time.perf_counter()
                for _ in range(5):
                    acc.dev_ca_register_lateral(img, out, w, h, cell, iters, 6.0, 0.02, 1)
                acc.synchronize()
                best = min(best, (time.perf_counter() - t0) / 5)
            return best

        few, many = took(400, 3), took(96, 3)
    assert few < 6 * many, f"{few * 1e6:.0f} us, {many * 1e6:.0f} us"

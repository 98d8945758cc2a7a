"""Blocks that disagree in pass after pass must not cost much more than the passes
in order alone: once a nyquist pass of a DCB call has given way, the later ones
run in order at once.  3000x2000 of clipped waves, eight iterations: 24 nyquist
passes, all of which disagree.  (With blocks and repairs in each of them the call
took 1.12 times as long as in order.)"""
import time

import pytest

from libraw_enhanced_b200 import scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_disagreeing_passes_cost_little():
    import libraw_enhanced_b200 as m

    h, w = 2000, 3000
    yy, xx = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"), indexing="ij")
    raw = ((torch.sin(xx / 90) + torch.cos(yy / 70)) * 12000 + 9000).clamp(0, 16383).contiguous()
    out = {}
    took = {}
    with m.CudaAccelerator(0) as acc:
        for limit in (0, 4_000_000_000):
            acc.set_wait_limit(limit)
            out[limit] = torch.zeros((h, w, 3), device="cuda")
            torch.cuda.synchronize()
            took[limit] = []
            for _ in range(8):
                t0 = time.perf_counter()
                acc.dev_demosaic_bayer_dcb(raw, out[limit], w, h, scenes.FILTERS["RGGB"], 16383.0, 8, False)
                acc.synchronize()
                took[limit].append(time.perf_counter() - t0)
            if limit == 0:
                assert acc.sweep_counts()[1] >= 24 * 8  # each nyquist pass ran in order
    blocks, in_order = (min(t[2:]) for t in took.values())
    assert torch.equal(*(o.view(torch.int32) for o in out.values()))
    assert blocks < 1.05 * in_order, f"{blocks * 1e3:.2f} ms, in order {in_order * 1e3:.2f} ms"

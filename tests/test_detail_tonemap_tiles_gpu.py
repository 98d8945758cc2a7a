"""The detail-preserving tone map at the edges of its tiles: column strips of
128 outputs, lanes of four columns (float4 when the width allows), row chunks
of 16 to 256 with steps of four, and frames narrower than the 25-px window.

The tolerance is the stage's acceptance tolerance (max-abs 1e-4, PSNR 90 dB):
window sums of at most 256 + 24 additions of values up to 2.56 * 25 carry an
error far below it, and the guided filter's eps of 0.0025 bounds what it
becomes in the result."""
import numpy as np
import pytest

import oracle
from libraw_enhanced_b200 import scenes
from tests._util import assert_parity

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def acc():
    import libraw_enhanced_b200 as m

    a = m.CudaAccelerator(0)
    yield a
    a.close()


@pytest.mark.parametrize("h,w", [(1, 1), (3, 2), (5, 27), (16, 128), (17, 129), (15, 127), (64, 256), (33, 1000),
                                 (700, 131), (257, 513)])
def test_detail_tonemap_tile_edges(acc, h, w):
    img = (scenes.scene_rgb(max(h, 64), max(w, 64), 90)[:h, :w] * np.float32(1.4)).astype(np.float32)
    assert_parity(acc.apply_detail_preserving_tonemap(img), oracle.detail_tonemap(img), what=f"{w}x{h}")


def test_detail_tonemap_unaligned_buffers(acc):
    import torch

    h, w = 60, 132
    img = (scenes.scene_rgb(h, w, 91) * np.float32(1.4)).astype(np.float32)
    src = torch.empty(h * w * 3 + 1, device="cuda")[1:].view(h, w, 3)
    src.copy_(torch.from_numpy(img))
    out = torch.empty((h, w, 3), device="cuda")
    torch.cuda.synchronize()
    acc.dev_detail_tonemap(src, out, w, h)
    acc.dev_detail_tonemap(src, src, w, h)  # in place
    acc.synchronize()
    assert torch.equal(out, src)
    assert_parity(out.cpu().numpy(), oracle.detail_tonemap(img))


@pytest.mark.parametrize("order,bits,defringe", [(0, 16, 0), (0, 32, 1), (1, 16, 1)])
def test_develop_detail_tonemap_in_reference_order(acc, order, bits, defringe):
    """Develops that end in 16-bit codes, or run defringe after the tone map,
    use the reference's scan order: the codes before defringe equal the
    oracle's tone map of the same image."""
    import libraw_enhanced_b200 as lre

    h, w = 150, 260
    m = scenes.bayer_scene(h, w, 92)
    wb = (2.0, 1.0, 1.5, 1.0)
    kw = dict(cfa="RGGB", cam_mul=wb, stage_order=order)
    got = acc.develop(m, lre.develop_params(tone_mapping=2, output_bits=bits, defringe=defringe, **kw))
    if order == 0:
        ref = oracle.detail_tonemap(acc.develop(m, lre.develop_params(**kw)))
        if defringe:
            ref = acc.defringe(ref)
    else:
        ref = oracle.detail_tonemap(acc.develop(m, lre.develop_params(defringe=1, **kw)))
    assert np.array_equal(got, ref if bits == 32 else oracle.quantize_u16(ref))

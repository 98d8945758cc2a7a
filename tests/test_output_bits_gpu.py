"""A 16-bit develop is the quantised 32-bit develop of the same chain, code for
code, for each tone map, stage order and set of corrections."""
import numpy as np
import pytest

import libraw_enhanced_b200 as lre
from libraw_enhanced_b200 import scenes

pytestmark = pytest.mark.gpu

WB = (2.0, 1.0, 1.5, 1.0)


@pytest.fixture(scope="module")
def acc():
    a = lre.CudaAccelerator(0)
    yield a
    a.close()


@pytest.mark.parametrize("tone", [0, 1, 2])
@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("stages", [{}, {"defringe": 1}, {"axial_ca_correction": 1},
                                    {"defringe": 1, "axial_ca_correction": 1, "lateral_ca_correction": 1}])
@pytest.mark.parametrize("h,w", [(97, 131), (600, 904)])
def test_codes_are_the_quantised_floats(acc, h, w, stages, order, tone):
    mos = scenes.bayer_scene(h, w, 114)
    out = {}
    for bits in (16, 32):
        p = lre.develop_params(cfa="RGGB", cam_mul=WB, stage_order=order, tone_mapping=tone, output_bits=bits, **stages)
        out[bits] = acc.develop(mos, p)
    assert out[16].dtype == np.uint16 and out[16].any()
    assert np.array_equal(out[16], acc.quantize(out[32]))

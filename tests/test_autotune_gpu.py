"""The batch autotuner does not choose between forms that are one and the same: at
axial radius 6 the strip width reaches no kernel and stays as it is."""
import numpy as np
import pytest

import libraw_enhanced_b200 as lre
from libraw_enhanced_b200 import scenes

pytestmark = pytest.mark.gpu


def tunings(radius, n):
    m = scenes.bayer_scene(96, 128, 150)
    p = lre.develop_params(cfa="RGGB", cam_mul=(2.0, 1.0, 1.5, 1.0), axial_ca_correction=1, axial_ca_radius=radius)
    out = []
    for _ in range(n):
        b = lre.Batch(0, lanes=1, use_graph=False, autotune=True)
        try:
            r = b.run([m], p)
            assert np.isfinite(r[0]).all()
            out.append(b.get_tuning())
        finally:
            b.close()
    return out


def test_strip_width_is_not_tuned_where_it_is_not_read():
    assert {t["axial_strip"] for t in tunings(6, 16)} == {128}


def test_other_radii_are_tuned():
    assert {t["axial_strip"] for t in tunings(3, 4)} <= {64, 128}

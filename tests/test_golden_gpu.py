"""Every stage against the reference's own outputs as stored in tests/golden (no
oracle build needed): bit for bit where the stage is, else within the parity
tolerance.  smoke() runs as it does without the oracle."""
import os

import numpy as np
import pytest

import libraw_enhanced_b200 as lre
import oracle
from libraw_enhanced_b200 import scenes
from tests._util import assert_parity

pytestmark = pytest.mark.gpu

WB = (2.0, 1.0, 1.5, 1.0)
F = scenes.FILTERS["RGGB"]


@pytest.fixture(scope="module")
def g():
    return dict(np.load(os.path.join(os.path.dirname(__file__), "golden", "develop_golden.npz")))


@pytest.fixture(scope="module")
def acc():
    a = lre.CudaAccelerator(0)
    yield a
    a.close()


EXACT = {
    "amaze_rggb": lambda a, g: a.demosaic_bayer_amaze(scenes.sparse_rgb(g["bayer_mosaic"], "RGGB"), F, WB),
    "u16": lambda a, g: a.quantize(g["tone"]),
    "black_pos": lambda a, g: a.black_level(g["raw4"], [10, 12, 14, 11, 2, 2, 100, 101, 102, 103], 0, 16383),
    "black_chan": lambda a, g: a.black_level(g["raw4"], [510, 512, 514, 511, 0, 0], 0, 16000),
    "wb_grbg": lambda a, g: a.apply_white_balance(g["raw4"], (2.1, 1.0, 1.7, 1.02), scenes.FILTERS["GRBG"]),
}
CLOSE = {
    "defringe": lambda a, g: a.defringe(g["amaze_rggb"]),
    "defringe_green_s4": lambda a, g: a.defringe(g["amaze_rggb"], strength=4.0, defringe_green=True),
    "axial": lambda a, g: a.ca_axial_cleanup(g["amaze_rggb"]),
    "tone": lambda a, g: a.tone_mapping(g["amaze_rggb"]),
    "detail": lambda a, g: a.apply_detail_preserving_tonemap(g["amaze_rggb"]),
    "micro": lambda a, g: a.enhance_micro_contrast(g["amaze_rggb"], 0.6, 8.0, 0.04),
    "lateral": lambda a, g: a.ca_register_lateral(g["lateral_in"], cell_size=32),
    "xtrans3": lambda a, g: a.demosaic_xtrans_3pass(scenes.sparse_rgb(g["xtrans_mosaic"], scenes.XTRANS_STD),
                                                    scenes.XTRANS_STD),
    "xtrans1": lambda a, g: a.demosaic_xtrans_1pass(scenes.sparse_rgb(g["xtrans_mosaic"], scenes.XTRANS_STD),
                                                    scenes.XTRANS_STD),
}


@pytest.mark.parametrize("key", EXACT)
def test_bits(acc, g, key):
    got = EXACT[key](acc, g)
    assert got.dtype == g[key].dtype and np.array_equal(got, g[key])


@pytest.mark.parametrize("key", CLOSE)
def test_values(acc, g, key):
    assert_parity(CLOSE[key](acc, g), g[key], what=key)


def test_develop_detail_tone_map_has_the_reference_bits(acc, g):
    out = acc.develop(g["bayer_mosaic"], lre.develop_params(cfa="RGGB", cam_mul=WB, tone_mapping=2))
    assert np.array_equal(out, g["detail"])


def test_smoke_without_the_oracle(monkeypatch, capsys):
    import __graft_entry__ as entry

    monkeypatch.setattr(oracle, "ref_available", lambda: False)
    entry.smoke()
    assert "stored reference outputs" in capsys.readouterr().out

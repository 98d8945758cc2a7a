"""Lateral CA either side of the lines between its forms, against the numpy
restatement and tolerance of test_lateral_cells_gpu: cells few enough for two CTAs
per SM (2 x 148 cells and one column of cells more; with cells of 160 pixels five),
and a remap of sixteen or four rows a thread (1184 and 1147 strips of 128 rows)."""
import numpy as np
import pytest

from tests.test_lateral_cells_gpu import acc, f32, lateral, scene  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w,cell,levels,iters", [
    (128, 1184, 32, 1, 3), (128, 1216, 32, 2, 3), (600, 1600, 160, 2, 1),
    (4095, 1184, 400, 1, 1), (3967, 1184, 400, 1, 1)])
def test_against_numpy(acc, h, w, cell, levels, iters):  # noqa: F811
    img = scene(h, w, 2000 + h + w)
    got = np.asarray(acc.ca_register_lateral(img, cell, iters, 6.0, 0.02, levels))
    ref = lateral(img, cell, iters, 6.0, 0.02, levels)
    assert np.array_equal(got[..., 1], img[..., 1])
    slope = max(np.abs(np.diff(img, axis=0)).max(), np.abs(np.diff(img, axis=1)).max())
    assert np.abs(got - ref).max() <= 2 * 2 * slope * np.spacing(f32(max(h, w))) + 4e-7

"""The table-driven logarithm has the bits of the one through CUDA's log in double
for every positive normal float (2.13e9 of them): where the middle of two floats
is too near to tell which one the table's double rounds to, it asks the other."""
import ctypes

import pytest

from tests.test_log_table_gpu import lib  # noqa: F401  (the fixture that builds the comparison)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lo", range(0x00800000, 0x7f800000, 0x10000000))
def test_every_normal_float(lib, lo):  # noqa: F811
    out = (ctypes.c_uint * 2)()
    assert lib.run(lo, min(lo + 0x10000000, 0x7f800000), 1, out) == 0
    assert out[0] == 0

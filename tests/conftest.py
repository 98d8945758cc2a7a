import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA sm_100 (B200) device")


# The oracle's reference libraries are built from a reference checkout.  Where
# there is neither, a test that asks for one is skipped, as the tests of the
# oracle itself are; with a checkout at hand a missing library is an error.
def _skip_if_no_reference(error):
    import oracle
    from __graft_entry__ import _reference_dir

    if isinstance(error, oracle.Missing) and not _reference_dir():
        pytest.skip(f"no reference checkout: {error}")


@pytest.hookimpl(wrapper=True)
def pytest_runtest_setup(item):
    try:
        return (yield)
    except FileNotFoundError as e:
        _skip_if_no_reference(e)
        raise


@pytest.hookimpl(wrapper=True)
def pytest_runtest_call(item):
    try:
        return (yield)
    except FileNotFoundError as e:
        _skip_if_no_reference(e)
        raise

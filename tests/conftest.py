import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200); run with -m gpu")


@pytest.hookimpl(wrapper=True)
def pytest_runtest_call(item):
    """A test that calls the reference library is skipped where that is not built: it has nothing to compare with."""
    from oracle import ref

    try:
        return (yield)
    except ref.NotBuilt as e:
        pytest.skip(str(e))

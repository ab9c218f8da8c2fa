import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)
TESTS = os.path.dirname(os.path.abspath(__file__))
if TESTS not in sys.path:
    sys.path.insert(0, TESTS)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs an sm_100 GPU and the built CUDA library")
    config.addinivalue_line("markers", "slow: long-running CPU test")


@pytest.hookimpl(wrapper=True)
def pytest_runtest_call(item):
    """A test that needs the reference's own build (oracle/_ref, made where the
    reference's sources are) is skipped where there is none."""
    try:
        return (yield)
    except OSError as error:
        build = os.path.join("oracle", "_ref")
        if build in str(error) and not os.path.isdir(os.path.join(ROOT, build)):
            pytest.skip(f"the reference's build is missing ({build})")
        raise

import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (ROOT, os.path.join(ROOT, "tests"), os.path.join(ROOT, "oracle")):
    if p not in sys.path:
        sys.path.insert(0, p)

GOLDEN = os.path.join(ROOT, "tests", "golden")
TOOLS = os.path.join(ROOT, "oracle", "_ref")  # built from the reference's sources, where they are


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200)")


@pytest.hookimpl(wrapper=True)
def pytest_pyfunc_call(pyfuncitem):
    """A test that gets as far as a tool built from the reference's sources, where
    those are absent, is skipped there, so that a run that stops at the first failure
    goes on to the tests that need none."""
    try:
        return (yield)
    except FileNotFoundError as e:
        name = os.fsdecode(e.filename or "")
        if os.path.dirname(name) == TOOLS and not os.path.exists(name):
            pytest.skip(f"{os.path.basename(name)} is not built (oracle/_ref)")
        raise


@pytest.fixture(scope="session")
def golden_dir():
    return GOLDEN


def golden(name):
    path = os.path.join(GOLDEN, name)
    if not os.path.exists(path):
        pytest.fail(f"golden fixture {name} missing (tests/golden/make_golden.py)")
    import numpy as np
    return dict(np.load(path))

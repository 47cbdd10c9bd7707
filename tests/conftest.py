import gc
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (ROOT, os.path.join(ROOT, "pytorch-lbm_gb300"), os.path.join(ROOT, "tests"),
          os.path.join(ROOT, "tests", "golden")):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (GB300) and the built native library")


@pytest.fixture(scope="session")
def built_lib():
    """Build (if stale) and load liblbm_gb300.so."""
    from lbm import _build, _native
    _build.build()
    return _native.lib()


@pytest.fixture(scope="module", autouse=True)
def _collect_solvers():
    """A solver and its wetting tables refer to each other: what a module's tests left gives its device arrays back at
    the module's end, not in the middle of a later module that watches memory."""
    yield
    gc.collect()

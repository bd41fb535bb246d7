import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA B200 device")
    config.addinivalue_line("markers", "slow: longer CPU test")


def pytest_collection_modifyitems(items):
    """The drop-in's GPU tests run the reference program beside it: without its
    binaries, which are built from the reference tree, they skip."""
    from oracle import reference
    if all(reference.available(b) for b in ("cmh_ref_f32", "cmh_ref_f64")):
        return
    for item in items:
        if item.path.name == "test_dropin.py" and item.get_closest_marker("gpu"):
            item.add_marker(pytest.mark.skip(reason="reference binaries not built"))


@pytest.fixture(scope="session")
def oracle_lib():
    from oracle import cpu
    cpu.lib()
    return cpu


@pytest.fixture(scope="session")
def native_lib():
    """The native library, built in-tree if it is missing."""
    from cm_halofinder_b200 import _abi, build
    if not os.path.exists(_abi.LIB_PATH):
        build.build()
    return _abi.lib()

import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))

# an empty folder in the place of elegant's sources is no reference tree
_tree = os.environ.get("ELEGANT_REFERENCE_TREE", "/root/reference")
if os.path.isdir(_tree) and not os.listdir(_tree):
    os.environ["ELEGANT_REFERENCE_TREE"] = os.path.join(_tree, "absent")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (runs the engine on the GPU)")


def _skip_without_reference():
    """Tests against elegant's own compiled code are skipped where it has not
    been compiled (oracle/Makefile.ref); their counterparts against the
    restatement run everywhere."""
    from reforacle import ReferenceMissing
    try:
        return (yield)
    except ReferenceMissing as e:
        pytest.skip(f"elegant's own code is not compiled here: {e}")


@pytest.hookimpl(wrapper=True)
def pytest_runtest_setup(item):
    return (yield from _skip_without_reference())


@pytest.hookimpl(wrapper=True)
def pytest_runtest_call(item):
    return (yield from _skip_without_reference())


@pytest.fixture(scope="session")
def ref_b2e():
    from reforacle import RefOracle
    return RefOracle("b2e")


@pytest.fixture(scope="session")
def ref_libm():
    from reforacle import RefOracle
    return RefOracle("libm")

import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")
    config.addinivalue_line("markers", "reference: needs the reference harness built from the reference sources")


def pytest_collection_modifyitems(items):
    # test_integration.py runs a binary built from the reference's sources and
    # fails where that could not be built: after all the others, so that a run
    # that stops at the first failure has run them
    items.sort(key=lambda item: item.path.name == "test_integration.py")


@pytest.fixture(scope="session")
def oracle_lib():
    from oracle import oracle as O
    O.build()
    return O


@pytest.fixture(scope="session")
def cuda_lib():
    """The CUDA path: built in-tree, loaded through ctypes; a missing build fails."""
    from caviar_b200 import build as B
    B.build()
    from caviar_b200 import _abi
    return _abi

import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)
HERE = os.path.dirname(os.path.abspath(__file__))
if HERE not in sys.path:
    sys.path.insert(0, HERE)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200); runs the CUDA kernels")
    config.addinivalue_line("markers", "slow: longer CPU test")


# modules whose every test compares with the translated reference
NEEDS_REFERENCE = ("test_gpu_noncie_hydro",)


def pytest_collection_modifyitems(items):
    """As the other tests of the translated reference: skipped where it is not
    built."""
    from oracle import ref_oracle
    if not ref_oracle.available():
        skip = pytest.mark.skip(reason="translated reference not built")
        for item in items:
            if item.module.__name__ in NEEDS_REFERENCE:
                item.add_marker(skip)


@pytest.fixture(scope="session")
def cuda_device():
    """The CUDA device for GPU tests.  Fails (does not skip) without one: a
    GPU test that cannot reach the kernels is a failure."""
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    torch.cuda.init()
    return torch.device("cuda:0")
